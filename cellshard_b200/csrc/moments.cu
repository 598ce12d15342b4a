// Row-label grouped per-feature moments over Blocked-ELL.
//
// For every kept row r with label g and every feature f:
//     sum[g][f] += x,  sumsq[g][f] += x*x   (x = fp16 value widened to fp32)
//
// Plan (all stream-ordered, no host synchronisation):
//   1. index     one warp per row block turns its ascending blockColIdx row
//                into a bitmap over column blocks plus per-32-block prefix
//                counts, so slot(rb, b) = prefix + popc(word & below(b)).
//   2. sort      stable counting sort of kept rows by label (tile histograms,
//                one-CTA group scan that also cuts each group's rows into
//                chunks, tile-local ranked scatter).
//   3. accumulate  grid (chunk, feature tile): each thread owns L consecutive
//                features of one column block and streams its chunk's rows
//                (all of one group), keeping its sums in registers; fp32 batch
//                sums of kBatch rows are folded into hi/lo two-sum pairs.
//                One partial (hi, lo) per (chunk, feature) goes to scratch.
//   4. combine   per (group, feature): add the group's chunk partials (fp64 or
//                fp32 by scheme), apply the feature mask, emit sum, sumsq,
//                mean and variance.
#include "common.cuh"
#include "moments_device.cuh"

#include <algorithm>
#include <cstring>

namespace csb {
namespace {

constexpr unsigned kTileRows = 1024;   // rows per sort tile
constexpr unsigned kSortThreads = 256; // 8 warps x 128 rows
constexpr unsigned kSortWarps = kSortThreads / 32;
constexpr unsigned kAccThreads = 256;
constexpr uint32_t kScanSteps = 4;
constexpr unsigned kBatch = 8;         // rows per fp32 batch sum
constexpr unsigned kDefaultChunkRows = 2048; // the most that is taken by default
constexpr unsigned kMaxChunkRows = 8192;
constexpr unsigned kIndexWarps = 4;
constexpr unsigned kMaxIndexWords = 2048; // column blocks / 32 per row block

struct chunk_desc {
    uint32_t group;
    uint32_t begin;
    uint32_t end;
    uint32_t pad;
};

struct moments_layout {
    uint2 *index;              // [row_blocks * words]
    uint32_t *tile_counts;     // [tiles * G]
    uint32_t *group_offsets;   // [G + 1]
    uint32_t *group_rows;      // [G]
    uint32_t *chunk_first;     // [G + 1]
    uint32_t *num_chunks;      // [1]
    chunk_desc *chunks;        // [max_chunks]
    uint32_t *sorted_rows;     // [rows]
    float *partials;           // [max_chunks * 4 * pstride]
    std::size_t bytes;
    uint32_t row_blocks, words, tiles, max_chunks, chunk_rows, col_blocks, pstride;
    bool short_chunks;         // see moments_accumulate_kernel
};

// Rows per chunk where the caller leaves it open.  A chunk's CTAs walk its rows
// one batch after the other, so a small matrix in chunks of 2,048 rows runs on a
// few SMs (8,192 x 2,000, 8 groups: 12 CTAs); every chunk costs 32 bytes of
// partials a column, 16 / chunk_rows of the rows' own bytes.  Halved to 256
// rows (6 %) while there are under 1,000 CTAs, and on to 64 only while there
// are under two per SM of this chip (written out, so that the order of the sums
// does not depend on the device).  Not past 250 chunks a group: the combine walks a
// group's chunks one after the other, 0.125 us each where columns and groups are few
// (600,000 x 2,000, one group: 484 us with 2,048 rows, 581 with 512).  us per call by
// 2,048 / 256 / 64 rows: 8,192 x 2,000 (8 groups) 99 / 52 / 36; 100,000 x 5,000 (16)
// 344 / 177 / 217; 20,000 x 8,000 (64) 78 / 76 / 83; 50,000 x 32,768 (64) 479 / 489 / 572
// (1,024: 480).
uint32_t default_chunk_rows(uint32_t rows, uint32_t col_blocks, uint32_t block_size, uint32_t groups) {
    const uint64_t segs = (uint64_t) col_blocks * ((block_size + 7u) / 8u);
    const uint64_t tiles = (segs + kAccThreads - 1u) / kAccThreads;
    // about half of the groups end in a chunk of their own
    auto ctas = [&](uint32_t chunk) { return (rows / chunk + groups / 2u) * tiles; };
    auto may_halve = [&](uint32_t chunk) { return rows / groups <= 250u * (chunk / 2u); };
    uint32_t chunk = kDefaultChunkRows;
    while (chunk > 256u && ctas(chunk) < 1000u && may_halve(chunk)) chunk /= 2u;
    while (chunk > 64u && ctas(chunk) < 296u && may_halve(chunk)) chunk /= 2u;
    return chunk;
}

// padded: the partials' columns in multiples of eight, for 16-byte stores.
bool make_layout(const cs_blocked_ell_view *src, const cs_group_moments_params *p, void *base, std::size_t cap,
                 moments_layout *lay, bool padded = true) {
    const uint32_t B = src->block_size;
    lay->row_blocks = (src->rows + B - 1u) / B;
    lay->col_blocks = (src->cols + B - 1u) / B;
    lay->words = (lay->col_blocks + 31u) / 32u;
    lay->tiles = (src->rows + kTileRows - 1u) / kTileRows;
    lay->chunk_rows =
        p->chunk_rows == 0u ? default_chunk_rows(src->rows, lay->col_blocks, B, p->group_count) : p->chunk_rows;
    const std::size_t G = p->group_count;
    lay->max_chunks = (uint32_t) ((src->rows + lay->chunk_rows - 1u) / lay->chunk_rows + G);
    lay->short_chunks = std::min<std::size_t>(lay->chunk_rows, G != 0u ? src->rows / G : 0u) <= 512u;
    scratch_carver c(base, cap);
    lay->index = c.take<uint2>((std::size_t) lay->row_blocks * lay->words + 1);
    lay->tile_counts = c.take<uint32_t>((std::size_t) lay->tiles * G + 1);
    lay->group_offsets = c.take<uint32_t>(G + 1);
    lay->group_rows = c.take<uint32_t>(G);
    lay->chunk_first = c.take<uint32_t>(G + 1);
    lay->num_chunks = c.take<uint32_t>(1);
    lay->chunks = c.take<chunk_desc>(lay->max_chunks);
    lay->sorted_rows = c.take<uint32_t>((std::size_t) src->rows + 1);
    lay->pstride = padded && src->cols <= 0xfffffff8u ? (src->cols + 7u) & ~7u : src->cols;
    lay->partials = c.take<float>((std::size_t) lay->max_chunks * 4u * lay->pstride + 1);
    lay->bytes = c.used;
    return c.fits();
}

// A smaller matrix may ask for more scratch than a larger one (shorter chunks),
// so scratch that was sized for the larger one, or for unpadded partials as the
// static array's limit counts them, takes longer chunks, at last of 2,048 rows
// without the padding.
template <typename Make>
bool fit_scratch(const cs_group_moments_params *params, Make make) {
    cs_group_moments_params p = *params;
    if (make(p, true)) return true;
    if (params->chunk_rows == 0u)
        for (p.chunk_rows = 128u; p.chunk_rows <= kDefaultChunkRows; p.chunk_rows *= 2u)
            if (make(p, true)) return true;
    p.chunk_rows = params->chunk_rows == 0u ? kDefaultChunkRows : params->chunk_rows;
    return make(p, false);
}

// ---------------------------------------------------------------------------
// 1. Column-block index per row block.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kIndexWarps * 32) moments_index_kernel(const uint32_t *__restrict__ block_col_idx,
                                                                         uint32_t row_blocks, uint32_t width,
                                                                         uint32_t col_blocks, uint32_t words,
                                                                         uint2 *__restrict__ index,
                                                                         uint32_t *status, bool vec4) {
    extern __shared__ uint32_t bitmap_smem[];
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    uint32_t *bits = bitmap_smem + (std::size_t) warp * words;
    for (uint32_t rb = blockIdx.x * kIndexWarps + warp; rb < row_blocks; rb += gridDim.x * kIndexWarps) {
        for (uint32_t w = lane; w < words; w += 32u) bits[w] = 0u;
        __syncwarp();
        const uint32_t *row = block_col_idx + (std::size_t) rb * width;
        uint32_t bad = 0u;
        auto mark = [&](uint32_t bc, uint32_t prev, bool has_prev) {
            if (bc == CS_INVALID_COL) return;
            if (bc >= col_blocks)
                bad |= CS_STATUS_INDEX_RANGE;
            else
                atomicOr(bits + (bc >> 5), 1u << (bc & 31u));
            if (has_prev && (prev == CS_INVALID_COL || prev >= bc)) bad |= CS_STATUS_BLOCK_COL_ORDER;
        };
        if (vec4) {
            // 4 entries per lane per step; the entry before a lane's first one is
            // the previous lane's last (or the previous step's lane 31)
            uint32_t carry = CS_INVALID_COL;
            for (uint32_t s0 = 0; s0 < width; s0 += 128u) {
                const uint32_t s = s0 + lane * 4u;
                uint4 q = make_uint4(CS_INVALID_COL, CS_INVALID_COL, CS_INVALID_COL, CS_INVALID_COL);
                if (s < width) q = __ldg(reinterpret_cast<const uint4 *>(row + s));
                uint32_t before = __shfl_up_sync(0xffffffffu, q.w, 1);
                if (lane == 0u) before = carry;
                if (s < width) {
                    mark(q.x, before, s > 0u);
                    mark(q.y, q.x, true);
                    mark(q.z, q.y, true);
                    mark(q.w, q.z, true);
                }
                carry = __shfl_sync(0xffffffffu, q.w, 31);
            }
        } else {
            for (uint32_t s = lane; s < width; s += 32u) mark(row[s], s > 0u ? row[s - 1u] : 0u, s > 0u);
        }
        bad = __reduce_or_sync(0xffffffffu, bad);
        if (lane == 0u) status_or(status, bad);
        __syncwarp();
        uint32_t carry = 0u;
        for (uint32_t w0 = 0; w0 < words; w0 += 32u) {
            const uint32_t w = w0 + lane;
            const uint32_t word = w < words ? bits[w] : 0u;
            const uint32_t cnt = __popc(word);
            uint32_t incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (unsigned) o) incl += t;
            }
            if (w < words) index[(std::size_t) rb * words + w] = make_uint2(word, carry + incl - cnt);
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// 2. Stable counting sort of kept rows by label.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t row_group(uint32_t r, uint32_t rows, const uint8_t *keep, const uint32_t *labels,
                                              uint32_t G) {
    if (r >= rows) return G;
    // both loads at once: the label does not wait for the mask
    const uint32_t g = labels != nullptr ? __ldg(labels + r) : 0u;
    const bool kept = keep == nullptr || __ldg(keep + r) != 0u;
    return kept && g < G ? g : G;
}

__global__ void __launch_bounds__(kSortThreads) moments_tile_hist_kernel(uint32_t rows, const uint8_t *__restrict__ keep,
                                                                         const uint32_t *__restrict__ labels, uint32_t G,
                                                                         uint32_t *__restrict__ tile_counts) {
    extern __shared__ uint32_t hist[];
    for (uint32_t g = threadIdx.x; g < G; g += blockDim.x) hist[g] = 0u;
    __syncthreads();
    const uint32_t base = blockIdx.x * kTileRows;
    // a small matrix is a few CTAs that wait for memory: all rows of a thread
    // are loaded before any is counted (here and in the scatter)
    uint32_t g[kTileRows / kSortThreads];
#pragma unroll
    for (uint32_t k = 0; k < kTileRows / kSortThreads; ++k)
        g[k] = row_group(base + k * kSortThreads + threadIdx.x, rows, keep, labels, G);
#pragma unroll
    for (uint32_t k = 0; k < kTileRows / kSortThreads; ++k)
        if (g[k] < G) atomicAdd(hist + g[k], 1u);
    __syncthreads();
    for (uint32_t g = threadIdx.x; g < G; g += blockDim.x)
        tile_counts[(std::size_t) blockIdx.x * G + g] = hist[g];
}

// A warp: exclusive scan of group g's per-tile counts (in place, group-relative)
// and the group's row total.
__device__ __forceinline__ void group_tiles(uint32_t g, uint32_t tiles, uint32_t G,
                                            uint32_t *__restrict__ tile_counts, uint32_t *__restrict__ group_rows) {
    const unsigned lane = threadIdx.x & 31u;
    uint32_t carry = 0u;
    for (uint32_t t0 = 0; t0 < tiles; t0 += 32u) {
        const uint32_t t = t0 + lane;
        const std::size_t k = (std::size_t) t * G + g;
        const uint32_t c = t < tiles ? tile_counts[k] : 0u;
        const uint32_t incl = warp_inclusive_scan(c);
        if (t < tiles) tile_counts[k] = carry + incl - c;
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0u) group_rows[g] = carry;
}

__global__ void __launch_bounds__(256) moments_group_tiles_kernel(uint32_t tiles, uint32_t G,
                                                                  uint32_t *__restrict__ tile_counts,
                                                                  uint32_t *__restrict__ group_rows) {
    const uint32_t g = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (g < G) group_tiles(g, tiles, G, tile_counts, group_rows);
}

// One CTA: group offsets, chunk cutting (each chunk holds rows of one group).
// kTiles: the groups' totals first.
template <bool kTiles>
__global__ void __launch_bounds__(1024) moments_group_scan_kernel(uint32_t G, uint32_t chunk_rows, uint32_t max_chunks,
                                                                  uint32_t tiles, uint32_t *tile_counts,
                                                                  uint32_t *group_rows,
                                                                  uint32_t *__restrict__ group_offsets,
                                                                  uint32_t *__restrict__ chunk_first,
                                                                  uint32_t *__restrict__ num_chunks,
                                                                  chunk_desc *__restrict__ chunks) {
    __shared__ uint32_t smem[33];
    __shared__ uint32_t first[1024], begin[1024], len[1024];
    if constexpr (kTiles) {
        for (uint32_t g = threadIdx.x >> 5; g < G; g += blockDim.x >> 5)
            group_tiles(g, tiles, G, tile_counts, group_rows);
        __syncthreads();
    }
    uint32_t carry_rows = 0u, carry_chunks = 0u;
    for (uint32_t g0 = 0; g0 < G; g0 += blockDim.x) {
        const uint32_t g = g0 + threadIdx.x;
        const uint32_t n = g < G ? group_rows[g] : 0u;
        const uint32_t nc = g < G ? (n + chunk_rows - 1u) / chunk_rows : 0u;
        uint32_t tot_n, tot_c;
        const uint32_t ex_n = block_exclusive_scan(n, smem, tot_n);
        const uint32_t ex_c = block_exclusive_scan(nc, smem, tot_c);
        const uint32_t off = carry_rows + ex_n, cf = carry_chunks + ex_c;
        if (g < G) {
            group_offsets[g] = off;
            chunk_first[g] = cf;
        }
        auto cut = [&](uint32_t id, uint32_t group, uint32_t from, uint32_t upto) {
            if (id < max_chunks) chunks[id] = chunk_desc{group, from, min(from + chunk_rows, upto), 0u};
        };
        if (__syncthreads_or(nc > 8u)) { // a thread per chunk: its group is the last that starts at or before it
            first[threadIdx.x] = ex_c;
            begin[threadIdx.x] = off;
            len[threadIdx.x] = n;
            __syncthreads();
            for (uint32_t c = threadIdx.x; c < tot_c; c += blockDim.x) {
                uint32_t lo = 0u, hi = blockDim.x - 1u;
                while (lo < hi) {
                    const uint32_t mid = (lo + hi + 1u) >> 1;
                    if (first[mid] <= c)
                        lo = mid;
                    else
                        hi = mid - 1u;
                }
                cut(carry_chunks + c, g0 + lo, begin[lo] + (c - first[lo]) * chunk_rows, begin[lo] + len[lo]);
            }
            __syncthreads();
        } else {
            for (uint32_t c = 0; c < nc; ++c) cut(cf + c, g, off + c * chunk_rows, off + n);
        }
        carry_rows += tot_n;
        carry_chunks += tot_c;
    }
    if (threadIdx.x == 0) {
        group_offsets[G] = carry_rows;
        chunk_first[G] = carry_chunks;
        *num_chunks = carry_chunks;
    }
}

__global__ void __launch_bounds__(kSortThreads) moments_tile_scatter_kernel(uint32_t rows,
                                                                            const uint8_t *__restrict__ keep,
                                                                            const uint32_t *__restrict__ labels,
                                                                            uint32_t G,
                                                                            const uint32_t *__restrict__ tile_base,
                                                                            const uint32_t *__restrict__ group_offsets,
                                                                            uint32_t *__restrict__ sorted_rows) {
    extern __shared__ uint32_t warp_counts[]; // [kSortWarps][G]
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    constexpr uint32_t rows_per_warp = kTileRows / kSortWarps, batches = rows_per_warp / 32u;
    const uint32_t wbase = blockIdx.x * kTileRows + warp * rows_per_warp;
    uint32_t group[batches], peers_of[batches];
#pragma unroll
    for (uint32_t b = 0; b < batches; ++b) group[b] = row_group(wbase + b * 32u + lane, rows, keep, labels, G);
    for (uint32_t i = threadIdx.x; i < kSortWarps * G; i += blockDim.x) warp_counts[i] = 0u;
    __syncthreads();
    uint32_t *my = warp_counts + (std::size_t) warp * G;
#pragma unroll
    for (uint32_t b = 0; b < batches; ++b) {
        const uint32_t g = group[b];
        const uint32_t peers = peers_of[b] = __match_any_sync(0xffffffffu, g);
        if (g < G && lane == (unsigned) (__ffs(peers) - 1)) my[g] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    for (uint32_t g = threadIdx.x; g < G; g += blockDim.x) {
        uint32_t run = tile_base[(std::size_t) blockIdx.x * G + g] + group_offsets[g];
        for (unsigned w = 0; w < kSortWarps; ++w) {
            const uint32_t c = warp_counts[(std::size_t) w * G + g];
            warp_counts[(std::size_t) w * G + g] = run;
            run += c;
        }
    }
    __syncthreads();
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (uint32_t b = 0; b < batches; ++b) {
        const uint32_t r = wbase + b * 32u + lane, g = group[b], peers = peers_of[b];
        uint32_t base = 0u;
        if (g < G) base = my[g];
        __syncwarp();
        if (g < G) {
            sorted_rows[base + __popc(peers & lt)] = r;
            if (lane == (unsigned) (__ffs(peers) - 1)) my[g] = base + __popc(peers);
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// 3. Accumulation.
// ---------------------------------------------------------------------------
// Where a sorted row's values and index entries live.  One partition: the
// row id and its row block's index offset, kept in shared memory as a uint2.
struct one_partition_rows {
    using entry = uint2;
    const uint16_t *__restrict__ val;
    const uint2 *__restrict__ index;
    const uint32_t *__restrict__ sorted_rows;
    uint32_t ell_cols, block_size, words;
    __device__ __forceinline__ entry fetch(uint32_t pos) const {
        const uint32_t r = sorted_rows[pos];
        return make_uint2(r, (r / block_size) * words);
    }
    __device__ __forceinline__ uint2 index_entry(const entry &e, uint32_t w) const { return __ldg(index + e.y + w); }
    __device__ __forceinline__ const uint16_t *row(const entry &e) const {
        return val + (std::size_t) e.x * ell_cols;
    }
};

// Several partitions (a shard): each sorted row's value row and index row
// addresses, precomputed by moments_row_ptrs_kernel.
struct many_partition_rows {
    using entry = ulonglong2;
    const ulonglong2 *__restrict__ row_ptrs;
    __device__ __forceinline__ entry fetch(uint32_t pos) const { return row_ptrs[pos]; }
    __device__ __forceinline__ uint2 index_entry(const entry &e, uint32_t w) const {
        return __ldg(reinterpret_cast<const uint2 *>(e.y) + w);
    }
    __device__ __forceinline__ const uint16_t *row(const entry &e) const {
        return reinterpret_cast<const uint16_t *>(e.x);
    }
};

// kVecStore: partials in 16-byte stores.  A thread's eight columns stand side by
// side, so a scalar store of a warp is 32 sectors for 128 bytes: half of the time
// of chunks of a dozen rows (3,000 x 20,000, 250 groups: 111 us, 52 with 16-byte
// stores), nothing at 2,048 rows, where the registers in fours cost the row loop
// 1.6 % (500,000 x 32,768, 64 groups: 3.99 and 4.06 ms).  Taken up to 512 rows;
// by these two figures the forms meet at about 1,200.
template <int L, bool COMP, bool kVecStore, typename Rows>
__global__ void __launch_bounds__(kAccThreads, 2) moments_accumulate_kernel(
    Rows rows_of, uint32_t block_size, uint32_t col_blocks, uint32_t cols, uint32_t pstride,
    const chunk_desc *__restrict__ chunks, const uint32_t *__restrict__ num_chunks, float *__restrict__ partials,
    const uint32_t *__restrict__ chunk_first, uint32_t g_lo, uint32_t g_hi) {
    using entry = typename Rows::entry;
    extern __shared__ __align__(16) unsigned char acc_smem[];
    entry *chunk_rows_smem = reinterpret_cast<entry *>(acc_smem);
    const uint32_t c = blockIdx.x;
    if (c >= *num_chunks) return;
    // with chunk_first: only the chunks of groups [g_lo, g_hi)
    if (chunk_first != nullptr && (c < chunk_first[g_lo] || c >= chunk_first[g_hi])) return;
    const chunk_desc d = chunks[c];
    const uint32_t n = d.end - d.begin;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) chunk_rows_smem[i] = rows_of.fetch(d.begin + i);
    __syncthreads();

    const uint32_t segs_per_block = block_size / L;
    const uint32_t seg = blockIdx.y * kAccThreads + threadIdx.x;
    const uint32_t b = seg / segs_per_block;
    const uint32_t part = seg - b * segs_per_block;
    if (b >= col_blocks) return;
    const uint32_t w = b >> 5;
    const uint32_t below = (1u << (b & 31u)) - 1u;
    const uint32_t bitmask = 1u << (b & 31u);
    const std::size_t lane_off = (std::size_t) part * L;

    float s_hi[L], s_lo[L], q_hi[L], q_lo[L];
#pragma unroll
    for (int j = 0; j < L; ++j) s_hi[j] = s_lo[j] = q_hi[j] = q_lo[j] = 0.0f;

    // two-stage software pipeline: the index entries of batch i+1 are in
    // flight while batch i's value loads are outstanding
    uint2 e_next[kBatch];
#pragma unroll
    for (unsigned u = 0; u < kBatch; ++u)
        e_next[u] = u < n ? rows_of.index_entry(chunk_rows_smem[u], w) : make_uint2(0u, 0u);
    uint32_t i = 0;
    for (; i + kBatch <= n; i += kBatch) {
        raw_vec<L> raw[kBatch];
#pragma unroll
        for (unsigned u = 0; u < kBatch; ++u) {
            const uint2 e = e_next[u];
            if (e.x & bitmask) {
                const uint32_t slot = e.y + __popc(e.x & below);
                load_raw<L>(rows_of.row(chunk_rows_smem[i + u]) + (std::size_t) slot * block_size + lane_off,
                            raw[u]);
            } else {
                zero_raw<L>(raw[u]);
            }
        }
#pragma unroll
        for (unsigned u = 0; u < kBatch; ++u) {
            const uint32_t k = i + kBatch + u;
            e_next[u] = k < n ? rows_of.index_entry(chunk_rows_smem[k], w) : make_uint2(0u, 0u);
        }
        if (COMP) {
            float bs[L], bq[L];
#pragma unroll
            for (int j = 0; j < L; ++j) bs[j] = bq[j] = 0.0f;
#pragma unroll
            for (unsigned u = 0; u < kBatch; ++u) {
                float x[L];
                unpack<L>(raw[u], x);
#pragma unroll
                for (int j = 0; j < L; ++j) {
                    bs[j] = __fadd_rn(bs[j], x[j]);
                    bq[j] = __fmaf_rn(x[j], x[j], bq[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < L; ++j) {
                two_sum_acc(s_hi[j], s_lo[j], bs[j]);
                two_sum_acc(q_hi[j], q_lo[j], bq[j]);
            }
        } else {
#pragma unroll
            for (unsigned u = 0; u < kBatch; ++u) {
                float x[L];
                unpack<L>(raw[u], x);
#pragma unroll
                for (int j = 0; j < L; ++j) {
                    s_hi[j] = __fadd_rn(s_hi[j], x[j]);
                    q_hi[j] = __fmaf_rn(x[j], x[j], q_hi[j]);
                }
            }
        }
    }
    // tail rows (fewer than a batch); their index entries are in e_next.  All
    // values are loaded before any is added: a group of few rows is all tail
    if (i < n) {
        raw_vec<L> raw[kBatch];
        uint32_t has = 0u;
#pragma unroll
        for (unsigned u = 0; u < kBatch; ++u) {
            const uint2 e = e_next[u]; // zero past the last row
            zero_raw<L>(raw[u]);
            if (e.x & bitmask) {
                has |= 1u << u;
                const uint32_t slot = e.y + __popc(e.x & below);
                load_raw<L>(rows_of.row(chunk_rows_smem[i + u]) + (std::size_t) slot * block_size + lane_off,
                            raw[u]);
            }
        }
#pragma unroll
        for (unsigned u = 0; u < kBatch; ++u) {
            if ((has >> u) & 1u) {
                float x[L];
                unpack<L>(raw[u], x);
#pragma unroll
                for (int j = 0; j < L; ++j) {
                    if (COMP) {
                        two_sum_acc(s_hi[j], s_lo[j], x[j]);
                        two_sum_acc(q_hi[j], q_lo[j], __fmul_rn(x[j], x[j]));
                    } else {
                        s_hi[j] = __fadd_rn(s_hi[j], x[j]);
                        q_hi[j] = __fmaf_rn(x[j], x[j], q_hi[j]);
                    }
                }
            }
        }
    }
    const std::size_t f0 = (std::size_t) b * block_size + lane_off;
    if (f0 >= cols) return;
    float *p = partials + (std::size_t) c * 4u * pstride + f0;
    // in padded columns a segment, which starts at a multiple of its L, ends inside them
    const bool vec = kVecStore && (pstride & 7u) == 0u && (reinterpret_cast<uintptr_t>(partials) & 15u) == 0u;
    auto store = [&](const float (&x)[L], uint32_t k) {
        float *to = p + (std::size_t) k * pstride;
        if constexpr (kVecStore && L % 4 == 0) {
            if (vec) {
#pragma unroll
                for (int j = 0; j < L; j += 4)
                    *reinterpret_cast<float4 *>(to + j) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
                return;
            }
        }
#pragma unroll
        for (int j = 0; j < L; ++j)
            if (f0 + j < cols) to[j] = x[j];
    };
    store(s_hi, 0u);
    store(s_lo, 1u);
    store(q_hi, 2u);
    store(q_lo, 3u);
}

// ---------------------------------------------------------------------------
// 4. Combine.
// ---------------------------------------------------------------------------
// a / b from y, the rounded 1 / b: the product corrected twice by its exact
// remainder, which is the correctly rounded quotient (P. Markstein, Computation
// of elementary functions on the IBM RISC System/6000 processor, 1990) where b
// is a whole number of 32 bits and nothing is near the ends of the double range;
// infinities and NaN pass through the product.
__device__ __forceinline__ double divide_by(double a, double b, double y) {
    const double q0 = a * y;
    const double q1 = fma(fma(-q0, b, a), y, q0);
    const double q2 = fma(fma(-q1, b, a), y, q1);
    return isinf(q0) ? q0 : q2;
}

// A thread adds C columns, 256 apart.  Bound by issue slots where a group has
// one or two chunks: two divisions an output, by the group's row counts, were
// half of the instructions; four columns share the reciprocals (250 groups of
// 20,000 columns: 58 -> 32 us).
// kLong: groups of many chunks (one column a thread).
template <int C, bool kLong>
__global__ void __launch_bounds__(256) moments_combine_kernel(
    uint32_t cols, uint32_t pstride, uint32_t G, uint32_t scheme, uint32_t ddof,
    const uint32_t *__restrict__ chunk_first, const uint32_t *__restrict__ group_rows,
    const float *__restrict__ partials, const uint8_t *__restrict__ feature_keep, float *__restrict__ out_sum,
    float *__restrict__ out_sumsq, float *__restrict__ out_mean, float *__restrict__ out_var,
    double *__restrict__ out_mean64, double *__restrict__ out_var64, uint32_t *__restrict__ out_group_rows,
    uint32_t g_base) {
    const uint32_t g = g_base + blockIdx.y;
    const uint32_t f0 = blockIdx.x * (256u * C) + threadIdx.x;
    if (g >= G) return;
    if (f0 == 0 && out_group_rows != nullptr) out_group_rows[g] = group_rows[g];
    const uint32_t c0 = chunk_first[g], c1 = chunk_first[g + 1];
    const uint32_t n = group_rows[g];
    bool kept[C];
#pragma unroll
    for (int k = 0; k < C; ++k) {
        const uint32_t f = f0 + 256u * k;
        kept[k] = f < cols && (feature_keep == nullptr || feature_keep[f] != 0u);
    }
    // kBatch consecutive chunks' partials of the thread's column (column 0's, unused,
    // where it has none).  A group of hundreds of chunks is a chain of their latencies:
    // loaded without a condition in the way, a batch is one (200,000 x 2,000 in one
    // group, 782 chunks: 98 us, 331 one by one).  Groups of few chunks go without: the
    // registers cost them more (6,000 x 8,000, 20 groups: 58 us a call, 62 with batches;
    // 20,000 x 33,000, 600 groups 482 and 534).
    constexpr uint32_t kBatchChunks = 16u;
    auto load_batch = [&](uint32_t c, float (&x)[kBatchChunks][4]) {
        const float *p = partials + (std::size_t) c * 4u * pstride + (kept[0] ? f0 : 0u);
#pragma unroll
        for (uint32_t u = 0; u < kBatchChunks; ++u)
#pragma unroll
            for (unsigned a = 0; a < 4u; ++a) x[u][a] = __ldg(p + (u * 4u + a) * (std::size_t) pstride);
    };
    float rs[C], rq[C], rm[C], rv[C];
    double dm[C], dv[C];
#pragma unroll
    for (int k = 0; k < C; ++k) {
        rs[k] = rq[k] = rm[k] = rv[k] = 0.0f;
        dm[k] = dv[k] = 0.0;
    }
    if (scheme == CS_MOMENTS_TWOSUM_F64_COMBINE) {
        double s[C], q[C];
#pragma unroll
        for (int k = 0; k < C; ++k) s[k] = q[k] = 0.0;
        uint32_t c = c0;
        if constexpr (kLong) {
            for (; c + kBatchChunks <= c1; c += kBatchChunks) {
                float x[kBatchChunks][4];
                load_batch(c, x);
#pragma unroll
                for (uint32_t u = 0; u < kBatchChunks; ++u) {
                    s[0] += (double) x[u][0] + (double) x[u][1];
                    q[0] += (double) x[u][2] + (double) x[u][3];
                }
            }
        }
#pragma unroll (8 / C)
        for (; c < c1; ++c) {
            const float *p = partials + (std::size_t) c * 4u * pstride + f0;
            float x[C][4];
#pragma unroll
            for (int k = 0; k < C; ++k)
#pragma unroll
                for (unsigned a = 0; a < 4u; ++a) x[k][a] = kept[k] ? p[a * (std::size_t) pstride + 256u * k] : 0.0f;
#pragma unroll
            for (int k = 0; k < C; ++k) {
                s[k] += (double) x[k][0] + (double) x[k][1];
                q[k] += (double) x[k][2] + (double) x[k][3];
            }
        }
        const double by_n = (double) n, by_dof = (double) (n > ddof ? n - ddof : 1u);
        const double inv_n = 1.0 / by_n, inv_dof = 1.0 / by_dof;
#pragma unroll
        for (int k = 0; k < C; ++k) {
            rs[k] = (float) s[k];
            rq[k] = (float) q[k];
            if (kept[k] && n > 0u) {
                dm[k] = C == 1 ? s[k] / by_n : divide_by(s[k], by_n, inv_n);
                if (n > ddof) {
                    double m2 = q[k] - s[k] * dm[k];
                    if (m2 < 0.0) m2 = 0.0;
                    dv[k] = C == 1 ? m2 / by_dof : divide_by(m2, by_dof, inv_dof);
                }
            }
            rm[k] = (float) dm[k];
            rv[k] = (float) dv[k];
        }
    } else {
#pragma unroll
        for (int k = 0; k < C; ++k) {
            if (!kept[k]) continue;
            float s_hi = 0.0f, s_lo = 0.0f, q_hi = 0.0f, q_lo = 0.0f;
            auto add = [&](const float (&x)[4]) {
                if (scheme == CS_MOMENTS_TWOSUM_F32) {
                    two_sum_acc(s_hi, s_lo, x[0]);
                    s_lo = __fadd_rn(s_lo, x[1]);
                    two_sum_acc(q_hi, q_lo, x[2]);
                    q_lo = __fadd_rn(q_lo, x[3]);
                } else {
                    s_hi = __fadd_rn(s_hi, x[0]);
                    q_hi = __fadd_rn(q_hi, x[2]);
                }
            };
            uint32_t c = c0;
            if constexpr (kLong) {
                for (; c + kBatchChunks <= c1; c += kBatchChunks) {
                    float x[kBatchChunks][4];
                    load_batch(c, x);
#pragma unroll
                    for (uint32_t u = 0; u < kBatchChunks; ++u) add(x[u]);
                }
            }
            for (; c < c1; ++c) {
                const float *p = partials + (std::size_t) c * 4u * pstride + f0 + 256u * k;
                const float x[4] = {p[0], p[pstride], p[2u * (std::size_t) pstride], p[3u * (std::size_t) pstride]};
                add(x);
            }
            rs[k] = __fadd_rn(s_hi, s_lo);
            rq[k] = __fadd_rn(q_hi, q_lo);
            if (n > 0u) {
                rm[k] = __fdiv_rn(rs[k], (float) n);
                if (n > ddof) {
                    float m2 = __fsub_rn(rq[k], __fmul_rn(rs[k], rm[k]));
                    if (m2 < 0.0f) m2 = 0.0f;
                    rv[k] = __fdiv_rn(m2, (float) (n - ddof));
                }
            }
            dm[k] = rm[k];
            dv[k] = rv[k];
        }
    }
#pragma unroll
    for (int k = 0; k < C; ++k) {
        const uint32_t f = f0 + 256u * k;
        if (f >= cols) continue;
        const std::size_t o = (std::size_t) g * cols + f;
        out_sum[o] = rs[k];
        out_sumsq[o] = rq[k];
        if (out_mean != nullptr) out_mean[o] = rm[k];
        if (out_var != nullptr) out_var[o] = rv[k];
        if (out_mean64 != nullptr) out_mean64[o] = dm[k];
        if (out_var64 != nullptr) out_var64[o] = dv[k];
    }
}

template <int L, bool COMP, typename Rows>
int launch_accumulate_rows(const Rows &rows_of, uint32_t block_size, uint32_t cols, const moments_layout &lay,
                           const uint32_t *chunk_first, uint32_t g_lo, uint32_t g_hi, cudaStream_t stream) {
    const uint32_t segs = lay.col_blocks * (block_size / L);
    dim3 grid(lay.max_chunks, (segs + kAccThreads - 1u) / kAccThreads);
    const std::size_t smem = (std::size_t) lay.chunk_rows * sizeof(typename Rows::entry);
    auto kern = lay.short_chunks ? moments_accumulate_kernel<L, COMP, true, Rows>
                                 : moments_accumulate_kernel<L, COMP, false, Rows>;
    if (smem > 48u * 1024u &&
        !cuda_ok(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem),
                 "moments smem attribute"))
        return 0;
    kern<<<grid, kAccThreads, smem, stream>>>(rows_of, block_size, lay.col_blocks, cols, lay.pstride, lay.chunks,
                                              lay.num_chunks, lay.partials, chunk_first, g_lo, g_hi);
    return launch_ok("moments_accumulate_kernel");
}

template <int L, bool COMP>
int launch_accumulate(const cs_blocked_ell_view *src, const moments_layout &lay, const uint32_t *chunk_first,
                      uint32_t g_lo, uint32_t g_hi, cudaStream_t stream) {
    const one_partition_rows rows_of{reinterpret_cast<const uint16_t *>(src->val), lay.index, lay.sorted_rows,
                                     src->ell_cols, src->block_size, lay.words};
    return launch_accumulate_rows<L, COMP>(rows_of, src->block_size, src->cols, lay, chunk_first, g_lo, g_hi, stream);
}

int validate(const cs_blocked_ell_view *src, const cs_group_moments_params *p) {
    if (src == nullptr || p == nullptr) {
        set_error("group_moments: null view or params");
        return 0;
    }
    if (src->block_size == 0u || src->ell_cols % src->block_size != 0u) {
        set_error("group_moments: block_size %u does not divide ell_cols %u", src->block_size, src->ell_cols);
        return 0;
    }
    if (p->group_count == 0u || p->group_count > CS_MAX_MOMENT_GROUPS) {
        set_error("group_moments: group_count %u outside [1, %u]", p->group_count, CS_MAX_MOMENT_GROUPS);
        return 0;
    }
    if (p->scheme > CS_MOMENTS_TWOSUM_F64_COMBINE) {
        set_error("group_moments: unknown scheme %u", p->scheme);
        return 0;
    }
    if (p->chunk_rows > kMaxChunkRows) {
        set_error("group_moments: chunk_rows %u above %u", p->chunk_rows, kMaxChunkRows);
        return 0;
    }
    const uint32_t col_blocks = (src->cols + src->block_size - 1u) / src->block_size;
    if ((col_blocks + 31u) / 32u > kMaxIndexWords) {
        set_error("group_moments: %u column blocks exceed the index limit", col_blocks);
        return 0;
    }
    return 1;
}

// A shard's partitions, passed to moments_row_ptrs_kernel by value (the
// table travels in the launch, so nothing of the host call outlives it).
struct moment_part {
    const uint16_t *val;
    const uint2 *index;
    uint32_t row0;     // first global row of the partition
    uint32_t ell_cols;
};
struct moment_part_table {
    moment_part p[CS_MOMENTS_MAX_PARTS];
    uint32_t count, block_size, words, pad;
};

// row_ptrs[i] = (address of sorted row i's values, address of its row
// block's index entries) for the kept rows of all groups.
__global__ void __launch_bounds__(256) moments_row_ptrs_kernel(moment_part_table T,
                                                              const uint32_t *__restrict__ sorted_rows,
                                                              const uint32_t *__restrict__ group_offsets, uint32_t G,
                                                              ulonglong2 *__restrict__ row_ptrs) {
    __shared__ uint32_t row0[CS_MOMENTS_MAX_PARTS];
    for (uint32_t k = threadIdx.x; k < T.count; k += blockDim.x) row0[k] = T.p[k].row0;
    __syncthreads();
    const uint32_t total = group_offsets[G];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const uint32_t r = sorted_rows[i];
        uint32_t lo = 0u, hi = T.count - 1u; // last partition whose first row is <= r
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1u) >> 1;
            if (row0[mid] <= r)
                lo = mid;
            else
                hi = mid - 1u;
        }
        const uint32_t local = r - row0[lo];
        const uint16_t *v = T.p[lo].val + (std::size_t) local * T.p[lo].ell_cols;
        const uint2 *x = T.p[lo].index + (std::size_t) (local / T.block_size) * T.words;
        row_ptrs[i] = make_ulonglong2((unsigned long long) v, (unsigned long long) x);
    }
}

// Stable sort of the kept rows [0, rows) by label into lay.sorted_rows, with
// each group's rows cut into chunks (prepare phase, after the index).
int sort_rows_by_label(const moments_layout &lay, uint32_t rows, const uint8_t *d_row_keep,
                       const uint32_t *d_row_labels, uint32_t G, cudaStream_t stream) {
    const std::size_t sort_smem = (std::size_t) kSortWarps * G * sizeof(uint32_t);
    // up to four steps of 32 tiles a warp the scan's one CTA totals the groups itself,
    // a launch less (us a call, two kernels / one: 8,000 x 1,000, 30 groups 34.1 / 30.1;
    // 20,000 rows, 100 groups 38.1 / 37.2; past it 20,000 rows, 250 groups 41.1 / 43.6)
    const bool fused = lay.tiles != 0u && (uint64_t) ((G + 31u) / 32u) * ((lay.tiles + 31u) / 32u) <= kScanSteps;
    if (lay.tiles != 0u) {
        const std::size_t hist_smem = (std::size_t) G * sizeof(uint32_t);
        moments_tile_hist_kernel<<<lay.tiles, kSortThreads, hist_smem, stream>>>(rows, d_row_keep, d_row_labels, G,
                                                                                lay.tile_counts);
        if (!launch_ok("moments_tile_hist_kernel")) return 0;
        if (!fused) {
            moments_group_tiles_kernel<<<(G + 7u) / 8u, 256, 0, stream>>>(lay.tiles, G, lay.tile_counts,
                                                                          lay.group_rows);
            if (!launch_ok("moments_group_tiles_kernel")) return 0;
        }
    } else if (!cuda_ok(cudaMemsetAsync(lay.group_rows, 0, (std::size_t) G * sizeof(uint32_t), stream),
                        "group rows memset")) {
        return 0;
    }
    auto scan = fused ? moments_group_scan_kernel<true> : moments_group_scan_kernel<false>;
    scan<<<1, 1024, 0, stream>>>(G, lay.chunk_rows, lay.max_chunks, lay.tiles, lay.tile_counts, lay.group_rows,
                                 lay.group_offsets, lay.chunk_first, lay.num_chunks, lay.chunks);
    if (!launch_ok("moments_group_scan_kernel")) return 0;
    if (lay.tiles != 0u) {
        if (sort_smem > 48u * 1024u &&
            !cuda_ok(cudaFuncSetAttribute(moments_tile_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int) sort_smem),
                     "scatter smem attribute"))
            return 0;
        moments_tile_scatter_kernel<<<lay.tiles, kSortThreads, sort_smem, stream>>>(
            rows, d_row_keep, d_row_labels, G, lay.tile_counts, lay.group_offsets, lay.sorted_rows);
        if (!launch_ok("moments_tile_scatter_kernel")) return 0;
    }
    return 1;
}

// Combine phase for groups [g_lo, g_hi).
int combine_groups(const moments_layout &lay, uint32_t cols, const cs_group_moments_params *params,
                   const uint8_t *d_feature_keep, const cs_group_moments_out *out, uint32_t g_lo, uint32_t g_hi,
                   cudaStream_t stream) {
    // four columns a thread once that still fills the device (two CTAs of 256 per SM)
    const uint32_t four = std::max(1u, (cols + 1023u) / 1024u), one = std::max(1u, (cols + 255u) / 256u);
    auto launch = [&](auto kern, uint32_t tiles) {
        kern<<<dim3(tiles, g_hi - g_lo), 256, 0, stream>>>(cols, lay.pstride, params->group_count, params->scheme,
                                                           params->ddof, lay.chunk_first, lay.group_rows, lay.partials,
                                                           d_feature_keep, out->sum, out->sumsq, out->mean, out->var,
                                                           out->mean64, out->var64, out->group_rows, g_lo);
    };
    const bool many_chunks = lay.max_chunks / params->group_count > 32u;
    if ((uint64_t) four * (g_hi - g_lo) >= 2u * (uint64_t) sm_count()) launch(moments_combine_kernel<4, false>, four);
    else if (many_chunks) launch(moments_combine_kernel<1, true>, one);
    else launch(moments_combine_kernel<1, false>, one);
    return launch_ok("moments_combine_kernel");
}

} // namespace
} // namespace csb

using namespace csb;

extern "C" int cs_b200_group_moments_scratch_bytes(const cs_blocked_ell_view *src, const cs_group_moments_params *params,
                                                   size_t *out_bytes) {
    if (!validate(src, params) || out_bytes == nullptr) {
        if (out_bytes == nullptr) set_error("group_moments_scratch_bytes: null output");
        return 0;
    }
    moments_layout lay;
    make_layout(src, params, nullptr, 0, &lay);
    *out_bytes = lay.bytes;
    return 1;
}

static int moments_run(const cs_blocked_ell_view *src, const uint8_t *d_row_keep, const uint8_t *d_feature_keep,
                       const uint32_t *d_row_labels, const cs_group_moments_params *params,
                       const cs_group_moments_out *out, void *d_scratch, size_t scratch_bytes, cs_stream_t s,
                       uint32_t phases, uint32_t g_lo = 0u, uint32_t g_hi = 0xffffffffu) {
    if (!validate(src, params)) return 0;
    if (out == nullptr || out->sum == nullptr || out->sumsq == nullptr) {
        set_error("group_moments: sum and sumsq outputs are required");
        return 0;
    }
    moments_layout lay;
    if (!fit_scratch(params, [&](const cs_group_moments_params &p, bool padded) {
            return make_layout(src, &p, d_scratch, scratch_bytes, &lay, padded);
        }) ||
        d_scratch == nullptr) {
        set_error("group_moments: scratch too small (%zu bytes, need %zu)", scratch_bytes, lay.bytes);
        return 0;
    }
    if (src->rows != 0u && src->ell_cols != 0u && (src->val == nullptr || src->blockColIdx == nullptr)) {
        set_error("group_moments: null view arrays");
        return 0;
    }
    cudaStream_t stream = as_stream(s);
    const uint32_t G = params->group_count;
    const uint32_t width = src->ell_cols / src->block_size;
    // a column-block index the caller built once for this partition replaces the scratch one
    const bool prebuilt = params->index != nullptr;
    if (prebuilt) lay.index = static_cast<uint2 *>(const_cast<void *>(params->index));
    // accumulate and combine may be restricted to groups [g_lo, g_hi)
    if (g_hi > G) g_hi = G;
    const bool all_groups = g_lo == 0u && g_hi == G;
    if (g_lo >= g_hi) return 1;
    const uint32_t *range_first = all_groups ? nullptr : lay.chunk_first;

    if ((phases & CS_MOMENTS_PHASE_PREPARE) && !prebuilt && lay.row_blocks != 0u && lay.words != 0u) {
        if (width != 0u) {
            const uint32_t blocks = (lay.row_blocks + kIndexWarps - 1u) / kIndexWarps;
            const std::size_t smem = (std::size_t) kIndexWarps * lay.words * sizeof(uint32_t);
            if (smem > 48u * 1024u &&
                !cuda_ok(cudaFuncSetAttribute(moments_index_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int) smem),
                         "index smem attribute"))
                return 0;
            moments_index_kernel<<<blocks, kIndexWarps * 32, smem, stream>>>(
                src->blockColIdx, lay.row_blocks, width, lay.col_blocks, lay.words, lay.index, out->status,
                (width % 4u) == 0u && (reinterpret_cast<uintptr_t>(src->blockColIdx) & 15u) == 0u);
            if (!launch_ok("moments_index_kernel")) return 0;
        } else if (!cuda_ok(cudaMemsetAsync(lay.index, 0, (std::size_t) lay.row_blocks * lay.words * sizeof(uint2),
                                            stream),
                            "index memset")) {
            return 0;
        }
    }

    if ((phases & CS_MOMENTS_PHASE_PREPARE) && !sort_rows_by_label(lay, src->rows, d_row_keep, d_row_labels, G, stream))
        return 0;

    if ((phases & CS_MOMENTS_PHASE_ACCUMULATE) && lay.col_blocks != 0u && lay.max_chunks != 0u && src->cols != 0u) {
        const bool comp = params->scheme != CS_MOMENTS_PLAIN_F32;
        const uint32_t B = src->block_size;
        const bool aligned16 = (reinterpret_cast<uintptr_t>(src->val) & 15u) == 0u;
        int ok;
#define CS_ACC(L_)                                                                                     \
    (comp ? launch_accumulate<L_, true>(src, lay, range_first, g_lo, g_hi, stream)                      \
          : launch_accumulate<L_, false>(src, lay, range_first, g_lo, g_hi, stream))
        if (B % 8u == 0u && aligned16)
            ok = CS_ACC(8);
        else if (B % 4u == 0u && (reinterpret_cast<uintptr_t>(src->val) & 7u) == 0u)
            ok = CS_ACC(4);
        else if (B % 2u == 0u && (reinterpret_cast<uintptr_t>(src->val) & 3u) == 0u)
            ok = CS_ACC(2);
        else
            ok = CS_ACC(1);
#undef CS_ACC
        if (!ok) return 0;
    }

    if ((phases & CS_MOMENTS_PHASE_COMBINE) && (src->cols != 0u || out->group_rows != nullptr) &&
        !combine_groups(lay, src->cols, params, d_feature_keep, out, g_lo, g_hi, stream))
        return 0;
    return 1;
}

namespace csb {

// Column-block index of a Blocked-ELL partition (index[rb * words + w] =
// (occupancy bits of column blocks 32w..32w+31, slots before them)), as the
// moments prepare phase builds it; used by the serving loop, which keeps one
// per staged partition.  words = ceil(ceil(cols / block_size) / 32).
int build_column_block_index(const cs_blocked_ell_view *src, uint2 *index, uint32_t *status, cudaStream_t stream) {
    const uint32_t B = src->block_size;
    const uint32_t row_blocks = (src->rows + B - 1u) / B;
    const uint32_t col_blocks = (src->cols + B - 1u) / B;
    const uint32_t words = (col_blocks + 31u) / 32u;
    if (row_blocks == 0u || words == 0u) return 1;
    const uint32_t width = src->ell_cols / B;
    if (width == 0u)
        return cuda_ok(cudaMemsetAsync(index, 0, (std::size_t) row_blocks * words * sizeof(uint2), stream),
                       "index memset");
    const uint32_t blocks = (row_blocks + kIndexWarps - 1u) / kIndexWarps;
    const std::size_t smem = (std::size_t) kIndexWarps * words * sizeof(uint32_t);
    if (smem > 48u * 1024u &&
        !cuda_ok(cudaFuncSetAttribute(moments_index_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem),
                 "index smem attribute"))
        return 0;
    moments_index_kernel<<<blocks, kIndexWarps * 32, smem, stream>>>(
        src->blockColIdx, row_blocks, width, col_blocks, words, index, status,
        (width % 4u) == 0u && (reinterpret_cast<uintptr_t>(src->blockColIdx) & 15u) == 0u);
    return launch_ok("moments_index_kernel");
}

std::size_t column_block_index_bytes(const cs_blocked_ell_view *src) {
    const uint32_t B = src->block_size;
    const std::size_t row_blocks = (src->rows + B - 1u) / B;
    const std::size_t words = (((std::size_t) src->cols + B - 1u) / B + 31u) / 32u;
    return (row_blocks * words + 1u) * sizeof(uint2);
}

// Scratch bytes the moments reduction needs at least for (src, params); 0 when the
// arguments are invalid (the error message is set).
std::size_t group_moments_scratch_needed(const cs_blocked_ell_view *src, const cs_group_moments_params *params) {
    if (!validate(src, params)) return 0;
    moments_layout lay;
    make_layout(src, params, nullptr, 0, &lay, false);
    return lay.bytes;
}

// The full reduction over caller-provided scratch (used by the entry points
// in this file and by the static-scratch entry point).
int group_moments_launch(const cs_blocked_ell_view *src, const uint8_t *d_row_keep, const uint8_t *d_feature_keep,
                         const uint32_t *d_row_labels, const cs_group_moments_params *params,
                         const cs_group_moments_out *out, void *d_scratch, size_t scratch_bytes, cs_stream_t s) {
    return moments_run(src, d_row_keep, d_feature_keep, d_row_labels, params, out, d_scratch, scratch_bytes, s,
                       CS_MOMENTS_PHASE_ALL);
}

} // namespace csb

extern "C" int cs_b200_group_moments_blocked_ell(const cs_blocked_ell_view *src, const uint8_t *d_row_keep,
                                                  const uint8_t *d_feature_keep, const uint32_t *d_row_labels,
                                                  const cs_group_moments_params *params,
                                                  const cs_group_moments_out *out, void *d_scratch,
                                                  size_t scratch_bytes, cs_stream_t s) {
    return moments_run(src, d_row_keep, d_feature_keep, d_row_labels, params, out, d_scratch, scratch_bytes, s,
                       CS_MOMENTS_PHASE_ALL);
}

extern "C" int cs_b200_group_moments_index_bytes(const cs_blocked_ell_view *src, size_t *out_bytes) {
    if (src == nullptr || out_bytes == nullptr || src->block_size == 0u) {
        set_error("group_moments_index_bytes: null argument or zero block size");
        return 0;
    }
    *out_bytes = column_block_index_bytes(src);
    return 1;
}

extern "C" int cs_b200_group_moments_build_index(const cs_blocked_ell_view *src, void *d_index, uint32_t *d_status,
                                                  cs_stream_t s) {
    if (src == nullptr || d_index == nullptr || src->block_size == 0u || src->ell_cols % src->block_size != 0u ||
        (src->rows != 0u && src->ell_cols != 0u && src->blockColIdx == nullptr)) {
        set_error("group_moments_build_index: null argument, zero block size or block size not dividing ell_cols");
        return 0;
    }
    const uint32_t col_blocks = (src->cols + src->block_size - 1u) / src->block_size;
    if ((col_blocks + 31u) / 32u > kMaxIndexWords) {
        set_error("group_moments_build_index: %u column blocks exceed the index limit", col_blocks);
        return 0;
    }
    return build_column_block_index(src, static_cast<uint2 *>(d_index), d_status, as_stream(s));
}

extern "C" int cs_b200_group_moments_phases(const cs_blocked_ell_view *src, const uint8_t *d_row_keep,
                                            const uint8_t *d_feature_keep, const uint32_t *d_row_labels,
                                            const cs_group_moments_params *params, const cs_group_moments_out *out,
                                            void *d_scratch, size_t scratch_bytes, uint32_t phases, cs_stream_t s) {
    if ((phases & ~(uint32_t) CS_MOMENTS_PHASE_ALL) != 0u) {
        set_error("group_moments_phases: unknown phase bits 0x%x", phases);
        return 0;
    }
    return moments_run(src, d_row_keep, d_feature_keep, d_row_labels, params, out, d_scratch, scratch_bytes, s,
                       phases);
}

// ---------------------------------------------------------------------------
// The reduction over a shard given as its partitions' views, in one call.
// ---------------------------------------------------------------------------
namespace {

struct parts_layout {
    moments_layout base;    // over all rows of the shard
    uint2 *part_index;      // per-partition column-block indexes built by the call
    ulonglong2 *row_ptrs;   // [rows]
    std::size_t bytes;
    uint32_t rows;
};

int validate_parts(const cs_blocked_ell_view *parts, uint32_t count, const cs_group_moments_params *params,
                   cs_blocked_ell_view *whole) {
    if (parts == nullptr || count == 0u || count > CS_MOMENTS_MAX_PARTS) {
        set_error("group_moments_parts: %u partitions (need 1..%u)", count, CS_MOMENTS_MAX_PARTS);
        return 0;
    }
    uint64_t rows = 0;
    for (uint32_t k = 0; k < count; ++k) {
        if (!validate(&parts[k], params)) return 0;
        if (parts[k].cols != parts[0].cols || parts[k].block_size != parts[0].block_size) {
            set_error("group_moments_parts: partition %u has cols %u / block size %u, partition 0 %u / %u", k,
                      parts[k].cols, parts[k].block_size, parts[0].cols, parts[0].block_size);
            return 0;
        }
        if (parts[k].rows != 0u && parts[k].ell_cols != 0u &&
            (parts[k].val == nullptr || parts[k].blockColIdx == nullptr)) {
            set_error("group_moments_parts: partition %u has null arrays", k);
            return 0;
        }
        rows += parts[k].rows;
    }
    if (rows >= 0xffffffffull) {
        set_error("group_moments_parts: %llu rows exceed the u32 row ids", (unsigned long long) rows);
        return 0;
    }
    *whole = parts[0];
    whole->rows = (uint32_t) rows;
    return 1;
}

bool make_parts_layout(const cs_blocked_ell_view *parts, uint32_t count, const cs_blocked_ell_view &whole,
                       const cs_group_moments_params *params, void *base, std::size_t cap, parts_layout *pl,
                       bool padded = true) {
    make_layout(&whole, params, base, cap, &pl->base, padded);
    const uint32_t B = whole.block_size;
    std::size_t blocks = 0;
    for (uint32_t k = 0; k < count; ++k) blocks += (parts[k].rows + B - 1u) / B;
    scratch_carver c(base, cap);
    c.used = pl->base.bytes;
    pl->part_index = c.take<uint2>(blocks * pl->base.words + 1u);
    pl->row_ptrs = c.take<ulonglong2>((std::size_t) whole.rows + 1u);
    pl->bytes = c.used;
    pl->rows = whole.rows;
    return c.fits();
}

} // namespace

extern "C" int cs_b200_group_moments_parts_scratch_bytes(const cs_blocked_ell_view *parts, uint32_t count,
                                                          const cs_group_moments_params *params, size_t *out_bytes) {
    cs_blocked_ell_view whole;
    if (out_bytes == nullptr) {
        set_error("group_moments_parts_scratch_bytes: null output");
        return 0;
    }
    if (!validate_parts(parts, count, params, &whole)) return 0;
    parts_layout pl;
    make_parts_layout(parts, count, whole, params, nullptr, 0, &pl);
    *out_bytes = pl.bytes;
    return 1;
}

extern "C" int cs_b200_group_moments_blocked_ell_parts(const cs_blocked_ell_view *parts, uint32_t count,
                                                       const void *const *d_indexes, const uint8_t *d_row_keep,
                                                       const uint8_t *d_feature_keep, const uint32_t *d_row_labels,
                                                       const cs_group_moments_params *params,
                                                       const cs_group_moments_out *out, void *d_scratch,
                                                       size_t scratch_bytes, cs_stream_t s) {
    cs_blocked_ell_view whole;
    if (!validate_parts(parts, count, params, &whole)) return 0;
    if (out == nullptr || out->sum == nullptr || out->sumsq == nullptr) {
        set_error("group_moments_parts: sum and sumsq outputs are required");
        return 0;
    }
    parts_layout pl;
    if (!fit_scratch(params, [&](const cs_group_moments_params &p, bool padded) {
            return make_parts_layout(parts, count, whole, &p, d_scratch, scratch_bytes, &pl, padded);
        }) ||
        d_scratch == nullptr) {
        set_error("group_moments_parts: scratch too small (%zu bytes, need %zu)", scratch_bytes, pl.bytes);
        return 0;
    }
    cudaStream_t stream = as_stream(s);
    const moments_layout &lay = pl.base;
    const uint32_t G = params->group_count, B = whole.block_size;
    moment_part_table T{};
    T.count = count;
    T.block_size = B;
    T.words = lay.words;
    uint32_t row0 = 0u;
    std::size_t built = 0;
    for (uint32_t k = 0; k < count; ++k) {
        const uint2 *idx = d_indexes != nullptr ? static_cast<const uint2 *>(d_indexes[k]) : nullptr;
        if (idx == nullptr) {
            uint2 *mine = pl.part_index + built * lay.words;
            built += (parts[k].rows + B - 1u) / B;
            if (!build_column_block_index(&parts[k], mine, out->status, stream)) return 0;
            idx = mine;
        }
        T.p[k] = moment_part{reinterpret_cast<const uint16_t *>(parts[k].val), idx, row0, parts[k].ell_cols};
        row0 += parts[k].rows;
    }
    if (!sort_rows_by_label(lay, whole.rows, d_row_keep, d_row_labels, G, stream)) return 0;
    if (whole.rows != 0u) {
        const unsigned grid = resident_grid(reinterpret_cast<const void *>(moments_row_ptrs_kernel), 256, 0,
                                            (whole.rows + 255u) / 256u);
        moments_row_ptrs_kernel<<<grid, 256, 0, stream>>>(T, lay.sorted_rows, lay.group_offsets, G, pl.row_ptrs);
        if (!launch_ok("moments_row_ptrs_kernel")) return 0;
    }
    if (lay.col_blocks != 0u && lay.max_chunks != 0u && whole.cols != 0u) {
        const bool comp = params->scheme != CS_MOMENTS_PLAIN_F32;
        bool a16 = true, a8 = true, a4 = true;
        for (uint32_t k = 0; k < count; ++k) {
            const uintptr_t v = reinterpret_cast<uintptr_t>(parts[k].val);
            const uint32_t rowb = parts[k].ell_cols * 2u; // a row's bytes: every row start keeps the base alignment
            a16 = a16 && (v & 15u) == 0u && rowb % 16u == 0u;
            a8 = a8 && (v & 7u) == 0u && rowb % 8u == 0u;
            a4 = a4 && (v & 3u) == 0u && rowb % 4u == 0u;
        }
        const many_partition_rows rows_of{pl.row_ptrs};
        int ok;
#define CS_ACCM(L_)                                                                                       \
    (comp ? launch_accumulate_rows<L_, true>(rows_of, B, whole.cols, lay, nullptr, 0u, G, stream)         \
          : launch_accumulate_rows<L_, false>(rows_of, B, whole.cols, lay, nullptr, 0u, G, stream))
        if (B % 8u == 0u && a16)
            ok = CS_ACCM(8);
        else if (B % 4u == 0u && a8)
            ok = CS_ACCM(4);
        else if (B % 2u == 0u && a4)
            ok = CS_ACCM(2);
        else
            ok = CS_ACCM(1);
#undef CS_ACCM
        if (!ok) return 0;
    }
    if (whole.cols != 0u || out->group_rows != nullptr)
        return combine_groups(lay, whole.cols, params, d_feature_keep, out, 0u, G, stream);
    return 1;
}

namespace {

// Copy stream and events of the host-delivery entry point, one set per host
// thread and device ordinal (created on first use on that device, kept for the
// thread's lifetime, so a thread that moves between devices creates nothing
// new after its first call on each).
struct host_copy_ctx {
    cudaStream_t copy = nullptr;
    cudaEvent_t ready = nullptr, done = nullptr;
};

constexpr int kCopyDevices = 64;

host_copy_ctx *host_copy_setup() {
    thread_local host_copy_ctx ctxs[kCopyDevices];
    int dev = 0;
    if (!cuda_ok(cudaGetDevice(&dev), "get device")) return nullptr;
    if (dev < 0 || dev >= kCopyDevices) {
        set_error("group_moments_to_host: device ordinal %d outside the supported range", dev);
        return nullptr;
    }
    host_copy_ctx &c = ctxs[dev];
    if (c.copy != nullptr && c.ready != nullptr && c.done != nullptr) return &c;
    // a set-up that failed partway keeps what it created and completes it now
    if (c.copy == nullptr && !cuda_ok(cudaStreamCreateWithFlags(&c.copy, cudaStreamNonBlocking), "copy stream"))
        return nullptr;
    if (c.ready == nullptr && !cuda_ok(cudaEventCreateWithFlags(&c.ready, cudaEventDisableTiming), "copy event"))
        return nullptr;
    if (c.done == nullptr && !cuda_ok(cudaEventCreateWithFlags(&c.done, cudaEventDisableTiming), "copy event"))
        return nullptr;
    return &c;
}

template <typename T>
bool copy_rows(T *h, const T *d, uint32_t g0, uint32_t g1, std::size_t row_elems, cudaStream_t copy) {
    if (h == nullptr || d == nullptr || g1 <= g0) return true;
    return cuda_ok(cudaMemcpyAsync(h + (std::size_t) g0 * row_elems, d + (std::size_t) g0 * row_elems,
                                   (std::size_t) (g1 - g0) * row_elems * sizeof(T), cudaMemcpyDeviceToHost, copy),
                   "moments D2H") != 0;
}

} // namespace

extern "C" int cs_b200_group_moments_to_host(const cs_blocked_ell_view *src, const uint8_t *d_row_keep,
                                             const uint8_t *d_feature_keep, const uint32_t *d_row_labels,
                                             const cs_group_moments_params *params, const cs_group_moments_out *d_out,
                                             const cs_group_moments_out *h_out, void *d_scratch,
                                             size_t scratch_bytes, uint32_t parts, cs_stream_t s) {
    if (h_out == nullptr || d_out == nullptr) {
        set_error("group_moments_to_host: null outputs");
        return 0;
    }
    const struct {
        const void *h, *d;
        const char *name;
    } fields[] = {{h_out->sum, d_out->sum, "sum"},          {h_out->sumsq, d_out->sumsq, "sumsq"},
                  {h_out->mean, d_out->mean, "mean"},       {h_out->var, d_out->var, "var"},
                  {h_out->mean64, d_out->mean64, "mean64"}, {h_out->var64, d_out->var64, "var64"},
                  {h_out->group_rows, d_out->group_rows, "group_rows"}};
    for (const auto &f : fields)
        if (f.h != nullptr && f.d == nullptr) {
            set_error("group_moments_to_host: host %s given without its device array", f.name);
            return 0;
        }
    if (!validate(src, params)) return 0;
    const uint32_t G = params->group_count;
    if (parts == 0u) parts = 2u;
    if (parts > G) parts = G;
    cudaStream_t stream = as_stream(s);
    if (!moments_run(src, d_row_keep, d_feature_keep, d_row_labels, params, d_out, d_scratch, scratch_bytes, s,
                     CS_MOMENTS_PHASE_PREPARE))
        return 0;
    host_copy_ctx *cp = host_copy_setup();
    if (cp == nullptr) return 0;
    host_copy_ctx &ctx = *cp;
    const std::size_t cols = src->cols;
    for (uint32_t k = 0; k < parts; ++k) {
        const uint32_t g0 = (uint32_t) ((uint64_t) k * G / parts), g1 = (uint32_t) ((uint64_t) (k + 1u) * G / parts);
        if (g1 <= g0) continue;
        // groups [g0, g1) accumulated and combined; their rows copy while the next part computes
        if (!moments_run(src, d_row_keep, d_feature_keep, d_row_labels, params, d_out, d_scratch, scratch_bytes, s,
                         CS_MOMENTS_PHASE_ACCUMULATE | CS_MOMENTS_PHASE_COMBINE, g0, g1) ||
            !cuda_ok(cudaEventRecord(ctx.ready, stream), "part event") ||
            !cuda_ok(cudaStreamWaitEvent(ctx.copy, ctx.ready, 0), "copy wait") ||
            !copy_rows(h_out->sum, d_out->sum, g0, g1, cols, ctx.copy) ||
            !copy_rows(h_out->sumsq, d_out->sumsq, g0, g1, cols, ctx.copy) ||
            !copy_rows(h_out->mean, d_out->mean, g0, g1, cols, ctx.copy) ||
            !copy_rows(h_out->var, d_out->var, g0, g1, cols, ctx.copy) ||
            !copy_rows(h_out->mean64, d_out->mean64, g0, g1, cols, ctx.copy) ||
            !copy_rows(h_out->var64, d_out->var64, g0, g1, cols, ctx.copy) ||
            !copy_rows(h_out->group_rows, d_out->group_rows, g0, g1, 1u, ctx.copy))
            return 0;
    }
    if (h_out->status != nullptr && d_out->status != nullptr &&
        !cuda_ok(cudaMemcpyAsync(h_out->status, d_out->status, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx.copy),
                 "status D2H"))
        return 0;
    // the caller's stream waits for the copies, so a sync on it covers them
    return cuda_ok(cudaEventRecord(ctx.done, ctx.copy), "copy done event") &&
           cuda_ok(cudaStreamWaitEvent(stream, ctx.done, 0), "stream wait");
}
