// Stable compressed transpose: CSR (cDim x uDim) -> CSC, row indices ascending
// inside every column -- the result of cusparseCsr2cscEx2 (ALG1), which the
// reference's build_compressed_transpose_raw uses as its primary path
// (src/convert/compressed_transpose_raw.cuh:43-81).  Its atomic fallback
// (:84-121) is order-nondeterministic and is not reproduced.
//
//   hist     rows are cut into T tiles; each CTA counts its tile's entries
//            per column in shared memory -> H[t][c].
//   colscan  per column, exclusive scan of H over tiles (in place) and the
//            column total; one device scan of the totals gives out_ptr.
//   scatter  each CTA replays its tile 16 rows at a time.  Round A sets, per
//            column, a 16-bit mask of which batch rows hold it (atomicOr in a
//            packed shared word: mask << 16 | running count); round B places
//            entry (r, c) at out_ptr[c] + H[t][c] + count + popc(mask below r);
//            round C advances the count.  Placement is therefore fixed by
//            (tile, row) order alone -- deterministic and stable.
// The one-pass path below is used only where the two-pass path (further down,
// the default) does not apply.  On the one-pass path a row that repeats a
// column sets CS_STATUS_DUPLICATE_COL in the status word at the start of the
// caller's scratch; the two-pass path keeps repeated entries, in row order.
#include "common.cuh"

#include <algorithm>
#include <type_traits>

namespace csb {
namespace {

constexpr unsigned kThreads = 512;
constexpr unsigned kBatchRows = 16;
constexpr uint32_t kColRange = 32768; // columns per shared-memory pass (128 KB)
constexpr uint32_t kMaxTileRows = 65535;

struct tr_layout {
    uint32_t *status;
    uint32_t *hist; // [tiles * uDim]
    void *scan_tmp;
    std::size_t scan_bytes;
    std::size_t bytes;
    uint32_t tiles, tile_rows, passes;
};

void make_layout(uint32_t cDim, uint32_t uDim, void *base, std::size_t cap, tr_layout *l) {
    const uint32_t sms = (uint32_t) sm_count();
    uint32_t tiles = cDim == 0u ? 1u : (cDim + 15u) / 16u;
    if (tiles > 2u * sms) tiles = 2u * sms;
    const uint32_t min_tiles = cDim == 0u ? 1u : (cDim + kMaxTileRows - 1u) / kMaxTileRows;
    if (tiles < min_tiles) tiles = min_tiles;
    if (tiles == 0u) tiles = 1u;
    l->tiles = tiles;
    l->tile_rows = cDim == 0u ? 0u : (cDim + tiles - 1u) / tiles;
    l->passes = uDim == 0u ? 0u : (uDim + kColRange - 1u) / kColRange;
    scratch_carver c(base, cap);
    l->status = c.take<uint32_t>(4);
    l->hist = c.take<uint32_t>((std::size_t) tiles * uDim + 1u);
    l->scan_bytes = scan_u32_scratch_bytes(uDim);
    l->scan_tmp = c.take<char>(l->scan_bytes);
    l->bytes = c.used;
}

__global__ void __launch_bounds__(kThreads) tr_hist_kernel(const uint32_t *__restrict__ ptr,
                                                          const uint32_t *__restrict__ idx, uint32_t cDim,
                                                          uint32_t uDim, uint32_t tile_rows,
                                                          uint32_t *__restrict__ hist, uint32_t *status) {
    extern __shared__ uint32_t tr_counts[];
    const uint32_t t = blockIdx.x;
    const uint32_t c0 = blockIdx.y * kColRange;
    const uint32_t cr = min(kColRange, uDim - c0);
    for (uint32_t k = threadIdx.x; k < cr; k += blockDim.x) tr_counts[k] = 0u;
    __syncthreads();
    const uint32_t r0 = t * tile_rows;
    const uint32_t r1 = min(cDim, r0 + tile_rows);
    uint32_t bad = 0u;
    if (r0 < r1) {
        const uint32_t a = ptr[r0], e = ptr[r1];
        for (uint32_t i = a + threadIdx.x; i < e; i += blockDim.x) {
            const uint32_t c = idx[i];
            if (c >= uDim) {
                bad |= CS_STATUS_INDEX_RANGE;
                continue;
            }
            if (c - c0 < cr) atomicAdd(tr_counts + (c - c0), 1u);
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < cr; k += blockDim.x) hist[(std::size_t) t * uDim + c0 + k] = tr_counts[k];
    if (bad) status_or(status, bad);
}

__global__ void __launch_bounds__(256) tr_colscan_kernel(uint32_t uDim, uint32_t tiles, uint32_t *__restrict__ hist,
                                                         uint32_t *__restrict__ totals) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= uDim) return;
    uint32_t run = 0u;
    for (uint32_t t = 0; t < tiles; ++t) {
        const std::size_t k = (std::size_t) t * uDim + c;
        const uint32_t v = hist[k];
        hist[k] = run;
        run += v;
    }
    totals[c] = run;
}

__global__ void __launch_bounds__(kThreads) tr_scatter_kernel(const uint32_t *__restrict__ ptr,
                                                             const uint32_t *__restrict__ idx,
                                                             const uint16_t *__restrict__ val, uint32_t cDim,
                                                             uint32_t uDim, uint32_t tile_rows,
                                                             const uint32_t *__restrict__ hist,
                                                             const uint32_t *__restrict__ out_ptr,
                                                             uint32_t *__restrict__ out_idx,
                                                             uint16_t *__restrict__ out_val, uint32_t *status) {
    extern __shared__ uint32_t tr_packed[]; // (mask << 16) | count per column of the pass
    __shared__ uint32_t rp[kBatchRows + 1];
    const uint32_t t = blockIdx.x;
    const uint32_t c0 = blockIdx.y * kColRange;
    const uint32_t cr = min(kColRange, uDim - c0);
    for (uint32_t k = threadIdx.x; k < cr; k += blockDim.x) tr_packed[k] = 0u;
    const uint32_t r0 = t * tile_rows;
    const uint32_t r1 = min(cDim, r0 + tile_rows);
    const uint32_t *hrow = hist + (std::size_t) t * uDim;
    uint32_t bad = 0u;
    for (uint32_t b0 = r0; b0 < r1; b0 += kBatchRows) {
        const uint32_t nb = min(kBatchRows, r1 - b0);
        __syncthreads();
        if (threadIdx.x <= nb) rp[threadIdx.x] = ptr[b0 + threadIdx.x];
        __syncthreads();
        const uint32_t a = rp[0], e = rp[nb];
        // round A: which batch rows hold each column
        for (uint32_t i = a + threadIdx.x; i < e; i += blockDim.x) {
            const uint32_t c = idx[i];
            if (c - c0 >= cr || c >= uDim) continue;
            uint32_t rl = 0u;
            while (rl + 1u < nb && rp[rl + 1u] <= i) ++rl;
            const uint32_t bit = 1u << (16u + rl);
            if (atomicOr(tr_packed + (c - c0), bit) & bit) bad |= CS_STATUS_DUPLICATE_COL;
        }
        __syncthreads();
        // round B: place
        for (uint32_t i = a + threadIdx.x; i < e; i += blockDim.x) {
            const uint32_t c = idx[i];
            if (c - c0 >= cr || c >= uDim) continue;
            uint32_t rl = 0u;
            while (rl + 1u < nb && rp[rl + 1u] <= i) ++rl;
            const uint32_t w = tr_packed[c - c0];
            const uint32_t mask = w >> 16;
            const uint32_t rank = (w & 0xffffu) + __popc(mask & ((1u << rl) - 1u));
            const uint32_t pos = out_ptr[c] + hrow[c] + rank;
            out_idx[pos] = b0 + rl;
            out_val[pos] = val[i];
        }
        __syncthreads();
        // round C: advance the per-column count, clear the mask
        for (uint32_t i = a + threadIdx.x; i < e; i += blockDim.x) {
            const uint32_t c = idx[i];
            if (c - c0 >= cr || c >= uDim) continue;
            uint32_t rl = 0u;
            while (rl + 1u < nb && rp[rl + 1u] <= i) ++rl;
            const uint32_t w = tr_packed[c - c0];
            const uint32_t mask = w >> 16;
            if (rl == (uint32_t) (__ffs(mask) - 1)) tr_packed[c - c0] = ((w & 0xffffu) + __popc(mask)) & 0xffffu;
        }
    }
    if (bad) status_or(status, bad);
}


// ---------------------------------------------------------------------------
// Two-pass stable transpose (default path).
//
// The one-pass scatter above appends to every column segment from every CTA
// at once; at 32,768 columns that leaves hundreds of MB of partially written
// sectors open, far beyond L2.  Here the column key is sorted in two stable
// counting-sort passes whose open write frontier is small:
//   pass 1  by bucket = column >> 8 (<= 1,024 buckets), tiles of 4,096 (COO:
//           8,192) consecutive entries; entries become packed words (row >> 5,
//           column & 255, row & 31) + values: the upper bits are the place of
//           the entry's bit in pass 2's bitmap.
//   pass 2  inside each bucket by column & 255, in chunks of <= 8,192 that
//           never cross a bucket, writing straight into the CSC.
// Each tile or chunk is reordered whole in shared memory and leaves as one
// run per digit, so global writes are long runs, not scattered entries.
// Both passes rank entries in input order (runs of a row's entries in one
// bucket; a bitmap of each column's rows, or ballots), so the result is the
// stable transpose.
// Needs cDim < 2^24 and uDim <= 262,144.
//
// The same two passes also put COO entries in row order (partition_rows_*
// below): the key is then the entry's row, the payload its column, and the low
// digit has LB = 8 to 11 bits so that up to 2,097,152 rows stay within the
// 1,024 pass-1 buckets.
// ---------------------------------------------------------------------------
constexpr unsigned kTpThreads = 256;
constexpr unsigned kTpWarps = kTpThreads / 32;
constexpr uint32_t kTpBucketBits = 8; // low digit of the transpose
constexpr uint32_t kTpMaxLowBits = 11;
constexpr uint32_t kTpMaxBuckets = 1024;
// entries per pass-1 tile (staged whole in shared memory): CSR rows leave runs of
// many entries even in small tiles, and more CTAs per SM overlap their phases
// (300,000 x 32,768: 4.69 ms against 4.98 with 8,192); COO entries are random,
// and a tile of twice the entries writes runs twice as long
constexpr uint32_t kTpTileCsr = 4096;
constexpr uint32_t kTpTileCoo = 8192;
constexpr uint32_t kTpChunk = 8192;  // entries per pass-2 chunk (staged whole in shared memory)
constexpr uint32_t kTpGran = 256;    // entries per warp per step; rows are looked up per granule

// Tiles or chunks per slice of the offset scan: 64, or 16 where that leaves only
// a few CTAs with a long chain each (365 tiles: 12 us by 64, 6 by 16).
constexpr uint32_t kTpShortSlices = 8192;
constexpr uint32_t tp_slice_len(uint32_t rows) { return rows <= kTpShortSlices ? 16u : 64u; }

// Counts of a pass, one row per tile or chunk and one column per digit, and
// what the scan over the rows of a segment makes of them: pass 1 has one
// segment (all tiles), pass 2 one per bucket (its chunks).
struct tp_counts {
    uint16_t *cnt;      // [rows][D]
    uint32_t *base;     // [rows][D] global slot of the row's first entry of the digit, less its start
    uint32_t *slices;   // [slices][D] sums, then exclusive prefixes inside the segment
    const uint32_t *start;   // [segments * D, `limit` of them] first slot of the digit; null where base has it
    const uint32_t *segment; // [rows] (null: one segment)
    uint32_t limit;
    // global slot of the row's first entry of digit d (kAdd: start is given)
    template <bool kAdd>
    __device__ __forceinline__ uint32_t first(uint32_t row, uint32_t D, uint32_t d) const {
        if constexpr (!kAdd) return base[(std::size_t) row * D + d];
        const std::size_t c = (segment != nullptr ? (std::size_t) segment[row] * D : 0u) + d;
        return base[(std::size_t) row * D + d] + (c < limit ? start[c] : 0u);
    }
};

struct tp2_layout {
    uint32_t *status;
    tp_counts one, two;
    uint32_t *total1;      // [K] entries of each bucket
    uint32_t *start1;      // [K + 1] first pass-1 slot of each bucket
    uint32_t *tmp_key;     // [nnz]
    uint16_t *tmp_val;     // [nnz]
    uint32_t *chunk_bucket; // [max_chunks]
    uint2 *chunk_range;     // [max_chunks] entries
    uint32_t *slice_bucket; // [max_slices]
    uint2 *slice_range;     // [max_slices] chunks
    uint32_t *slice_first;  // [K + 1]
    uint32_t *gran_row;     // [nnz / kTpGran + 1] row holding entry j * kTpGran
    void *scan_tmp;
    std::size_t scan_bytes, bytes;
    uint32_t K, tiles1, max_chunks, most_chunks, slice1, slice2, slices1, max_slices, low_bits;
};

bool tp2_applicable(uint32_t cDim, uint32_t uDim) {
    return cDim < (1u << 24) && uDim <= kTpMaxBuckets * 256u;
}

void tp2_make_layout(uint32_t uDim, uint32_t nnz, uint32_t low_bits, bool granules, void *base, std::size_t cap,
                     tp2_layout *l) {
    const uint32_t D = 1u << low_bits;
    l->low_bits = low_bits;
    l->K = (uint32_t) (((uint64_t) uDim + D - 1u) >> low_bits);
    if (l->K == 0u) l->K = 1u;
    const uint32_t tile = granules ? kTpTileCsr : kTpTileCoo;
    l->tiles1 = nnz == 0u ? 1u : (uint32_t) (((std::size_t) nnz + tile - 1u) / tile);
    l->max_chunks = nnz / kTpChunk + l->K + 1u;
    l->most_chunks = std::min(l->max_chunks, nnz / kTpChunk + 2u); // of one bucket
    l->slice1 = tp_slice_len(l->tiles1);
    l->slice2 = tp_slice_len(l->max_chunks);
    l->slices1 = (l->tiles1 + l->slice1 - 1u) / l->slice1;
    l->max_slices = l->max_chunks / l->slice2 + l->K + 1u;
    scratch_carver c(base, cap);
    l->status = c.take<uint32_t>(4);
    auto counts = [&](tp_counts *t, std::size_t rows, std::size_t slices, std::size_t digits) {
        t->cnt = c.take<uint16_t>(rows * digits);
        t->base = c.take<uint32_t>(rows * digits);
        t->slices = c.take<uint32_t>(slices * digits);
    };
    // room for the short slices of fewer rows too: scratch for many entries does for fewer
    counts(&l->one, l->tiles1, std::max(l->slices1, std::min(l->tiles1, kTpShortSlices) / 16u), l->K);
    counts(&l->two, l->max_chunks, std::max(l->max_slices, std::min(l->max_chunks, kTpShortSlices) / 16u + l->K + 1u),
           D);
    l->total1 = c.take<uint32_t>(l->K);
    l->start1 = c.take<uint32_t>((std::size_t) l->K + 1u);
    l->tmp_key = c.take<uint32_t>((std::size_t) nnz + 1u);
    l->tmp_val = c.take<uint16_t>((std::size_t) nnz + 8u);
    l->gran_row = granules ? c.take<uint32_t>((std::size_t) nnz / kTpGran + 1u) : nullptr;
    l->chunk_bucket = c.take<uint32_t>(l->max_chunks);
    l->chunk_range = c.take<uint2>(l->max_chunks);
    l->slice_bucket = c.take<uint32_t>(std::max(l->max_slices, kTpShortSlices / 16u + l->K + 1u));
    l->slice_range = c.take<uint2>(std::max(l->max_slices, kTpShortSlices / 16u + l->K + 1u));
    l->slice_first = c.take<uint32_t>((std::size_t) l->K + 1u);
    l->one.start = l->two.start = nullptr; // see tp_offsets
    l->one.segment = nullptr;
    l->one.limit = l->K;
    l->two.segment = l->chunk_bucket;
    l->two.limit = uDim;
    l->scan_bytes = scan_u32_scratch_bytes(uDim);
    l->scan_tmp = c.take<char>(l->scan_bytes);
    l->bytes = c.used;
}

// gran_row[j] = the row holding entry j * kTpGran (rows own the granules that
// start inside them).
__global__ void __launch_bounds__(256) tp_gran_rows_kernel(const uint32_t *__restrict__ ptr, uint32_t cDim,
                                                          uint32_t *__restrict__ gran_row) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= cDim) return;
    const uint32_t lo = ptr[r], hi = ptr[r + 1u];
    for (std::size_t j = ((std::size_t) lo + kTpGran - 1u) / kTpGran; j * kTpGran < hi; ++j) gran_row[j] = r;
}

// Pass-1 histogram: tile t is entries [t * TILE, (t + 1) * TILE).  A
// thread's whole share is in flight at once, 16 bytes a load where the keys
// are aligned, and neighbouring entries of one bucket are added together.
// 393 M entries in 128 buckets: 285 us (361 with an atomic per entry and four
// 4-byte loads in flight).
template <uint32_t TILE, bool VEC>
__global__ void __launch_bounds__(kTpThreads) tp_hist1_kernel(const uint32_t *__restrict__ idx, uint32_t nnz,
                                                             uint32_t uDim, uint32_t low_bits, uint32_t K,
                                                             uint16_t *__restrict__ cnt, uint32_t *status) {
    extern __shared__ uint32_t tp_h[];
    const uint32_t a = blockIdx.x * TILE, n = min(nnz - a, TILE);
    constexpr unsigned V = TILE / (4u * kTpThreads); // vectors per thread
    uint32_t c[V][4];
    if (VEC && n == TILE) {
#pragma unroll
        for (unsigned v = 0; v < V; ++v) {
            const uint4 x = __ldg(reinterpret_cast<const uint4 *>(idx + a) + v * kTpThreads + threadIdx.x);
            c[v][0] = x.x;
            c[v][1] = x.y;
            c[v][2] = x.z;
            c[v][3] = x.w;
        }
    } else {
#pragma unroll
        for (unsigned v = 0; v < V; ++v)
#pragma unroll
            for (unsigned j = 0; j < 4u; ++j) {
                const uint32_t i = (v * kTpThreads + threadIdx.x) * 4u + j;
                c[v][j] = i < n ? __ldg(idx + a + i) : uDim;
            }
    }
    for (uint32_t k = threadIdx.x; k < K; k += blockDim.x) tp_h[k] = 0u;
    __syncthreads();
    uint32_t bad = 0u;
#pragma unroll
    for (unsigned v = 0; v < V; ++v) {
        uint32_t k = 0u, run = 0u;
#pragma unroll
        for (unsigned j = 0; j < 4u; ++j) {
            const uint32_t x = c[v][j];
            if (x >= uDim) {
                if ((v * kTpThreads + threadIdx.x) * 4u + j < n) bad = CS_STATUS_INDEX_RANGE;
                continue;
            }
            if ((x >> low_bits) != k) {
                if (run != 0u) atomicAdd(tp_h + k, run);
                k = x >> low_bits;
                run = 0u;
            }
            ++run;
        }
        if (run != 0u) atomicAdd(tp_h + k, run);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < K; k += blockDim.x) cnt[(std::size_t) blockIdx.x * K + k] = (uint16_t) tp_h[k];
    if (bad) status_or(status, bad);
}

// The offset scan, over slices of 16 or 64 rows so that a segment of many rows
// is not one serial chain: slice sums, a scan of each segment's slices, then
// the rows of every slice.  Rows are D counters wide and a warp reads 32 of
// them together (the counts used to lie digit by digit, one sector apart for a
// CTA that wants its row of them; scanned as one array of 12 M words they took
// 100 us and 256 scattered reads per chunk at 300,000 x 32,768).
__device__ __forceinline__ uint2 tp_slice_rows(const uint2 *__restrict__ range, uint32_t rows, uint32_t len) {
    if (range != nullptr) return range[blockIdx.x];
    return make_uint2(blockIdx.x * len, min(rows, (blockIdx.x + 1u) * len));
}

__global__ void __launch_bounds__(256) tp_slice_sums_kernel(const uint16_t *__restrict__ cnt, uint32_t D,
                                                            uint32_t rows, uint32_t len,
                                                            const uint2 *__restrict__ range,
                                                            uint32_t *__restrict__ slices) {
    const uint2 r = tp_slice_rows(range, rows, len);
    const uint32_t d = blockIdx.y * blockDim.x + threadIdx.x;
    if (d < D) {
        uint32_t sum = 0u;
#pragma unroll 16
        for (uint32_t i = r.x; i < r.y; ++i) sum += __ldg(cnt + (std::size_t) i * D + d);
        slices[(std::size_t) blockIdx.x * D + d] = sum;
    }
}

// One segment (blockIdx.x) and 32 digits (blockIdx.y) per CTA: 32 threads per
// digit, each over a run of the segment's slices.  totals[segment * D + d] for
// digits below `limit` in all.
__global__ void __launch_bounds__(1024) tp_slice_scan_kernel(uint32_t *__restrict__ slices, uint32_t D,
                                                             const uint32_t *__restrict__ seg_first, uint32_t n_slices,
                                                             uint32_t limit, uint32_t *__restrict__ totals) {
    __shared__ uint32_t part[32][33];
    const uint32_t x = threadIdx.x & 31u, y = threadIdx.x >> 5, d = blockIdx.y * 32u + x;
    const uint32_t s0 = seg_first != nullptr ? seg_first[blockIdx.x] : 0u;
    const uint32_t s1 = seg_first != nullptr ? seg_first[blockIdx.x + 1u] : n_slices;
    const uint32_t per = (s1 - s0 + 31u) / 32u;
    const uint32_t a = min(s1, s0 + y * per), e = min(s1, a + per);
    uint32_t sum = 0u;
    if (d < D)
        for (uint32_t i = a; i < e; ++i) sum += slices[(std::size_t) i * D + d];
    part[y][x] = sum;
    __syncthreads();
    // warp y scans digit y of the 32
    {
        const uint32_t v = part[x][y], incl = warp_inclusive_scan(v);
        part[x][y] = incl - v;
        const std::size_t c = (std::size_t) blockIdx.x * D + blockIdx.y * 32u + y;
        if (x == 31u && blockIdx.y * 32u + y < D && c < limit) totals[c] = incl;
    }
    __syncthreads();
    if (d < D) {
        uint32_t run = part[y][x];
        for (uint32_t i = a; i < e; ++i) {
            const uint32_t v = slices[(std::size_t) i * D + d];
            slices[(std::size_t) i * D + d] = run;
            run += v;
        }
    }
}

// The same, or (T = uint16_t) the scan of the rows themselves, by a thread per
// digit: many segments of few slices or rows each, which the CTAs of 1,024
// threads above mostly leave idle.  range: null where seg_first counts in's rows.
template <typename T>
__global__ void __launch_bounds__(256) tp_segment_scan_kernel(const T *in, uint32_t D,
                                                              const uint32_t *__restrict__ seg_first,
                                                              const uint2 *__restrict__ range, uint32_t limit,
                                                              uint32_t *out, uint32_t *__restrict__ totals) {
    const uint32_t d = blockIdx.y * blockDim.x + threadIdx.x;
    if (d >= D) return;
    uint32_t r0 = seg_first[blockIdx.x], r1 = seg_first[blockIdx.x + 1u];
    if (range != nullptr) {
        const uint32_t s0 = r0, s1 = r1;
        r0 = s0 < s1 ? range[s0].x : 0u;
        r1 = s0 < s1 ? range[s1 - 1u].y : 0u;
    }
    constexpr uint32_t U = 8; // loads in flight; `out` may be `in`
    uint32_t run = 0u;
    for (uint32_t i0 = r0; i0 < r1; i0 += U) {
        uint32_t v[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) v[u] = i0 + u < r1 ? (uint32_t) in[(std::size_t) (i0 + u) * D + d] : 0u;
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            if (i0 + u < r1) out[(std::size_t) (i0 + u) * D + d] = run;
            run += v[u];
        }
    }
    const std::size_t c = (std::size_t) blockIdx.x * D + d;
    if (c < limit) totals[c] = run;
}

// start[segment * D + d]: global slot of the digit's first entry
__global__ void __launch_bounds__(256) tp_slice_apply_kernel(const uint16_t *__restrict__ cnt, uint32_t D,
                                                             uint32_t rows, uint32_t len,
                                                             const uint2 *__restrict__ range,
                                                             const uint32_t *__restrict__ segment,
                                                             const uint32_t *__restrict__ slices,
                                                             const uint32_t *__restrict__ start, uint32_t limit,
                                                             uint32_t *__restrict__ base) {
    const uint2 r = tp_slice_rows(range, rows, len);
    const std::size_t c0 = (segment != nullptr ? (std::size_t) segment[blockIdx.x] : 0u) * D;
    const uint32_t d = blockIdx.y * blockDim.x + threadIdx.x;
    if (d < D) {
        uint32_t run = slices[(std::size_t) blockIdx.x * D + d] + (c0 + d < limit ? start[c0 + d] : 0u);
#pragma unroll 16
        for (uint32_t i = r.x; i < r.y; ++i) {
            base[(std::size_t) i * D + d] = run;
            run += __ldg(cnt + (std::size_t) i * D + d);
        }
    }
}

// The three at once for few rows: a segment and 32 digits per CTA as in
// tp_slice_scan_kernel, over the rows themselves.  A digit's 32 threads walk
// rows / 32 each, twice, and the scatter adds the digits' starts (two dependent
// loads in every CTA): four launches fewer, for up to 1,024 tiles or chunks.  us
// a call by three kernels / this: transposes of 43 tiles 126 / 110, of 240
// 121 / 99, of 733 154 / 135, of 2,929 260 / 256, of 8,789 573 / 606, of 24,000
// 1,329 / 1,467.  A scatter that asks at run time whether to add costs the large
// COO partitions 2 %, so it is compiled both ways.
constexpr uint32_t kTpDirectRows = 1024;
__global__ void __launch_bounds__(1024) tp_rows_scan_kernel(const uint16_t *__restrict__ cnt, uint32_t D,
                                                            uint32_t rows, const uint32_t *__restrict__ seg_first,
                                                            const uint2 *__restrict__ range, uint32_t limit,
                                                            uint32_t *__restrict__ base,
                                                            uint32_t *__restrict__ totals) {
    __shared__ uint32_t part[32][33];
    const uint32_t x = threadIdx.x & 31u, y = threadIdx.x >> 5, d = blockIdx.y * 32u + x;
    uint32_t r0 = 0u, r1 = rows;
    if (seg_first != nullptr) {
        const uint32_t s0 = seg_first[blockIdx.x], s1 = seg_first[blockIdx.x + 1u];
        r0 = s0 < s1 ? range[s0].x : 0u;
        r1 = s0 < s1 ? range[s1 - 1u].y : 0u;
    }
    const uint32_t per = (r1 - r0 + 31u) / 32u;
    const uint32_t a = min(r1, r0 + y * per), e = min(r1, a + per);
    uint32_t sum = 0u;
    if (d < D) {
#pragma unroll 8
        for (uint32_t i = a; i < e; ++i) sum += __ldg(cnt + (std::size_t) i * D + d);
    }
    part[y][x] = sum;
    __syncthreads();
    {
        const uint32_t v = part[x][y], incl = warp_inclusive_scan(v);
        part[x][y] = incl - v;
        const std::size_t c = (std::size_t) blockIdx.x * D + blockIdx.y * 32u + y;
        if (x == 31u && blockIdx.y * 32u + y < D && c < limit) totals[c] = incl;
    }
    __syncthreads();
    if (d < D) {
        uint32_t run = part[y][x];
#pragma unroll 8
        for (uint32_t i = a; i < e; ++i) {
            base[(std::size_t) i * D + d] = run;
            run += __ldg(cnt + (std::size_t) i * D + d);
        }
    }
}

// Block-wide exclusive scan of n <= Q * blockDim.x values in place (each
// thread scans up to Q consecutive entries); out[n] receives the total.
template <int Q>
__device__ __forceinline__ void block_scan_small(uint32_t *v, uint32_t n, uint32_t *smem33) {
    const uint32_t t = threadIdx.x;
    uint32_t loc[Q], sum = 0u;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const uint32_t k = t * (unsigned) Q + q;
        loc[q] = k < n ? v[k] : 0u;
        sum += loc[q];
    }
    uint32_t tot;
    uint32_t run = block_exclusive_scan(sum, smem33, tot);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const uint32_t k = t * (unsigned) Q + q;
        if (k < n) v[k] = run;
        run += loc[q];
    }
    if (t == 0) v[n] = tot;
    __syncthreads();
}

// An entry between the passes: its payload (row; COO: column) around the low digit.
__device__ __forceinline__ uint32_t tp_pack(uint32_t pay, uint32_t digit, uint32_t low_bits) {
    return (pay >> 5) << (low_bits + 5u) | digit << 5 | (pay & 31u);
}
template <int LB>
__device__ __forceinline__ uint32_t tp_digit(uint32_t key) {
    return key >> 5 & ((1u << LB) - 1u);
}
template <int LB>
__device__ __forceinline__ uint32_t tp_payload(uint32_t key) {
    return key >> (LB + 5) << 5 | (key & 31u);
}

constexpr uint32_t kTpSub = 2048;                        // entries counted and placed per step
constexpr unsigned kTpBatches = kTpSub / kTpWarps / 32; // 32-entry batches per warp per step

// lanes of the warp holding the same digit (valid lanes only; 0 if invalid).
// match.any is cheaper than one ballot per digit bit when a batch holds few
// distinct digits (pass 1: consecutive entries of a row share a bucket); with
// ~30 distinct digits per batch (pass 2) the ballots win.
__device__ __forceinline__ uint32_t tp_peers(uint32_t d, bool valid) {
    const uint32_t m = __match_any_sync(0xffffffffu, valid ? d : 0xffffffffu);
    return valid ? m : 0u;
}

// last major r in [0, cDim) with ptr[r] <= i
__device__ __forceinline__ uint32_t major_of(const uint32_t *__restrict__ ptr, uint32_t cDim, uint32_t i) {
    uint32_t lo = 0u, hi = cDim - 1u;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1u) >> 1;
        if (__ldg(ptr + mid) <= i)
            lo = mid;
        else
            hi = mid - 1u;
    }
    return lo;
}

// Stable in-CTA reorder shared by both passes.  The tile's per-digit counts
// are known up front (from the pass's histogram), so `lb` holds each digit's
// first staging slot.  Each step of kTpSub entries gives every warp
// kTpBatches batches of 32 held in registers: the warp counts them per digit
// (peer masks from warp_match_digit), the CTA turns the per-warp counts into
// staging slots (digit base + entries already placed + earlier warps), and
// the warp places its entries in order.  Counters are u16: one warp places at
// most kTpSub / kTpWarps entries per step and the stage holds <= 65535.
struct tp_stage {
    uint16_t *cnt;  // [kTpWarps][D]
    uint16_t *bas;  // [kTpWarps][D]
    uint32_t *lb;   // [D + 1]
    uint32_t *fill; // [D]
};

template <unsigned WARPS>
__device__ __forceinline__ void tp_stage_prefix(const tp_stage &sg, uint32_t D) {
    for (uint32_t d = threadIdx.x; d < D; d += blockDim.x) {
        uint32_t t = sg.lb[d] + sg.fill[d];
        const uint32_t t0 = t;
#pragma unroll
        for (unsigned w = 0; w < WARPS; ++w) {
            const uint32_t c = sg.cnt[w * D + d];
            sg.cnt[w * D + d] = 0u;
            sg.bas[w * D + d] = (uint16_t) t;
            t += c;
        }
        sg.fill[d] += t - t0;
    }
}

// Pass 1 of the transpose: the key is the CSR entry's column, the payload its
// row.  Consecutive entries of a row ascend, so the entries of one bucket stand
// in runs (~10 at 1,311 entries in 128 buckets), and what is sorted is the
// tile's list of runs: heads by a shuffle and a ballot per 32 entries, the runs
// ranked by bucket (per-warp counts, then in order), and every entry moves by
// its run's displacement.  Rows in any column order only make the runs shorter.
// Row starts inside the tile are bits over its entries too: the row of an entry
// is the number of starts up to it, looked up in the tile's list of rows.
// 60,000 x 32,768, 79 M entries: 435 us; 457 with match.any on every 32 entries,
// two barriers per 2,048 entries and a row pointer read per batch; 481 ranking
// entry by entry at run ends.  Bound by the phases that a CTA goes through one
// after the other (load 80, rank 190, write 120 us when run alone).
constexpr unsigned kTpThreads1 = 256;
constexpr unsigned kTpWarps1 = kTpThreads1 / 32;
constexpr unsigned kTpBatches1 = kTpTileCsr / kTpThreads1; // 32-entry batches per warp
constexpr uint32_t kTpTileWords = kTpTileCsr / 32u;
static_assert(kTpTileWords <= kTpThreads1, "a thread per word of the tile's bits");
constexpr uint32_t kTpTileRows = 2048;                   // listed rows: a tile with more, or in a gap of more
constexpr uint32_t kTpTileSpan = 32768;                  // empty rows than this, searches the row pointers

struct tp_tile_smem {
    union {
        unsigned long long st[kTpTileCsr]; // staged entries: packed word | value << 32 | bucket << 48
        struct {
            uint32_t runs[kTpTileCsr];     // first entry | bucket << 16
            uint32_t cnt[kTpWarps1 * kTpMaxBuckets / 2u]; // [warp][K2] pairs of u16: counts, then staging slots
        };
    };
    uint16_t move[kTpTileCsr];             // a run's staging slot - its first entry
    uint32_t heads[kTpTileWords], starts[kTpTileWords]; // bits: run heads, row starts
    uint16_t heads_pre[kTpTileWords], starts_pre[kTpTileWords];
    uint16_t row_of[kTpTileRows];        // row - the tile's first row
    uint32_t scan33[33];
};

template <bool kAdd>
__global__ void __launch_bounds__(kTpThreads1, 4)
    tp_scatter1_csr_kernel(const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ idx,
                           const uint16_t *__restrict__ val, uint32_t cDim, uint32_t uDim, uint32_t nnz, uint32_t K,
                           const tp_counts one, const uint32_t *__restrict__ gran_row, uint32_t *__restrict__ tmp_key,
                           uint16_t *__restrict__ tmp_val) {
    extern __shared__ __align__(16) unsigned char tp_ts[];
    tp_tile_smem &sm = *reinterpret_cast<tp_tile_smem *>(tp_ts);
    uint32_t *run = reinterpret_cast<uint32_t *>(tp_ts + sizeof(tp_tile_smem)); // [K] global base per bucket
    uint32_t *lb = run + K;                                                     // [K + 1]
    constexpr uint32_t kNone = 0xffffu; // bucket of an entry out of range or past the tile
    const uint32_t K2 = (K + 1u) / 2u;
    const unsigned t = threadIdx.x, warp = t >> 5, lane = t & 31u;
    const unsigned le = 0xffffffffu >> (31u - lane);
    const uint32_t a = blockIdx.x * kTpTileCsr, n = min(nnz - a, kTpTileCsr), e = a + n;
    const uint32_t w0 = warp * (kTpBatches1 * 32u); // the warp's first entry in the tile
    uint32_t cc[kTpBatches1], vv[kTpBatches1 / 2u];
    if (n == kTpTileCsr) {
#pragma unroll
        for (unsigned q = 0; q < kTpBatches1; ++q) cc[q] = __ldcs(idx + a + w0 + q * 32u + lane);
#pragma unroll
        for (unsigned q = 0; q < kTpBatches1; q += 2u) {
            const unsigned short *p = reinterpret_cast<const unsigned short *>(val) + a + w0 + q * 32u + lane;
            vv[q / 2u] = (uint32_t) __ldcs(p) | (uint32_t) __ldcs(p + 32) << 16;
        }
    } else {
#pragma unroll
        for (unsigned q = 0; q < kTpBatches1; ++q) {
            const uint32_t i = w0 + q * 32u + lane;
            cc[q] = i < n ? __ldcs(idx + a + i) : 0xffffffffu;
            const uint32_t v = i < n ? (uint32_t) __ldcs(reinterpret_cast<const unsigned short *>(val) + a + i) : 0u;
            vv[q / 2u] = (q & 1u) ? vv[q / 2u] | v << 16 : v;
        }
    }
    for (uint32_t k = t; k < K; k += kTpThreads1) {
        run[k] = one.first<kAdd>(blockIdx.x, K, k);
        lb[k] = one.cnt[(std::size_t) blockIdx.x * K + k];
    }
    for (uint32_t k = t; k < kTpWarps1 * K2; k += kTpThreads1) sm.cnt[k] = 0u;
    if (t < kTpTileWords) sm.starts[t] = 0u;
    // rows that may start inside the tile; the tile's first entry lies in r_begin
    const uint32_t r_begin = min(__ldg(gran_row + a / kTpGran), cDim - 1u);
    const uint32_t r_end = e < nnz ? min(__ldg(gran_row + e / kTpGran), cDim - 1u) : major_of(ptr, cDim, e - 1u);
    const bool near = r_end < r_begin || r_end - r_begin <= kTpTileSpan;
    __syncthreads();
    block_scan_small<4>(lb, K, sm.scan33);
    // run heads (a warp's first entry is one) and row starts (of rows with entries)
#pragma unroll
    for (unsigned q = 0; q < kTpBatches1; ++q) {
        const uint32_t k = cc[q] < uDim ? cc[q] >> kTpBucketBits : kNone;
        uint32_t up = __shfl_up_sync(0xffffffffu, k, 1);
        if (q != 0u) {
            const uint32_t before = __shfl_sync(0xffffffffu, cc[q - (q != 0u)], 31);
            if (lane == 0u) up = before < uDim ? before >> kTpBucketBits : kNone;
        }
        const uint32_t h = __ballot_sync(0xffffffffu, k != up || (q == 0u && lane == 0u));
        if (lane == 0u) sm.heads[w0 / 32u + q] = h;
    }
    for (uint32_t r = r_begin + 1u + t; near && r <= r_end; r += kTpThreads1) {
        const uint32_t x = __ldg(ptr + r) - a;
        if (x < n && x != 0u && __ldg(ptr + r + 1u) != x + a) atomicOr(sm.starts + (x >> 5), 1u << (x & 31u));
    }
    __syncthreads();
    uint32_t n_runs, n_starts;
    {
        const uint32_t both = t < kTpTileWords ? __popc(sm.heads[t]) | __popc(sm.starts[t]) << 16 : 0u;
        uint32_t total; // both counts are at most kTpTileCsr
        const uint32_t before = block_exclusive_scan(both, sm.scan33, total);
        if (t < kTpTileWords) {
            sm.heads_pre[t] = (uint16_t) before;
            sm.starts_pre[t] = (uint16_t) (before >> 16);
        }
        n_runs = total & 0xffffu;
        n_starts = total >> 16;
    }
    __syncthreads();
    const bool listed = near && n_starts < kTpTileRows;
#pragma unroll
    for (unsigned q = 0; q < kTpBatches1; ++q) {
        const uint32_t word = w0 / 32u + q, h = sm.heads[word];
        const uint32_t k = cc[q] < uDim ? cc[q] >> kTpBucketBits : kNone;
        if (h >> lane & 1u) sm.runs[sm.heads_pre[word] + __popc(h & (le >> 1))] = (w0 + q * 32u + lane) | k << 16;
    }
    if (listed) {
        if (t == 0u) sm.row_of[0] = 0u;
        for (uint32_t r = r_begin + 1u + t; r <= r_end; r += kTpThreads1) {
            const uint32_t x = __ldg(ptr + r) - a;
            if (x < n && x != 0u && __ldg(ptr + r + 1u) != x + a)
                sm.row_of[sm.starts_pre[x >> 5] + __popc(sm.starts[x >> 5] & ((1u << (x & 31u)) - 1u)) + 1u] =
                    (uint16_t) (r - r_begin);
        }
    }
    __syncthreads();
    // each warp takes consecutive runs: entries per bucket, staging slots, then
    // its runs in order
    uint32_t *my_cnt = sm.cnt + warp * K2;
    uint16_t *my_bas = reinterpret_cast<uint16_t *>(my_cnt);
    const uint32_t per = (n_runs + kTpThreads1 - 1u) / kTpThreads1 * 32u;
    const uint32_t u0 = min(n_runs, warp * per), u1 = min(n_runs, u0 + per);
    auto length = [&](uint32_t u, uint32_t rec) {
        return (u + 1u < n_runs ? sm.runs[u + 1u] & 0xffffu : kTpTileCsr) - (rec & 0xffffu);
    };
    for (uint32_t u = u0 + lane; u < u1; u += 32u) {
        const uint32_t rec = sm.runs[u], k = rec >> 16;
        if (k != kNone) atomicAdd(my_cnt + (k >> 1), length(u, rec) << (16u * (k & 1u)));
    }
    __syncthreads();
    for (uint32_t k2 = t; k2 < K2; k2 += kTpThreads1) {
        uint32_t s0 = lb[2u * k2], s1 = 2u * k2 + 1u < K ? lb[2u * k2 + 1u] : 0u;
#pragma unroll
        for (unsigned w = 0; w < kTpWarps1; ++w) {
            const uint32_t c = sm.cnt[w * K2 + k2];
            sm.cnt[w * K2 + k2] = s0 | s1 << 16;
            s0 += c & 0xffffu;
            s1 += c >> 16;
        }
    }
    __syncthreads();
    for (uint32_t v0 = u0; v0 < u1; v0 += 32u) {
        const uint32_t u = v0 + lane;
        const uint32_t rec = u < u1 ? sm.runs[u] : kNone << 16, k = rec >> 16;
        // entries in the bucket's earlier runs of the 32, a run per turn; the last
        // run of each bucket moves the bucket on.  Columns in any order leave up to
        // 32 runs in eight buckets (200,000 x 2,000 of 100: 393 us, 427 with the
        // bucket's slot read and written by every run in turn)
        const uint32_t peers = tp_peers(k, k != kNone), len = u < u1 ? length(u, rec) : 0u;
        uint32_t before = 0u;
        for (uint32_t left = peers & (le >> 1); __any_sync(0xffffffffu, left != 0u); left &= left - 1u) {
            const uint32_t v = __shfl_sync(0xffffffffu, len, left != 0u ? __ffs(left) - 1 : 0);
            if (left != 0u) before += v;
        }
        uint32_t slot = 0u;
        if (k != kNone) slot = my_bas[k] + before;
        __syncwarp();
        if (k != kNone) {
            sm.move[u] = (uint16_t) (slot - (rec & 0xffffu));
            if ((peers & ~le) == 0u) my_bas[k] = (uint16_t) (slot + len);
        }
        __syncwarp();
    }
    __syncthreads(); // the stage takes the place of the runs and the counts
    auto in_place = [](uint32_t r) { return r >> 5 << (kTpBucketBits + 5u) | (r & 31u); };
    // the row that goes on into the next batch, as its bits of the packed word
    uint32_t row_bits = listed ? in_place(r_begin + sm.row_of[sm.starts_pre[w0 / 32u]]) : 0u;
#pragma unroll
    for (unsigned q = 0; q < kTpBatches1; ++q) {
        const uint32_t word = w0 / 32u + q, c = cc[q], pos = w0 + q * 32u + lane;
        const uint32_t sb = sm.starts[word];
        if (!listed)
            row_bits = in_place(major_of(ptr, cDim, min(a + pos, e - 1u)));
        else if (sb != 0u)
            row_bits = in_place(r_begin + sm.row_of[sm.starts_pre[word] + __popc(sb & le)]);
        const uint32_t lp = (pos + sm.move[sm.heads_pre[word] + __popc(sm.heads[word] & le) - 1u]) & 0xffffu;
        if (c < uDim)
            sm.st[lp] = (unsigned long long) (row_bits | (c & 255u) << 5) |
                        (unsigned long long) (((q & 1u) ? vv[q / 2u] >> 16 : vv[q / 2u] & 0xffffu) |
                                              c >> kTpBucketBits << 16)
                            << 32;
        if (sb != 0u) row_bits = __shfl_sync(0xffffffffu, row_bits, 31);
    }
    __syncthreads();
    const uint32_t placed = min(lb[K], kTpTileCsr);
    for (uint32_t k = t; k < K; k += kTpThreads1) run[k] -= lb[k]; // the global slot of staging slot 0
    __syncthreads();
#pragma unroll 4
    for (uint32_t j = t; j < placed; j += kTpThreads1) {
        const unsigned long long v = sm.st[j];
        const uint32_t g = run[(uint32_t) (v >> 48)] + j;
        tmp_key[g] = (uint32_t) v;
        tmp_val[g] = (uint16_t) (v >> 32);
    }
}

std::size_t tp_scatter1_csr_smem(uint32_t K) { return sizeof(tp_tile_smem) + ((std::size_t) 2u * K + 1u) * 4u; }

// Pass 1 of COO entries: the key is the entry's row, the payload its (mapped)
// column.  Random rows leave nothing to rank by but the counters themselves: a
// thread's entries take their places in a bucket by shared atomics, in any
// order, which costs ~50 warp instructions per 32 entries against ~230 of the
// ballots below.  Only a repeated (row, column) needs the order of the entries;
// the shape pass that follows finds those, and the ballot kernels then run.
constexpr unsigned kTpThreadsCoo = 512;
constexpr unsigned kTpPerCoo = kTpTileCoo / kTpThreadsCoo;

template <bool kAdd>
__global__ void __launch_bounds__(kTpThreadsCoo, 2)
    tp_scatter1_coo_kernel(const uint32_t *__restrict__ key, const uint16_t *__restrict__ val,
                           const uint32_t *__restrict__ pay, const uint32_t *__restrict__ pay_map, uint32_t uDim,
                           uint32_t nnz, uint32_t low_bits, uint32_t K, const tp_counts one,
                           uint32_t *__restrict__ tmp_key, uint16_t *__restrict__ tmp_val) {
    extern __shared__ __align__(16) uint32_t tp_s[];
    __shared__ uint32_t scan33[33];
    // staged entry: packed word | value << 32 | bucket << 48
    unsigned long long *st = reinterpret_cast<unsigned long long *>(tp_s); // [kTpTileCoo]
    uint32_t *run = reinterpret_cast<uint32_t *>(st + kTpTileCoo);         // [K] global base per bucket
    uint32_t *at = run + K;                                                // [K + 1] next staging slot
    const unsigned t = threadIdx.x;
    const uint32_t a = blockIdx.x * kTpTileCoo, n = min(nnz - a, kTpTileCoo);
    uint32_t rr[kTpPerCoo], pp[kTpPerCoo], vv[kTpPerCoo / 2u];
#pragma unroll
    for (unsigned q = 0; q < kTpPerCoo; ++q) {
        const uint32_t i = q * kTpThreadsCoo + t;
        rr[q] = i < n ? __ldcs(key + a + i) : 0xffffffffu;
        pp[q] = i < n ? __ldcs(pay + a + i) : 0u;
        const uint32_t v = i < n ? (uint32_t) __ldcs(reinterpret_cast<const unsigned short *>(val) + a + i) : 0u;
        vv[q / 2u] = (q & 1u) ? vv[q / 2u] | v << 16 : v;
    }
    for (uint32_t k = t; k < K; k += kTpThreadsCoo) {
        run[k] = one.first<kAdd>(blockIdx.x, K, k);
        at[k] = one.cnt[(std::size_t) blockIdx.x * K + k];
    }
    if (pay_map != nullptr)
#pragma unroll
        for (unsigned q = 0; q < kTpPerCoo; ++q)
            if (rr[q] < uDim) pp[q] = __ldg(pay_map + pp[q]);
    __syncthreads();
    block_scan_small<2>(at, K, scan33);
    const uint32_t placed = min(at[K], kTpTileCoo);
    for (uint32_t k = t; k < K; k += kTpThreadsCoo) run[k] -= at[k]; // the global slot of staging slot 0
    __syncthreads();
    const uint32_t low_mask = (1u << low_bits) - 1u;
#pragma unroll
    for (unsigned q = 0; q < kTpPerCoo; ++q) {
        if (rr[q] >= uDim) continue;
        const uint32_t k = rr[q] >> low_bits;
        const uint32_t lp = atomicAdd(at + k, 1u);
        if (lp < kTpTileCoo)
            st[lp] = (unsigned long long) tp_pack(pp[q], rr[q] & low_mask, low_bits) |
                     (unsigned long long) (((q & 1u) ? vv[q / 2u] >> 16 : vv[q / 2u] & 0xffffu) | k << 16) << 32;
    }
    __syncthreads();
#pragma unroll 4
    for (uint32_t j = t; j < placed; j += kTpThreadsCoo) {
        const unsigned long long v = st[j];
        const uint32_t g = run[(uint32_t) (v >> 48)] + j;
        tmp_key[g] = (uint32_t) v;
        tmp_val[g] = (uint16_t) (v >> 32);
    }
}

std::size_t tp_scatter1_coo_smem(uint32_t K) {
    return (std::size_t) kTpTileCoo * 8u + ((std::size_t) 2u * K + 1u) * 4u;
}

// The same in the order of the entries (stable): a tile's entries are ranked in
// 32-entry batches by ballots, one per bucket bit.
template <bool kAdd>
__global__ void __launch_bounds__(kTpThreads) tp_scatter1_coo_stable_kernel(
    const uint32_t *__restrict__ idx, const uint16_t *__restrict__ val, const uint32_t *__restrict__ pay,
    const uint32_t *__restrict__ pay_map, uint32_t uDim, uint32_t nnz, uint32_t low_bits, uint32_t K,
    const tp_counts one, uint32_t *__restrict__ tmp_key, uint16_t *__restrict__ tmp_val) {
    extern __shared__ __align__(16) uint32_t tp_s[];
    __shared__ uint32_t scan33[33];
    // staged entry: key | value << 32 | bucket << 48
    unsigned long long *st = reinterpret_cast<unsigned long long *>(tp_s); // [kTpTileCoo]
    uint32_t *run = reinterpret_cast<uint32_t *>(st + kTpTileCoo);           // [K] global base per bucket
    tp_stage sg;
    sg.lb = run + K;                                                       // [K + 1]
    sg.fill = sg.lb + K + 1u;                                              // [K]
    sg.cnt = reinterpret_cast<uint16_t *>(sg.fill + K);                    // [kTpWarps][K]
    sg.bas = sg.cnt + kTpWarps * K;                                        // [kTpWarps][K]
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t a = blockIdx.x * kTpTileCoo, e = min(nnz - a, kTpTileCoo) + a;
    for (uint32_t k = threadIdx.x; k < K; k += blockDim.x) {
        run[k] = one.first<kAdd>(blockIdx.x, K, k);
        sg.lb[k] = one.cnt[(std::size_t) blockIdx.x * K + k];
        sg.fill[k] = 0u;
    }
    for (uint32_t k = threadIdx.x; k < kTpWarps * K; k += blockDim.x) sg.cnt[k] = 0u;
    __syncthreads();
    block_scan_small<4>(sg.lb, K, scan33);
    const unsigned lt = (1u << lane) - 1u;
    uint16_t *my_cnt = sg.cnt + warp * K;
    uint16_t *my_bas = sg.bas + warp * K;
    uint32_t ncc[kTpBatches], npp[kTpBatches];
    const uint32_t low_mask = (1u << low_bits) - 1u;
    uint16_t nvv[kTpBatches];
    auto fetch = [&](uint32_t sc) {
        const uint32_t n = min(kTpSub, e - sc);
        const uint32_t wa = sc + min(n, warp * kTpGran), we = sc + min(n, (warp + 1u) * kTpGran);
#pragma unroll
        for (unsigned q = 0; q < kTpBatches; ++q) {
            const uint32_t i = wa + q * 32u + lane;
            const bool in = i < we;
            ncc[q] = in ? __ldg(idx + i) : uDim;
            nvv[q] = in ? __ldg(reinterpret_cast<const unsigned short *>(val) + i) : (uint16_t) 0u;
            npp[q] = in ? __ldg(pay + i) : 0u;
        }
    };
    fetch(a);
    for (uint32_t sc0 = a; sc0 < e; sc0 += kTpSub) {
        uint32_t cc[kTpBatches], pk[kTpBatches], rl[kTpBatches];
        uint16_t vv[kTpBatches];
#pragma unroll
        for (unsigned q = 0; q < kTpBatches; ++q) {
            cc[q] = ncc[q];
            vv[q] = nvv[q];
            rl[q] = pay_map != nullptr && cc[q] < uDim ? __ldg(pay_map + npp[q]) : npp[q];
        }
        if (sc0 + kTpSub < e) fetch(sc0 + kTpSub);
#pragma unroll
        for (unsigned q = 0; q < kTpBatches; ++q) {
            const bool ok = cc[q] < uDim;
            const uint32_t k = cc[q] >> low_bits;
            pk[q] = warp_match_digit<10>(k, ok);
            if (ok && lane == (unsigned) (__ffs(pk[q]) - 1)) my_cnt[k] += (uint16_t) __popc(pk[q]);
            __syncwarp();
        }
        __syncthreads();
        tp_stage_prefix<kTpWarps>(sg, K);
        __syncthreads();
#pragma unroll
        for (unsigned q = 0; q < kTpBatches; ++q) {
            const bool ok = cc[q] < uDim;
            const uint32_t k = cc[q] >> low_bits;
            uint32_t lp = 0u;
            if (ok) lp = my_bas[k] + __popc(pk[q] & lt);
            __syncwarp();
            if (ok) {
                if (lp < kTpTileCoo)
                    st[lp] = (unsigned long long) tp_pack(rl[q], cc[q] & low_mask, low_bits) |
                             ((unsigned long long) vv[q] << 32) | ((unsigned long long) k << 48);
                if (lane == (unsigned) (__ffs(pk[q]) - 1)) my_bas[k] += (uint16_t) __popc(pk[q]);
            }
            __syncwarp();
        }
    }
    __syncthreads();
    const uint32_t placed = min(sg.lb[K], kTpTileCoo);
    // run[k] - lb[k]: the global slot of staging slot 0 for bucket k
    for (uint32_t k = threadIdx.x; k < K; k += blockDim.x) run[k] -= sg.lb[k];
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < placed; j += blockDim.x) {
        const unsigned long long v = st[j];
        const uint32_t g = run[(uint32_t) (v >> 48)] + j;
        tmp_key[g] = (uint32_t) v;
        tmp_val[g] = (uint16_t) (v >> 32);
    }
}

std::size_t tp_scatter1_smem(uint32_t K) {
    return (std::size_t) kTpTileCoo * 8u + ((std::size_t) 3u * K + 1u) * 4u + (std::size_t) 2u * kTpWarps * K * 2u;
}

// One CTA: bucket starts from their totals, then every bucket's entry range is
// cut at the multiples of kTpChunk and its chunks into slices; a scan of the
// buckets' chunk counts, and a thread per chunk finds its bucket in it (a
// thread per bucket writing its chunks one by one took 84 us for 48,000).
__device__ __forceinline__ uint32_t tp_find(const uint32_t *first, uint32_t K, uint32_t id) {
    uint32_t lo = 0u, hi = K - 1u; // last k with first[k] <= id
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1u) >> 1;
        if (first[mid] <= id)
            lo = mid;
        else
            hi = mid - 1u;
    }
    return lo;
}

__global__ void __launch_bounds__(1024) tp_chunks_kernel(const tp2_layout l) {
    __shared__ uint32_t smem[33];
    __shared__ uint32_t first[kTpMaxBuckets + 1u], begin[kTpMaxBuckets + 1u], slice[kTpMaxBuckets + 1u];
    const uint32_t k = threadIdx.x, K = l.K; // K <= kTpMaxBuckets == blockDim.x
    uint32_t total;
    const uint32_t n = k < K ? l.total1[k] : 0u;
    const uint32_t b = block_exclusive_scan(n, smem, total);
    if (k < K) begin[k] = l.start1[k] = b;
    if (k == 0u) begin[K] = l.start1[K] = total;
    const uint32_t nc = n != 0u ? (b + n - 1u) / kTpChunk + 1u - b / kTpChunk : 0u;
    uint32_t chunks, slices;
    const uint32_t fc = block_exclusive_scan(nc, smem, chunks);
    const uint32_t fs = block_exclusive_scan((nc + l.slice2 - 1u) / l.slice2, smem, slices);
    if (k < K) {
        first[k] = fc;
        slice[k] = l.slice_first[k] = fs;
    }
    if (k == 0u) {
        first[K] = chunks;
        slice[K] = l.slice_first[K] = slices;
    }
    __syncthreads();
    for (uint32_t id = threadIdx.x; id < l.max_chunks; id += blockDim.x) {
        uint32_t bk = 0u;
        uint2 r = make_uint2(0u, 0u); // unused chunks are empty
        if (id < chunks) {
            bk = tp_find(first, K, id);
            const uint32_t cell = begin[bk] / kTpChunk + (id - first[bk]);
            r.x = max(begin[bk], cell * kTpChunk);
            r.y = cell == 0xffffffffu / kTpChunk ? begin[bk + 1u] : min(begin[bk + 1u], (cell + 1u) * kTpChunk);
        }
        l.chunk_bucket[id] = bk;
        l.chunk_range[id] = r;
    }
    for (uint32_t id = threadIdx.x; id < l.max_slices; id += blockDim.x) {
        uint32_t bk = 0u;
        uint2 r = make_uint2(0u, 0u);
        if (id < slices) {
            bk = tp_find(slice, K, id);
            r.x = first[bk] + (id - slice[bk]) * l.slice2;
            r.y = min(first[bk + 1u], r.x + l.slice2);
        }
        l.slice_bucket[id] = bk;
        l.slice_range[id] = r;
    }
}

// one histogram per warp while eight of them fit (LB = 8), one per CTA above
template <int LB>
__global__ void __launch_bounds__(kTpThreads) tp_hist2_kernel(const uint32_t *__restrict__ tmp_key,
                                                             const uint2 *__restrict__ chunk_range,
                                                             uint16_t *__restrict__ cnt) {
    constexpr uint32_t D = 1u << LB;
    constexpr unsigned kCopies = LB == 8 ? kTpWarps : 1u;
    __shared__ uint32_t h[kCopies][D];
    const unsigned copy = (threadIdx.x >> 5) % kCopies;
    for (uint32_t d = threadIdx.x; d < kCopies * D; d += blockDim.x) (&h[0][0])[d] = 0u;
    __syncthreads();
    const uint32_t b = chunk_range[blockIdx.x].x, e = chunk_range[blockIdx.x].y;
    constexpr unsigned U = 4;
    for (uint32_t i0 = b; i0 < e; i0 += U * blockDim.x) {
        uint32_t kk[U];
#pragma unroll
        for (unsigned u = 0; u < U; ++u) {
            const uint32_t i = i0 + u * blockDim.x + threadIdx.x;
            kk[u] = i < e ? __ldg(tmp_key + i) : 0xffffffffu; // no packed key: see partition_low_bits
        }
#pragma unroll
        for (unsigned u = 0; u < U; ++u)
            if (kk[u] != 0xffffffffu) atomicAdd(&h[copy][tp_digit<LB>(kk[u])], 1u);
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < D; d += blockDim.x) {
        uint32_t t = 0u;
#pragma unroll
        for (unsigned w = 0; w < kCopies; ++w) t += h[w][d];
        cnt[(std::size_t) blockIdx.x * D + d] = (uint16_t) t;
    }
}

// Stable ranking of one pass-2 chunk [b, e) into the stage by ballots: each
// step gives every warp 256 consecutive entries in eight 32-entry batches; a
// batch's peers (lanes with the same digit) come from one ballot per digit bit.
// lb holds each digit's first staging slot; fill and cnt are zero on entry.
template <int LB, unsigned WARPS>
__device__ void tp_rank_ballots(const uint32_t *__restrict__ tmp_key, const uint16_t *__restrict__ tmp_val, uint32_t b,
                                uint32_t e, const tp_stage &sg, uint32_t *st_key, uint16_t *st_val) {
    constexpr uint32_t D = 1u << LB;
    constexpr uint32_t kStep = WARPS * kTpGran;
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const unsigned lt = (1u << lane) - 1u;
    uint16_t *my_cnt = sg.cnt + warp * D;
    uint16_t *my_bas = sg.bas + warp * D;
    uint32_t nkk[kTpBatches];
    uint16_t nvv[kTpBatches];
    auto fetch = [&](uint32_t sc) {
        const uint32_t n = min(kStep, e - sc);
        const uint32_t wa = sc + min(n, warp * kTpGran), we = sc + min(n, (warp + 1u) * kTpGran);
#pragma unroll
        for (unsigned q = 0; q < kTpBatches; ++q) {
            const uint32_t i = wa + q * 32u + lane;
            const bool in = i < we;
            nkk[q] = in ? __ldg(tmp_key + i) : 0u;
            nvv[q] = in ? __ldg(reinterpret_cast<const unsigned short *>(tmp_val) + i) : (uint16_t) 0u;
        }
    };
    fetch(b);
    for (uint32_t sc0 = b; sc0 < e; sc0 += kStep) {
        const uint32_t n = min(kStep, e - sc0);
        const uint32_t wa = sc0 + min(n, warp * kTpGran);
        const uint32_t we = sc0 + min(n, (warp + 1u) * kTpGran);
        uint32_t kk[kTpBatches], pk[kTpBatches];
        uint16_t vv[kTpBatches];
#pragma unroll
        for (unsigned q = 0; q < kTpBatches; ++q) {
            kk[q] = nkk[q];
            vv[q] = nvv[q];
        }
        if (sc0 + kStep < e) fetch(sc0 + kStep);
#pragma unroll
        for (unsigned q = 0; q < kTpBatches; ++q) {
            const bool in = wa + q * 32u + lane < we;
            const uint32_t d = tp_digit<LB>(kk[q]);
            pk[q] = warp_match_digit<LB>(d, in);
            if (in && lane == (unsigned) (__ffs(pk[q]) - 1)) my_cnt[d] += (uint16_t) __popc(pk[q]);
            __syncwarp();
        }
        __syncthreads();
        tp_stage_prefix<WARPS>(sg, D);
        __syncthreads();
#pragma unroll
        for (unsigned q = 0; q < kTpBatches; ++q) {
            const bool in = wa + q * 32u + lane < we;
            const uint32_t d = tp_digit<LB>(kk[q]);
            uint32_t lp = 0u;
            if (in) lp = my_bas[d] + __popc(pk[q] & lt);
            __syncwarp();
            if (in) {
                if (lp < kTpChunk) {
                    st_key[lp] = kk[q];
                    st_val[lp] = vv[q];
                }
                if (lane == (unsigned) (__ffs(pk[q]) - 1)) my_bas[d] += (uint16_t) __popc(pk[q]);
            }
            __syncwarp();
        }
    }
}

// Pass 2 by ballots: a chunk of one bucket reordered by the low digit in shared
// memory (stable), then written out as one run per key.  Sparse transposes, and
// COO entries whose order counts.
template <int LB, bool kAdd>
__global__ void __launch_bounds__(kTpThreads) tp_scatter2_kernel(const uint32_t *__restrict__ tmp_key,
                                                                const uint16_t *__restrict__ tmp_val,
                                                                const uint2 *__restrict__ chunk_range,
                                                                const tp_counts two, uint32_t *__restrict__ out_idx,
                                                                uint16_t *__restrict__ out_val) {
    extern __shared__ __align__(16) uint32_t tp_s2[];
    constexpr uint32_t D = 1u << LB;
    __shared__ uint32_t gbase[D];
    __shared__ uint32_t lb[D + 1u];
    __shared__ uint32_t fill[D];
    __shared__ uint32_t scan33[33];
    uint32_t *st_key = tp_s2;                                              // [kTpChunk]
    uint16_t *st_val = reinterpret_cast<uint16_t *>(st_key + kTpChunk);   // [kTpChunk]
    tp_stage sg;
    sg.cnt = st_val + kTpChunk;                                            // [kTpWarps][D]
    sg.bas = sg.cnt + kTpWarps * D;                                        // [kTpWarps][D]
    sg.lb = lb;
    sg.fill = fill;
    const uint32_t b = chunk_range[blockIdx.x].x, e = chunk_range[blockIdx.x].y;
    if (b >= e) return;
    for (uint32_t d = threadIdx.x; d < D; d += kTpThreads) {
        lb[d] = two.cnt[(std::size_t) blockIdx.x * D + d];
        gbase[d] = two.first<kAdd>(blockIdx.x, D, d);
        fill[d] = 0u;
#pragma unroll
        for (unsigned w = 0; w < kTpWarps; ++w) sg.cnt[w * D + d] = 0u;
    }
    __syncthreads();
    block_scan_small<(D / kTpThreads)>(lb, D, scan33);
    tp_rank_ballots<LB, kTpWarps>(tmp_key, tmp_val, b, e, sg, st_key, st_val);
    // global slot of staging slot 0 for digit d
    for (uint32_t d = threadIdx.x; d < D; d += kTpThreads) gbase[d] -= lb[d];
    __syncthreads();
    const uint32_t n = min(e - b, kTpChunk);
    for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) {
        const uint32_t key = st_key[j];
        const uint32_t g = gbase[tp_digit<LB>(key)] + j;
        out_idx[g] = tp_payload<LB>(key);
        out_val[g] = st_val[j];
    }
}

// Pass 2 of COO entries, in any order inside a row: as tp_scatter1_coo_kernel,
// by shared atomics on the row's next staging slot.
template <int LB, bool kAdd>
__global__ void __launch_bounds__(kTpThreadsCoo, 2)
    tp_scatter2_coo_kernel(const uint32_t *__restrict__ tmp_key, const uint16_t *__restrict__ tmp_val,
                           const uint2 *__restrict__ chunk_range, const tp_counts two, uint32_t *__restrict__ out_idx,
                           uint16_t *__restrict__ out_val) {
    extern __shared__ __align__(16) uint32_t tp_s2[];
    constexpr uint32_t D = 1u << LB;
    __shared__ uint32_t scan33[33];
    uint32_t *st_key = tp_s2;                                            // [kTpChunk]
    uint16_t *st_val = reinterpret_cast<uint16_t *>(st_key + kTpChunk); // [kTpChunk]
    uint32_t *gbase = reinterpret_cast<uint32_t *>(st_val + kTpChunk);  // [D]
    uint32_t *at = gbase + D;                                           // [D + 1] next staging slot
    const unsigned t = threadIdx.x;
    const uint32_t b = chunk_range[blockIdx.x].x, e = chunk_range[blockIdx.x].y;
    if (b >= e) return;
    const uint32_t n = min(e - b, kTpChunk);
    constexpr unsigned kPer = kTpChunk / kTpThreadsCoo;
    uint32_t kk[kPer], vv[kPer / 2u];
#pragma unroll
    for (unsigned q = 0; q < kPer; ++q) {
        const uint32_t i = q * kTpThreadsCoo + t;
        kk[q] = i < n ? __ldcs(tmp_key + b + i) : 0xffffffffu; // no packed key: see partition_low_bits
        const uint32_t v = i < n ? (uint32_t) __ldcs(reinterpret_cast<const unsigned short *>(tmp_val) + b + i) : 0u;
        vv[q / 2u] = (q & 1u) ? vv[q / 2u] | v << 16 : v;
    }
    for (uint32_t d = t; d < D; d += kTpThreadsCoo) {
        at[d] = two.cnt[(std::size_t) blockIdx.x * D + d];
        gbase[d] = two.first<kAdd>(blockIdx.x, D, d);
    }
    __syncthreads();
    block_scan_small<(D + kTpThreadsCoo - 1u) / kTpThreadsCoo>(at, D, scan33);
    for (uint32_t d = t; d < D; d += kTpThreadsCoo) gbase[d] -= at[d]; // global slot of staging slot 0
    __syncthreads();
#pragma unroll
    for (unsigned q = 0; q < kPer; ++q) {
        if (kk[q] == 0xffffffffu) continue;
        const uint32_t lp = atomicAdd(at + tp_digit<LB>(kk[q]), 1u);
        if (lp < kTpChunk) {
            st_key[lp] = kk[q];
            st_val[lp] = (uint16_t) ((q & 1u) ? vv[q / 2u] >> 16 : vv[q / 2u]);
        }
    }
    __syncthreads();
#pragma unroll 4
    for (uint32_t j = t; j < n; j += kTpThreadsCoo) {
        const uint32_t key = st_key[j];
        const uint32_t g = gbase[tp_digit<LB>(key)] + j;
        out_idx[g] = tp_payload<LB>(key);
        out_val[g] = st_val[j];
    }
}

constexpr std::size_t tp_scatter2_coo_smem(uint32_t low_bits) {
    return (std::size_t) kTpChunk * 6u + ((std::size_t) 2u << low_bits) * 4u + 4u;
}

// Pass 2 of the transpose.  Pass 1 is stable, so the rows of a chunk never
// decrease, and the rank of an entry among its column's is the number of
// earlier ROWS of the chunk that hold the column: a bitmap over (32-row word,
// column) filled by atomicOr in any order, popcounts prefixed per column (the
// prefix starts at the column's staging slot, so one lookup gives the slot).
// The bitmap covers 32 * kTpSpanWords rows; a chunk that spans more goes round
// by round (rows ascending), one that would take over kTpRounds by ballots.
// A row that holds a column twice leaves fewer bits than entries: its chunk is
// ranked by ballots.  A matrix with under kTpRowsKernelMin entries per row and
// 256 columns takes the ballot kernel for all chunks: at 300,000 x 32,768 and
// density 0.02 (5 entries) the whole transpose takes 2.76 ms this way and 2.96
// by ballots, at 0.01 (2.6) 1.64 and 1.61, at 0.006 1.12 and 1.06.
// 300,000 x 32,768, 393 M entries: 1.80 ms (4.7 GB) where ballots in every
// chunk took 2.45; bound by shared-memory wavefronts (34 per 32 entries).
constexpr double kTpRowsKernelMin = 3.0;
constexpr unsigned kTpThreads2 = 512;
constexpr unsigned kTpWarps2 = kTpThreads2 / 32;
constexpr uint32_t kTpSpanWords = 36; // two CTAs per SM with the stage
constexpr uint32_t kTpSpanKeys = kTpSpanWords << (kTpBucketBits + 5u); // packed words of a span
constexpr uint32_t kTpRounds = 4;
constexpr unsigned kTpPerThread = kTpChunk / kTpThreads2;

struct tp_rows_smem {
    uint32_t key[kTpChunk];                // staged words
    uint32_t bits[kTpSpanWords * 256];     // ballots: cnt, bas
    uint16_t pre[kTpSpanWords * 256];
    uint16_t val[kTpChunk];                // staged values
    uint32_t gbase[256], lb[257], fill[256], scan33[33], dup;
};
static_assert(0xffffffffu - kTpRounds * kTpSpanKeys >= kTpSpanKeys, "no entry is past every span of a chunk");
static_assert(sizeof(uint32_t) * kTpSpanWords * 256u >= 2u * kTpWarps2 * 256u * sizeof(uint16_t),
              "the ballot counters fit the bitmap's place");

template <bool kAdd>
__global__ void __launch_bounds__(kTpThreads2, 2)
    tp_scatter2_rows_kernel(const uint32_t *__restrict__ tmp_key, const uint16_t *__restrict__ tmp_val,
                            const uint2 *__restrict__ chunk_range, const tp_counts two,
                            uint32_t *__restrict__ out_idx, uint16_t *__restrict__ out_val) {
    extern __shared__ __align__(16) unsigned char tp_rs[];
    tp_rows_smem &sm = *reinterpret_cast<tp_rows_smem *>(tp_rs);
    constexpr int LB = (int) kTpBucketBits;
    const uint32_t b = chunk_range[blockIdx.x].x, e = chunk_range[blockIdx.x].y;
    if (b >= e) return;
    const unsigned t = threadIdx.x;
    const uint32_t n = min(e - b, kTpChunk);
    // consecutive lanes take consecutive entries: ~3 rows of ascending columns,
    // few of which meet in one bitmap word
    uint32_t kk[kTpPerThread];
    uint32_t vv[kTpPerThread / 2u];
    const uint32_t *kp = tmp_key + b + t;
    const unsigned short *vp = reinterpret_cast<const unsigned short *>(tmp_val) + b + t;
    if (n == kTpChunk) {
#pragma unroll
        for (unsigned q = 0; q < kTpPerThread; ++q) kk[q] = __ldcs(kp + q * kTpThreads2);
#pragma unroll
        for (unsigned q = 0; q < kTpPerThread; q += 2u)
            vv[q / 2u] = (uint32_t) __ldcs(vp + q * kTpThreads2) | (uint32_t) __ldcs(vp + (q + 1u) * kTpThreads2) << 16;
    } else {
        // no entry: the word before the first span.  A round's k0 lies at most kTpRounds spans
        // behind it, so the difference wraps to near 2^32, past every span (the word of all
        // ones would be inside a span that starts in the last 36 * 32 rows below 2^24)
        const uint32_t none = (__ldg(tmp_key + b) >> (LB + 5) << (LB + 5)) - 1u;
#pragma unroll
        for (unsigned q = 0; q < kTpPerThread; ++q) {
            const bool in = q * kTpThreads2 + t < n;
            kk[q] = in ? __ldcs(kp + q * kTpThreads2) : none;
            const uint32_t v = in ? (uint32_t) __ldcs(vp + q * kTpThreads2) : 0u;
            vv[q / 2u] = (q & 1u) ? vv[q / 2u] | v << 16 : v;
        }
    }
    if (t < 256u) {
        sm.lb[t] = two.cnt[(std::size_t) blockIdx.x * 256u + t];
        sm.gbase[t] = two.first<kAdd>(blockIdx.x, 256u, t);
    }
    if (t == 0u) sm.dup = 0u;
    const uint32_t w_first = __ldg(tmp_key + b) >> (LB + 5), w_last = __ldg(tmp_key + e - 1u) >> (LB + 5);
    __syncthreads();
    block_scan_small<1>(sm.lb, 256u, sm.scan33);
    if (t < 256u) {
        sm.fill[t] = sm.lb[t];
        sm.gbase[t] -= sm.lb[t]; // global slot of staging slot 0
    }
    bool ballots = (w_last - w_first) / kTpSpanWords >= kTpRounds;
    if (!ballots) {
        for (uint32_t w0 = w_first; w0 <= w_last; w0 += kTpSpanWords) {
            const uint32_t words = min(kTpSpanWords, w_last - w0 + 1u), k0 = w0 << (LB + 5);
            const uint32_t span = words << (LB + 5); // the words past it are not cleared
            for (uint32_t w = t; w < words * 64u; w += kTpThreads2)
                reinterpret_cast<uint4 *>(sm.bits)[w] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
#pragma unroll
            for (unsigned q = 0; q < kTpPerThread; ++q) {
                const uint32_t x = kk[q] - k0;
                if (x < span) atomicOr(sm.bits + (x >> 5), 1u << (x & 31u));
            }
            __syncthreads();
            // two threads per column, each with half of the words: the prefix
            // starts at the column's next staging slot
            {
                constexpr uint32_t kHalf = kTpSpanWords / 2u;
                const uint32_t d = t >> 1, h = t & 1u;
                uint32_t c[kHalf], sum = 0u;
#pragma unroll
                for (uint32_t w = 0; w < kHalf; ++w) {
                    c[w] = h * kHalf + w < words ? __popc(sm.bits[(h * kHalf + w) * 256u + d]) : 0u;
                    sum += c[w];
                }
                const uint32_t other = __shfl_xor_sync(0xffffffffu, sum, 1);
                uint32_t run = sm.fill[d] + (h ? other : 0u);
#pragma unroll
                for (uint32_t w = 0; w < kHalf; ++w) {
                    sm.pre[(h * kHalf + w) * 256u + d] = (uint16_t) run;
                    run += c[w];
                }
                __syncwarp();
                if (h) sm.fill[d] = run;
            }
            __syncthreads();
#pragma unroll
            for (unsigned q = 0; q < kTpPerThread; ++q) {
                const uint32_t x = kk[q] - k0;
                if (x < span) {
                    const uint32_t lp = sm.pre[x >> 5] + __popc(sm.bits[x >> 5] & ((1u << (x & 31u)) - 1u));
                    sm.key[lp] = kk[q]; // lp < n: the column's slots start at lb and hold its entries
                    sm.val[lp] = (uint16_t) ((q & 1u) ? vv[q / 2u] >> 16 : vv[q / 2u]);
                }
            }
            __syncthreads();
        }
        if (t < 256u && sm.fill[t] != sm.lb[t + 1u]) sm.dup = 1u;
        __syncthreads();
        ballots = sm.dup != 0u;
    }
    if (ballots) {
        __syncthreads();
        tp_stage sg;
        sg.cnt = reinterpret_cast<uint16_t *>(sm.bits);
        sg.bas = sg.cnt + kTpWarps2 * 256u;
        sg.lb = sm.lb;
        sg.fill = sm.fill;
        if (t < 256u) sm.fill[t] = 0u;
        for (uint32_t w = t; w < kTpWarps2 * 256u; w += kTpThreads2) sg.cnt[w] = 0u;
        __syncthreads();
        tp_rank_ballots<LB, kTpWarps2>(tmp_key, tmp_val, b, e, sg, sm.key, sm.val);
        __syncthreads();
    }
#pragma unroll 4
    for (uint32_t j = t; j < n; j += kTpThreads2) {
        const uint32_t key = sm.key[j];
        const uint32_t g = sm.gbase[tp_digit<LB>(key)] + j;
        out_idx[g] = tp_payload<LB>(key);
        out_val[g] = sm.val[j];
    }
}

constexpr std::size_t tp_scatter2_smem(uint32_t low_bits) {
    return (std::size_t) kTpChunk * 6u + ((std::size_t) 2u * kTpWarps * 2u << low_bits);
}

enum class tp_rank { rows, ballots, any }; // how a pass-2 chunk is ranked

template <typename K>
int tp_smem(K kernel, std::size_t smem, const char *what) {
    return cuda_ok(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem), what);
}

// The totals of `t`'s digits, and its offsets: complete but for the digits'
// starts, which the scatter then adds (t->start), where the rows are few (in each
// segment, or kTpDirectRows in all); else tp_offsets_apply adds them once they are
// scanned.  rows [0, rows) in slices of len, or the segments' slices `range`; a
// segment has at most most_rows of the total_rows.
// us of a transpose into 262,144 columns (1,024 buckets; 1 M / 2 M / 6 M entries):
// 101 / 121 / 233, with 32 threads a digit in every segment 144 / 163 / 279 (44 of
// them in 8,192 CTAs of the second pass's scan).
int tp_offsets(tp_counts *t, uint32_t D, uint32_t rows, uint32_t total_rows, uint32_t most_rows, uint32_t len,
               uint32_t slices, uint32_t segments, const uint32_t *seg_first, const uint2 *range, uint32_t limit,
               uint32_t *totals, const uint32_t *start, cudaStream_t stream) {
    const dim3 grid(segments, (D + 31u) / 32u), by_digit(segments, (D + 255u) / 256u);
    // a serial step per 8 rows of the longest segment there can be against 8 CTAs of 1,024
    // threads a segment, two to an SM: they cost the same at about four segments a row
    auto few = [&](uint32_t n) { return segments > 1u && n <= segments / 4u; };
    if (few(most_rows)) {
        t->start = start;
        tp_segment_scan_kernel<<<by_digit, 256, 0, stream>>>(t->cnt, D, seg_first, range, limit, t->base, totals);
        return launch_ok("tp_segment_scan_kernel");
    }
    if (total_rows <= kTpDirectRows) {
        t->start = start;
        tp_rows_scan_kernel<<<grid, 1024, 0, stream>>>(t->cnt, D, rows, seg_first, range, limit, t->base, totals);
        return launch_ok("tp_rows_scan_kernel");
    }
    const dim3 by_slice(slices, (D + 255u) / 256u);
    tp_slice_sums_kernel<<<by_slice, 256, 0, stream>>>(t->cnt, D, rows, len, range, t->slices);
    if (!launch_ok("tp_slice_sums_kernel")) return 0;
    if (few(most_rows / len + 2u)) {
        tp_segment_scan_kernel<<<by_digit, 256, 0, stream>>>((const uint32_t *) t->slices, D, seg_first, nullptr, limit,
                                                             t->slices, totals);
        return launch_ok("tp_segment_scan_kernel");
    }
    tp_slice_scan_kernel<<<grid, 1024, 0, stream>>>(t->slices, D, seg_first, slices, limit, totals);
    return launch_ok("tp_slice_scan_kernel");
}

int tp_offsets_apply(const tp_counts &t, uint32_t D, uint32_t rows, uint32_t len, uint32_t slices, const uint2 *range,
                     const uint32_t *segment, uint32_t limit, const uint32_t *start, cudaStream_t stream) {
    if (t.start != nullptr) return 1;
    tp_slice_apply_kernel<<<dim3(slices, (D + 255u) / 256u), 256, 0, stream>>>(t.cnt, D, rows, len, range, segment,
                                                                                  t.slices, start, limit, t.base);
    return launch_ok("tp_slice_apply_kernel");
}

// Counts and pass 2 of `l`'s pass-1 result (low digit of LB bits).  rows: the
// payloads of a bucket never decrease (the transpose); any: entries of one key
// in any order (COO); ballots: in their own order.
template <int LB, tp_rank kRank>
int tp_second_pass(uint32_t uDim, const tp2_layout &l, uint32_t *out_ptr, uint32_t *out_idx, uint16_t *out_val,
                   cudaStream_t stream) {
    static_assert(kRank != tp_rank::rows || LB == (int) kTpBucketBits, "the row ranking has 256 digits");
    tp_hist2_kernel<LB><<<l.max_chunks, kTpThreads, 0, stream>>>(l.tmp_key, l.chunk_range, l.two.cnt);
    if (!launch_ok("tp_hist2_kernel")) return 0;
    constexpr uint32_t D = 1u << LB;
    tp_counts two = l.two;
    if (!tp_offsets(&two, D, 0u, l.max_chunks, l.most_chunks, l.slice2, l.max_slices, l.K, l.slice_first,
                    l.slice_range, uDim, out_ptr, out_ptr, stream) ||
        !scan_exclusive_u32(out_ptr, out_ptr, uDim, true, l.scan_tmp, l.scan_bytes, stream) ||
        !tp_offsets_apply(two, D, 0u, 0u, l.max_slices, l.slice_range, l.slice_bucket, uDim, out_ptr, stream))
        return 0;
    const bool add = two.start != nullptr;
    auto launch = [&](auto kern, unsigned threads, std::size_t smem) {
        if (!tp_smem(kern, smem, "scatter2 smem attribute")) return 0;
        kern<<<l.max_chunks, threads, smem, stream>>>(l.tmp_key, l.tmp_val, l.chunk_range, two, out_idx, out_val);
        return launch_ok("tp_scatter2_kernel");
    };
    if constexpr (kRank == tp_rank::rows)
        return launch(add ? tp_scatter2_rows_kernel<true> : tp_scatter2_rows_kernel<false>, kTpThreads2,
                      sizeof(tp_rows_smem));
    else if constexpr (kRank == tp_rank::any)
        return launch(add ? tp_scatter2_coo_kernel<LB, true> : tp_scatter2_coo_kernel<LB, false>, kTpThreadsCoo,
                      tp_scatter2_coo_smem(LB));
    else
        return launch(add ? tp_scatter2_kernel<LB, true> : tp_scatter2_kernel<LB, false>, kTpThreads,
                      tp_scatter2_smem(LB));
}

// Pass 1: `ptr` is null for COO (payloads `pay` through `pay_map`; `stable`
// keeps the entries' order).
int tp_first_pass(uint32_t cDim, uint32_t uDim, uint32_t nnz, const uint32_t *ptr, const uint32_t *key,
                  const uint16_t *val, const uint32_t *pay, const uint32_t *pay_map, bool stable, const tp2_layout &l,
                  cudaStream_t stream) {
    const bool csr = ptr != nullptr, vec = (reinterpret_cast<uintptr_t>(key) & 15u) == 0u;
    auto hist1 = csr ? (vec ? tp_hist1_kernel<kTpTileCsr, true> : tp_hist1_kernel<kTpTileCsr, false>)
                     : (vec ? tp_hist1_kernel<kTpTileCoo, true> : tp_hist1_kernel<kTpTileCoo, false>);
    hist1<<<l.tiles1, kTpThreads, (std::size_t) l.K * 4u, stream>>>(key, nnz, uDim, l.low_bits, l.K, l.one.cnt,
                                                                    l.status);
    if (!launch_ok("tp_hist1_kernel")) return 0;
    tp_counts one = l.one;
    if (!tp_offsets(&one, l.K, l.tiles1, l.tiles1, l.tiles1, l.slice1, l.slices1, 1u, nullptr, nullptr, l.K, l.total1,
                    l.start1, stream))
        return 0;
    tp_chunks_kernel<<<1, 1024, 0, stream>>>(l);
    if (!launch_ok("tp_chunks_kernel") ||
        !tp_offsets_apply(one, l.K, l.tiles1, l.slice1, l.slices1, nullptr, nullptr, l.K, l.start1, stream))
        return 0;
    const bool add = one.start != nullptr;
    if (csr) {
        auto kern = add ? tp_scatter1_csr_kernel<true> : tp_scatter1_csr_kernel<false>;
        const std::size_t smem = tp_scatter1_csr_smem(l.K);
        if (!tp_smem(kern, smem, "scatter1 smem attribute")) return 0;
        kern<<<l.tiles1, kTpThreads1, smem, stream>>>(ptr, key, val, cDim, uDim, nnz, l.K, one, l.gran_row, l.tmp_key,
                                                      l.tmp_val);
    } else {
        auto any = add ? tp_scatter1_coo_kernel<true> : tp_scatter1_coo_kernel<false>;
        auto in_order = add ? tp_scatter1_coo_stable_kernel<true> : tp_scatter1_coo_stable_kernel<false>;
        auto kern = stable ? in_order : any;
        const std::size_t smem = stable ? tp_scatter1_smem(l.K) : tp_scatter1_coo_smem(l.K);
        if (!tp_smem(kern, smem, "scatter1 smem attribute")) return 0;
        kern<<<l.tiles1, stable ? kTpThreads : kTpThreadsCoo, smem, stream>>>(key, val, pay, pay_map, uDim, nnz,
                                                                              l.low_bits, l.K, one, l.tmp_key,
                                                                              l.tmp_val);
    }
    return launch_ok("tp_scatter1_kernel");
}

int transpose2_launch(uint32_t cDim, uint32_t uDim, uint32_t nnz, const uint32_t *ptr, const uint32_t *idx,
                      const uint16_t *val, uint32_t *out_ptr, uint32_t *out_idx, uint16_t *out_val,
                      const tp2_layout &l, cudaStream_t stream) {
    tp_gran_rows_kernel<<<(cDim + 255u) / 256u, 256, 0, stream>>>(ptr, cDim, l.gran_row);
    if (!launch_ok("tp_gran_rows_kernel")) return 0;
    return tp_first_pass(cDim, uDim, nnz, ptr, idx, val, nullptr, nullptr, false, l, stream) &&
           ((double) nnz >= kTpRowsKernelMin * (double) cDim * (double) l.K
                ? tp_second_pass<(int) kTpBucketBits, tp_rank::rows>(uDim, l, out_ptr, out_idx, out_val, stream)
                : tp_second_pass<(int) kTpBucketBits, tp_rank::ballots>(uDim, l, out_ptr, out_idx, out_val, stream));
}

uint32_t bits_below(uint64_t v) { // bits that hold 0 .. v - 1
    uint32_t b = 0u;
    while (((uint64_t) 1u << b) < v) ++b;
    return b;
}

// Low digit of the row partition: the fewest bits that keep the buckets within
// kTpMaxBuckets; 0 where the partition does not apply (more rows than that
// allows, or a column and the digit do not fit one packed word together, with
// the word of all ones left over as "no entry").
uint32_t partition_low_bits(uint32_t rows, uint32_t cols) {
    uint32_t lb = kTpBucketBits;
    while (lb <= kTpMaxLowBits && (uint64_t) rows > ((uint64_t) kTpMaxBuckets << lb)) ++lb;
    return lb <= kTpMaxLowBits && bits_below((uint64_t) cols + 1u) + lb <= 32u ? lb : 0u;
}

} // namespace

int transpose_launch(uint32_t cDim, uint32_t uDim, uint32_t nnz, const uint32_t *ptr, const uint32_t *idx,
                     const uint16_t *val, uint32_t *out_ptr, uint32_t *out_idx, uint16_t *out_val, void *scratch,
                     std::size_t scratch_bytes, cudaStream_t stream) {
    if (tp2_applicable(cDim, uDim)) {
        tp2_layout l2;
        tp2_make_layout(uDim, nnz, kTpBucketBits, true, scratch, scratch_bytes, &l2);
        if (scratch == nullptr || l2.bytes > scratch_bytes) {
            set_error("compressed_transpose: scratch %zu < %zu bytes", scratch_bytes, l2.bytes);
            return 0;
        }
        if (!cuda_ok(cudaMemsetAsync(l2.status, 0, 16, stream), "transpose status memset") ||
            !cuda_ok(cudaMemsetAsync(out_ptr, 0, ((std::size_t) uDim + 1u) * 4u, stream), "transpose out_ptr memset"))
            return 0;
        if (nnz == 0u || cDim == 0u || uDim == 0u) return 1;
        return transpose2_launch(cDim, uDim, nnz, ptr, idx, val, out_ptr, out_idx, out_val, l2, stream);
    }
    tr_layout l;
    make_layout(cDim, uDim, scratch, scratch_bytes, &l);
    if (scratch == nullptr || l.bytes > scratch_bytes) {
        set_error("compressed_transpose: scratch %zu < %zu bytes", scratch_bytes, l.bytes);
        return 0;
    }
    if (!cuda_ok(cudaMemsetAsync(l.status, 0, 16, stream), "transpose status memset") ||
        !cuda_ok(cudaMemsetAsync(out_ptr, 0, ((std::size_t) uDim + 1u) * 4u, stream), "transpose out_ptr memset"))
        return 0;
    if (nnz == 0u || cDim == 0u || uDim == 0u) return 1;
    const std::size_t smem = (std::size_t) min(uDim, kColRange) * sizeof(uint32_t);
    if (!cuda_ok(cudaFuncSetAttribute(tr_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem),
                 "hist smem attribute") ||
        !cuda_ok(cudaFuncSetAttribute(tr_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem),
                 "scatter smem attribute"))
        return 0;
    dim3 grid(l.tiles, l.passes);
    tr_hist_kernel<<<grid, kThreads, smem, stream>>>(ptr, idx, cDim, uDim, l.tile_rows, l.hist, l.status);
    if (!launch_ok("tr_hist_kernel")) return 0;
    tr_colscan_kernel<<<(uDim + 255u) / 256u, 256, 0, stream>>>(uDim, l.tiles, l.hist, out_ptr);
    if (!launch_ok("tr_colscan_kernel")) return 0;
    if (!scan_exclusive_u32(out_ptr, out_ptr, uDim, true, l.scan_tmp, l.scan_bytes, stream)) return 0;
    tr_scatter_kernel<<<grid, kThreads, smem, stream>>>(ptr, idx, val, cDim, uDim, l.tile_rows, l.hist, out_ptr,
                                                        out_idx, out_val, l.status);
    return launch_ok("tr_scatter_kernel");
}

// COO entries by rows: row pointers, columns (through `map` when given) and
// values, a row's entries in any order or, `stable`, in their own.  Every row
// is below `rows` and every mapped column below `cols`.  Two passes move 22 bytes
// an entry in runs; the two stable 32-bit sorts and the random gathers that this
// replaces moved over 100, most of them one sector per entry.
std::size_t partition_rows_scratch_bytes(uint32_t n, uint32_t rows, uint32_t cols) {
    const uint32_t lb = partition_low_bits(rows, cols);
    if (n == 0u || rows == 0u || lb == 0u) return 0u;
    tp2_layout l;
    tp2_make_layout(rows, n, lb, false, nullptr, 0, &l);
    return l.bytes;
}

int partition_rows(uint32_t n, uint32_t rows, uint32_t cols, const uint32_t *row, const uint32_t *col,
                   const uint32_t *map, const uint16_t *val, bool stable, uint32_t *out_ptr, uint32_t *out_col,
                   uint16_t *out_val, void *scratch, std::size_t scratch_bytes, cudaStream_t stream) {
    const uint32_t lb = partition_low_bits(rows, cols);
    if (n == 0u || rows == 0u || lb == 0u) {
        set_error("partition_rows: %u rows by %u columns outside its range", rows, cols);
        return 0;
    }
    tp2_layout l;
    tp2_make_layout(rows, n, lb, false, scratch, scratch_bytes, &l);
    if (scratch == nullptr || l.bytes > scratch_bytes) {
        set_error("partition_rows: scratch %zu < %zu bytes", scratch_bytes, l.bytes);
        return 0;
    }
    if (!cuda_ok(cudaMemsetAsync(l.status, 0, 16, stream), "partition status memset") ||
        !tp_first_pass(0u, rows, n, nullptr, row, val, col, map, stable, l, stream))
        return 0;
    auto second = [&](auto low) {
        constexpr int LB = decltype(low)::value;
        return stable ? tp_second_pass<LB, tp_rank::ballots>(rows, l, out_ptr, out_col, out_val, stream)
                      : tp_second_pass<LB, tp_rank::any>(rows, l, out_ptr, out_col, out_val, stream);
    };
    switch (lb) {
        case 8u: return second(std::integral_constant<int, 8>{});
        case 9u: return second(std::integral_constant<int, 9>{});
        case 10u: return second(std::integral_constant<int, 10>{});
        default: return second(std::integral_constant<int, 11>{});
    }
}

std::size_t transpose_scratch(uint32_t cDim, uint32_t uDim, uint32_t nnz) {
    if (tp2_applicable(cDim, uDim)) {
        tp2_layout l2;
        tp2_make_layout(uDim, nnz, kTpBucketBits, true, nullptr, 0, &l2);
        return l2.bytes;
    }
    tr_layout l;
    make_layout(cDim, uDim, nullptr, 0, &l);
    return l.bytes;
}

// CSC (cols-major) -> CSR (rows-major) into fresh device buffers (used by the
// host conversion wrappers for column-compressed input).
int transpose_csc_to_csr_staged(const cs_compressed_view *src, uint32_t **d_ptr, uint32_t **d_idx, uint16_t **d_val,
                                cudaStream_t stream) {
    const uint32_t cDim = src->cols, uDim = src->rows;
    void *scratch = nullptr;
    const std::size_t sb = transpose_scratch(cDim, uDim, src->nnz);
    if (!cuda_ok(cudaMalloc((void **) d_ptr, ((std::size_t) uDim + 1u) * 4u), "transpose ptr") ||
        !cuda_ok(cudaMalloc((void **) d_idx, (std::size_t) src->nnz * 4u + 16u), "transpose idx") ||
        !cuda_ok(cudaMalloc((void **) d_val, (std::size_t) src->nnz * 2u + 16u), "transpose val") ||
        !cuda_ok(cudaMalloc(&scratch, sb), "transpose scratch"))
        return 0;
    int ok = transpose_launch(cDim, uDim, src->nnz, src->majorPtr, src->minorIdx, src->val, *d_ptr, *d_idx, *d_val,
                              scratch, sb, stream);
    uint32_t status = 0u;
    if (ok)
        ok = cuda_ok(cudaMemcpyAsync(&status, scratch, 4, cudaMemcpyDeviceToHost, stream), "transpose status") &&
             cuda_ok(cudaStreamSynchronize(stream), "transpose sync");
    cudaFree(scratch);
    if (ok && status != 0u) {
        set_error("column-compressed input rejected (status 0x%x)", status);
        ok = 0;
    }
    return ok;
}

} // namespace csb

using namespace csb;

extern "C" int cs_b200_compressed_transpose_scratch_bytes(uint32_t cDim, uint32_t uDim, uint32_t nnz,
                                                          size_t *out_bytes) {
    if (out_bytes == nullptr) {
        set_error("compressed_transpose_scratch_bytes: null output");
        return 0;
    }
    *out_bytes = transpose_scratch(cDim, uDim, nnz);
    return 1;
}

extern "C" int cs_b200_build_compressed_transpose(uint32_t cDim, uint32_t uDim, uint32_t nnz, const uint32_t *d_cAxPtr,
                                                  const uint32_t *d_uAxIdx, const uint16_t *d_val,
                                                  uint32_t *d_out_uAxPtr, uint32_t *d_heads, uint32_t *d_out_cAxIdx,
                                                  uint16_t *d_out_val, void *d_scan_tmp, size_t scan_bytes,
                                                  cs_stream_t s) {
    (void) d_heads;
    if (d_out_uAxPtr == nullptr || (nnz != 0u && (d_cAxPtr == nullptr || d_uAxIdx == nullptr || d_val == nullptr ||
                                                  d_out_cAxIdx == nullptr || d_out_val == nullptr))) {
        set_error("compressed_transpose: null device array");
        return 0;
    }
    return transpose_launch(cDim, uDim, nnz, d_cAxPtr, d_uAxIdx, d_val, d_out_uAxPtr, d_out_cAxIdx, d_out_val,
                            d_scan_tmp, scan_bytes, as_stream(s));
}
