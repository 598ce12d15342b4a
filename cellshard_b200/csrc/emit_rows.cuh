// Sliced-ELL row emission of the single-partition and batched converters: row r
// owns the w slots [base, base + w) of its slice; its n real (column, value)
// pairs go into the first n slots in CSR order, the rest is padding
// (CS_INVALID_COL, 0) -- sliced_ell_from_compressed.cuh:49-80.
//
// A group of GL lanes (GL in {32, 16, 8, 4}) writes one row.  Real slots are
// copied lane by lane, so loads and stores are whole lines whatever the two
// rows' alignments, kEmitFlight of them in flight per lane before the first is
// stored: a row is one latency per GL * kEmitFlight entries, and with 24 warps
// an SM that latency is what bounds the copy.  (Four slots a lane with 16-byte
// stores took eight scattered loads and one latency per 4 * GL slots.)  The
// padding needs no loads: 16-byte column and 8-byte value stores between an
// unaligned head and tail.  Requires col_idx 16-byte and val 8-byte aligned.
#pragma once

#include "common.cuh"

namespace csb {

constexpr unsigned kEmitFlight = 8;

template <unsigned GL>
__device__ __forceinline__ void sell_emit_row_vec(const uint32_t *__restrict__ idx, const uint16_t *__restrict__ val,
                                                  uint32_t a, uint32_t n, uint32_t w, std::size_t base,
                                                  uint32_t *__restrict__ col_idx, uint16_t *__restrict__ out_val,
                                                  unsigned gl) {
    if (n > w) n = w;
    const uint32_t *ip = idx + a;
    const unsigned short *vp = reinterpret_cast<const unsigned short *>(val) + a;
    uint32_t *cp = col_idx + base;
    uint16_t *op = out_val + base;
    for (uint32_t k0 = gl; k0 < n; k0 += GL * kEmitFlight) {
        uint32_t c[kEmitFlight];
        uint16_t v[kEmitFlight];
#pragma unroll
        for (unsigned u = 0; u < kEmitFlight; ++u) {
            const uint32_t k = k0 + GL * u;
            if (k < n) {
                c[u] = __ldcs(ip + k);
                v[u] = __ldcs(vp + k);
            }
        }
#pragma unroll
        for (unsigned u = 0; u < kEmitFlight; ++u) {
            const uint32_t k = k0 + GL * u;
            if (k < n) {
                __stcs(cp + k, c[u]);
                __stcs(reinterpret_cast<unsigned short *>(op) + k, (unsigned short) v[u]);
            }
        }
    }
    // padding [n, w): up to three slots to a vector boundary, vectors, a tail
    const uint32_t head = min(w, n + ((4u - (uint32_t) ((base + n) & 3u)) & 3u));
    const uint32_t body_end = head + ((w - head) & ~3u);
    if (n + gl < head) {
        cp[n + gl] = CS_INVALID_COL;
        op[n + gl] = 0u;
    }
    for (uint32_t k = head + 4u * gl; k < body_end; k += 4u * GL) {
        __stcs(reinterpret_cast<uint4 *>(cp + k),
               make_uint4(CS_INVALID_COL, CS_INVALID_COL, CS_INVALID_COL, CS_INVALID_COL));
        __stcs(reinterpret_cast<uint2 *>(op + k), make_uint2(0u, 0u));
    }
    if (body_end + gl < w) {
        cp[body_end + gl] = CS_INVALID_COL;
        op[body_end + gl] = 0u;
    }
}

// The same for short rows that a group of lanes covers in one or two steps: four
// slots a lane, 16-byte column and 8-byte value stores from the first aligned
// slot, the unaligned head and the tail one slot at a time.  A row of under 100
// entries has no second latency to hide and keeps the wider stores (500,000 rows
// of 25, eight lanes: 135 us a call, 144 lane by lane; 300,000 of 150 by 32 lanes 250 and
// 245).
template <unsigned GL>
__device__ __forceinline__ void sell_emit_short_row_vec(const uint32_t *__restrict__ idx,
                                                        const uint16_t *__restrict__ val, uint32_t a, uint32_t n,
                                                        uint32_t w, std::size_t base, uint32_t *__restrict__ col_idx,
                                                        uint16_t *__restrict__ out_val, unsigned gl) {
    if (n > w) n = w;
    const uint32_t *ip = idx + a;
    const unsigned short *vp = reinterpret_cast<const unsigned short *>(val) + a;
    uint32_t *cp = col_idx + base;
    uint16_t *op = out_val + base;
    auto col = [&](uint32_t k) { return k < n ? __ldg(ip + k) : CS_INVALID_COL; };
    auto value = [&](uint32_t k) { return k < n ? (uint32_t) __ldg(vp + k) : 0u; };
    auto one = [&](uint32_t k) {
        cp[k] = col(k);
        op[k] = (uint16_t) value(k);
    };
    const uint32_t head = min((4u - (uint32_t) (base & 3u)) & 3u, w);
    const uint32_t body_end = head + ((w - head) & ~3u);
    if (gl < head) one(gl);
    for (uint32_t k = head + 4u * gl; k < body_end; k += 4u * GL) {
        *reinterpret_cast<uint4 *>(cp + k) = make_uint4(col(k), col(k + 1u), col(k + 2u), col(k + 3u));
        *reinterpret_cast<uint2 *>(op + k) =
            make_uint2(value(k) | value(k + 1u) << 16, value(k + 2u) | value(k + 3u) << 16);
    }
    for (uint32_t k = body_end + gl; k < w; k += GL) one(k);
}

} // namespace csb
