// Expert rows as pieces for the block-scaled expert kernel (moe_mx_tc.cu): written by a kernel of their own, or by the one that routes a small batch.
#pragma once

#include "mx_common.cuh"

namespace oxq {

constexpr int MM_BK = 128; // columns of a stage
inline int moe_mx_stages(int k) { return (k + MM_BK - 1) / MM_BK; }

// q: [pair][piece][rows_cap][k]; sfx: [pair][stage][rows_cap], a byte per 32 columns; second: [stage][rows_cap], which rows have a second pair.
// That pair is written where a row has one, and not at all elsewhere; then *any = mark. k is a multiple of 32.
struct MoeMxPieces {
    int k, stages, rows_cap;
    unsigned char *q, *sfx, *second;
    unsigned long long *any, mark;
};
inline MoeMxPieces moe_mx_pieces(int k, int rows_cap, void *pieces, void *sfx, void *second, unsigned long long mark)
{
    return {k, moe_mx_stages(k), rows_cap, (unsigned char *)pieces, (unsigned char *)sfx, (unsigned char *)second + 8, (unsigned long long *)second, mark};
}

// Sixteen lanes hold 128 columns of a row; row r is src[from(r)]. Every thread of the first `ctas` CTAs.
template <typename From> __device__ __forceinline__ void moe_mx_split_rows(const __nv_bfloat16 *src, int rows, const MoeMxPieces &p, int ctas, From from)
{
    const int lane = threadIdx.x & 15;
    for (int item = (blockIdx.x * blockDim.x + threadIdx.x) >> 4; (item & ~1) < rows * p.stages; item += (ctas * blockDim.x) >> 4) {
        const bool real = item < rows * p.stages; // the other half of a warp may be past the end: it stays for the shuffles
        const int row = real ? item / p.stages : 0, st = real ? item - row * p.stages : 0, c = st * MM_BK + lane * 8;
        uint4 raw = make_uint4(0u, 0u, 0u, 0u);
        if (c < p.k) raw = ld_produced(reinterpret_cast<const uint4 *>(src + (size_t)from(row) * p.k + c));
        const MxBlock b = mx_block(raw);
        auto store = [&](int pair, uint2 hi, uint2 lo, uint32_t s) {
            if (!real || c >= p.k) return;
            unsigned char *dst = p.q + ((size_t)pair * 2 * p.rows_cap + row) * p.k + c;
            *reinterpret_cast<uint2 *>(dst) = hi;
            *reinterpret_cast<uint2 *>(dst + (size_t)p.rows_cap * p.k) = lo;
            if ((lane & 3) == 0) p.sfx[((size_t)(pair * p.stages + st) * p.rows_cap + row) * 4 + (lane >> 2)] = (unsigned char)s;
        };
        float v[8];
        uint2 hi, lo;
        const uint32_t s = mx_first_pair(raw, b, v, hi, lo);
        store(0, hi, lo, s);
        const unsigned half = 0xFFFFu << (threadIdx.x & 16); // the row's lanes of this warp
        const unsigned ask = __ballot_sync(0xFFFFFFFFu, b.second != MX_ONE_PAIR), e5m2 = __ballot_sync(0xFFFFFFFFu, b.second == MX_SECOND_E5M2);
        if (real && lane == 0) p.second[(size_t)st * p.rows_cap + row] = (unsigned char)(!(ask & half) ? MX_ONE_PAIR : (e5m2 & half) ? MX_SECOND_E5M2 : MX_SECOND_E4M3);
        if (ask) { // some row of the warp
            const uint32_t s2 = mx_second_pair(raw, v, s, (e5m2 & half) != 0, hi, lo);
            if (ask & half) store(1, hi, lo, s2);
            if (real && lane == 0) *p.any = p.mark;
        }
    }
}

} // namespace oxq
