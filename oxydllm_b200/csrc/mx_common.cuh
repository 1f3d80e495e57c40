// Block-scaled 8-bit tensor-core MMA (tcgen05 kind::mxf8f6f4) with bf16 activations: PTX wrappers, and how bf16 values become pairs
// of 8-bit numbers.
//
// kind::mxf8f6f4 multiplies elements of at most 8 bits at twice the rate of bf16 and takes one power-of-two scale (E8M0) per
// row and 32 elements of k for each operand; it accumulates in f32. A bf16 value has 8 significant bits, an E4M3 number 4, so a
// block of 32 activations is written as hi + lo / 16, both scaled so that the block's largest magnitude lies in [128, 256): hi is
// the nearest E4M3 number and the remainder of at most 4 significant bits is lo exactly. Two MMAs (or one with both as columns)
// then cost what one bf16 MMA costs, and the weights can stay in the few bits that they have.
//
// That is exact for values of at least 2^-13 of their block's largest; smaller ones are off by up to 2^-21 of that largest. Where
// half of the block is within 2^-9 of the largest such an error is below 2^-12 of an ordinary value of the block, less than bf16's own
// rounding, and is let be. Elsewhere (an outlier among small values, whose weight may be zero) what is missing becomes a second pair
// with a scale of its own, exact for another 13 binades, and the stage of k is multiplied a second time with it. Infinities and NaN
// have no E4M3 form: they are zero in the first pair, and the second pair of their tile is then E5M2, which has both (its numbers
// have 3 significant bits, the rest of such a tile is right to 2^-27 of a block's largest).
#pragma once

#include <atomic>

#include <cuda_fp8.h>

#include "tc_common.cuh"

namespace oxq {

// D[tmem] (+)= (A * 2^(sfa-127)) (B * 2^(sfb-127)), K = 32; which byte of the scale words counts is in idesc.
__device__ __forceinline__ void umma_mxf8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                          uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], %1, %2, %3, [%4], [%5], p;\n\t}"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
                 : "memory");
}
// Scales of 128 rows and four 32-wide blocks of k: 512 bytes, row r's four at (r % 32) * 16 + (r / 32) * 4, to four columns
// of tensor memory. Ordered before the MMAs that the same thread issues behind it.
__device__ __forceinline__ void tmem_cp_scales(uint32_t taddr, uint32_t smem_addr)
{
    const uint64_t desc = (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46);
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}
// Four columns of this warp's quarter of tensor memory, the same word everywhere.
__device__ __forceinline__ void tmem_fill4(uint32_t taddr, uint32_t v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %1, %1, %1};" ::"r"(taddr), "r"(v) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// 8 columns of this warp's quarter of tensor memory.
__device__ __forceinline__ void tmem_ld_x8(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

constexpr int MX_E4M3 = 0, MX_E5M2 = 1, MX_E2M1 = 5;
// Instruction descriptor: A and B element types, E8M0 scales; bits 29 and 4 up choose the byte of A's and B's scale words.
__host__ __device__ constexpr uint32_t mx_idesc(int a_type, int n)
{
    return ((uint32_t)a_type << 7) | ((uint32_t)MX_E4M3 << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) |
           ((128u >> 4) << 24);
}
constexpr uint32_t MX_IDESC_B_E5M2 = (uint32_t)(MX_E5M2 ^ MX_E4M3) << 10; // turns B's type
__host__ __device__ constexpr uint32_t mx_idesc_blocks(int a_block, int b_block) { return ((uint32_t)a_block << 29) | ((uint32_t)b_block << 4); }

// Whether a stage of a tile has a second pair of pieces, and of which type.
constexpr int MX_ONE_PAIR = 0, MX_SECOND_E4M3 = 1, MX_SECOND_E5M2 = 2;

// What a block of 32 values needs; this lane has eight of them, the other three of four neighbouring lanes the rest.
struct MxBlock {
    uint32_t e; // biased exponent of the largest finite magnitude
    int second; // MX_...
};
__device__ __forceinline__ MxBlock mx_block(const uint4 &raw)
{
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    // Largest magnitude and smallest but for zeros (which become 0xFFFF), two at a time. Most warps have nothing that needs a closer look.
    uint32_t hi2 = 0, lo2 = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t a = w[i] & 0x7FFF7FFFu;
        hi2 = __vmaxu2(hi2, a);
        lo2 = __vminu2(lo2, __vsub2(a, 0x00010001u));
    }
    uint32_t both = (max(hi2 >> 16, hi2 & 0xFFFFu) << 16) | (0xFFFFu - min(lo2 >> 16, lo2 & 0xFFFFu));
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) both = __vmaxu2(both, __shfl_xor_sync(0xFFFFFFFFu, both, o));
    MxBlock b;
    b.e = both >> 23;
    b.second = MX_ONE_PAIR;
    const uint32_t least = 0xFFFFu - (both & 0xFFFFu); // magnitude less one; 0xFFFF: all zero
    if (!__any_sync(0xFFFFFFFFu, b.e == 255u || (least != 0xFFFFu && b.e - (least + 1u >> 7) > 13u))) return b;
    uint32_t h[8], amax = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        h[i] = ((i & 1) ? w[i >> 1] : w[i >> 1] << 16) & 0x7FFF0000u;
        if (h[i] < 0x7F800000u) amax = max(amax, h[i]);
    }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) amax = max(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
    b.e = amax >> 23;
    // a byte each: values within 2^-9 of the largest, those farther off, those below 2^-13, infinities and NaN
    uint32_t count = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t d = b.e - (h[i] >> 23);
        if (h[i] >= 0x7F800000u) count += 1u << 24;
        else if (h[i] != 0u) count += d > 13u ? 0x010100u : d > 8u ? 0x000100u : 1u;
    }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) count += __shfl_xor_sync(0xFFFFFFFFu, count, o);
    b.second = count >> 24 ? MX_SECOND_E5M2 : (count >> 16) && (count >> 8 & 0xFFu) > (count & 0xFFu) ? MX_SECOND_E4M3 : MX_ONE_PAIR;
    return b;
}

template <__nv_fp8_interpretation_t TYPE> __device__ __forceinline__ float2 mx_decode(uint16_t two)
{
    const __half2_raw r = __nv_cvt_fp8x2_to_halfraw2(two, TYPE);
    return __half22float2(*reinterpret_cast<const __half2 *>(&r));
}
// v times mul as hi + lo / 16; v becomes what is missing.
template <__nv_fp8_interpretation_t TYPE> __device__ __forceinline__ void mx_pair(float (&v)[8], float mul, uint2 &hi, uint2 &lo)
{
    uint16_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float a = v[2 * i] * mul, b = v[2 * i + 1] * mul;
        h[i] = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, TYPE);
        const float2 f = mx_decode<TYPE>(h[i]);
        a -= f.x;
        b -= f.y;
        l[i] = __nv_cvt_float2_to_fp8x2(make_float2(a * 16.0f, b * 16.0f), __NV_SATFINITE, TYPE);
        const float2 g = mx_decode<TYPE>(l[i]);
        v[2 * i] = fmaf(g.x, -0.0625f, a);
        v[2 * i + 1] = fmaf(g.y, -0.0625f, b);
    }
    hi = make_uint2((uint32_t)h[0] | ((uint32_t)h[1] << 16), (uint32_t)h[2] | ((uint32_t)h[3] << 16));
    lo = make_uint2((uint32_t)l[0] | ((uint32_t)l[1] << 16), (uint32_t)l[2] | ((uint32_t)l[3] << 16));
}
// The first pair, infinities and NaN as zero; returns the block's scale byte (lo's is four less). v: what is missing, in units of that scale.
__device__ __forceinline__ uint32_t mx_first_pair(const uint4 &raw, const MxBlock &b, float (&v)[8], uint2 &hi, uint2 &lo)
{
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 8; i++) {
        v[i] = __uint_as_float((i & 1) ? w[i >> 1] & 0xFFFF0000u : w[i >> 1] << 16);
        if (b.second == MX_SECOND_E5M2 && !(fabsf(v[i]) < INFINITY)) v[i] = 0.0f;
    }
    const uint32_t sf = b.e < 11u ? 4u : b.e - 7u;
    mx_pair<__NV_E4M3>(v, __uint_as_float((254u - sf) << 23), hi, lo);
    return sf;
}
// The second pair of what mx_first_pair has left, as E4M3 or, with infinities and NaN, as E5M2; the scale byte as above.
__device__ __forceinline__ uint32_t mx_second_pair(const uint4 &raw, float (&v)[8], uint32_t sf, bool e5m2, uint2 &hi, uint2 &lo)
{
    float rmax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) rmax = fmaxf(rmax, fabsf(v[i]));
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) rmax = fmaxf(rmax, __shfl_xor_sync(0xFFFFFFFFu, rmax, o));
    // the largest goes to [128, 256), in E5M2 to [2^14, 2^15); scale bytes stay at 4 and more, factors finite
    const int up = rmax == 0.0f ? 0 : min(min((e5m2 ? 14 : 7) - ((int)(__float_as_uint(rmax) >> 23) - 127), 120), (int)sf - 4);
    const float mul = __uint_as_float((uint32_t)(127 + up) << 23);
    if (e5m2) {
        mx_pair<__NV_E5M2>(v, mul, hi, lo);
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
        uint32_t h[2] = {hi.x, hi.y};
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t bits = (i & 1) ? w[i >> 1] & 0xFFFF0000u : w[i >> 1] << 16, mag = bits & 0x7FFF0000u;
            if (mag >= 0x7F800000u) h[i >> 2] |= (bits >> 24 & 0x80u | (mag == 0x7F800000u ? 0x7Cu : 0x7Fu)) << (8 * (i & 3)); // the byte is zero
        }
        hi = make_uint2(h[0], h[1]);
    } else mx_pair<__NV_E4M3>(v, mul, hi, lo);
    return sf - (uint32_t)up;
}

// A number that no other call of this process has had, in no order that a stale value would have by chance, 56 bits.
inline unsigned long long mx_call_mark()
{
    static std::atomic<unsigned long long> calls{0};
    return ((calls.fetch_add(1, std::memory_order_relaxed) + 1) * 0x9E3779B97F4A7C15ull) >> 8;
}

// ---- waits and arrivals of roles that run as whole warps ------------------------------------------------------------------------
__device__ __forceinline__ void mx_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait of a whole warp; the outcome is the same in all lanes (and known to be, so that the loops around it stay uniform).
__device__ __forceinline__ bool mx_wait(uint32_t bar, uint32_t parity, int *flag, int code)
{
    if (__all_sync(0xFFFFFFFFu, mbar_test(bar, parity))) return true;
    return __all_sync(0xFFFFFFFFu, mbar_wait(bar, parity, flag, code));
}
// The same for two or three barriers: the polls are under way together (one takes about a hundred clocks from the address to the
// branch, whether or not the phase has long been complete).
__device__ __forceinline__ bool mx_wait2(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, int *flag, int code)
{
    const bool t0 = mbar_test(b0, p0), t1 = mbar_test(b1, p1);
    if (__all_sync(0xFFFFFFFFu, t0 && t1)) return true;
    bool ok = mbar_wait(b0, p0, flag, code);
    ok = ok && mbar_wait(b1, p1, flag, code);
    return __all_sync(0xFFFFFFFFu, ok);
}
__device__ __forceinline__ bool mx_wait3(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, uint32_t b2, uint32_t p2, int *flag, int code)
{
    const bool t0 = mbar_test(b0, p0), t1 = mbar_test(b1, p1), t2 = mbar_test(b2, p2);
    if (__all_sync(0xFFFFFFFFu, t0 && t1 && t2)) return true;
    bool ok = mbar_wait(b0, p0, flag, code);
    ok = ok && mbar_wait(b1, p1, flag, code);
    ok = ok && mbar_wait(b2, p2, flag, code);
    return __all_sync(0xFFFFFFFFu, ok);
}

} // namespace oxq
