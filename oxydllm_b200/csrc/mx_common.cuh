// Block-scaled 8-bit tensor-core MMA (tcgen05 kind::mxf8f6f4) with exact bf16 activations: PTX wrappers, and how a bf16 value
// becomes two E4M3 numbers.
//
// kind::mxf8f6f4 multiplies elements of at most 8 bits at twice the rate of bf16 and takes one power-of-two scale (E8M0) per
// row and 32 elements of k for each operand; it accumulates in f32. A bf16 value has 8 significant bits, an E4M3 number 4, so a
// block of 32 activations is written as hi + lo / 16, both scaled so that the block's largest magnitude lies in [128, 256): hi is
// the nearest E4M3 number and the remainder of at most 4 significant bits is lo exactly. Two MMAs (or one with both as columns)
// then cost what one bf16 MMA costs, and the weights can stay in the few bits that they have. Elements below 2^-13 of their block's
// largest come out E4M3-subnormal: the error of the sum of both is at most 2^-21 of that largest. An infinite or NaN activation
// gives NaN.
#pragma once

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

constexpr int MX_E4M3 = 0, MX_E2M1 = 5;
// Instruction descriptor: A and B element types, E8M0 scales; bits 29 and 4 up choose the byte of A's and B's scale words.
__host__ __device__ constexpr uint32_t mx_idesc(int a_type, int n)
{
    return ((uint32_t)a_type << 7) | ((uint32_t)MX_E4M3 << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) |
           ((128u >> 4) << 24);
}
__host__ __device__ constexpr uint32_t mx_idesc_blocks(int a_block, int b_block) { return ((uint32_t)a_block << 29) | ((uint32_t)b_block << 4); }

// Eight neighbouring values of a block whose largest magnitude has the bits `amax`: hi and lo as E4M3 bytes, and the block's
// scale byte (lo's is four less).
__device__ __forceinline__ uint32_t mx_split8(const float (&v)[8], uint32_t amax, uint2 &hi, uint2 &lo)
{
    const uint32_t e = amax >> 23; // biased exponent
    const uint32_t sf = e < 11u ? 4u : e - 7u;
    const float mul = __uint_as_float((254u - sf) << 23);
    uint16_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float a = v[2 * i] * mul, b = v[2 * i + 1] * mul;
        if (e == 255u) { a += a - a; b += b - b; } // infinite -> NaN (the conversion would saturate)
        h[i] = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
        const __half2_raw back = __nv_cvt_fp8x2_to_halfraw2(h[i], __NV_E4M3);
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&back));
        l[i] = __nv_cvt_float2_to_fp8x2(make_float2((a - f.x) * 16.0f, (b - f.y) * 16.0f), __NV_SATFINITE, __NV_E4M3);
    }
    hi = make_uint2((uint32_t)h[0] | ((uint32_t)h[1] << 16), (uint32_t)h[2] | ((uint32_t)h[3] << 16));
    lo = make_uint2((uint32_t)l[0] | ((uint32_t)l[1] << 16), (uint32_t)l[2] | ((uint32_t)l[3] << 16));
    return sf;
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
