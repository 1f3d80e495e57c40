// GGUF Q6_K decode GEMV (1 <= m <= 32), tuned variant.
//
// Q6_K super-block (210 B / 256 weights): u8 ql[128] (low 4 bits), u8 qh[64] (high 2 bits), i8
// scales[16] (one per 16 weights), f16 d. For half h (0, 1), quad q (0..3) and l (0..31), weight
// 128h + 32q + l has low bits in ql[64h + 32(q&1) + l] (low nibble for q < 2, high nibble else),
// high bits in qh[32h + l] >> 2q, scale scales[8h + 2q + l/16]; w = d * scale * (6-bit - 32).
//
// Same decomposition as the other row-format kernels: warps of a CTA = row tiles x k parts, a
// thread-block cluster adds further k slices, partial sums meet in (distributed) shared memory and
// are added in a fixed order; tokens beyond 8 per CTA go to neighbouring CTAs that stream the same
// weights. One mma.sync.m16n8k16 step covers the 16 consecutive weights that share a scale: lane c
// of the quad that feeds one operand row takes l = 16s + 4c .. 16s + 4c + 3, i.e. one 32-bit word of
// ql per quad parity and one of qh per (h, s), which serve the four quads. The 6-bit values are
// assembled four at a time with shifts and lop3, become f16 by byte permute (0x6400 | v = 1024 + v)
// and the offset 1024 + 32 comes out in f32 with the sums of x over each 16 weights when the step
// is folded with d * scale. Super-blocks are 210 bytes, so every other one starts 2 bytes off a
// word boundary: its words are read as two halfwords. Rows must hold an even number of
// super-blocks (4-byte aligned rows).
#include <cooperative_groups.h>

#include <cstdio>
#include <cstdlib>

#include "oxq_common.cuh"
#include "tc_common.cuh"

namespace oxq {

namespace cg = cooperative_groups;

struct Q6kGemvParams {
    const __nv_bfloat16 *x;
    const uint8_t *blocks; // [n][k/256][210]
    const void *bias;
    void *y;
    int bias_dtype, y_dtype;
    int m, k, n;
    int row_tiles, k_warps; // warps of a CTA = row_tiles x k_warps
    int token_split;        // neighbouring CTAs that share their rows and take 8 tokens each (>= 1)
};

__device__ __forceinline__ void q6k_mma_f16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2])
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// 32-bit word at a 2-byte aligned address (warp-uniform alignment).
__device__ __forceinline__ uint32_t q6k_ld32(const uint8_t *p)
{
    if (reinterpret_cast<uintptr_t>(p) & 2) {
        const unsigned short *h = reinterpret_cast<const unsigned short *>(p);
        return (uint32_t)__ldg(h) | ((uint32_t)__ldg(h + 1) << 16);
    }
    return __ldg(reinterpret_cast<const uint32_t *>(p));
}

// The words of one (half h, sixteen s) combination for one row: ql of even quads, ql of odd quads, qh.
struct Q6kCombo {
    uint32_t ql_even, ql_odd, qh;
};

__device__ __forceinline__ void q6k_load_combo(Q6kCombo &w, const uint8_t *blk, int combo, int c)
{
    const int h = combo >> 1, s = combo & 1;
    const uint8_t *ql = blk + 64 * h + 16 * s + 4 * c;
    w.ql_even = q6k_ld32(ql);
    w.ql_odd = q6k_ld32(ql + 32);
    w.qh = q6k_ld32(blk + 128 + 32 * h + 16 * s + 4 * c);
}

// Exact float of a signed byte without the conversion unit.
__device__ __forceinline__ float q6k_i8_to_f32(uint32_t byte)
{
    return __uint_as_float(0x4B000000u | (byte ^ 0x80u)) - 8388736.0f; // 2^23 + 128
}

__global__ void __launch_bounds__(256, 3) q6k_gemv_kernel(const Q6kGemvParams p)
{
    extern __shared__ __align__(16) unsigned char smem[];
    pdl_launch_dependents();
    cg::cluster_group cluster = cg::this_cluster();
    const int nrt = p.row_tiles, ks = (int)gridDim.y, rank = (int)blockIdx.y; // cluster = the y extent of the grid
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int rt = warp % nrt, kw = warp / nrt;
    const int zt = blockIdx.x % p.token_split, bx = blockIdx.x / p.token_split;
    const int m0 = zt * 8, m_loc = min(8, p.m - m0); // this CTA's tokens [m0, m0 + m_loc)
    const int n0 = (bx * nrt + rt) * 16;
    const int nsb = p.k >> 8;                        // super-blocks per row
    const int sl = nsb / ks, sb_cta = rank * sl;     // this CTA's super-blocks
    const int wsb = sl / p.k_warps, sb_off = kw * wsb; // this warp's part of them
    const int kl = sl << 8, k_cta = sb_cta << 8;
    const int xrow = kl + 16; // halves; 32 bytes of padding: the 8-byte fragment reads of a half warp hit distinct banks
    __half *xs = reinterpret_cast<__half *>(smem);
    float *sx = reinterpret_cast<float *>(smem + (size_t)m_loc * xrow * 2); // [kl/16][8]: sums of x per 16 k and token
    float *red = sx + (size_t)(kl >> 4) * 8;                                // [warp][4][lane]
    float *zeros = red + blockDim.x * 4; // 16 bytes of zeros: what lanes without a token read as x

    const int r0 = min(n0 + g, p.n - 1), r1 = min(n0 + g + 8, p.n - 1); // past-the-end rows re-read the last row
    const uint8_t *q0 = p.blocks + ((size_t)r0 * nsb + sb_cta + sb_off) * 210;
    const uint8_t *q1 = p.blocks + ((size_t)r1 * nsb + sb_cta + sb_off) * 210;

    Q6kCombo cur0, cur1;
    if (wsb > 0) {
        q6k_load_combo(cur0, q0, 0, c);
        q6k_load_combo(cur1, q1, 0, c);
    }

    // Stage the slice of x as f16 with the sums of the staged values over each 16 k: four neighbouring
    // threads hold one. Rows without a token keep zero sums.
    if (tid < 4) zeros[tid] = 0.0f;
    for (int idx = tid; idx < (kl >> 4) * 8; idx += blockDim.x) sx[idx] = 0.0f;
    __syncthreads();
    pdl_wait(); // x may come from the kernel before this one; the first weights are already on their way
    for (int row = 0; row < m_loc; row++) {
        const uint2 *src = reinterpret_cast<const uint2 *>(p.x + (size_t)(m0 + row) * p.k + k_cta);
        uint2 *dst = reinterpret_cast<uint2 *>(xs + (size_t)row * xrow);
        for (int q4 = tid; q4 < (kl >> 2); q4 += blockDim.x) { // kl / 4 is a multiple of 64: whole warps
            const uint2 raw = ld_produced(src + q4);
            uint2 o;
            o.x = f32x2_to_f16x2_sat(bf16_lo_f32(raw.x), bf16_hi_f32(raw.x));
            o.y = f32x2_to_f16x2_sat(bf16_lo_f32(raw.y), bf16_hi_f32(raw.y));
            dst[q4] = o;
            const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&o.x));
            const float2 b = __half22float2(*reinterpret_cast<const __half2 *>(&o.y)); // sum what the tensor cores will see
            float sum = (a.x + a.y) + (b.x + b.y);
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
            if ((lane & 3) == 0) sx[(q4 >> 2) * 8 + row] = sum;
        }
    }
    __syncthreads();

    // This lane's x for fragment column g (four halves per step), or the zeros (stride 0).
    const bool real = g < m_loc;
    const __half *xbase = real ? xs + (size_t)g * xrow + (sb_off << 8) + 4 * c : reinterpret_cast<const __half *>(zeros);
    const int xmul = real ? 1 : 0;
    const float *sxb = sx + (size_t)(sb_off << 4) * 8 + 2 * c; // sums of tokens 2c, 2c+1 (the accumulator's columns)

    float tot[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int sb = 0; sb < wsb; sb++) {
        const uint8_t *blk0 = q0 + (size_t)sb * 210, *blk1 = q1 + (size_t)sb * 210;
        uint32_t sc0[4], sc1[4]; // the 16 signed scales of each row's super-block
#pragma unroll
        for (int i = 0; i < 4; i++) {
            sc0[i] = q6k_ld32(blk0 + 192 + 4 * i);
            sc1[i] = q6k_ld32(blk1 + 192 + 4 * i);
        }
        const float d0 = __half2float(__ushort_as_half(__ldg(reinterpret_cast<const unsigned short *>(blk0 + 208))));
        const float d1 = __half2float(__ushort_as_half(__ldg(reinterpret_cast<const unsigned short *>(blk1 + 208))));
#pragma unroll
        for (int combo = 0; combo < 4; combo++) {
            const Q6kCombo w0 = cur0, w1 = cur1;
            if (combo < 3) { // next combination on its way while this one is consumed
                q6k_load_combo(cur0, blk0, combo + 1, c);
                q6k_load_combo(cur1, blk1, combo + 1, c);
            } else if (sb + 1 < wsb) {
                q6k_load_combo(cur0, blk0 + 210, 0, c);
                q6k_load_combo(cur1, blk1 + 210, 0, c);
            }
            const int h = combo >> 1, s = combo & 1;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t l0 = (q & 1) ? w0.ql_odd : w0.ql_even, l1 = (q & 1) ? w1.ql_odd : w1.ql_even;
                const uint32_t v0 = ((q < 2 ? l0 : l0 >> 4) & 0x0F0F0F0Fu) | (((w0.qh >> (2 * q)) & 0x03030303u) << 4);
                const uint32_t v1 = ((q < 2 ? l1 : l1 >> 4) & 0x0F0F0F0Fu) | (((w1.qh >> (2 * q)) & 0x03030303u) << 4);
                // bytes of v = weights k0 + 4c .. k0 + 4c + 3 (0..63 each) -> f16 pairs 1024 + v
                const uint32_t a[4] = {__byte_perm(v0, 0x64646464u, 0x5140), __byte_perm(v1, 0x64646464u, 0x5140),
                                       __byte_perm(v0, 0x64646464u, 0x7362), __byte_perm(v1, 0x64646464u, 0x7362)};
                const int k0 = (sb << 8) + 128 * h + 32 * q + 16 * s; // first k of the step within the warp's range
                const uint2 xv = *reinterpret_cast<const uint2 *>(xbase + xmul * k0);
                const float2 sxv = *reinterpret_cast<const float2 *>(sxb + (size_t)(k0 >> 4) * 8);
                float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                const uint32_t b[2] = {xv.x, xv.y};
                q6k_mma_f16(acc, a, b);
                const int si = 8 * h + 2 * q + s; // scale index
                const float f0 = d0 * q6k_i8_to_f32((sc0[si >> 2] >> (8 * (si & 3))) & 0xFFu);
                const float f1 = d1 * q6k_i8_to_f32((sc1[si >> 2] >> (8 * (si & 3))) & 0xFFu);
                tot[0] = fmaf(f0, fmaf(-1056.0f, sxv.x, acc[0]), tot[0]);
                tot[1] = fmaf(f0, fmaf(-1056.0f, sxv.y, acc[1]), tot[1]);
                tot[2] = fmaf(f1, fmaf(-1056.0f, sxv.x, acc[2]), tot[2]);
                tot[3] = fmaf(f1, fmaf(-1056.0f, sxv.y, acc[3]), tot[3]);
            }
        }
    }

#pragma unroll
    for (int e = 0; e < 4; e++) red[(warp * 4 + e) * 32 + lane] = tot[e];
    if (ks > 1) cluster.sync(); else __syncthreads();

    // Every (row tile, accumulator slot, lane) is summed by one thread of the cluster, in ascending k.
    const int slots = nrt * 4 * 32;
    for (int o = rank * blockDim.x + tid; o < slots; o += ks * blockDim.x) {
        const int ln = o & 31, e = (o >> 5) & 3, wt = o >> 7;
        const int nn = (bx * nrt + wt) * 16 + (ln >> 2) + 8 * (e >> 1), row = 2 * (ln & 3) + (e & 1);
        if (nn < p.n && row < m_loc) {
            float sum = 0.0f;
            for (int q = 0; q < ks; q++) {
                const float *src = ks > 1 ? cluster.map_shared_rank(red, q) : red;
                for (int w = 0; w < p.k_warps; w++) sum += src[((w * nrt + wt) * 4 + e) * 32 + ln];
            }
            if (p.bias) sum += load_as_f32(p.bias, p.bias_dtype, nn);
            store_as(p.y, p.y_dtype, (size_t)(m0 + row) * p.n + nn, sum);
        }
    }
    if (ks > 1) cluster.sync(); // nobody leaves while a peer may still read its shared memory
}

// ---------------------------------------------------------------------------------------------------------------
// Wide layers (the vocabulary projection), m <= 8: one CTA per SM walks 16-row tiles, x staged once for all of them.
//
// A CTA holds two engines that take its tiles in turn: a producer warp that copies stages of 16 rows x 8 super-blocks
// (16 bulk copies of 1680 bytes) into the engine's ring, and eight warps that take one super-block of the stage each, so the k
// split is the warp and a row's alignment (every other super-block starts 2 bytes off a word) is a constant of the warp. The rows'
// pitch of 420 words puts the 8 rows x 4 words of a fragment read on distinct banks. 6-bit values become f16 1024 + v, minus 1056
// exactly, so no sums of x are needed; a step's accumulators are multiplied by d * scale in f32.
//
// What bounds it: instruction issue (the kernel above spends 9.1 per weight: it stages x in every CTA, loads every word of a misaligned
// super-block as halfwords from global memory and folds sums of x; 5.2 here while every lane converted all scales of its rows and
// read x 8 bytes at a time). 128256 x 4096 at 3 / 8 tokens 105.9 / 113.0 us then, 90.9 / 95.2 now.
constexpr int Q6W_ROWS = 16, Q6W_SB = 8, Q6W_ENGINES = 2, Q6W_WARPS = 8;
constexpr int Q6W_ROW_BYTES = Q6W_SB * 210, Q6W_STAGE_BYTES = Q6W_ROWS * Q6W_ROW_BYTES;
constexpr int Q6W_THREADS = Q6W_ENGINES * (Q6W_WARPS + 1) * 32, Q6W_MAX_RING = 4;
constexpr int Q6W_RED = Q6W_WARPS * 4 * 32; // floats of one tile's partial sums
static_assert(Q6W_ROW_BYTES % 16 == 0, "bulk copies");

__device__ int g_q6k_gemv_flag; // a bounded wait ran out

struct Q6kWideParams {
    const __nv_bfloat16 *x;
    const uint8_t *blocks;
    const void *bias;
    void *y;
    int bias_dtype, y_dtype;
    int m, k, n, tiles, ring;
    int test_skip_loads; // self-test: no stage is ever loaded
};

__device__ __forceinline__ uint32_t q6w_lds32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
// 32-bit word at addr, which is 2 bytes off a word where ODD.
template <bool ODD> __device__ __forceinline__ uint32_t q6w_word(uint32_t addr)
{
    if (!ODD) return q6w_lds32(addr);
    return __byte_perm(q6w_lds32(addr - 2), q6w_lds32(addr + 2), 0x5432);
}
__device__ __forceinline__ uint32_t q6w_sub(uint32_t v) // f16 pairs 1024 + v -> v - 32, exact
{
    const uint32_t off = 0x64206420u; // 1056
    const __half2 d = __hsub2(*reinterpret_cast<const __half2 *>(&v), *reinterpret_cast<const __half2 *>(&off));
    return *reinterpret_cast<const uint32_t *>(&d);
}

// One super-block of 16 rows at blk (this lane: rows g and g + 8, words 4c of every piece) times x, in halves of 128 weights: the 8
// scales a row has there are multiplied by d once, by the lane that loads them, and handed to the row's other lanes through `scr`
// (this warp's 16 x 8 floats; a row's two sets of four change places in every other group of four rows, so that the 8 rows of a
// 16-byte read take distinct banks). Every lane used to work out all 32 for itself, 6 of about 40 instructions per 16 weights of k.
template <bool ODD>
__device__ __forceinline__ void q6w_superblock(float (&tot)[4], uint32_t blk, float *scr, int lane, const __half *xp, int xmul)
{
    const int g = lane >> 2, c = lane & 3;
    const uint32_t blk0 = blk + (uint32_t)(g * Q6W_ROW_BYTES), blk1 = blk0 + 8 * Q6W_ROW_BYTES;
    const uint32_t mine = blk + (uint32_t)((lane >> 1) * Q6W_ROW_BYTES); // the row whose scales this lane converts
    uint16_t dr;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(dr) : "r"(mine + 208));
    const float d = __half2float(__ushort_as_half(dr));
    float *put = scr + (lane >> 1) * 8 + 2 * (lane & 1);
    const int put_s = 4 * ((lane >> 3) & 1), get_s = 4 * ((g >> 2) & 1);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t sc = q6w_word<ODD>(mine + 192 + 8 * h + 4 * (lane & 1)) ^ 0x80808080u; // signed byte + 128
        float f[4]; // sixteens 2 (lane & 1) + {0, 0, 1, 1} of the pairs, s = 0, 1, 0, 1
#pragma unroll
        for (int i = 0; i < 4; i++) f[i] = d * (__uint_as_float(__byte_perm(sc, 0x4B000000u, 0x7440 + i)) - 8388736.0f); // 2^23 + 128
        __syncwarp(); // the half before, or the tile's partial sums, have been read
        *reinterpret_cast<float2 *>(put + put_s) = make_float2(f[0], f[2]);
        *reinterpret_cast<float2 *>(put + (put_s ^ 4)) = make_float2(f[1], f[3]);
        __syncwarp();
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const uint32_t at = 64 * h + 16 * s + 4 * c, hat = 128 + 32 * h + 16 * s + 4 * c;
            const uint32_t le0 = q6w_word<ODD>(blk0 + at), lo0 = q6w_word<ODD>(blk0 + at + 32), qh0 = q6w_word<ODD>(blk0 + hat);
            const uint32_t le1 = q6w_word<ODD>(blk1 + at), lo1 = q6w_word<ODD>(blk1 + at + 32), qh1 = q6w_word<ODD>(blk1 + hat);
            const float4 s0 = *reinterpret_cast<const float4 *>(scr + g * 8 + (get_s ^ (4 * s)));
            const float4 s1 = *reinterpret_cast<const float4 *>(scr + (g + 8) * 8 + (get_s ^ (4 * s)));
            const float f0[4] = {s0.x, s0.y, s0.z, s0.w}, f1[4] = {s1.x, s1.y, s1.z, s1.w};
            uint4 xv;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t l0 = (q & 1) ? lo0 : le0, l1 = (q & 1) ? lo1 : le1;
                const uint32_t b0 = (q == 0 ? qh0 << 4 : q == 1 ? qh0 << 2 : q == 2 ? qh0 : qh0 >> 2) & 0x30303030u;
                const uint32_t b1 = (q == 0 ? qh1 << 4 : q == 1 ? qh1 << 2 : q == 2 ? qh1 : qh1 >> 2) & 0x30303030u;
                const uint32_t v0 = ((q < 2 ? l0 : l0 >> 4) & 0x0F0F0F0Fu) | b0, v1 = ((q < 2 ? l1 : l1 >> 4) & 0x0F0F0F0Fu) | b1;
                const uint32_t a[4] = {q6w_sub(__byte_perm(v0, 0x64646464u, 0x5140)), q6w_sub(__byte_perm(v1, 0x64646464u, 0x5140)),
                                       q6w_sub(__byte_perm(v0, 0x64646464u, 0x7362)), q6w_sub(__byte_perm(v1, 0x64646464u, 0x7362))};
                if ((q & 1) == 0) xv = *reinterpret_cast<const uint4 *>(xp + xmul * (128 * h + 64 * s + 16 * q));
                const uint32_t b[2] = {(q & 1) ? xv.z : xv.x, (q & 1) ? xv.w : xv.y};
                float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                q6k_mma_f16(acc, a, b);
                tot[0] = fmaf(f0[q], acc[0], tot[0]);
                tot[1] = fmaf(f0[q], acc[1], tot[1]);
                tot[2] = fmaf(f1[q], acc[2], tot[2]);
                tot[3] = fmaf(f1[q], acc[3], tot[3]);
            }
        }
    }
}

__global__ void __launch_bounds__(Q6W_THREADS, 1) q6k_gemv_wide_kernel(const Q6kWideParams p)
{
    extern __shared__ __align__(16) unsigned char smem[];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int engine = warp / (Q6W_WARPS + 1), ew = warp % (Q6W_WARPS + 1); // ew == Q6W_WARPS: the engine's producer
    const int chunks = p.k / (Q6W_SB * 256), xrow = p.k + 32;
    const size_t row_bytes = (size_t)chunks * Q6W_ROW_BYTES;
    // rings of both engines | partial sums (two tiles per engine) | barriers | zeros | x
    const uint32_t base = smem_u32(smem);
    const uint32_t ring = base + (uint32_t)(engine * p.ring * Q6W_STAGE_BYTES);
    unsigned char *rest = smem + (size_t)Q6W_ENGINES * p.ring * Q6W_STAGE_BYTES;
    float *red = reinterpret_cast<float *>(rest) + engine * 2 * Q6W_RED;
    rest += Q6W_ENGINES * 2 * Q6W_RED * sizeof(float);
    const uint32_t bars = smem_u32(rest) + (uint32_t)(engine * 2 * Q6W_MAX_RING * 8);
    auto full = [&](int r) { return bars + 8u * r; };
    auto empty = [&](int r) { return bars + 8u * (Q6W_MAX_RING + r); };
    rest += Q6W_ENGINES * 2 * Q6W_MAX_RING * 8;
    float *zeros = reinterpret_cast<float *>(rest); // 16 bytes: what lanes without a token read as x
    __half *xs = reinterpret_cast<__half *>(rest + 16);

    if (ew == Q6W_WARPS && lane < Q6W_MAX_RING) {
        mbar_init(full(lane), 1);
        mbar_init(empty(lane), Q6W_WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 4) zeros[threadIdx.x] = 0.0f;
    __syncthreads();

    const int first = (int)blockIdx.x + engine * (int)gridDim.x, step = Q6W_ENGINES * (int)gridDim.x; // this engine's tiles
    if (ew == Q6W_WARPS) {
        // ---- producer: weights are read before the previous kernel has finished; lane r copies row r -------------
        int r = 0;
        uint32_t ph = 0;
        long long it = 0;
        bool ok = true;
        for (int t = first; t < p.tiles && ok; t += step) {
            const int row = min(t * Q6W_ROWS + min(lane, Q6W_ROWS - 1), p.n - 1); // past-the-end rows re-read the last row
            const uint8_t *src = p.blocks + (size_t)row * row_bytes;
            for (int ch = 0; ch < chunks && ok; ch++, it++) {
                if (it == p.ring) pdl_wait(); // slots come free only after x: that time must not count as this wait
                if (it >= p.ring) ok = __all_sync(0xFFFFFFFFu, mbar_wait(empty(r), ph ^ 1u, &g_q6k_gemv_flag, 1));
                if (ok && !p.test_skip_loads) {
                    if (lane == 0) mbar_arrive_expect_tx(full(r), Q6W_STAGE_BYTES);
                    __syncwarp();
                    if (lane < Q6W_ROWS)
                        bulk_copy_g2s(ring + (uint32_t)(r * Q6W_STAGE_BYTES + lane * Q6W_ROW_BYTES), src + (size_t)ch * Q6W_ROW_BYTES,
                                      Q6W_ROW_BYTES, full(r));
                }
                if (++r == p.ring) { r = 0; ph ^= 1u; }
            }
        }
        return;
    }

    // ---- x as f16, once for all tiles; the first stages are on their way --------------------------------------------
    pdl_wait(); // x may come from the kernel before this one, y may still be read by it
    {
        const int ct = (engine * Q6W_WARPS + ew) * 32 + lane, per_row = p.k / 4;
        for (int idx = ct; idx < p.m * per_row; idx += Q6W_ENGINES * Q6W_WARPS * 32) {
            const int row = idx / per_row, q4 = idx - row * per_row;
            const uint2 raw = ld_produced(reinterpret_cast<const uint2 *>(p.x + (size_t)row * p.k) + q4);
            uint2 o;
            o.x = f32x2_to_f16x2_sat(bf16_lo_f32(raw.x), bf16_hi_f32(raw.x));
            o.y = f32x2_to_f16x2_sat(bf16_lo_f32(raw.y), bf16_hi_f32(raw.y));
            // [half][sixteen of a pair][two pairs][word c][pair][4]: a lane reads two steps' words as 16 bytes
            const int at = (q4 & ~63) | (q4 & 32) | ((q4 & 4) << 2) | ((q4 & 16) >> 1) | ((q4 & 3) << 1) | ((q4 & 8) >> 3);
            reinterpret_cast<uint2 *>(xs + (size_t)row * xrow)[at] = o;
        }
    }
    asm volatile("bar.sync 3, %0;" ::"n"(Q6W_ENGINES * Q6W_WARPS * 32) : "memory"); // all but the producers

    const int g = lane >> 2, c = lane & 3;
    const bool real = g < p.m;
    const __half *xbase = real ? xs + (size_t)g * xrow + ew * 256 + 8 * c : reinterpret_cast<const __half *>(zeros);
    const int xmul = real ? 1 : 0;
    int r = 0, buf = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int t = first; t < p.tiles; t += step, buf ^= 1) {
        float tot[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        float *mine = red + buf * Q6W_RED, *scr = mine + ew * 128; // the warp's own part, not yet written, holds scales till then
        for (int ch = 0; ch < chunks && ok; ch++) {
            ok = __all_sync(0xFFFFFFFFu, mbar_wait(full(r), ph, &g_q6k_gemv_flag, 2));
            if (!ok) break;
            const uint32_t blk = ring + (uint32_t)(r * Q6W_STAGE_BYTES + ew * 210);
            const __half *xp = xbase + xmul * (ch * Q6W_SB * 256);
            if (ew & 1) q6w_superblock<true>(tot, blk, scr, lane, xp, xmul);
            else q6w_superblock<false>(tot, blk, scr, lane, xp, xmul);
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty(r)) : "memory");
            if (++r == p.ring) { r = 0; ph ^= 1u; }
        }
        // the engine's warps meet once per tile (also after a wait gave up); the other buffer is free again by then
#pragma unroll
        for (int e = 0; e < 4; e++) mine[(ew * 4 + e) * 32 + lane] = tot[e];
        asm volatile("bar.sync %0, %1;" ::"r"(1 + engine), "n"(Q6W_WARPS * 32) : "memory");
        const int o = ew * 32 + lane; // 0 .. 255: accumulator slot and lane, in ascending k over the warps
        if (o < 4 * 32 && ok) {
            const int ln = o & 31, e = o >> 5;
            const int nn = t * Q6W_ROWS + (ln >> 2) + 8 * (e >> 1), row = 2 * (ln & 3) + (e & 1);
            if (nn < p.n && row < p.m) {
                float sum = 0.0f;
#pragma unroll
                for (int w = 0; w < Q6W_WARPS; w++) sum += mine[(w * 4 + e) * 32 + ln];
                if (p.bias) sum += load_as_f32(p.bias, p.bias_dtype, nn);
                store_as(p.y, p.y_dtype, (size_t)row * p.n + nn, sum);
            }
        }
    }
}

static size_t q6w_fixed(int m, int k)
{
    return (size_t)Q6W_ENGINES * 2 * Q6W_RED * 4 + Q6W_ENGINES * 2 * Q6W_MAX_RING * 8 + 16 + (size_t)m * (k + 32) * 2;
}

// Ring depth of an engine, 0 where the kernel does not apply: rows of whole stages (8 super-blocks), at least four tiles per
// SM (below that the last wave costs more than the staging saves), room for two stages per engine beside x.
static int q6w_ring(int m, int k, int n, const void *blocks)
{
    if (m > 8 || k % (Q6W_SB * 256) != 0 || !aligned(blocks, 16) || ceil_div(n, Q6W_ROWS) < 4 * sm_count()) return 0;
    const long long room = 227 * 1024 - (long long)q6w_fixed(m, k);
    const int ring = room > 0 ? (int)(room / (Q6W_ENGINES * Q6W_STAGE_BYTES)) : 0;
    return ring < 2 ? 0 : ring < Q6W_MAX_RING ? ring : Q6W_MAX_RING;
}

static int launch_q6k_wide(const Q6kGemvParams &g, int ring, cudaStream_t st, int test_skip_loads = 0)
{
    Q6kWideParams p = {g.x, g.blocks, g.bias, g.y, g.bias_dtype, g.y_dtype, g.m, g.k, g.n, ceil_div(g.n, Q6W_ROWS), ring, test_skip_loads};
    const size_t smem = (size_t)Q6W_ENGINES * ring * Q6W_STAGE_BYTES + q6w_fixed(g.m, g.k);
    static size_t configured[64] = {};
    int device = 0;
    OXQ_CUDA(cudaGetDevice(&device));
    if (device >= 64 || configured[device] < smem) {
        OXQ_CUDA(cudaFuncSetAttribute(q6k_gemv_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (device < 64) configured[device] = smem;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count(), 1, 1);
    cfg.blockDim = dim3(Q6W_THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    allow_early_start(attr, cfg.numAttrs);
    OXQ_CUDA(cudaLaunchKernelEx(&cfg, q6k_gemv_wide_kernel, p));
    return OXQ_OK;
}

// The code of a bounded wait that ran out since the last call, 0 if none (synchronises the device's copy).
int q6k_gemv_take_flag(int &flag)
{
    OXQ_CUDA(cudaMemcpyFromSymbol(&flag, g_q6k_gemv_flag, sizeof(int)));
    if (flag != 0) {
        const int zero = 0;
        OXQ_CUDA(cudaMemcpyToSymbol(g_q6k_gemv_flag, &zero, sizeof(int)));
    }
    return OXQ_OK;
}

static size_t q6k_smem(int m_cta, int kl, int warps)
{
    return (size_t)m_cta * (kl + 16) * 2 + (size_t)(kl / 16) * 8 * 4 + (size_t)warps * 4 * 32 * 4 + 16;
}

static int launch_q6k(const Q6kGemvParams &p, int ks, cudaStream_t st)
{
    const int nw = p.row_tiles * p.k_warps;
    const size_t smem = q6k_smem(p.m < 8 ? p.m : 8, p.k / ks, nw);
    auto kern = q6k_gemv_kernel;
    static size_t configured[64] = {};
    int device = 0;
    OXQ_CUDA(cudaGetDevice(&device));
    if (device >= 64 || configured[device] < smem) {
        OXQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (device < 64) configured[device] = smem;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ceil_div(p.n, 16 * p.row_tiles) * p.token_split, ks, 1);
    cfg.blockDim = dim3(nw * 32, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = ks;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ks > 1 ? 1 : 0;
    allow_early_start(attr, cfg.numAttrs);
    OXQ_CUDA(cudaLaunchKernelEx(&cfg, kern, p));
    return OXQ_OK;
}

// Picks warps-per-CTA x cluster so that the k split divides the super-blocks of a row evenly.
static bool q6k_pick(int m, int k, int &nrt, int &kw, int &ks)
{
    const int nsb = k / 256;
    static const int few[][3] = {{1, 8, 1}, {2, 4, 1}, {1, 6, 1}, {1, 5, 1}, {2, 3, 1}, {2, 2, 1}, {1, 7, 1}, {2, 1, 1}, {1, 1, 1}};
    static const int many[][3] = {{2, 4, 1}, {4, 2, 1}, {2, 3, 1}, {8, 1, 2}, {8, 1, 1}};
    const int(*cand)[3] = m <= 8 ? few : many;
    const int count = m <= 8 ? 9 : 5;
    for (int t = 0; t < count; t++)
        if (nsb % (cand[t][1] * cand[t][2]) == 0) { nrt = cand[t][0]; kw = cand[t][1]; ks = cand[t][2]; return true; }
    return false;
}

// True when the tuned kernel applies; otherwise the caller uses the generic row-format kernel.
bool q6k_gemv_supported(int m, int k, const void *blocks)
{
    int a, b, c;
    return m <= 32 && k % 512 == 0 && (reinterpret_cast<uintptr_t>(blocks) & 3) == 0 && q6k_pick(m, k, a, b, c) &&
           q6k_smem(m < 8 ? m : 8, k, 8) <= 160 * 1024;
}

int q6k_gemv(const void *x, const void *blocks, const void *bias, int bias_dtype, void *y, int y_dtype, int m, int k, int n,
             cudaStream_t st)
{
    Q6kGemvParams p;
    p.x = (const __nv_bfloat16 *)x; p.blocks = (const uint8_t *)blocks; p.bias = bias; p.y = y;
    p.bias_dtype = bias_dtype; p.y_dtype = y_dtype; p.m = m; p.k = k; p.n = n;
    if (const int ring = q6w_ring(m, k, n, blocks)) return launch_q6k_wide(p, ring, st);
    int nrt = 2, kw = 4, ks = 1;
    q6k_pick(m, k, nrt, kw, ks);
    if (const char *env = tuning_env("OXQ_Q6K_GEMV_TUNE")) { // bench-harness knob: "row_tiles,k_warps,cluster"
        int a = 0, b = 0, cc = 0;
        if (sscanf(env, "%d,%d,%d", &a, &b, &cc) == 3 && a >= 1 && b >= 1 && a * b <= 8 && cc >= 1 && cc <= 8 &&
            (cc & (cc - 1)) == 0 && (k / 256) % (b * cc) == 0) {
            nrt = a; kw = b; ks = cc;
        }
    }
    p.row_tiles = nrt; p.k_warps = kw;
    p.token_split = ceil_div(m, 8); // 8 tokens per CTA; more on neighbouring CTAs
    return launch_q6k(p, ks, st);
}

} // namespace oxq

// Self-test of the wide kernel's abort path: one tile (16 rows x 2048) whose stage never comes. The eight warps that wait for it give up
// after two seconds, side by side, the flag takes their code and the kernel returns; oxq_awq_gemv_check reports it.
OXQ_EXPORT int oxq_selftest_q6k_wait_expiry(void *scratch, size_t scratch_bytes, void *stream)
{
    oxq::clear_error();
    OXQ_REQUIRE(scratch && scratch_bytes >= (1u << 18) && oxq::aligned(scratch, 256), OXQ_ERR_WORKSPACE,
                "oxq_selftest_q6k_wait_expiry: 256-byte aligned scratch of at least 256 KiB needed");
    unsigned char *b = reinterpret_cast<unsigned char *>(scratch);
    oxq::Q6kGemvParams p = {};
    p.x = reinterpret_cast<__nv_bfloat16 *>(b); p.blocks = b + (1 << 16); p.y = b + (3 << 16);
    p.y_dtype = OXQ_F32; p.m = 1; p.k = oxq::Q6W_SB * 256; p.n = oxq::Q6W_ROWS;
    return oxq::launch_q6k_wide(p, 2, (cudaStream_t)stream, 1);
}
