// GGUF matmul (Q4_0, Q8_0, Q4_K, Q6_K) from one token to a few hundred: blocks streamed from HBM through shared memory into mma.sync.
//
// One CTA per SM walks its share of all (tile, unit) pairs: a tile is 128 out features x at most 64 tokens, a unit 256 input features. A
// producer warp keeps up to eight boxes (128 rows x 256 weights as stored, and the tokens' 256 activations) on their way with two TMA copies each.
// 4 KQ warps multiply: 32 rows x 256 / KQ weights of a box each, codes turned into exact bf16 integers by byte permutes (128 + code,
// less the offset) in the order in which they lie, so that lane c of a row takes activations 4 c .. 4 c + 3 of every 16 with one load. A scale block's
// sum (32 weights, 16 for Q6_K) is multiplied by its scale in f32. For the K types two more warps turn the packed scales of a box into
// f32 ahead of the multiplication (by the multiplying warps that would be 160 instructions a warp and box), for Q4_K also the sums of x that the
// minima multiply. Parts of a tile meet as in stream_common.cuh. Nothing is rounded between the codes and the f32 sums, x is bf16 as given.
//
// What bounds it: up to 16 tokens instruction issue and the start and end of a launch (about 6 us: pipeline filling from a cold memory system, and putting
// shared tiles together); ncu on 4096 x 64000, Q4_0, one token: 374 warp instructions per 32 rows x 128 weights, issue slots 55 % with two
// warps a scheduler; four (KQ = 4) were no faster. From 32 tokens the tensor cores: mma.sync takes 8.8 clocks a scheduler, 930 multiply-adds a clock
// and SM. Loads do not bound it (boxes of whole 128-byte lines, and no copies of x at all, took the same time). Figures at the rules below.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "formats.cuh"
#include "stream_common.cuh"

namespace oxq {

constexpr int SR_ROWS = 128, SR_BOX = 256; // out features of a tile; weights of a row of a box
constexpr int SR_PLANE = SR_ROWS + 4;      // floats from one token's row of a tile to the next in shared memory
constexpr int SR_X_PITCH = 544;            // bytes from one token's 256 activations to the next: eight 32-byte reads fall into distinct banks
constexpr int SR_MAX_STAGES = 8;
constexpr int SR_MAX_BLOCK = 64;           // tokens of a tile

// BYTES: of 256 weights; PITCH: of a row of a box in shared memory (16-byte pieces, rows in distinct banks); SUB: weights that share a
// scale; TABLE: bytes of the scales of a row in f32 where they are unpacked ahead of the multiplication, else 0.
template <int TYPE> struct SrFormat;
template <> struct SrFormat<OXQ_GGML_Q4_0> { static constexpr int BYTES = 144, PITCH = 144, SUB = 32, TABLE = 0; };
template <> struct SrFormat<OXQ_GGML_Q8_0> { static constexpr int BYTES = 272, PITCH = 272, SUB = 32, TABLE = 0; };
template <> struct SrFormat<OXQ_GGML_Q4_K> { static constexpr int BYTES = 144, PITCH = 144, SUB = 32, TABLE = 64; };
template <> struct SrFormat<OXQ_GGML_Q6_K> { static constexpr int BYTES = 210, PITCH = 240, SUB = 16, TABLE = 64; };

struct StreamRowsParams {
    const __nv_bfloat16 *x;
    const uint8_t *blocks;
    int k, stages;
    int *flag;
    StreamOut out;
};

// Q4_K weights are multiplied in two parts, d sc q and dmin mn, which an infinite activation turns into infinity less infinity. Where a sum
// is not finite it is computed again from whole weights.
__device__ __noinline__ float sr_whole_q4k(const uint8_t *row, const __nv_bfloat16 *x, int k)
{
    float sum = 0.0f;
    for (int i = 0; i < k; i++) sum = fmaf(gguf_decode_elem<OXQ_GGML_Q4_K>(row + (size_t)(i >> 8) * 144, i & 255), __bfloat162float(x[i]), sum);
    return sum;
}
template <int TYPE> struct SrMend {
    const __nv_bfloat16 *x;
    const uint8_t *blocks;
    int k;
    __device__ __forceinline__ float operator()(float v, int tok, int row) const
    {
        if (TYPE != OXQ_GGML_Q4_K || fabsf(v) < INFINITY) return v;
        return sr_whole_q4k(blocks + (size_t)row * (k / 256) * 144, x + (size_t)tok * k, k);
    }
};

// Byte i (and i + 1) of v as the bf16 pair 128 + byte, bytes below 128.
__device__ __forceinline__ uint32_t sr_pair01(uint32_t v, uint32_t magic) { return __byte_perm(v, magic, 0x4140); }
__device__ __forceinline__ uint32_t sr_pair23(uint32_t v, uint32_t magic) { return __byte_perm(v, magic, 0x4342); }
// Four bytes from an address that is a multiple of four, or (ODD) of two only.
template <bool ODD> __device__ __forceinline__ uint32_t sr_word(const unsigned char *p)
{
    if constexpr (!ODD) return st_lds<uint32_t>(p);
    return __byte_perm(st_lds<uint32_t>(p - 2), st_lds<uint32_t>(p + 2), 0x5432);
}
__device__ __forceinline__ float sr_f16(const unsigned char *p) { return half_bits_to_f32(st_lds<uint16_t>(p)); }

// MT: eights of tokens of a tile; KQ: parts of a box that warps take (with four groups of 32 rows, 4 KQ warps multiply).
template <int TYPE, int MT, int KQ>
__global__ void __launch_bounds__(KQ * 128 + 128, 1)
    gguf_stream_kernel(const StreamRowsParams p, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap)
{
    using Fm = SrFormat<TYPE>;
    constexpr int W_BYTES = SR_ROWS * Fm::PITCH, X_BYTES = MT * 8 * SR_X_PITCH, TABLE_BYTES = SR_ROWS * Fm::TABLE;
    constexpr bool SUMS = TYPE == OXQ_GGML_Q4_K; // of x, which minima and the 128 of the operands multiply
    constexpr int SUM_BYTES = SUMS ? 8 * 8 * MT * 4 : 0, SLOT = W_BYTES + X_BYTES + TABLE_BYTES + SUM_BYTES;
    constexpr int SR_CONSUMERS = KQ * 128, PART = SR_BOX / KQ; // threads; weights of a row that a warp takes of a box
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long bars[3 * SR_MAX_STAGES];
    __shared__ uint32_t last, helped;
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = p.stages;
    // shared memory: slots (rows of blocks, x, unpacked scales, sums of x) | partial tiles [part]
    unsigned char *slots = smem_raw + (((smem_u32(smem_raw) + 127u) & ~127u) - smem_u32(smem_raw));
    const uint32_t base = smem_u32(slots);
    float *red = reinterpret_cast<float *>(slots + S * SLOT);
    const uint32_t full = smem_u32(bars), ready = full + 8 * SR_MAX_STAGES, empty = ready + 8 * SR_MAX_STAGES;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(full + 8 * s, 1);
            mbar_init(ready + 8 * s, 2);
            mbar_init(empty + 8 * s, KQ * 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&wmap) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
    }
    __syncthreads();
    pdl_wait();

    const int G = p.out.units_per_tile;
    const int u0 = st_share(p.out, gridDim.x, blockIdx.x), u1 = st_share(p.out, gridDim.x, blockIdx.x + 1);
    int s = 0;
    uint32_t ph = 0;
    constexpr int PRODUCER = KQ * 4, SCALER = PRODUCER + 1, HELPER = PRODUCER + 3; // warps
    const bool help = st_needs_help(p.out, u0, u1);
    if (warp == HELPER) {
        if (help) st_help<SR_CONSUMERS>(p.out, u0 / G, &helped);
        return;
    }
    if (warp == PRODUCER) {
        // ---- producer ----------------------------------------------------------------------------------------------
        for (int u = u0; u < u1; u++) {
            if (!mx_wait(empty + 8 * s, ph ^ 1u, p.flag, ST_CODE + 1)) return;
            const int tile = u / G, chunk = u - tile * G;
            const int row0 = tile / p.out.tok_blocks * SR_ROWS, tok0 = tile % p.out.tok_blocks * p.out.tok_step;
            const uint32_t slot = base + (uint32_t)(s * SLOT), bar = full + 8 * s;
            if (elect_one()) {
                mbar_arrive_expect_tx(bar, W_BYTES + X_BYTES);
                tma_load_2d(slot, &wmap, bar, (chunk * Fm::BYTES & ~15) / 4, row0);
                tma_load_2d(slot + W_BYTES, &xmap, bar, chunk * (SR_BOX / 2), tok0);
            }
            __syncwarp();
            if (++s == S) { s = 0; ph ^= 1u; }
        }
        return;
    }
    if (warp >= SCALER) {
        // ---- scales in f32, and sums of x: two warps, half of the rows and of the sums each --------------------------
        if constexpr (Fm::TABLE != 0) {
            const int h = warp - SCALER;
            for (int u = u0; u < u1; u++) {
                if (!mx_wait(full + 8 * s, ph, p.flag, ST_CODE + 3)) return;
                unsigned char *slot = slots + s * SLOT, *table = slot + W_BYTES + X_BYTES;
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int row = h * 64 + i * 32 + lane;
                    if constexpr (TYPE == OXQ_GGML_Q4_K) {
                        const uint4 v = st_lds<uint4>(slot + row * Fm::PITCH); // d, dmin | 6-bit scales and minima
                        const float2 dm = st_f16x2(v.x);
                        const uint32_t sc[2] = {v.y & 0x3F3F3F3Fu, (v.w & 0x0F0F0F0Fu) | (v.y >> 2 & 0x30303030u)};
                        const uint32_t mn[2] = {v.z & 0x3F3F3F3Fu, (v.w >> 4 & 0x0F0F0F0Fu) | (v.z >> 2 & 0x30303030u)};
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            // an integer below 2^23 in the low bits of 2^23
                            const float q = __uint_as_float(0x4B000000u | (sc[j >> 2] >> (8 * (j & 3)) & 0x3Fu)) - 8388608.0f;
                            const float m = __uint_as_float(0x4B000000u | (mn[j >> 2] >> (8 * (j & 3)) & 0x3Fu)) - 8388608.0f;
                            const float ds = dm.x * q, u128 = fmaf(128.0f, ds, dm.y * m);
                            reinterpret_cast<float2 *>(table)[j * SR_ROWS + row] = make_float2(ds, u128);
                        }
                    } else {
                        // the blocks of a box begin 0 to 14 bytes behind its first
                        const unsigned char *blk = slot + row * Fm::PITCH + ((u % G * Fm::BYTES) & 15);
                        const bool odd = (u % G * Fm::BYTES) & 2;
                        const unsigned char *at = blk + 192 - (odd ? 2 : 0);
                        const float d = sr_f16(blk + 208);
                        uint32_t w[4], lo = st_lds<uint32_t>(at);
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const uint32_t hi = st_lds<uint32_t>(at + 4 * q + 4);
                            w[q] = odd ? __byte_perm(lo, hi, 0x5432) : lo;
                            lo = hi;
                        }
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            const float q = __uint_as_float(0x4B000000u | ((w[j >> 2] >> (8 * (j & 3)) & 0xFFu) ^ 0x80u)) - 8388736.0f;
                            reinterpret_cast<float *>(table)[j * SR_ROWS + row] = d * q;
                        }
                    }
                }
                if constexpr (SUMS) {
                    const unsigned char *xs = slot + W_BYTES + (lane >> 2) * SR_X_PITCH + (lane & 3) * 8;
                    float *sums = reinterpret_cast<float *>(table + TABLE_BYTES);
#pragma unroll
                    for (int i = h * 4; i < h * 4 + 4; i++)
#pragma unroll
                        for (int mt = 0; mt < MT; mt++) {
                            const uint2 b0 = st_lds<uint2>(xs + mt * 8 * SR_X_PITCH + i * 64), b1 = st_lds<uint2>(xs + mt * 8 * SR_X_PITCH + i * 64 + 32);
                            float a[4];
                            st_mma_first(a, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u, b0.x, b0.y);
                            st_mma(a, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u, b1.x, b1.y);
                            if (lane < 4) *reinterpret_cast<float2 *>(sums + i * 8 * MT + mt * 8 + 2 * lane) = make_float2(a[0], a[1]);
                        }
                }
                __syncwarp();
                if (lane == 0) mx_arrive(ready + 8 * s);
                if (++s == S) { s = 0; ph ^= 1u; }
            }
        }
        return;
    }

    // ---- unpack and multiply: 32 rows, one part of every box ---------------------------------------------------------
    const int rg = warp & 3, kq = warp >> 2, g = lane >> 2, c = lane & 3;
    // Q6_K blocks interleave the 32-weight quarters of a half: with four parts a warp takes quarters kq % 2 and kq % 2 + 2 of half kq / 2
    constexpr bool Q6 = TYPE == OXQ_GGML_Q6_K;
    const int x_part = Q6 ? (KQ == 4 ? kq >> 1 : kq) * 128 : kq * PART;
    uint32_t magic; // kept opaque so that it stays in a register
    asm volatile("mov.b32 %0, 0x43434343;" : "=r"(magic));
    const int row_off = (rg * 32 + g) * Fm::PITCH + 4 * c, x_off = W_BYTES + g * SR_X_PITCH + x_part * 2 + 8 * c;
    const SrMend<TYPE> mend{p.x, p.blocks, p.k};
    float tot[2][MT][4];
    bool ok = true;
    bool others = false;
    for (int u = u0; u < u1;) {
        const int tile = u / G, seg_end = min(u1, (tile + 1) * G), first_unit = u;
#pragma unroll
        for (int t = 0; t < 2; t++)
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int i = 0; i < 4; i++) tot[t][mt][i] = 0.0f;
#pragma unroll 1
        for (; u < seg_end; u++) {
            if (u + 1 == seg_end && seg_end == u1 && warp == 0) others = st_others(p.out, tile, st_owner(p.out, gridDim.x, tile * G), st_owner(p.out, gridDim.x, (tile + 1) * G - 1));
            if (Fm::TABLE) ok = ok && mx_wait2(full + 8 * s, ph, ready + 8 * s, ph, p.flag, ST_CODE + 2);
            else ok = ok && mx_wait(full + 8 * s, ph, p.flag, ST_CODE + 2);
            if (!ok) continue;
            const unsigned char *slot = slots + s * SLOT, *xs = slot + x_off;
            const unsigned char *w0 = slot + row_off; // row g of this warp's 32; rows 8, 16 and 24 further follow at 8 PITCH each
            const unsigned char *table = slot + W_BYTES + X_BYTES + (rg * 32 + g) * (Fm::TABLE / (SR_BOX / Fm::SUB));
            float acc[2][MT][4];
            // 16 weights of rows g and g + 8 of the two row tiles (pairs a[t][h][0], a[t][h][1]) times x at `at` weights into the half
            auto multiply = [&](const uint32_t (&a)[2][2][2], int at, bool begin) {
#pragma unroll
                for (int mt = 0; mt < MT; mt++) {
                    const uint2 b = st_lds<uint2>(xs + mt * 8 * SR_X_PITCH + at * 2);
#pragma unroll
                    for (int t = 0; t < 2; t++) {
                        if (begin) st_mma_first(acc[t][mt], a[t][0][0], a[t][1][0], a[t][0][1], a[t][1][1], b.x, b.y);
                        else st_mma(acc[t][mt], a[t][0][0], a[t][1][0], a[t][0][1], a[t][1][1], b.x, b.y);
                    }
                }
            };
            auto fold = [&](const float (&ds)[2][2]) {
#pragma unroll
                for (int t = 0; t < 2; t++)
#pragma unroll
                    for (int mt = 0; mt < MT; mt++)
#pragma unroll
                        for (int i = 0; i < 4; i++) tot[t][mt][i] = fmaf(ds[t][i >> 1], acc[t][mt][i], tot[t][mt][i]);
            };
            if constexpr (TYPE == OXQ_GGML_Q4_K) {
#pragma unroll
                for (int j = 0; j < PART / 32; j++) { // sub-blocks of 32: low nibbles of 32 bytes, then their high nibbles
#pragma unroll
                    for (int hb = 0; hb < 2; hb++) {
                        uint32_t a[2][2][2];
#pragma unroll
                        for (int r = 0; r < 4; r++) {
                            const uint32_t w = st_lds<uint32_t>(w0 + r * 8 * Fm::PITCH + 16 + kq * (PART / 2) + (j >> 1) * 32 + hb * 16);
                            const uint32_t v = ((j & 1) ? w >> 4 : w) & 0x0F0F0F0Fu;
                            a[r >> 1][r & 1][0] = sr_pair01(v, magic);
                            a[r >> 1][r & 1][1] = sr_pair23(v, magic);
                        }
                        multiply(a, j * 32 + hb * 16, hb == 0);
                    }
                    float ds[2][2], um[2][2];
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const float2 v = st_lds<float2>(table + ((kq * (PART / 32) + j) * SR_ROWS + r * 8) * 8);
                        ds[r >> 1][r & 1] = v.x;
                        um[r >> 1][r & 1] = v.y;
                    }
                    fold(ds);
                    const unsigned char *sums = slot + W_BYTES + X_BYTES + TABLE_BYTES + ((kq * (PART / 32) + j) * 8 * MT + 2 * c) * 4;
#pragma unroll
                    for (int mt = 0; mt < MT; mt++) {
                        const float2 sv = st_lds<float2>(sums + mt * 32);
#pragma unroll
                        for (int t = 0; t < 2; t++)
#pragma unroll
                            for (int i = 0; i < 4; i++) tot[t][mt][i] = fmaf(-um[t][i >> 1], (i & 1) ? sv.y : sv.x, tot[t][mt][i]);
                    }
                }
            } else if constexpr (TYPE == OXQ_GGML_Q4_0) {
                constexpr uint32_t off = 0x43084308u; // 128 + 8
#pragma unroll
                for (int j = 0; j < PART / 32; j++) { // blocks of 18 bytes
                    uint32_t w[4];
                    float ds[2][2];
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const unsigned char *blk = w0 + r * 8 * Fm::PITCH + kq * (PART / 32) * 18 + j * 18;
                        w[r] = (j & 1) ? sr_word<false>(blk + 2) : sr_word<true>(blk + 2);
                        ds[r >> 1][r & 1] = sr_f16(blk - 4 * c);
                    }
#pragma unroll
                    for (int hb = 0; hb < 2; hb++) { // low nibbles: weights 0 .. 15 of the block
                        uint32_t a[2][2][2];
#pragma unroll
                        for (int r = 0; r < 4; r++) {
                            const uint32_t v = (hb ? w[r] >> 4 : w[r]) & 0x0F0F0F0Fu;
                            a[r >> 1][r & 1][0] = st_sub2(sr_pair01(v, magic), off);
                            a[r >> 1][r & 1][1] = st_sub2(sr_pair23(v, magic), off);
                        }
                        multiply(a, j * 32 + hb * 16, hb == 0);
                    }
                    fold(ds);
                }
            } else if constexpr (TYPE == OXQ_GGML_Q8_0) {
#pragma unroll
                for (int j = 0; j < PART / 32; j++) { // blocks of 34 bytes
                    float ds[2][2];
#pragma unroll
                    for (int hb = 0; hb < 2; hb++) {
                        uint32_t a[2][2][2];
#pragma unroll
                        for (int r = 0; r < 4; r++) {
                            const unsigned char *blk = w0 + r * 8 * Fm::PITCH + kq * (PART / 32) * 34 + j * 34;
                            const uint32_t v = (j & 1) ? sr_word<false>(blk + 2 + hb * 16) : sr_word<true>(blk + 2 + hb * 16);
                            if (hb == 0) ds[r >> 1][r & 1] = sr_f16(blk - 4 * c);
                            // b = (b & 127) - (b & 128): 128 + (b & 127) less 128 or 256
#pragma unroll
                            for (int q = 0; q < 2; q++) {
                                const uint32_t two = q ? sr_pair23(v, magic) : sr_pair01(v, magic);
                                a[r >> 1][r & 1][q] = st_sub2(two & 0xFF7FFF7Fu, two & 0xFF80FF80u);
                            }
                        }
                        multiply(a, j * 32 + hb * 16, hb == 0);
                    }
                    fold(ds);
                }
            } else {
                constexpr uint32_t off = 0x43204320u; // 128 + 32
                const int behind = ((u - tile * G) * Fm::BYTES) & 15, half = KQ == 4 ? kq >> 1 : kq;
                const unsigned char *wb = w0 + behind; // blocks begin 0 to 14 bytes behind the box's first
                auto quants = [&](auto odd) {
#pragma unroll
                    for (int hb = 0; hb < 2; hb++) {
                        uint32_t qh[4];
#pragma unroll
                        for (int r = 0; r < 4; r++) qh[r] = sr_word<decltype(odd)::value != 0>(wb + r * 8 * Fm::PITCH + 128 + half * 32 + hb * 16);
#pragma unroll
                        for (int lq = 0; lq < (KQ == 4 ? 1 : 2); lq++) { // the first or the second 32 bytes of the half's 64: quarters lo and lo + 2
                            const int lo = KQ == 4 ? kq & 1 : lq;
                            uint32_t ql[4];
#pragma unroll
                            for (int r = 0; r < 4; r++) ql[r] = sr_word<decltype(odd)::value != 0>(wb + r * 8 * Fm::PITCH + half * 64 + lo * 32 + hb * 16);
#pragma unroll
                            for (int up = 0; up < 2; up++) {
                                const int j = lo + 2 * up;
                                uint32_t a[2][2][2];
                                float ds[2][2];
#pragma unroll
                                for (int r = 0; r < 4; r++) {
                                    const uint32_t two = up ? qh[r] >> (2 * lo) : qh[r] << (4 - 2 * lo);
                                    const uint32_t v = ((up ? ql[r] >> 4 : ql[r]) & 0x0F0F0F0Fu) | (two & 0x30303030u);
                                    a[r >> 1][r & 1][0] = st_sub2(sr_pair01(v, magic), off);
                                    a[r >> 1][r & 1][1] = st_sub2(sr_pair23(v, magic), off);
                                    ds[r >> 1][r & 1] = st_lds<float>(table + ((half * 8 + 2 * j + hb) * SR_ROWS + r * 8) * 4);
                                }
                                multiply(a, j * 32 + hb * 16, true);
                                fold(ds);
                            }
                        }
                    }
                };
                if (behind & 2) quants(std::integral_constant<int, 1>());
                else quants(std::integral_constant<int, 0>());
            }
            __syncwarp();
            if (lane == 0) mx_arrive(empty + 8 * s);
            if (++s == S) { s = 0; ph ^= 1u; }
        }
        if (first_unit != u0) asm volatile("bar.sync 1, %0;" ::"n"(SR_CONSUMERS) : "memory"); // the segment before has been read out of red
        float *mine = red + (size_t)kq * (8 * MT) * SR_PLANE + (2 * c) * SR_PLANE + rg * 32 + g;
#pragma unroll
        for (int t = 0; t < 2; t++)
#pragma unroll
            for (int mt = 0; mt < MT; mt++) {
                float *at = mine + mt * 8 * SR_PLANE + t * 16;
                at[0] = tot[t][mt][0];
                at[SR_PLANE] = tot[t][mt][1];
                at[8] = tot[t][mt][2];
                at[SR_PLANE + 8] = tot[t][mt][3];
            }
        st_finish<SR_CONSUMERS, SR_ROWS, SR_PLANE>(p.out, mend, red, KQ, 8 * MT * SR_PLANE, tile, first_unit, seg_end, seg_end == u1, others, ok, &last);
    }
    if (help) st_helped<SR_CONSUMERS, SR_ROWS>(p.out, mend, u0 / G, ok, &helped);
}

static int sr_block_tokens(int m) // tokens of a tile
{
    const int blocks = ceil_div(m, SR_MAX_BLOCK);
    return ceil_div(ceil_div(m, blocks), 8) * 8;
}
static size_t sr_flag_bytes(int tiles) { return ((size_t)(sm_count() + tiles) * sizeof(unsigned long long) + 255) / 256 * 256; }

bool gguf_stream_supported(int type, int m, int k, int n, const void *x, const void *blocks)
{
    if (m < 1 || k < SR_BOX || k % SR_BOX != 0 || n < 1 || !aligned(x, 16) || !aligned(blocks, 16)) return false;
    switch (type) {
    case OXQ_GGML_Q4_0: case OXQ_GGML_Q8_0: case OXQ_GGML_Q4_K: break;
    case OXQ_GGML_Q6_K: if (k % (8 * SR_BOX) != 0) return false; break; // rows of a multiple of 16 bytes
    default: return false;
    }
    return n % 2 == 0 && m <= 512;
}

size_t gguf_stream_scratch_bytes(int m, int n)
{
    const int step = sr_block_tokens(m), tiles = ceil_div(n, SR_ROWS) * ceil_div(m, step);
    return sr_flag_bytes(tiles) + (size_t)(sm_count() + tiles) * step * SR_ROWS * sizeof(float);
}

template <int TYPE, int MT, int KQ>
static int sr_launch(StreamRowsParams &p, const CUtensorMap &wmap, const CUtensorMap &xmap, int ctas, cudaStream_t st)
{
    using Fm = SrFormat<TYPE>;
    auto kern = gguf_stream_kernel<TYPE, MT, KQ>;
    const size_t slot = SR_ROWS * (Fm::PITCH + Fm::TABLE) + MT * 8 * SR_X_PITCH + (TYPE == OXQ_GGML_Q4_K ? 8 * 8 * MT * 4 : 0);
    const size_t red = (size_t)KQ * 8 * MT * SR_PLANE * sizeof(float);
    p.stages = (int)((226 * 1024 - 512 - red) / slot);
    if (p.stages > SR_MAX_STAGES) p.stages = SR_MAX_STAGES;
    if (const char *e = tuning_env("SR_STAGES")) p.stages = atoi(e) < p.stages ? atoi(e) : p.stages;
    const size_t smem = p.stages * slot + red + 128;
    static size_t configured[64] = {};
    int device = 0;
    OXQ_CUDA(cudaGetDevice(&device));
    if (device >= 64 || configured[device] < smem) {
        OXQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (device < 64) configured[device] = smem;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(KQ * 128 + 128, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    allow_early_start(attr, cfg.numAttrs);
    OXQ_CUDA(cudaLaunchKernelEx(&cfg, kern, p, wmap, xmap));
    return OXQ_OK;
}

template <int TYPE>
static int sr_run(StreamRowsParams &p, const void *x, const void *blocks, int k, cudaStream_t st)
{
    using Fm = SrFormat<TYPE>;
    const StreamOut &o = p.out;
    const uint64_t row_bytes = (uint64_t)(k / SR_BOX) * Fm::BYTES;
    const int mt = o.tok_step <= 8 ? 1 : o.tok_step <= 16 ? 2 : o.tok_step <= 32 ? 4 : 8;
    CUtensorMap wmap, xmap;
    CUresult r = encode_tiled_2d(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, blocks, row_bytes / 4, (uint64_t)o.n, row_bytes, Fm::PITCH / 4, SR_ROWS,
                                 CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (blocks) failed with CUresult %d", (int)r);
    r = encode_tiled_2d(&xmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, x, (uint64_t)k / 2, (uint64_t)o.m, (uint64_t)k * 2, SR_X_PITCH / 4, 8 * mt,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (x) failed with CUresult %d", (int)r);
    // a unit, in hundredths of a us: 55 up to eight tokens, 65 / 85 / 175 at 16 / 32 / 64
    const int more = o.tok_step > 8 ? o.tok_step - 8 : 0;
    const int ctas = st_ctas(p.out, o.tok_step > 32 ? 85 + (o.tok_step - 32) * 45 / 16 : 55 + more * 5 / 4, 150 + 6 * more, 10 + more * 5 / 4, 450 + 16 * more);
    const char *e4 = tuning_env("SR_KQ");
    const int kq = e4 ? atoi(e4) : 2;
    switch (mt) {
    case 1: return kq == 4 ? sr_launch<TYPE, 1, 4>(p, wmap, xmap, ctas, st) : sr_launch<TYPE, 1, 2>(p, wmap, xmap, ctas, st);
    case 2: return kq == 4 ? sr_launch<TYPE, 2, 4>(p, wmap, xmap, ctas, st) : sr_launch<TYPE, 2, 2>(p, wmap, xmap, ctas, st);
    case 4: return kq == 4 ? sr_launch<TYPE, 4, 4>(p, wmap, xmap, ctas, st) : sr_launch<TYPE, 4, 2>(p, wmap, xmap, ctas, st);
    default: return sr_launch<TYPE, 8, 2>(p, wmap, xmap, ctas, st);
    }
}

int gguf_stream_matmul(int type, const void *x, const void *blocks, const void *bias, int bias_dtype, void *y, int y_dtype, int m, int k, int n,
                       int *flag, void *scratch, cudaStream_t st)
{
    StreamRowsParams p = {};
    p.x = reinterpret_cast<const __nv_bfloat16 *>(x); p.blocks = reinterpret_cast<const uint8_t *>(blocks);
    p.k = k; p.flag = flag;
    StreamOut &o = p.out;
    o.bias = bias; o.y = y; o.bias_dtype = bias_dtype; o.y_dtype = y_dtype; o.m = m; o.n = n; o.ldy = n;
    o.tok_step = sr_block_tokens(m);
    o.tok_blocks = ceil_div(m, o.tok_step);
    o.pairs = y_dtype == OXQ_BF16 && aligned(y, 4);
    o.units_per_tile = k / SR_BOX;
    const int tiles = ceil_div(n, SR_ROWS) * o.tok_blocks;
    o.total = tiles * o.units_per_tile;
    o.mark = mx_call_mark();
    o.flags = reinterpret_cast<unsigned long long *>(scratch);
    o.partials = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(scratch) + sr_flag_bytes(tiles));
    switch (type) {
    case OXQ_GGML_Q4_0: return sr_run<OXQ_GGML_Q4_0>(p, x, blocks, k, st);
    case OXQ_GGML_Q8_0: return sr_run<OXQ_GGML_Q8_0>(p, x, blocks, k, st);
    case OXQ_GGML_Q4_K: return sr_run<OXQ_GGML_Q4_K>(p, x, blocks, k, st);
    default: return sr_run<OXQ_GGML_Q6_K>(p, x, blocks, k, st);
    }
}

} // namespace oxq

using namespace oxq;

// Where the other kernels are the faster ones. Up to 32 tokens those are the GEMVs: on small layers, with few tokens, us there / here, in graphs of calls on
// different weights. Q4_0: 2048 x 1024 at 4 / 8 tokens 6.0 / 8.6 against 6.5 / 7.3, 2048 x 2560 at 2 / 4 6.8 / 8.2 against 7.3, 4096 x 1024 at 1 / 2 6.6 / 7.9 against
// 7.3, 2048 x 6144 at 2 / 4 8.4 / 10.5 against 9.1, 2048 x 11264 at one 13.4 against 9.7. Q8_0: 2048 x 1024 at 2 / 4 6.4 / 7.6 against 6.6, 4096 x 1024 at one 11.5 against
// 8.1. Q4_K: 2048 x 1024 at 8 / 12 / 16 / 32 6.6 / 10.5 / 12.7 / 12.8 against 7.7 / 9.7 / 10.3 / 14.5, 4096 x 4096 at 1 / 8 / 12 5.6 / 9.8 / 13.4 against 10.1 / 11.0 / 13.0, 2048 x 6144
// at 2 / 4 7.9 / 10.1 against 9.4, 2048 x 11264 at 1 / 2 10.1 / 11.6 against 10.6, 14336 x 4096 at 1 / 2 / 4 14.6 / 16.7 / 31.6 against 18.1, 14336 x 1024 at 1 / 2 9.9 / 12.5
// against 10.5, 4096 x 14336 at one 19.0 against 17.2. Q6_K, which has a kernel of its own for wide layers (4096 x 14336 at 1 / 8 14.7 / 17.3 against 19.4): 4096 x 1024 at
// 4 / 8 7.6 / 11.2 against 8.7 / 9.4, 4096 x 4096 at one 12.6 against 11.2, 4096 x 6144 at 1 / 2 12.9 / 14.2 against 13.4.
// Above 32 tokens they are the dense copy and its GEMM, about 0.9 us a million weights and 4 us a thousand of k (4096 x 4096 31 us, 14336 x 4096 111 at 64 and
// 128 tokens), against 20 us and 0.0133 (Q4_0) to 0.0225 (Q4_K) a unit of 64 tokens here (4096 x 14336 at 64 tokens 36.5 to 57.8 us, 68 to 70 there).
static bool gguf_stream_faster(int type, int m, int k, int n)
{
    if (const char *e = tuning_env("SR_ROUTE")) return atoi(e) != 0;
    const long long w = (long long)k * n, mw = m * w;
    if (m <= 32) {
        switch (type) {
        case OXQ_GGML_Q4_0:
            if (k >= 4096) return mw >= 8000000;
            return m >= 8 ? mw >= 14000000 : w >= (m >= 4 ? 5000000 : 20000000);
        case OXQ_GGML_Q8_0: return mw >= (k >= 4096 ? 4000000 : k >= 2048 ? 5000000 : 12000000);
        case OXQ_GGML_Q4_K:
            if (m >= 12) return w >= (m <= 16 ? 2000000 : 4000000);
            if (m >= 4) return k > 4096 || n >= 6144;
            if (m >= 2) return n >= 10240 || (k >= 12288 && n <= 2048);
            return n >= 12288 && w >= 50000000;
        default:
            if (m <= 8 && n >= 9472) return false;
            if (m >= 8) return mw >= 30000000;
            return k >= 4096 && w >= 14000000 && (m >= 2 || n <= k);
        }
    }
    const int slope = type == OXQ_GGML_Q4_0 ? 133 : type == OXQ_GGML_Q8_0 ? 155 : type == OXQ_GGML_Q4_K ? 225 : 180;
    const long long units = (long long)ceil_div(n, SR_ROWS) * (k / SR_BOX) * ceil_div(m, sr_block_tokens(m));
    return m <= 256 && 20 * 10000 + slope * units < w * 9 / 1000 + k * 40;
}

OXQ_EXPORT size_t oxq_gguf_scratch_bytes(int ggml_type, int m, int k, int n)
{
    return gguf_stream_supported(ggml_type, m, k, n, nullptr, nullptr) && gguf_stream_faster(ggml_type, m, k, n) ? gguf_stream_scratch_bytes(m, n) : 0;
}

OXQ_EXPORT int oxq_gguf_matmul(int ggml_type, const void *x, int x_dtype, const void *blocks, const void *bias, int bias_dtype, void *y,
                               int y_dtype, int m, int k, int n, void *flag_word, void *scratch, size_t scratch_bytes, void *stream)
{
    clear_error();
    OXQ_REQUIRE(x && blocks && y && flag_word && scratch, OXQ_ERR_NULL, "oxq_gguf_matmul: null pointer");
    OXQ_REQUIRE(x_dtype == OXQ_BF16, OXQ_ERR_UNSUPPORTED, "oxq_gguf_matmul: activations must be bf16");
    OXQ_REQUIRE(valid_dtype(y_dtype) && (!bias || valid_dtype(bias_dtype)), OXQ_ERR_UNSUPPORTED, "oxq_gguf_matmul: unsupported dtype");
    OXQ_REQUIRE(aligned(scratch, 256) && aligned(flag_word, 4), OXQ_ERR_BAD_ALIGN, "oxq_gguf_matmul: scratch must be 256-byte aligned");
    OXQ_REQUIRE(gguf_stream_supported(ggml_type, m, k, n, x, blocks), OXQ_ERR_UNSUPPORTED,
                "oxq_gguf_matmul: type %d, [%d, %d] x [%d, %d] or the alignment are not served", ggml_type, m, k, n, k);
    OXQ_REQUIRE(scratch_bytes >= gguf_stream_scratch_bytes(m, n), OXQ_ERR_WORKSPACE, "oxq_gguf_matmul: scratch of %zu bytes needed, got %zu",
                gguf_stream_scratch_bytes(m, n), scratch_bytes);
    return gguf_stream_matmul(ggml_type, x, blocks, bias, bias_dtype, y, y_dtype, m, k, n, reinterpret_cast<int *>(flag_word), scratch,
                              (cudaStream_t)stream);
}
