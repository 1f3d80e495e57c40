// AWQ and GPTQ 4-bit matmul of decode-sized batches: packed words streamed from HBM through shared memory into mma.sync.
//
// One CTA per SM walks its share of all (tile, unit) pairs: a tile is 256 out features (two halves of 128; for a gated projection 128 gates and their partners) x at
// most 16 tokens, a unit 128 input rows. Three k groups of four warps take thirds of a segment, each with a ring and a producer warp of its own, so that nothing
// but the end of a tile is common to them. The unpacked weight is q - z, exact in bf16: an AWQ word holds eight out features of one input row; a transposed 8 x 8 load
// of its 16-bit halves gives a lane two input rows of four out features, and each nibble position is one operand register of mma.sync, so that seven
// instructions make eight weights (byte permutes of two words: nine). A GPTQ word is eight input rows of one out feature and takes activations in the order of its
// nibbles. A group's sum is multiplied by its scale in f32. Parts of a tile meet as in stream_common.cuh.
//
// What bounds it: instruction issue up to 8 tokens (about 330 warp instructions per 64 rows x 64 out features, of which the unpack is 112 at half
// rate and the subtraction of zero points 64 at two clocks; the loads alone ran at 6 TB/s), beside 3.5 us until the first unit is there and 2 to 3 us for a shared tile.
// Units of 64 rows took 22.7 us on 4096 x 28672 at one token, of 128 rows 18.9; without the subtraction (128 + z times the sum of x taken off in f32, not exact) 17.9.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "stream_common.cuh"

namespace oxq {

constexpr int S4_COLS = 256, S4_PLANE = S4_COLS + 2;   // out features of a tile; floats from one token's row of it to the next in shared memory
constexpr int S4_UNIT = 128;                           // input rows of a unit
constexpr int S4_HALF_BYTES = S4_UNIT * 64;            // packed words of a unit, 128 out features
constexpr int S4_W_BYTES = 2 * S4_HALF_BYTES;
constexpr int S4_X_BYTES = 8 * 64 * 2;                 // eight tokens, 64 input rows
constexpr int S4_KG = 3;                               // k groups of four warps, each with a ring and a producer of its own
constexpr int S4_CONSUMERS = S4_KG * 128, S4_THREADS = S4_CONSUMERS + S4_KG * 32 + 32;
constexpr int S4_MAX_STAGES = 4;
constexpr int S4_MAX_BLOCK = 16;                       // tokens of a tile

struct Stream4Params {
    int sym, n;
    int gshift;       // log2(group size)
    int stages;
    int half1;        // out feature at which the second half of tile 0 begins
    int tile_step;    // out features from a tile to the next
    int *flag;
    StreamOut out;
};

struct Stream4Maps { CUtensorMap words, x, scales, zeros; };

// NG: quantization groups of a unit, 1, 2 or 4. MT: eights of tokens.
template <bool GPTQ, int NG, int MT>
__global__ void __launch_bounds__(S4_THREADS, 1)
    packed4_stream_kernel(const Stream4Params p, const __grid_constant__ Stream4Maps maps)
{
    constexpr int KG = S4_KG, SLOT = S4_W_BYTES + 2 * MT * S4_X_BYTES; // x: [64 rows][eight tokens]
    constexpr int Z_AT = 2 * NG * 256, META = (2 * NG * (256 + 64) + 127) / 128 * 128; // scales [group][half][128], zero points [group][half][16 words]
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long bars[KG * S4_MAX_STAGES * 2];
    __shared__ uint32_t last, helped;
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, S = p.stages;
    // shared memory: slots [k group][stage] | scales and zero points [k group][stage] | partial tiles [k group]
    unsigned char *slots = smem_raw + (((smem_u32(smem_raw) + 1023u) & ~1023u) - smem_u32(smem_raw)), *metas = slots + KG * S * SLOT;
    float *red = reinterpret_cast<float *>(metas + KG * S * META);
    const int kg = warp < 4 * KG ? warp >> 2 : warp < 5 * KG ? warp - 4 * KG : 0;
    const uint32_t full = smem_u32(bars) + (uint32_t)(kg * S4_MAX_STAGES * 16), empty = full + 8 * S4_MAX_STAGES;
    if (warp >= 4 * KG && warp < 5 * KG && lane == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(full + 8 * s, 1);
            mbar_init(empty + 8 * s, 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.words) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.x) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.scales) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.zeros) : "memory");
    }
    __syncthreads();
    pdl_wait();

    const int G = p.out.units_per_tile;
    const int u0 = st_share(p.out, gridDim.x, blockIdx.x), u1 = st_share(p.out, gridDim.x, blockIdx.x + 1);
    const bool help = st_needs_help(p.out, u0, u1);
    int s = 0;
    uint32_t ph = 0;
    if (warp == 5 * KG) {
        if (help) st_help<S4_CONSUMERS>(p.out, u0 / G, &helped);
        return;
    }
    if (warp >= 4 * KG) {
        // ---- producer of one k group: four copies a unit (about 130 clocks each to issue; eight, for each half and group: 19.0 us, with four 18.6, 4096 x 28672) -----------------------------
        const uint32_t bytes = S4_W_BYTES + 2 * MT * S4_X_BYTES + (uint32_t)NG * (p.sym ? 512u : 640u);
        for (int u = u0; u < u1;) {
            const int tile = u / G, seg_end = min(u1, (tile + 1) * G), cnt = seg_end - u;
            const int ft = tile / p.out.tok_blocks, block = p.out.gate ? ft : 2 * ft, tok0 = tile % p.out.tok_blocks * p.out.tok_step; // block: of 128 out features
            int kb = u + cnt * kg / KG - tile * G;
            for (const int end = u + cnt * (kg + 1) / KG - tile * G; kb < end; kb++) {
                if (!mx_wait(empty + 8 * s, ph ^ 1u, p.flag, ST_CODE + 1)) return;
                const uint32_t slot = smem_u32(slots) + (uint32_t)((kg * S + s) * SLOT), sc = smem_u32(metas) + (uint32_t)((kg * S + s) * META), bar = full + 8 * s;
                if (elect_one()) {
                    mbar_arrive_expect_tx(bar, bytes);
                    const int group = (kb * S4_UNIT) >> p.gshift;
                    if constexpr (GPTQ) st_load_3d(slot, &maps.words, bar, kb * (S4_UNIT / 8), block * 4);
                    else st_load_4d(slot, &maps.words, bar, kb * S4_UNIT, block, 0);
                    st_load_3d(slot + S4_W_BYTES, &maps.x, bar, tok0, 2 * kb);
                    st_load_4d(sc, &maps.scales, bar, block, 0, group);
                    if (!p.sym) st_load_4d(sc + Z_AT, &maps.zeros, bar, block, 0, group);
                }
                __syncwarp();
                if (++s == S) { s = 0; ph ^= 1u; }
            }
            u = seg_end;
        }
        return;
    }

    // ---- unpack and multiply: 64 out features, this k group's units --------------------------------------------------
    const int cg = warp & 3, half = cg >> 1, g = lane >> 2, c = lane & 3;
    uint32_t mask, magic; // opaque to constant propagation so that they stay in registers
    asm volatile("mov.b32 %0, 0x000F000F;\n\tmov.b32 %1, 0x43004300;" : "=r"(mask), "=r"(magic));
    // AWQ: a transposed 8 x 8 load gives a lane the 16-bit halves of two input rows, four out features each
    const int ar = ((lane >> 4) << 3) + (lane & 7);
    const uint32_t a_off = (uint32_t)(half * S4_HALF_BYTES + ar * 64 + (((2 * (cg & 1) + ((lane >> 3) & 1)) ^ ((ar >> 1) & 3)) << 4));
    // GPTQ: four neighbouring out features of a packed row (eight input rows); [block of 32 features][16 packed rows][128 bytes], swizzled
    const int q_off = half * S4_HALF_BYTES + (cg & 1) * 4096;
    const uint32_t odd = (g & 1) ? 0x7632u : 0x5410u;
    const int sc_off = half * 256 + (cg & 1) * 128 + (GPTQ ? g * 8 : (g >> 1) * 16);
    const int z_off = Z_AT + half * 64 + (cg & 1) * 32 + (g >> 1) * 4;
    float tot[4][MT][4];
    bool ok = true;
    bool others = false;
    for (int u = u0; u < u1;) {
        const int tile = u / G, seg_end = min(u1, (tile + 1) * G), cnt = seg_end - u;
        int b = u + cnt * kg / KG;
        const int e = u + cnt * (kg + 1) / KG;
#pragma unroll
        for (int t = 0; t < 4; t++)
#pragma unroll
            for (int mt = 0; mt < MT; mt++) tot[t][mt][0] = tot[t][mt][1] = tot[t][mt][2] = tot[t][mt][3] = 0.0f;
#pragma unroll 1
        for (; b < e; b++) {
            if (b + 1 == e && seg_end == u1 && warp == 0) others = st_others(p.out, tile, st_owner(p.out, gridDim.x, tile * G), st_owner(p.out, gridDim.x, (tile + 1) * G - 1));
            ok = ok && mx_wait(full + 8 * s, ph, p.flag, ST_CODE + 2);
            if (!ok) break;
            const unsigned char *slot = slots + (kg * S + s) * SLOT, *sc = metas + (kg * S + s) * META;
            const uint32_t slot_a = smem_u32(slots) + (uint32_t)((kg * S + s) * SLOT);
#pragma unroll
            for (int grp = 0; grp < NG; grp++) {
                constexpr int PAIRS = 4 / NG; // of steps of 16 input rows
                // zero points: bf16 pairs 128 + z. AWQ: out features of 16-bit halves g and g + 8; GPTQ: 4 g .. 4 g + 3 of the two blocks of 32
                uint32_t zz[8];
                {
                    const unsigned char *at = sc + z_off + grp * 128;
                    const bool none = GPTQ && p.sym;
                    const uint32_t w[2] = {none ? 0x77777777u : st_lds<uint32_t>(at), none ? 0x77777777u : st_lds<uint32_t>(at + 16)};
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint32_t z4 = __byte_perm(w[h], 0, (g & 1) ? 0x3232 : 0x1010);
#pragma unroll
                        for (int j = 0; j < 4; j++) zz[4 * h + j] = st_and_or(z4 >> (4 * j), mask, magic) + (GPTQ ? 0x00010001u : 0u);
                    }
                }
                float acc[4][MT][4];
#pragma unroll
                for (int pr = 0; pr < PAIRS; pr++) {
                    const int at = grp * PAIRS + pr; // 32 input rows of the unit
                    uint32_t xb[MT][4];
                    if constexpr (!GPTQ) {
                        uint32_t r[2][4];
                        st_ldmatrix_t(r[0], slot_a + a_off + (uint32_t)(at * 2048));
                        st_ldmatrix_t(r[1], slot_a + a_off + (uint32_t)(at * 2048 + 1024));
#pragma unroll
                        for (int mt = 0; mt < MT; mt++)
                            st_ldmatrix(xb[mt], slot_a + S4_W_BYTES + (uint32_t)(((at >> 1) * MT + mt) * S4_X_BYTES + (lane & 7) * 128 + ((((at & 1) * 4 + (lane >> 3)) ^ (lane & 7)) << 4)));
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const bool first = pr == 0 && h == 0;
#pragma unroll
                            for (int j = 0; j < 4; j++) {
                                uint32_t a[4];
#pragma unroll
                                for (int i = 0; i < 4; i++) a[i] = st_sub2(st_and_or(r[h][i] >> (4 * j), mask, magic), zz[4 * (i & 1) + j]);
#pragma unroll
                                for (int mt = 0; mt < MT; mt++) {
                                    if (first) st_mma_first(acc[j][mt], a[0], a[1], a[2], a[3], xb[mt][0], xb[mt][1]);
                                    else st_mma(acc[j][mt], a[0], a[1], a[2], a[3], xb[mt][2 * h], xb[mt][2 * h + 1]);
                                }
                            }
                        }
                    } else {
                        // packed rows of a step: every second one, so that no two lanes meet in a bank; in order where groups are of 32
                        const int sub = at >> 1, row = NG == 4 ? 4 * (at & 1) + c : 2 * c + (at & 1);
#pragma unroll
                        for (int mt = 0; mt < MT; mt++) {
                            const uint4 v = st_lds<uint4>(slot + S4_W_BYTES + (sub * MT + mt) * S4_X_BYTES + g * 128 + ((row ^ g) << 4));
                            xb[mt][0] = __byte_perm(v.x, v.z, 0x5410); // input rows 0 and 4, 1 and 5, 2 and 6, 3 and 7 of the word
                            xb[mt][1] = __byte_perm(v.x, v.z, 0x7632);
                            xb[mt][2] = __byte_perm(v.y, v.w, 0x5410);
                            xb[mt][3] = __byte_perm(v.y, v.w, 0x7632);
                        }
#pragma unroll
                        for (int blk = 0; blk < 2; blk++) {
                            const uint4 wv = st_lds<uint4>(slot + q_off + blk * 2048 + sub * 1024 + row * 128 + ((g ^ row) << 4));
                            const uint32_t w[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
                            for (int jj = 0; jj < 2; jj++)
#pragma unroll
                                for (int ss = 0; ss < 2; ss++) {
                                    uint32_t a[4];
#pragma unroll
                                    for (int i = 0; i < 4; i++)
                                        a[i] = st_sub2(st_and_or(w[2 * jj + (i & 1)] >> (8 * ss + 4 * (i >> 1)), mask, magic), zz[4 * blk + 2 * jj + (i & 1)]);
#pragma unroll
                                    for (int mt = 0; mt < MT; mt++) {
                                        float (&d)[4] = acc[2 * blk + jj][mt];
                                        if (pr == 0 && ss == 0) st_mma_first(d, a[0], a[1], a[2], a[3], xb[mt][0], xb[mt][1]);
                                        else st_mma(d, a[0], a[1], a[2], a[3], xb[mt][2 * ss], xb[mt][2 * ss + 1]);
                                    }
                                }
                        }
                    }
                }
                // scales of the accumulator rows g and g + 8 of the four products
                const unsigned char *at = sc + sc_off + grp * 512;
                float2 s01[2], s23[2];
                if constexpr (!GPTQ) {
                    const uint4 lo = st_lds<uint4>(at), hi = st_lds<uint4>(at + 64);
                    s01[0] = st_f16x2(__byte_perm(lo.x, lo.y, odd)); s23[0] = st_f16x2(__byte_perm(lo.z, lo.w, odd));
                    s01[1] = st_f16x2(__byte_perm(hi.x, hi.y, odd)); s23[1] = st_f16x2(__byte_perm(hi.z, hi.w, odd));
                } else { // products 0 and 1: the first block, out features 4 g + {0, 1} and 4 g + {2, 3}
                    const uint2 lo = st_lds<uint2>(at), hi = st_lds<uint2>(at + 64);
                    s01[0] = st_f16x2(__byte_perm(lo.x, lo.y, 0x5410)); s01[1] = st_f16x2(__byte_perm(lo.x, lo.y, 0x7632));
                    s23[0] = st_f16x2(__byte_perm(hi.x, hi.y, 0x5410)); s23[1] = st_f16x2(__byte_perm(hi.x, hi.y, 0x7632));
                }
#pragma unroll
                for (int t = 0; t < 4; t++)
#pragma unroll
                    for (int mt = 0; mt < MT; mt++)
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float2 pair = t < 2 ? s01[i >> 1] : s23[i >> 1];
                            tot[t][mt][i] = fmaf((t & 1) ? pair.y : pair.x, acc[t][mt][i], tot[t][mt][i]);
                        }
            }
            __syncwarp();
            if (lane == 0) mx_arrive(empty + 8 * s);
            if (++s == S) { s = 0; ph ^= 1u; }
        }
        if (u != u0) asm volatile("bar.sync 1, %0;" ::"n"(S4_CONSUMERS) : "memory"); // the segment before has been read out of red
        float *mine = red + (size_t)kg * (8 * MT) * S4_PLANE;
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const int col = GPTQ ? cg * 64 + (t >> 1) * 32 + 4 * g + 2 * (t & 1) : cg * 64 + 8 * (g >> 1) + (g & 1) + 2 * t;
            const int next = GPTQ ? 1 : 32; // accumulator row g + 8
#pragma unroll
            for (int mt = 0; mt < MT; mt++) {
                float *at = mine + (8 * mt + 2 * c) * S4_PLANE + col;
                at[0] = tot[t][mt][0];
                at[S4_PLANE] = tot[t][mt][1];
                at[next] = tot[t][mt][2];
                at[S4_PLANE + next] = tot[t][mt][3];
            }
        }
        st_finish<S4_CONSUMERS, S4_COLS, S4_PLANE>(p.out, StKeep(), red, KG, 8 * MT * S4_PLANE, tile, u, seg_end, seg_end == u1, others, ok, &last);
        u = seg_end;
    }
    if (help) st_helped<S4_CONSUMERS, S4_COLS>(p.out, StKeep(), u0 / G, ok, &helped);
}

bool stream4_supported(int m, int k, int n, int group_size, int scales_dtype, const void *x, const void *qweight, const void *qzeros,
                       const void *scales, int gate)
{
    return m >= 1 && m <= 64 && n % (gate ? 256 : 128) == 0 && k % S4_UNIT == 0 && group_size >= 32 && (group_size & (group_size - 1)) == 0 &&
           k % group_size == 0 && scales_dtype == OXQ_F16 && aligned(x, 16) && aligned(qweight, 16) && aligned(qzeros, 16) && aligned(scales, 16);
}

// Batches that this kernel is the best one for; measured per call in graphs of calls on different weights, us in the kernel that took the call before / here.
//   AWQ, groups from 64 on, up to 8 tokens, against the GEMV, which starts before the kernel ahead has finished: 4096 x 28672 at 1 / 8 tokens 21.3 / 32.9 against
//   18.9 / 19.5, 14336 x 1024 12.2 / 16.2 against 10.6 / 13.3, 10240 x 2048 12.4 / 14.5 against 10.0 / 13.2; not 12288 x 1024 9.6 against 10.0 at one token, 8192 x 2048 8.9
//   against 9.5, 4096 x 6144 8.3 / 9.8 against 10.7 / 12.4. Where the GEMV cannot split k, and beyond its batches, against the grouped kernel: 5632 x 256 11.1 / 11.5
//   against 8.3 / 11.0, 13824 x 5120 23.8 / 24.0 against 15.3 / 16.8, 1152 x 1152 10.8 / 11.0 against 7.5 / 7.8.
//   From 9 tokens on against the grouped kernel: 4096 x 28672 at 16 30.4 against 23.8, 18944 x 3584 at 12 / 16 22.4 / 22.5 against 20.9 / 23.4; groups of 64
//   3072 x 16384 at 16 19.8 against 18.7.
//   GPTQ, groups from 64 on, against the grouped and the block-scaled kernel: 4096 x 14336 at 1 / 8 / 16 tokens 19.3 / 19.5 / 19.8 against 14.7 / 15.9 / 20.1,
//   2048 x 512 at 3 / 7 8.7 / 8.8 against 7.0 / 9.0, 4096 x 512 at 7 10.7 against 9.8, 4096 x 28672 at 16 35.3 against 24.6; groups of 64 4096 x 14336 at 8 / 16 25.2 / 25.1
//   against 16.7 / 21.2.
//   Groups of 32, which only GEMVs and a dense copy served: AWQ 4096 x 28672 at 8 / 16 / 32 / 48 / 64 tokens 38 / 65 / 114 / 138 / 138 against 22 / 28 / 53 / 78 / 87, 7168 x
//   2048 at 1 / 8 12.5 / 15.6 against 9.9 / 12.4, not 4096 x 6144 at 8 (11.1 against 12.5) nor 2048 x 512 at 32 (10.8 against 13.2); GPTQ 4096 x 4096 at 1 / 8 / 16 / 64 29 /
//   70 / 27 / 28 against 10 / 12 / 16 / 22, 14336 x 4096 at 1 / 8 165 / 756 against 16 / 18, not 512 x 512 at 1 / 2 (3.9 / 4.7 against 5.5).
bool stream4_faster(int m, int k, int n, int group_size, int gptq)
{
    if (const char *e = tuning_env("S4_ROUTE")) return atoi(e) != 0;
    const long long w = (long long)k * n;
    if (group_size == 32 && m > 8) return k >= 4096 || w >= (m <= 48 ? 4000000 : 24000000) || (!gptq && m <= 16 && k >= 2048);
    if (m > 16) return false;
    if (gptq) {
        if (group_size == 32) return m >= 4 || k * m >= 2048;
        if (m <= 8) return m <= 6 || k >= 4096 || w >= 10000000;
        return w >= (group_size == 64 ? 40000000 : 80000000);
    }
    if (m <= 8) {
        if (group_size == 32) return k >= 7168 || w >= 26000000;
        if (oxq_awq_gemv_max_m(k, n, group_size) < m || k > 12288 || (k >= 10240 && w >= 20000000) || (k >= 8192 && w >= 28000000)) return true;
        return w >= (group_size > 64 ? 40000000 : m >= 6 ? 45000000 : 55000000);
    }
    if (group_size == 64) return w >= 45000000 || (m <= 12 && k >= 8192 && w >= 28000000);
    return w >= 80000000 || (m <= 12 && k >= 12288 && w >= 40000000);
}

static int s4_block_tokens(int m) // tokens of a tile
{
    const int blocks = ceil_div(m, S4_MAX_BLOCK);
    return blocks > 1 ? ceil_div(ceil_div(m, blocks), 8) * 8 : m;
}
static size_t s4_flag_bytes(int tiles) { return ((size_t)(sm_count() + tiles) * sizeof(unsigned long long) + 255) / 256 * 256; }

// Scratch that a call of this size needs.
size_t stream4_scratch_bytes(int m, int n)
{
    const int step = s4_block_tokens(m), tiles = ceil_div(n, S4_COLS) * ceil_div(m, step);
    return s4_flag_bytes(tiles) + (size_t)(sm_count() + tiles) * step * S4_COLS * sizeof(float);
}

template <bool GPTQ, int NG, int MT>
static int s4_launch(Stream4Params &p, const Stream4Maps &maps, int ctas, cudaStream_t st)
{
    auto kern = packed4_stream_kernel<GPTQ, NG, MT>;
    const size_t slot = S4_W_BYTES + 2 * MT * S4_X_BYTES + (2 * NG * (256 + 64) + 127) / 128 * 128;
    const size_t red = (size_t)S4_KG * 8 * MT * S4_PLANE * sizeof(float);
    p.stages = (int)((226 * 1024 - 1024 - 512 - red) / (S4_KG * slot));
    if (p.stages > S4_MAX_STAGES) p.stages = S4_MAX_STAGES;
    const size_t smem = (size_t)S4_KG * p.stages * slot + red + 1024;
    static size_t configured[64] = {};
    int device = 0;
    OXQ_CUDA(cudaGetDevice(&device));
    if (device >= 64 || configured[device] < smem) {
        OXQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (device < 64) configured[device] = smem;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(S4_THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    allow_early_start(attr, cfg.numAttrs);
    OXQ_CUDA(cudaLaunchKernelEx(&cfg, kern, p, maps));
    return OXQ_OK;
}

// gate: n is [gate | up], y = act(gate) * up (1 SiLU, 2 GeLU-tanh).
int stream4_matmul(const void *x, const uint32_t *qweight, const uint32_t *qzeros, const void *scales, const void *bias, int bias_dtype, void *y,
                   int y_dtype, int m, int k, int n, int group_size, int col_base, int ldy, int *flag, cudaStream_t st, int gptq, int sym, int gate,
                   void *scratch, size_t scratch_bytes)
{
    if (!scratch || scratch_bytes < stream4_scratch_bytes(m, n)) return OXQ_ERR_UNSUPPORTED;
    Stream4Params p = {};
    p.sym = (gptq && (sym || qzeros == nullptr)) ? 1 : 0;
    p.n = n; p.flag = flag;
    while ((1 << p.gshift) < group_size) p.gshift += 1;
    p.tile_step = gate ? S4_COLS / 2 : S4_COLS;
    p.half1 = gate ? n / 2 : S4_COLS / 2;
    StreamOut &o = p.out;
    o.bias = bias ? (const unsigned char *)bias + (size_t)col_base * dtype_size(bias_dtype) : nullptr;
    o.y = (unsigned char *)y + (size_t)col_base * dtype_size(y_dtype);
    o.bias_dtype = bias_dtype; o.y_dtype = y_dtype; o.m = m; o.n = n; o.ldy = ldy; o.gate = gate;
    o.tok_step = s4_block_tokens(m);
    o.tok_blocks = ceil_div(m, o.tok_step);
    o.pairs = y_dtype == OXQ_BF16 && ldy % 2 == 0 && aligned(o.y, 4);
    o.units_per_tile = k / S4_UNIT;
    const int tiles = ceil_div(n, S4_COLS) * o.tok_blocks;
    o.total = tiles * o.units_per_tile;
    o.mark = mx_call_mark();
    o.flags = reinterpret_cast<unsigned long long *>(scratch);
    o.partials = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(scratch) + s4_flag_bytes(tiles));
    const int ctas = st_ctas(o, o.tok_step <= 8 ? 40 : 55, 235 + 13 * o.tok_step, 12 + 17 * o.tok_step / 10, 600 + 45 * o.tok_step);

    const int mt = o.tok_step <= 8 ? 1 : 2;
    Stream4Maps maps;
    const int rc = st_packed4_maps(maps.words, maps.scales, maps.zeros, qweight, p.sym ? nullptr : qzeros, scales, k, n, group_size, gptq, gate);
    if (rc) return rc;
    const CUresult r = encode_tiled_3d(&maps.x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x, 64, (uint64_t)m, (uint64_t)k / 64, (uint64_t)k * 2, 128, 64, 8 * mt, 2,
                                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (x) failed with CUresult %d", (int)r);
    const int ng = group_size >= 128 ? 1 : group_size == 64 ? 2 : 4;
#define S4_RUN(GPTQ_, MT_)                                                                                                      \
    return ng == 1 ? s4_launch<GPTQ_, 1, MT_>(p, maps, ctas, st) : ng == 2 ? s4_launch<GPTQ_, 2, MT_>(p, maps, ctas, st) \
                                                                       : s4_launch<GPTQ_, 4, MT_>(p, maps, ctas, st)
    if (gptq && mt == 1) S4_RUN(true, 1);
    if (gptq) S4_RUN(true, 2);
    if (mt == 1) S4_RUN(false, 1);
    S4_RUN(false, 2);
#undef S4_RUN
}

} // namespace oxq
