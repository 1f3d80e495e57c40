// AWQ and GPTQ 4-bit matmul of ten to some two hundred tokens: packed words streamed through shared memory, unpacked into tensor memory, tcgen05.mma.
//
// A tile is 256 out features (two halves of 128; of a gated projection 128 gates and their partners) x up to 96 tokens, a unit 128 input rows. The operand that meets
// the activations is q - z, exact in bf16; a quantization group's product leaves tensor memory once and is added to the totals with its scale, in f32. Roles of a CTA:
//   warps 0, 2    TMA, one copy each of a unit's words, zero points, activations, scales;
//   warps 1, 3    tcgen05.mma kind::f16, a half each: weights [128 x 16] from tensor memory times activations [16 x tokens] from shared memory;
//   warps 4..19   unpack, two sets that take the units in turn; a warp has 32 out features of a half. AWQ: a transposed 8 x 8 load of 16-bit halves gives a lane two
//                 input rows of four out features, which is the operand's layout for 16 x 128-bit stores (11 instructions for eight weights);
//   warps 20..27  fold, a half each warpgroup, the totals of an out feature in a thread's registers.
// Tensor memory: 256 columns of accumulators, 2 x 2 x 64 of operands. Where the tiles are fewer than the SMs, up to eight CTAs, a cluster, share a tile's units and
// put it together through each other's shared memory, each a part of the tokens; shares that cross tile borders meet in scratch as in stream_common.cuh.
//
// What bounds it: instruction issue, 850 (32 tokens) to 1030 (80) warp instructions a unit and scheduler in 1100 to 1400 clocks (leaving out the unpack's arithmetic, its
// stores, the fold's or seven eighths of the MMAs changed a call by 0 to 8 %); from 65 tokens also the chain of an accumulator, one a half there: MMAs, fold, next
// MMAs. Beside that 8 us to fill the pipeline and to end. On the way: eight unpack warps, each on every unit, 35 to 44 us (4096 x 28672 at 32 / 77 tokens; now 26.6 / 33.6), one
// warp with eight copies a unit 29.4 / 34.9, one issuing warp for both halves 40 / 55, scales read from L2 by the fold 43 / 61.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <atomic>

#include "stream_common.cuh"

namespace oxq {

constexpr int W4_COLS = 256;                           // out features of a tile, in two halves
constexpr int W4_UNIT = 128;                           // input rows of a unit
constexpr int W4_HALF_BYTES = W4_UNIT * 64, W4_W_BYTES = 2 * W4_HALF_BYTES;
constexpr int W4_Z_BYTES = 1024, W4_S_BYTES = 2048;    // zero points and scales of a unit: [group][half][16 words], [group][half][128], up to four groups
constexpr int W4_MAX_TOK = 96, W4_MAX_STAGES = 8;
constexpr int W4_A_AT = 256, W4_A_COLS = 64;           // tensor memory: accumulators in columns 0 .. 255, then operands [stage][half][64 columns]
constexpr int W4_UNPACK_WARP0 = 4, W4_FOLD_WARP0 = 20;
constexpr int W4_FOLD = 256, W4_THREADS = W4_FOLD_WARP0 * 32 + W4_FOLD;
// Registers a thread: 72 at launch, then by role, for tiles of up to 64 tokens and of more: control 40 / 32, unpack 56 / 48, fold 112 / 136.
template <int CH> struct W4Regs { static constexpr int CONTROL = CH > 4 ? 32 : 40, UNPACK = CH > 4 ? 48 : 56, FOLD = CH > 4 ? 136 : 112; };
static_assert(128 * (W4Regs<4>::CONTROL + 4 * W4Regs<4>::UNPACK + 2 * W4Regs<4>::FOLD) <= W4_THREADS * 72 &&
                  128 * (W4Regs<6>::CONTROL + 4 * W4Regs<6>::UNPACK + 2 * W4Regs<6>::FOLD) <= W4_THREADS * 72, "registers of the block");

struct Wide4Params {
    int scales_f16, sym, n;
    int gshift, groups; // log2(group size); groups of a unit
    int stages, npad;   // npad: tokens of a tile, a multiple of 16
    int half1, tile_step;
    int cluster;        // above 1: so many CTAs share a tile, one cluster, and put it together through their shared memory
    int *flag;
    StreamOut out;
};

template <int V> struct W4Int { static constexpr int value = V; };
struct Wide4Maps { CUtensorMap words, x, scales, zeros; };

__device__ __forceinline__ void w4_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void w4_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float w4_peer(uint32_t addr, int rank) // shared memory of a CTA of the cluster
{
    float v;
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}" : "=f"(v) : "r"(addr), "r"(rank) : "memory");
    return v;
}
__device__ __forceinline__ void w4_umma(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// 16 lanes x 16 columns: register 2 i holds row lane / 4, column 4 i + lane % 4; register 2 i + 1 the row eight further on.
__device__ __forceinline__ void w4_st_16x16(uint32_t taddr, const uint32_t (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void w4_st_32x16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

// CH: sixteens of tokens of a tile; a fold warpgroup takes half of them.
template <bool GPTQ, int CH>
__global__ void __launch_bounds__(W4_THREADS, 1)
    packed4_wide_kernel(const Wide4Params p, const __grid_constant__ Wide4Maps maps)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long bars[2 * W4_MAX_STAGES + 16];
    __shared__ uint32_t tmem_slot, last, helped;
    pdl_launch_dependents();
    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, S = p.stages;
    unsigned char *slots = smem_raw + (((smem_u32(smem_raw) + 1023u) & ~1023u) - smem_u32(smem_raw));
    const int slot_bytes = W4_W_BYTES + p.npad * W4_UNIT * 2 + W4_Z_BYTES + W4_S_BYTES, z_at = W4_W_BYTES + p.npad * W4_UNIT * 2, s_at = z_at + W4_Z_BYTES;
    // full: a unit's words, zero points, scales and activations have landed; empty: its eight unpacking warps and the fold are done with them (the fold comes
    // after its MMAs). Of each half: afull / aempty [stage]: an operand is in tensor memory, has been multiplied; dfull / dempty [slot]: an accumulator is
    // complete, has been read
    const uint32_t full = smem_u32(bars), empty = full + 8 * W4_MAX_STAGES, afull = empty + 8 * W4_MAX_STAGES, aempty = afull + 32, dfull = aempty + 32,
                   dempty = dfull + 32;
    if (warp == 0 && lane == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(full + 8 * s, 2);
            mbar_init(empty + 8 * s, 8 + W4_FOLD / 32);
        }
        for (int s = 0; s < 4; s++) {
            mbar_init(afull + 8 * s, 4);
            mbar_init(aempty + 8 * s, 1);
            mbar_init(dfull + 8 * s, 1);
            mbar_init(dempty + 8 * s, W4_FOLD / 64);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.words) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.x) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.scales) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.zeros) : "memory");
    }
    if (warp == 3) {
        tmem_alloc(smem_u32(&tmem_slot), 512u);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_wait();

    const int G = p.out.units_per_tile, NG = p.groups;
    const int u0 = st_share(p.out, gridDim.x, blockIdx.x), u1 = st_share(p.out, gridDim.x, blockIdx.x + 1);
    const bool help = st_needs_help(p.out, u0, u1);
    constexpr int ACCS = CH > 4 ? 1 : 2; // accumulators of a half
    auto halves_of = [&](int tile) { return tile / p.out.tok_blocks * p.tile_step + p.half1 < p.n ? 2 : 1; };

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(W4Regs<CH>::CONTROL));
        if (warp == 0 || warp == 2) {
            // ---- TMA: warp 0 words and zero points, warp 2 activations and scales (a copy takes a warp about 130 clocks to issue; one warp with eight
            // copies a unit, one for each half and group, held the kernel to 1200 clocks a unit) ------------------------------------------------
            const bool leader = elect_one();
            const uint32_t bytes = warp == 0 ? W4_W_BYTES + (p.sym ? 0 : NG * 128) : p.npad * W4_UNIT * 2 + NG * 512;
            int s = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int u = u0, kb = u0 % G, tile = u0 / G; u < u1 && ok; tile++, kb = 0) {
                const int seg_end = min(u1, (tile + 1) * G), ft = tile / p.out.tok_blocks, tok0 = tile % p.out.tok_blocks * p.out.tok_step;
                const int block = p.out.gate ? ft : 2 * ft; // of 128 out features
                for (; u < seg_end && ok; u++, kb++) {
                    ok = mx_wait(empty + 8 * s, ph, p.flag, ST_CODE + 1);
                    const uint32_t slot = smem_u32(slots) + (uint32_t)(s * slot_bytes), bar = full + 8 * s;
                    if (ok && leader) {
                        mbar_arrive_expect_tx(bar, bytes);
                        const int group = (kb * W4_UNIT) >> p.gshift;
                        if (warp == 0) {
                            if constexpr (GPTQ) st_load_3d(slot, &maps.words, bar, kb * (W4_UNIT / 8), block * 4);
                            else st_load_4d(slot, &maps.words, bar, kb * W4_UNIT, block, 0);
                            if (!p.sym) st_load_4d(slot + z_at, &maps.zeros, bar, block, 0, group);
                        } else {
                            st_load_3d(slot + W4_W_BYTES, &maps.x, bar, tok0, 2 * kb);
                            st_load_4d(slot + s_at, &maps.scales, bar, block, 0, group);
                        }
                    }
                    __syncwarp();
                    if (++s == S) { s = 0; ph ^= 1u; }
                }
            }
            if (warp == 2 && help) st_help<W4_FOLD>(p.out, u0 / G, &helped);
        } else if (warp == 1 || warp == 3) {
            // ---- MMA issue, one half each: from one unit's MMAs to the next an issuing warp takes about 900 clocks -------------------------
            const bool leader = elect_one();
            const int h = warp >> 1;
            const uint32_t idesc = tc_idesc(128, 16 * CH);
            constexpr uint32_t SUB = 16 * CH * 128 >> 4; // 64 input rows of activations, in units of 16 bytes
            int s = 0, st = 0, d = 0;
            uint32_t ph = 0, aph = 0, dph = 1;
            bool ok = true;
            for (int u = u0, tile = u0 / G; u < u1 && ok; tile++) {
              const int seg_end = min(u1, (tile + 1) * G);
              for (; u < seg_end && ok; u++) {
                { // (a half that lies beyond n is multiplied as it lies in shared memory and goes nowhere)
                    const uint64_t xd = kmajor_sw128_desc(smem_u32(slots) + (uint32_t)(s * slot_bytes + W4_W_BYTES));
                    const uint32_t a = tmem + W4_A_AT + (uint32_t)((2 * st + h) * W4_A_COLS), abar = 8 * (2 * h + st);
                    for (int g = 0; g < NG && ok; g++) {
                        const uint32_t dt = tmem + (uint32_t)((h * ACCS + d) * 16 * CH), dbar = 8 * (2 * h + d);
                        ok = g == 0 ? mx_wait3(full + 8 * s, ph, afull + abar, aph, dempty + dbar, dph, p.flag, ST_CODE + 4) : mx_wait(dempty + dbar, dph, p.flag, ST_CODE + 4);
                        if (!ok) break;
                        tc_fence_after();
                        if (leader) {
                            if (NG == 1) {
#pragma unroll
                                for (int i = 0; i < 8; i++) w4_umma(dt, a + 8 * i, xd + (uint64_t)((i >> 2) * SUB + 2 * (i & 3)), idesc, i != 0);
                            } else if (NG == 2) {
                                const uint32_t ag = a + 32 * g;
                                const uint64_t xg = xd + (uint64_t)(g * SUB);
#pragma unroll
                                for (int i = 0; i < 4; i++) w4_umma(dt, ag + 8 * i, xg + (uint64_t)(2 * i), idesc, i != 0);
                            } else {
                                const uint32_t ag = a + 16 * g;
                                const uint64_t xg = xd + (uint64_t)((g >> 1) * SUB + 4 * (g & 1));
#pragma unroll
                                for (int i = 0; i < 2; i++) w4_umma(dt, ag + 8 * i, xg + (uint64_t)(2 * i), idesc, i != 0);
                            }
                            umma_commit(dfull + dbar);
                            if (g == NG - 1) umma_commit(aempty + abar);
                        }
                        __syncwarp();
                        if (++d == ACCS) { d = 0; dph ^= 1u; }
                    }
                    st ^= 1;
                    if (st == 0) aph ^= 1u;
                }
                if (++s == S) { s = 0; ph ^= 1u; }
              }
            }
        }
    } else if (warp < W4_FOLD_WARP0) {
        // ---- unpack: 32 out features of one half of every second unit, q - z as bf16 -------------------------------------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(W4Regs<CH>::UNPACK));
        const int st = (warp - W4_UNPACK_WARP0) >> 3, h = ((warp - W4_UNPACK_WARP0) >> 2) & 1, q = warp & 3, g8 = lane >> 2;
        uint32_t mask, magic; // opaque to constant propagation so that they stay in registers
        asm volatile("mov.b32 %0, 0x000F000F;\n\tmov.b32 %1, 0x43004300;" : "=r"(mask), "=r"(magic));
        const int zoff = z_at + h * 64 + q * 16 + (GPTQ ? (lane >> 3) * 4 : (g8 >> 1) * 4);
        const int per = (W4_UNIT / 32) / NG; // 32 input rows a step, steps of a group
        const uint32_t a = tmem + W4_A_AT + (uint32_t)((2 * st + h) * W4_A_COLS) + ((uint32_t)(32 * q) << 16), abar = 8 * (2 * h + st);
        int s = st; // S is even: a slot always meets the same warps, which see every phase of its barriers
        uint32_t ph = 0, aph = 1;
        for (int u = u0 + st; u < u1; u += 2) {
            if (!mx_wait2(full + 8 * s, ph, aempty + abar, aph, p.flag, ST_CODE + 2)) break;
            {
                tc_fence_after();
                const unsigned char *slot = slots + s * slot_bytes;
                const uint32_t words = smem_u32(slot) + (uint32_t)(h * W4_HALF_BYTES + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4)); // 32 input rows further on: the same swizzle
                uint32_t zz[GPTQ ? 1 : 4], raw[4][4];
#pragma unroll
                for (int at = 0; at < 4; at++) {
                    if constexpr (GPTQ) {
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const int r = 4 * at + i;
                            raw[at][i] = st_lds<uint32_t>(slot + h * W4_HALF_BYTES + q * 2048 + r * 128 + ((g8 ^ (r & 7)) << 4) + (lane & 3) * 4);
                        }
                    } else st_ldmatrix_t(raw[at], words + (uint32_t)(at * 2048));
                }
#pragma unroll
                for (int at = 0; at < 4; at++) {
                    if (at % per == 0) {
                        const uint32_t w = GPTQ && p.sym ? 0x77777777u : st_lds<uint32_t>(slot + zoff + at / per * 128);
                        if constexpr (GPTQ) {
                            const uint32_t z = w >> (4 * (lane & 7)) & 15u;
                            zz[0] = (z | z << 16) + (magic + 0x00010001u);
                        } else {
                            const uint32_t z4 = __byte_perm(w, 0, (g8 & 1) ? 0x3232 : 0x1010);
#pragma unroll
                            for (int j = 0; j < 4; j++) zz[j] = st_and_or(z4 >> (4 * j), mask, magic);
                        }
                    }
                    if constexpr (GPTQ) {
                        uint32_t o[16];
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const uint32_t w = raw[at][i];
                            uint32_t t[4]; // input rows j and j + 4
#pragma unroll
                            for (int j = 0; j < 4; j++) t[j] = st_sub2(st_and_or(w >> (4 * j), mask, magic), zz[0]);
                            o[4 * i] = __byte_perm(t[0], t[1], 0x5410);
                            o[4 * i + 1] = __byte_perm(t[2], t[3], 0x5410);
                            o[4 * i + 2] = __byte_perm(t[0], t[1], 0x7632);
                            o[4 * i + 3] = __byte_perm(t[2], t[3], 0x7632);
                        }
                        w4_st_32x16(a + 16 * at, o);
                    } else {
                        // a transposed 8 x 8 load gives a lane the 16-bit half g8 of two input rows: out features 8 (g8 / 2) + g8 % 2 + 2 j
                        const uint32_t (&r)[4] = raw[at];
                        uint32_t lo[8], hi[8];
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            lo[2 * i] = st_sub2(st_and_or(r[i], mask, magic), zz[0]);
                            lo[2 * i + 1] = st_sub2(st_and_or(r[i] >> 4, mask, magic), zz[1]);
                            hi[2 * i] = st_sub2(st_and_or(r[i] >> 8, mask, magic), zz[2]);
                            hi[2 * i + 1] = st_sub2(st_and_or(r[i] >> 12, mask, magic), zz[3]);
                        }
                        w4_st_16x16(a + 16 * at, lo);
                        w4_st_16x16(a + 16 * at + (16u << 16), hi);
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
            }
            __syncwarp();
            if (lane == 0) {
                mx_arrive(afull + abar);
                mx_arrive(empty + 8 * s);
            }
            aph ^= 1u;
            s += 2;
            if (s >= S) { s -= S; ph ^= 1u; }
        }
    } else {
        // ---- fold: a group's products times its scale into the totals, a half to each of the two warpgroups ---------------------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(W4Regs<CH>::FOLD));
        const int q = warp & 3, h = (warp - W4_FOLD_WARP0) >> 2, ft = threadIdx.x - W4_FOLD_WARP0 * 32;
        // lane -> out feature of its half
        const int of = 32 * q + (GPTQ ? lane : 8 * ((lane & 7) >> 1) + (lane & 1) + 2 * (lane >> 3));
        const uint32_t dcol = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(h * ACCS * 16 * CH);
        struct Tile { int f0, f1, halves, tokens, first; float b0, b1; };
        auto tile_of = [&](int tile) {
            Tile t;
            t.f0 = tile / p.out.tok_blocks * p.tile_step + of; t.f1 = t.f0 + p.half1;
            t.halves = halves_of(tile);
            t.tokens = st_tokens(p.out, tile); t.first = tile % p.out.tok_blocks * p.out.tok_step;
            t.b0 = p.out.bias ? load_as_f32(p.out.bias, p.out.bias_dtype, t.f0) : 0.0f;
            t.b1 = p.out.bias && t.halves > 1 ? load_as_f32(p.out.bias, p.out.bias_dtype, t.f1) : 0.0f;
            return t;
        };
        auto output = [&](const Tile &t, int tok, float a, float b) {
            const size_t at = (size_t)(t.first + tok) * p.out.ldy;
            if (p.out.gate) {
                store_as(p.out.y, p.out.y_dtype, at + t.f0, st_act(a, b, p.out.gate));
                return;
            }
            store_as(p.out.y, p.out.y_dtype, at + t.f0, a + t.b0);
            if (t.halves > 1) store_as(p.out.y, p.out.y_dtype, at + t.f1, b + t.b1);
        };
        float tot[16 * CH];
        int s = 0, d = 0;
        uint32_t ph = 0, dph = 0;
        bool ok = true;
        // the sums of CTAs i_lo .. of a tile in scratch, in ascending k; a warpgroup takes every second eight tokens
        auto together = [&](int tile, int i_lo, int parts) {
            const Tile t = tile_of(tile);
            const size_t stride = (size_t)p.out.tok_step * W4_COLS;
            const float *src = p.out.partials + (size_t)(i_lo + tile) * stride + 32 * q + lane;
#pragma unroll 1
            for (int i0 = 8 * h; i0 < t.tokens; i0 += 16) {
                float a[8], b[8];
#pragma unroll
                for (int i = 0; i < 8; i++) a[i] = b[i] = 0.0f;
#pragma unroll 1
                for (int x0 = 0; x0 < parts; x0 += 2) { // 32 loads under way together
                    float va[2][8], vb[2][8];
#pragma unroll
                    for (int y = 0; y < 2; y++)
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            va[y][i] = vb[y][i] = 0.0f;
                            if (x0 + y < parts && i0 + i < t.tokens) {
                                const float *at = src + (size_t)(x0 + y) * stride + (i0 + i) * W4_COLS;
                                va[y][i] = __ldcg(at);
                                vb[y][i] = __ldcg(at + W4_COLS / 2);
                            }
                        }
#pragma unroll
                    for (int y = 0; y < 2; y++)
#pragma unroll
                        for (int i = 0; i < 8; i++) { a[i] += va[y][i]; b[i] += vb[y][i]; }
                }
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (i0 + i < t.tokens) output(t, i0 + i, a[i], b[i]);
            }
        };
        for (int u = u0; u < u1;) {
            const int tile = u / G, seg_end = min(u1, (tile + 1) * G);
#pragma unroll
            for (int i = 0; i < 16 * CH; i++) tot[i] = 0.0f;
#pragma unroll 1
            for (int b = u; b < seg_end && ok; b++) {
                const unsigned char *scales = slots + s * slot_bytes + s_at + h * 256 + of * 2;
#pragma unroll 1
                for (int g = 0; g < NG && ok; g++) {
                    const uint32_t dbar = 8 * (2 * h + d);
                    ok = g == 0 ? mx_wait2(full + 8 * s, ph, dfull + dbar, dph, p.flag, ST_CODE + 5) : mx_wait(dfull + dbar, dph, p.flag, ST_CODE + 5);
                    if (!ok) break;
                    const uint16_t bits = st_lds<uint16_t>(scales + g * 512);
                    const float sc = p.scales_f16 ? half_bits_to_f32(bits) : bf16_lo_f32(bits);
                    tc_fence_after();
                    constexpr int PART = CH > 4 ? 4 : 2 * CH < 4 ? 2 * CH : 4; // eights of columns in flight
#pragma unroll
                    for (int c0 = 0; c0 < 2 * CH; c0 += PART) {
                        uint32_t v[PART][8];
#pragma unroll
                        for (int c = 0; c < PART; c++)
                            if (c0 + c < 2 * CH) tmem_ld_x8(dcol + (uint32_t)(d * 16 * CH + 8 * (c0 + c)), v[c]);
                        tmem_ld_wait();
                        if (c0 + PART >= 2 * CH) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) {
                                mx_arrive(dempty + dbar);
                                if (g == NG - 1) mx_arrive(empty + 8 * s);
                            }
                        }
#pragma unroll
                        for (int c = 0; c < PART; c++)
#pragma unroll
                            for (int i = 0; i < 8; i++)
                                if (c0 + c < 2 * CH) tot[8 * (c0 + c) + i] = fmaf(sc, __uint_as_float(v[c][i]), tot[8 * (c0 + c) + i]);
                    }
                    if (++d == ACCS) { d = 0; dph ^= 1u; }
                }
                if (++s == S) { s = 0; ph ^= 1u; }
            }
            // the end of a segment: as st_finish, with the sums in registers
            const int i_lo = st_owner(p.out, gridDim.x, tile * G), i_hi = st_owner(p.out, gridDim.x, (tile + 1) * G - 1);
            const Tile t = tile_of(tile);
            if (p.cluster > 1) { // the units of this share are done with by both warpgroups: the ring is free
                asm volatile("bar.sync 1, %0;" ::"n"(W4_FOLD) : "memory");
                float *mine = reinterpret_cast<float *>(slots) + 128 * h + 32 * q + lane;
#pragma unroll
                for (int i = 0; i < 16 * CH; i++) mine[i * W4_COLS] = tot[i];
                __syncwarp();
                w4_cluster_arrive();
                w4_cluster_wait();
                const int rank = (int)blockIdx.x % p.cluster, tokens = ok ? t.tokens : 0;
                const uint32_t at = smem_u32(slots) + (uint32_t)((32 * q + lane) * 4);
                auto merge = [&](auto ranks_, auto toks_) { // in ascending k; 32 loads under way together (one token at a time: 4 us for 80 tokens of two CTAs)
                    constexpr int R = decltype(ranks_)::value, T = decltype(toks_)::value;
#pragma unroll 1
                    for (int tok = h + 2 * rank; tok < tokens; tok += 2 * p.cluster * T) {
                        float va[T][R], vb[T][R];
#pragma unroll
                        for (int i = 0; i < T; i++)
#pragma unroll
                            for (int r = 0; r < R; r++) {
                                const int t1 = tok + 2 * p.cluster * i;
                                va[i][r] = vb[i][r] = 0.0f;
                                if (r < p.cluster && t1 < tokens) {
                                    va[i][r] = w4_peer(at + (uint32_t)(t1 * W4_COLS * 4), r);
                                    vb[i][r] = w4_peer(at + (uint32_t)(t1 * W4_COLS * 4 + W4_COLS * 2), r);
                                }
                            }
#pragma unroll
                        for (int i = 0; i < T; i++) {
                            float a = 0.0f, b = 0.0f;
#pragma unroll
                            for (int r = 0; r < R; r++) { a += va[i][r]; b += vb[i][r]; }
                            if (tok + 2 * p.cluster * i < tokens) output(t, tok + 2 * p.cluster * i, a, b);
                        }
                    }
                };
                if (p.cluster <= 2) merge(W4Int<2>(), W4Int<8>());
                else if (p.cluster <= 4) merge(W4Int<4>(), W4Int<4>());
                else merge(W4Int<8>(), W4Int<2>());
            } else if (i_lo == i_hi && !p.out.gate) {
                if (ok && h < t.halves) {
                    const int col = h ? t.f1 : t.f0;
                    const float bias = h ? t.b1 : t.b0;
#pragma unroll
                    for (int i = 0; i < 16 * CH; i++)
                        if (i < t.tokens) store_as(p.out.y, p.out.y_dtype, (size_t)(t.first + i) * p.out.ldy + col, tot[i] + bias);
                }
            } else { // (gates and their partners are with different warpgroups: a whole tile takes this way too)
                if (ok) {
                    float *part = p.out.partials + (size_t)(blockIdx.x + tile) * p.out.tok_step * W4_COLS + 128 * h + 32 * q + lane;
#pragma unroll
                    for (int i = 0; i < 16 * CH; i++)
                        if (i < t.tokens) part[i * W4_COLS] = tot[i];
                }
                bool now = i_lo == i_hi;
                if (!now && seg_end != u1) asm volatile("bar.arrive 2, %0;" ::"n"(W4_FOLD + 32) : "memory"); // the helping warp sets the flag
                else {
                    asm volatile("bar.sync 1, %0;" ::"n"(W4_FOLD) : "memory");
                    if (!now) {
                        if (ft < 32) {
                            const bool all = st_arrive(p.out, tile, i_lo, i_hi);
                            if (all) st_clear(p.out, tile, i_lo, i_hi);
                            if (ft == 0) *(volatile uint32_t *)&last = all;
                        }
                        asm volatile("bar.sync 1, %0;" ::"n"(W4_FOLD) : "memory");
                        now = *(volatile uint32_t *)&last;
                    }
                }
                if (now && ok) together(tile, i_lo, i_hi - i_lo + 1);
            }
            u = seg_end;
        }
        if (help) { // a first segment whose tile the helping warp found complete
            asm volatile("bar.sync 3, %0;" ::"n"(W4_FOLD + 32) : "memory");
            const int tile = u0 / G, i_lo = st_owner(p.out, gridDim.x, tile * G);
            if (*(volatile uint32_t *)&helped && ok) together(tile, i_lo, st_owner(p.out, gridDim.x, (tile + 1) * G - 1) - i_lo + 1);
        }
    }
    if (p.cluster > 1) {
        // Every warp of the cluster's CTAs comes to this barrier twice: the fold's came to it first when their sums were in shared memory, and nobody
        // leaves while a peer may still read them.
        __syncwarp();
        if (warp < W4_FOLD_WARP0) {
            w4_cluster_arrive();
            w4_cluster_wait();
        }
        w4_cluster_arrive();
        w4_cluster_wait();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 3) tmem_dealloc(tmem, 512u);
}

bool wide4_supported(int m, int k, int n, int group_size, int scales_dtype, const void *x, const void *qweight, const void *qzeros, const void *scales, int gate)
{
    return m >= 1 && m <= 3 * W4_MAX_TOK && n % (gate ? 256 : 128) == 0 && k % W4_UNIT == 0 && group_size >= 32 && (group_size & (group_size - 1)) == 0 &&
           k % group_size == 0 && (scales_dtype == OXQ_F16 || scales_dtype == OXQ_BF16) && aligned(x, 16) && aligned(qweight, 16) && aligned(qzeros, 16) &&
           aligned(scales, 16);
}

// Batches that this kernel is the best one for, us in a graph of calls on different weights, the kernel that took the call before / here. (Over the linears of layers of
// 2048 to 4096 features, 5632 to 14336 in between, at 9 to 256 tokens, and GPTQ 2048 .. 14336 x 1024 .. 14336 at 3 to 256: 1.17 times as fast on the average, 7 % slower at worst.)
//   Groups from 64 on, 9 to 96 tokens, against the grouped kernel (csrc/group_tc.cu) or the one on rounded weights (csrc/fused_tc.cu): AWQ 4096 x 4096 at 16 / 32 / 64 /
//   96 tokens 11.5 / 12.0 / 15.1 / 17.1 against 10.2 / 11.2 / 12.9 / 14.9, 4096 x 28672 at 32 / 64 / 96 32.3 / 39.9 / 49.5 against 26.6 / 31.3 / 37.8, 2048 x 2048 at 64 12.1 against
//   9.3, groups of 64 4096 x 28672 at 64 58.0 against 39.2; GPTQ 14336 x 4096 at 32 / 96 22.6 / 29.6 against 21.6 / 26.2. Not: groups of 64 on 65 to 96 tokens where k is short
//   and the other kernel's tiles of 128 out features fill one round (3072 x 16384 at 80 23.7 against 24.0); 75 to 111 tiles, which leave a quarter of the SMs or more
//   idle (2560 x 19456, groups of 64, at 16 / 32 18.0 / 22.5 against 22.0 / 23.0); up to 16 tokens what csrc/stream4.cu does better: 4096 x 28672 at 12 23.9 against
//   24.1, groups of 64 26.6 against 32.4, 14336 x 4096 at 12 21.2 against 22.4, GPTQ of groups of 64 4096 x 14336 at 12 20.0 against 20.8.
//   Up to 8 tokens: wide AWQ layers of short k (2048 x 11264 at 3 / 8 11.5 / 12.8 against 10.4 / 10.6), small GPTQ layers (4096 x 1024 at 3 / 8 8.2 / 9.8 against 7.8 / 8.0,
//   2048 x 6144 at 8 10.3 against 9.3, 4096 x 4096 at 5 10.3 against 10.5).
//   97 to 192 tokens in two blocks, to 256 in three, where the tiles are few (4096 x 4096 at 128 / 192 19.3 / 19.5 against 14.6 / 17.2 and at 224 20.9 against 21.4, 2048 x
//   11264 at 128 16.5 against 19.7, 4096 x 6144 at 256 30.2 against 23.4).
//   Groups of 32: 2048 x 2560 at 12 / 48 / 64 12.1 / 14.2 / 18.8 against 8.7 / 10.7 / 11.5, 4096 x 4096 at 12 / 32 / 64 / 128 13.8 / 16.8 / 21.7 / 34.6 against 14.6 / 15.9 / 18.2 /
//   21.5, 4096 x 28672 at 32 52.8 against 48.5, but 14336 x 4096 at 32 / 64 30.8 / 49.2 against 37.2 / 51.4 (at 80 113.6 against 60.6), 2048 x 11264 at 48 16.3 against 17.8.
bool wide4_faster(int m, int k, int n, int group_size, int gptq)
{
    if (const char *e = tuning_env("W4_ROUTE")) return atoi(e) != 0;
    if (k < 1024) return false; // 512 x 2048 at 16 5.3 against 6.3, 1024 x 1024 at 17 7.5 against 6.5
    const long long w = (long long)k * n;
    const int tiles = ceil_div(n, W4_COLS); // of a block of tokens
    const bool idle = tiles > 74 && tiles < (m <= 16 ? 120 : 112);
    if (group_size == 32) {
        if (m <= 16) return m > 8 && w <= 8000000;
        if (m <= 64) return k <= 4096 && (w <= 20000000 || w >= 80000000 || m > 48);
        if (m <= W4_MAX_TOK) return m <= 80 || !idle;
        if (m <= 128) return tiles <= 16 || w >= 80000000;
        return m <= 2 * W4_MAX_TOK && tiles <= 16 && (!gptq || k >= 8192);
    }
    if (gptq && k <= 2048 && tiles > 37) return false;
    if (m <= 8) {
        if (!gptq) return k <= 2048 && n >= 10240 && m >= (group_size > 64 ? 3 : 6);
        return k >= 2048 && (w <= 6000000 ? m >= (group_size > 64 ? 3 : 4) : w <= 13000000 && m >= (group_size > 64 ? 5 : 7));
    }
    if (m <= 16) {
        if (w >= 80000000) return false;
        if (group_size > 64) return true;
        return gptq ? w < 40000000 : !idle && (m > 12 || k < 8192 || w < 28000000);
    }
    if (m <= W4_MAX_TOK) {
        if (group_size > 64) return !idle || k < 4096;
        return m <= 32 ? !idle : m <= 64 || k > 3072 || n <= 10240 || n > 18944;
    }
    if (m <= 2 * W4_MAX_TOK) return tiles <= 18 || (tiles <= 24 && (k < 4096 || (k == 4096 && group_size > 64 && m > 128)));
    return m <= 256 && k <= 8192 && (tiles <= 12 || (tiles >= 18 && tiles <= 24 && k <= 4096));
}

static int w4_pad(int m) { return ceil_div(ceil_div(m, ceil_div(m, W4_MAX_TOK)), 16) * 16; } // tokens of a tile
static size_t w4_flag_bytes(int tiles) { return ((size_t)(sm_count() + tiles) * sizeof(unsigned long long) + 255) / 256 * 256; }

// How many clusters of c such CTAs the device holds at a time (SMs come in groups of 16 to 20, which no cluster spans): 16 clusters of 8 would be 128 CTAs but
// take two rounds (4096 x 4096, 17 to 32 tokens: 8 to a tile 20 us, 6 to a tile 11.2).
static int w4_clusters(int c)
{
    static std::atomic<int> known[64][9];
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device >= 64) return 0;
    int n = known[device][c].load(std::memory_order_relaxed);
    if (n) return n - 1;
    auto kern = packed4_wide_kernel<false, 6>;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(c, 1, 1);
    cfg.blockDim = dim3(W4_THREADS, 1, 1);
    cfg.dynamicSmemBytes = 226 * 1024;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    known[device][c].store(n + 1, std::memory_order_relaxed);
    return n;
}

// How many CTAs take a call and how they share tiles (o.grain, cluster).
static int w4_plan(StreamOut &o, int npad, int groups, int &cluster)
{
    const int tiles = o.total / o.units_per_tile;
    // In hundredths of a microsecond: a unit takes `unit`, putting together a tile that a cluster shares 150, shares that cross tile borders `cross` (4096 x
    // 28672, 24 units a CTA, against whole tiles of 32, one a CTA: at 17 / 77 tokens 29.8 / 43 us against 26.0 / 33.6; 14336 x 1024 at 96 tokens, 38 shares a tile, 104 us).
    const int sms = sm_count(), unit = 45 + npad * 45 / 100 + (groups - 1) * (15 + npad * 9 / 10), shares = ceil_div(sms, tiles) + 1;
    const int cross = 500 + npad * (15 + (shares > 2 ? 3 * (shares - 2) : 0));
    int ctas = tiles < sms ? tiles : sms, best = ceil_div(tiles, sms) * o.units_per_tile * unit;
    cluster = 1;
    o.grain = o.units_per_tile;
    for (int c = 2; c <= 8 && tiles * c <= sms && c <= o.units_per_tile; c++) {
        const int cost = ceil_div(o.units_per_tile, c) * unit + 150;
        if (cost < best && tiles <= w4_clusters(c)) { best = cost; ctas = tiles * c; cluster = c; o.grain = 1; }
    }
    if (o.total >= 2 * sms && tiles % sms != 0) {
        const int cost = ceil_div(o.total, sms) * unit + cross;
        if (cost < best) { best = cost; ctas = sms; cluster = 1; o.grain = 1; }
    }
    if (const char *e = tuning_env("W4_CONF")) { // cluster size, 0: equal shares
        const int c = atoi(e);
        if (c == 0) { ctas = sms < o.total ? sms : o.total; cluster = 1; o.grain = 1; }
        else if (tiles * c <= sms && c <= o.units_per_tile) { ctas = tiles * c; cluster = c; o.grain = c > 1 ? 1 : o.units_per_tile; }
    }
    return ctas;
}

static int w4_groups(int group_size) { return group_size >= W4_UNIT ? 1 : W4_UNIT / group_size; } // of a unit

// Scratch that a call of this size needs: marks and sums, where tiles meet there.
size_t wide4_scratch_bytes(int m, int k, int n, int group_size, int gate)
{
    StreamOut o = {};
    const int npad = w4_pad(m), tiles = ceil_div(n, W4_COLS) * ceil_div(m, npad);
    int cluster = 1;
    o.units_per_tile = k / W4_UNIT;
    o.total = tiles * o.units_per_tile;
    const int ctas = w4_plan(o, npad, w4_groups(group_size), cluster);
    if (cluster > 1 || (o.grain == o.units_per_tile && !gate)) return 256;
    return w4_flag_bytes(tiles) + (size_t)(ctas + tiles) * npad * W4_COLS * sizeof(float);
}

template <bool GPTQ, int CH>
static int w4_launch(Wide4Params &p, const Wide4Maps &maps, int ctas, cudaStream_t st)
{
    auto kern = packed4_wide_kernel<GPTQ, CH>;
    const size_t slot = W4_W_BYTES + (size_t)p.npad * W4_UNIT * 2 + W4_Z_BYTES + W4_S_BYTES;
    p.stages = (int)((226 * 1024 - 1024) / slot);
    p.stages = p.stages > W4_MAX_STAGES ? W4_MAX_STAGES : p.stages & ~1;
    const size_t smem = p.stages * slot + 1024;
    static size_t configured[64] = {};
    int device = 0;
    OXQ_CUDA(cudaGetDevice(&device));
    if (device >= 64 || configured[device] < smem) {
        OXQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (device < 64) configured[device] = smem;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(W4_THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    allow_early_start(attr, cfg.numAttrs);
    if (p.cluster > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = p.cluster;
        attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
        cfg.numAttrs += 1;
    }
    OXQ_CUDA(cudaLaunchKernelEx(&cfg, kern, p, maps));
    return OXQ_OK;
}

// gate: n is [gate | up], y = act(gate) * up (1 SiLU, 2 GeLU-tanh).
int wide4_matmul(const void *x, const uint32_t *qweight, const uint32_t *qzeros, const void *scales, int scales_dtype, const void *bias, int bias_dtype,
                 void *y, int y_dtype, int m, int k, int n, int group_size, int col_base, int ldy, int *flag, cudaStream_t st, int gptq, int sym, int gate,
                 void *scratch, size_t scratch_bytes)
{
    if (!scratch || scratch_bytes < wide4_scratch_bytes(m, k, n, group_size, gate)) return OXQ_ERR_UNSUPPORTED;
    Wide4Params p = {};
    p.scales_f16 = scales_dtype == OXQ_F16;
    p.sym = (gptq && (sym || qzeros == nullptr)) ? 1 : 0;
    p.n = n; p.flag = flag;
    while ((1 << p.gshift) < group_size) p.gshift += 1;
    p.groups = w4_groups(group_size);
    p.tile_step = gate ? W4_COLS / 2 : W4_COLS;
    p.half1 = gate ? n / 2 : W4_COLS / 2;
    p.npad = w4_pad(m);
    StreamOut &o = p.out;
    o.bias = bias ? (const unsigned char *)bias + (size_t)col_base * dtype_size(bias_dtype) : nullptr;
    o.y = (unsigned char *)y + (size_t)col_base * dtype_size(y_dtype);
    o.bias_dtype = bias_dtype; o.y_dtype = y_dtype; o.m = m; o.n = n; o.ldy = ldy; o.gate = gate;
    o.tok_step = p.npad;
    o.tok_blocks = ceil_div(m, o.tok_step);
    o.units_per_tile = k / W4_UNIT;
    const int tiles = ceil_div(n, W4_COLS) * o.tok_blocks;
    o.total = tiles * o.units_per_tile;
    o.mark = mx_call_mark();
    o.flags = reinterpret_cast<unsigned long long *>(scratch);
    o.partials = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(scratch) + w4_flag_bytes(tiles));
    const int ctas = w4_plan(o, p.npad, p.groups, p.cluster);
    Wide4Maps maps;
    const int rc = st_packed4_maps(maps.words, maps.scales, maps.zeros, qweight, p.sym ? nullptr : qzeros, scales, k, n, group_size, gptq, gate);
    if (rc) return rc;
    const CUresult r = encode_tiled_3d(&maps.x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x, 64, (uint64_t)m, (uint64_t)k / 64, (uint64_t)k * 2, 128, 64, (uint32_t)p.npad, 2,
                                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (x) failed with CUresult %d", (int)r);
#define W4_RUN(GPTQ_)                                                                   \
    switch (p.npad / 16) {                                                              \
    case 1: return w4_launch<GPTQ_, 1>(p, maps, ctas, st);                        \
    case 2: return w4_launch<GPTQ_, 2>(p, maps, ctas, st);                        \
    case 3: return w4_launch<GPTQ_, 3>(p, maps, ctas, st);                        \
    case 4: return w4_launch<GPTQ_, 4>(p, maps, ctas, st);                        \
    case 5: return w4_launch<GPTQ_, 5>(p, maps, ctas, st);                        \
    default: return w4_launch<GPTQ_, 6>(p, maps, ctas, st);                       \
    }
    if (gptq) W4_RUN(true);
    W4_RUN(false);
#undef W4_RUN
}

} // namespace oxq
