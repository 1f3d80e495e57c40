// Grouped expert matmul of the GPT-OSS MoE layer on MXFP4 weights for small batches, on the block-scaled tensor cores: E2M1
// codes and E8M0 scales are operands as they are, nothing is unpacked. Same table, same outputs as csrc/moe_fused_tc.cu, which
// writes bf16 weights into its operand tile and is the faster one from a few dozen rows per expert on.
// Mirrors the expert half of MoeFeedForward::forward (moe.rs:466-499, dispatch_sparse 563-607).
//
// Activations are two E4M3 pieces with block scales (mx_common.cuh), written by a kernel in front; a stage in which a token block has
// outliers, infinities or NaN comes a second time, at the unit's end, with a second pair of pieces. A unit of work is (token
// block of one expert: up to 48 expert-sorted rows) x (128 out features); CTA b takes units b, b + grid, ... of the device-side
// table, feature tiles fastest. The pieces are neighbouring columns of one MMA (hi | lo), and stages of 128 input columns go to two
// accumulators in turn, so that two warps issue them; the epilogue adds the four. Roles:
//   warp 0        TMA: packed nibbles (128 out features x 64 bytes), as far ahead as the ring allows;
//   warp 2        TMA: both pieces of the block's rows for a stage;
//   warps 1, 3    tcgen05.mma kind::mxf8f6f4 and the copies of the block scales to tensor memory, even and odd stages;
//   warps 4..15   three teams of four warps that take the stages in turn: eight packed bytes (16 codes) to each 16-byte chunk of the operand
//                 row, as the MMA wants 4-bit elements, and the block scales of weights and rows in tensor-memory order;
//   warps 16..19  epilogue of the previous unit while the next one accumulates: bias, clamped SwiGLU (even row gate, odd row up).
//
// What bounds it: a stage's chain of polls, operand rows and arrival in a team. us a layer at 13 / 50 / 200 / 340 tokens, 32 experts of
// 2880 x 2880, with two teams 122 / 148 / 167 / 194, with three 108 / 130 / 144 / 170, with what outliers need 119 / 131 / 146 / 173; packed
// weights alone take 66 from HBM. With an outlier in every block of 32 columns 50 tokens take 183.
#include "moe_mx_split.cuh"

namespace oxq {

constexpr int MM_ROWS = 128;                 // out features per unit
constexpr int MM_MAX_TOK = 48;               // rows of a token block
constexpr int MM_TEAMS = 3, MM_ISSUERS = 2, MM_TEAM_WARPS = 4, MM_UNPACK_WARPS = MM_TEAMS * MM_TEAM_WARPS, MM_EPI_WARPS = 4;
constexpr int MM_EPI_WARP0 = 4 + MM_UNPACK_WARPS;
constexpr int MM_THREADS = (MM_EPI_WARP0 + MM_EPI_WARPS) * 32;
constexpr int MM_SLOTS = 6, MM_RAW = 6;
constexpr int MM_A_BYTES = MM_ROWS * MM_BK;  // 16 codes per 16-byte chunk
constexpr int MM_RAW_BYTES = MM_ROWS * MM_BK / 2;
constexpr int MM_XBOX_ROWS = 16, MM_XBOX_BYTES = MM_XBOX_ROWS * MM_BK, MM_X_BYTES = 2 * MM_MAX_TOK * MM_BK;
constexpr int MM_SF_BYTES = 512;             // scales of 128 rows and 128 k
constexpr int MM_SF_COLS = 64, MM_ACC_COLS = 2 * MM_MAX_TOK; // tensor memory: scales | accumulators [unit parity][stage parity]
constexpr int MM_NUM_BARS = 2 * MM_RAW + 2 * MM_SLOTS + 4;
constexpr size_t MM_SMEM = 1024 + (size_t)MM_SLOTS * (MM_A_BYTES + MM_X_BYTES + 2 * MM_SF_BYTES) + MM_RAW * MM_RAW_BYTES + 8 * MM_NUM_BARS + 16;
constexpr int MM_CODE = 60;                  // wait codes 61 .. 67: oxq_gemm_check names them
static_assert(MM_SMEM <= 227 * 1024, "operand slots and the ring must fit one CTA's shared memory");
static_assert(MM_SLOTS % MM_TEAMS == 0 && MM_SLOTS % MM_ISSUERS == 0 && MM_RAW % MM_TEAMS == 0 && MM_EPI_WARP0 % 4 == 0, "a slot always meets the same team and issuer: a parity wait tells a phase from the next one only");
static_assert(8 * MM_SLOTS <= MM_SF_COLS && MM_SF_COLS + 4 * MM_ACC_COLS <= 512, "tensor memory");

struct MoeMxParams {
    const int4 *entries;   // token blocks: {first row in the expert-sorted matrix, rows, expert, -}
    const int *n_blocks;   // how many
    const uint8_t *scales; // [experts, n, k / 32]
    const uint32_t *sfx;   // [pair][stage][rows_cap] block scales of the rows' hi pieces
    const unsigned char *second;   // [stage][rows_cap] MX_...: whether the row has a second pair of pieces there
    const unsigned char *pieces;   // [pair][piece][rows_cap][k]
    const unsigned long long *any; // `mark` where some have
    unsigned long long mark;
    const void *bias;      // [experts, n] or null
    void *out;
    int *flag;
    int n, k, nkb, stages, rows_cap; // out features per expert, in features, scale bytes per row, stages per unit
    int scale_bytes;       // a row's scales are read this many at a time (its length and their alignment allow it)
    int tiles_n, bias_dtype, ldo, epi;
    float limit;
    int test_skip_loads;   // self-test only: the weight producer issues nothing
};

// ---- rows -> pieces and block scales ---------------------------------------------------------------------------------------------
// Row r is src[perm[r] / top_k] (perm null: src[r]).
__global__ void __launch_bounds__(256)
    moe_mx_split_kernel(const __nv_bfloat16 *src, const int *perm, int top_k, const int *total_rows, const MoeMxPieces q)
{
    pdl_wait();
    pdl_launch_dependents();
    moe_mx_split_rows(src, ld_produced(total_rows), q, gridDim.x, [&](int row) { return perm ? ld_produced(perm + row) / top_k : row; });
}

// Stages in which rows of a token block have a second pair, in order, E4M3 before E5M2: body(stage, MX_...), until it returns false.
template <typename Body> __device__ __forceinline__ bool mm_second_stages(const MoeMxParams &p, int4 en, Body body)
{
    for (int t = 0; t < p.stages; t += 32) {
        const int at = t + (int)(threadIdx.x & 31);
        unsigned kinds = 0; // of the rows, four at a time: all loads are under way together
        if (at < p.stages) {
            const size_t first = (size_t)at * p.rows_cap + en.x;
            const unsigned *words = reinterpret_cast<const unsigned *>(p.second + (first & ~(size_t)3));
            const int skip = (int)(first & 3), span = skip + en.y;
#pragma unroll
            for (int w = 0; w < MM_MAX_TOK / 4 + 1; w++)
                if (4 * w < span) {
                    unsigned v = ld_produced(words + w);
                    if (w == 0) v &= ~0u << (8 * skip);
                    if (4 * w + 4 > span) v &= ~0u >> (8 * (4 * w + 4 - span));
                    kinds |= v;
                }
            kinds |= kinds >> 16;
            kinds |= kinds >> 8;
        }
        const unsigned e4m3 = __ballot_sync(0xFFFFFFFFu, kinds & MX_SECOND_E4M3), e5m2 = __ballot_sync(0xFFFFFFFFu, kinds & MX_SECOND_E5M2);
        for (unsigned hit = e4m3 | e5m2; hit; hit &= hit - 1) {
            const int i = __ffs(hit) - 1;
            if ((e4m3 >> i & 1u) && !body(t + i, MX_SECOND_E4M3)) return false;
            if ((e5m2 >> i & 1u) && !body(t + i, MX_SECOND_E5M2)) return false;
        }
    }
    return true;
}
// A unit's stages as all roles walk them: body(stage, pair, MX_...), until it returns false.
template <bool SECOND, typename Body> __device__ __forceinline__ bool mm_stages(const MoeMxParams &p, int4 en, Body body)
{
    bool ok = true;
    for (int it = 0; it < p.stages && ok; it++) ok = body(it, 0, MX_ONE_PAIR);
    if (SECOND && ok) ok = mm_second_stages(p, en, [&](int it, int kind) { return body(it, 1, kind); });
    return ok;
}

// Shared memory behind `base`: A slots | rows' slots | ring of packed boxes | scales of A and of the rows per slot | barriers | tensor-memory
// address.
constexpr int MM_BARS = MM_SLOTS * (MM_A_BYTES + MM_X_BYTES + 2 * MM_SF_BYTES) + MM_RAW * MM_RAW_BYTES;

// What the warps do; SECOND: with stages that come a second time.
template <bool SECOND>
__device__ __forceinline__ void moe_mx_roles(const MoeMxParams &p, const CUtensorMap &wmap, const CUtensorMap &xmap, uint32_t base, uint32_t tmem_base, int n_units)
{
    const uint32_t x_base = base + MM_SLOTS * MM_A_BYTES, raw_base = x_base + MM_SLOTS * MM_X_BYTES;
    const uint32_t sf_base = raw_base + MM_RAW * MM_RAW_BYTES, bars = base + MM_BARS;
    const uint32_t rawfull = bars, rawempty = rawfull + 8 * MM_RAW, full = rawempty + 8 * MM_RAW, empty = full + 8 * MM_SLOTS,
                   tfull = empty + 8 * MM_SLOTS, tempty = tfull + 16;
    const uint32_t tmem_acc = tmem_base + MM_SF_COLS;
    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, T = p.stages;
    if (warp == 0) {
        // ---- packed nibbles --------------------------------------------------------------------------------------------
        const bool leader = elect_one();
        int r = 0;
        uint32_t ph = 1; // a fresh barrier passes parity 1
        bool ok = true;
        for (int u = blockIdx.x; ok && u < n_units && !p.test_skip_loads; u += gridDim.x) {
            const int tb = u / p.tiles_n, f = u - tb * p.tiles_n;
            const int4 en = ld_produced(p.entries + tb);
            const int rowbase = en.z * p.n + f * MM_ROWS;
            ok = mm_stages<SECOND>(p, en, [&](int it, int, int) {
                const bool ok = mx_wait(rawempty + 8 * r, ph, p.flag, MM_CODE + 1);
                if (ok && leader) {
                    mbar_arrive_expect_tx(rawfull + 8 * r, MM_RAW_BYTES);
                    tma_load_2d(raw_base + (uint32_t)(r * MM_RAW_BYTES), &wmap, rawfull + 8 * r, it * (MM_BK / 2), rowbase);
                }
                __syncwarp();
                if (++r == MM_RAW) { r = 0; ph ^= 1u; }
                return ok;
            });
        }
    } else if (warp == 2) {
        // ---- both pieces of the block's rows ----------------------------------------------------------------------------------
        const bool leader = elect_one();
        int s = 0, done = 0;
        uint32_t ph = 1;
        bool ok = true;
        for (int u = blockIdx.x; ok && u < n_units; u += gridDim.x) {
            const int tb = u / p.tiles_n;
            const int4 en = ld_produced(p.entries + tb);
            const int boxes = (en.y + MM_XBOX_ROWS - 1) / MM_XBOX_ROWS;
            ok = mm_stages<SECOND>(p, en, [&](int it, int pair, int kind) {
                const bool ok = mx_wait(empty + 8 * s, ph, p.flag, MM_CODE + 2);
                if (SECOND && pair && ok) { // 16 bytes at a time, zeros where the row has no second pair of this kind; lo's rows follow hi's
                    constexpr int AHEAD = 4; // rows that a lane has on their way
                    const int j = lane & 7, col = it * MM_BK + 16 * j, n16 = boxes * MM_XBOX_ROWS;
                    for (int r0 = lane >> 3; r0 < n16; r0 += 4 * AHEAD) {
                        uint4 v[2][AHEAD];
                        bool has[AHEAD];
#pragma unroll
                        for (int i = 0; i < AHEAD; i++) {
                            const int r = r0 + 4 * i;
                            has[i] = r < en.y && col < p.k && ld_produced(p.second + (size_t)it * p.rows_cap + en.x + r) == kind;
                        }
#pragma unroll
                        for (int i = 0; i < AHEAD; i++)
#pragma unroll
                            for (int piece = 0; piece < 2; piece++) {
                                v[piece][i] = make_uint4(0u, 0u, 0u, 0u);
                                if (has[i])
                                    v[piece][i] = ld_produced(reinterpret_cast<const uint4 *>(p.pieces + ((size_t)(2 + piece) * p.rows_cap + en.x + r0 + 4 * i) * p.k + col));
                            }
#pragma unroll
                        for (int i = 0; i < AHEAD; i++)
#pragma unroll
                            for (int piece = 0; piece < 2; piece++) {
                                const int at = piece * n16 + r0 + 4 * i;
                                if (r0 + 4 * i < n16)
                                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(x_base + (uint32_t)(s * MM_X_BYTES + at * MM_BK + ((j ^ (at & 7)) << 4))),
                                                 "r"(v[piece][i].x), "r"(v[piece][i].y), "r"(v[piece][i].z), "r"(v[piece][i].w) : "memory");
                            }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic-proxy stores -> visible to the MMA
                    __syncwarp();
                    if (leader) mx_arrive(full + 8 * s);
                } else if (ok && leader) {
                    mbar_arrive_expect_tx(full + 8 * s, (uint32_t)(2 * boxes * MM_XBOX_BYTES));
                    const uint32_t dst = x_base + (uint32_t)(s * MM_X_BYTES);
                    for (int b = 0; b < 2 * boxes; b++) { // lo's rows follow hi's
                        const int lo = b >= boxes;
                        tma_load_2d(dst + (uint32_t)(b * MM_XBOX_BYTES), &xmap, full + 8 * s, it * MM_BK,
                                    lo * p.rows_cap + en.x + (b - lo * boxes) * MM_XBOX_ROWS);
                    }
                }
                __syncwarp();
                if (++s == MM_SLOTS) { s = 0; ph ^= 1u; }
                done++;
                return ok;
            });
        }
        // The commits of the last stages arrive here asynchronously: the CTA stays until they have.
        for (int left = min(MM_SLOTS, done), q = done - left; left > 0 && ok; left--, q++)
            ok = mx_wait(empty + 8 * (q % MM_SLOTS), (uint32_t)(q / MM_SLOTS) & 1u, p.flag, MM_CODE + 7);
    } else if (warp < 4) {
        // ---- MMA issue: warp 1 even stages, warp 3 odd ones, each into its own accumulator; stages are counted over all units -------
        const bool leader = elect_one();
        const int me = warp >> 1;
        const uint64_t da0 = kmajor_sw128_desc(base), db0 = kmajor_sw128_desc(x_base);
        int s = 0, ul = 0;
        uint32_t ph = 0, parity = 0; // parity: of the stages counted so far
        bool ok = true;
        for (int u = blockIdx.x; ok && u < n_units; u += gridDim.x, ul++) {
            const int4 en = ld_produced(p.entries + u / p.tiles_n);
            const int n16 = (en.y + 15) & ~15;
            const uint32_t idesc0 = mx_idesc(MX_E2M1, 2 * n16);
            const int buf = ul & 1;
            const uint32_t d = tmem_acc + (uint32_t)((2 * buf + me) * MM_ACC_COLS);
            ok = mx_wait(tempty + 8 * buf, (((uint32_t)ul >> 1) & 1u) ^ 1u, p.flag, MM_CODE + 3);
            bool first = true;
            ok = ok && mm_stages<SECOND>(p, en, [&](int it, int, int kind) {
                bool ok = true;
                if (parity == (uint32_t)me) {
                    ok = mx_wait(full + 8 * s, ph, p.flag, MM_CODE + 4);
                    if (ok) {
                        tc_fence_after();
                        if (leader) {
                            const uint32_t idesc = kind == MX_SECOND_E5M2 ? idesc0 ^ MX_IDESC_B_E5M2 : idesc0;
                            const uint32_t sfa = tmem_base + 8u * s, sfs = sf_base + (uint32_t)(s * 2 * MM_SF_BYTES);
                            tmem_cp_scales(sfa, sfs);
                            tmem_cp_scales(sfa + 4, sfs + MM_SF_BYTES);
                            const uint64_t da = da0 + (uint64_t)(s * (MM_A_BYTES >> 4)), db = db0 + (uint64_t)(s * (MM_X_BYTES >> 4));
                            const int steps = min(MM_BK, p.k - it * MM_BK) / 32;
#pragma unroll
                            for (int kk = 0; kk < MM_BK / 32; kk++)
                                if (kk < steps)
                                    umma_mxf8(d, da + 2 * kk, db + 2 * kk, idesc | mx_idesc_blocks(kk, kk), sfa, sfa + 4, !(first && kk == 0));
                            umma_commit(empty + 8 * s);
                        }
                        __syncwarp();
                        first = false;
                    }
                }
                parity ^= 1u;
                if (++s == MM_SLOTS) { s = 0; ph ^= 1u; }
                return ok;
            });
            if (ok && leader) umma_commit(tfull + 8 * buf);
            __syncwarp();
        }
    } else if (warp < MM_EPI_WARP0) {
        // ---- operand rows and scales ---------------------------------------------------------------------------------------
        const int team = (warp - 4) / MM_TEAM_WARPS, ut = threadIdx.x - (4 + team * MM_TEAM_WARPS) * 32; // 0 .. 127
        const uint32_t src0 = (uint32_t)ut * 16u; // 16 packed bytes: block ut % 4 of rows ut / 4 + 32 i
        const uint32_t row = (uint32_t)ut >> 2, q = (uint32_t)ut & 3u;
        const uint32_t dst0 = (row >> 3) * 1024u + (row & 7) * 128u, c0 = ((2 * q) ^ (row & 7)) << 4, c1 = ((2 * q + 1) ^ (row & 7)) << 4;
        const uint32_t sf_at = (uint32_t)(ut & 31) * 16u + (uint32_t)(ut >> 5) * 4u; // row ut's scales
        int s = 0;
        uint32_t ph = 0;
        int turn = 0; // of the stages counted so far
        bool ok = true, reused = false; // reused: the slots have been used before
        static_assert(MM_SLOTS == MM_RAW, "one slot counter for both rings");
        for (int u = blockIdx.x; ok && u < n_units; u += gridDim.x) {
            const int tb = u / p.tiles_n, f = u - tb * p.tiles_n;
            const int4 en = ld_produced(p.entries + tb);
            const int n16 = (en.y + 15) & ~15;
            const uint8_t *srow = f * MM_ROWS + ut < p.n ? p.scales + ((size_t)en.z * p.n + f * MM_ROWS + ut) * p.nkb : nullptr;
            // rows of hi, then of lo, in the order of the columns
            const bool has_row = ut < en.y;
            const uint32_t *xrow = p.sfx + en.x + (has_row ? ut : 0);
            const int lo_row = n16 + ut;
            const uint32_t lo_at = (uint32_t)(lo_row & 31) * 16u + (uint32_t)(lo_row >> 5) * 4u;
            ok = mm_stages<SECOND>(p, en, [&](int it, int pair, int kind) {
                if (turn == team) {
                    // the scales come straight from L2 and are asked for ahead of the polls, which hide their latency; past the last
                    // out feature and past k: 1.0 (never used there, but no NaN)
                    uint32_t sa = 0x7F7F7F7Fu;
                    if (srow != nullptr) {
                        const uint8_t *sp = srow + it * 4;
                        if (p.scale_bytes == 4) sa = __ldg(reinterpret_cast<const uint32_t *>(sp));
                        else if (p.scale_bytes == 2) {
                            sa = __ldg(reinterpret_cast<const uint16_t *>(sp));
                            sa |= (it * 4 + 2 < p.nkb ? (uint32_t)__ldg(reinterpret_cast<const uint16_t *>(sp) + 1) : 0x7F7Fu) << 16;
                        } else {
                            sa = 0;
#pragma unroll
                            for (int j = 0; j < 4; j++) sa |= (it * 4 + j < p.nkb ? (uint32_t)__ldg(sp + j) : 127u) << (8 * j);
                        }
                    }
                    uint32_t sx = 0x7F7F7F7Fu;
                    if (has_row && (!SECOND || !pair || ld_produced(p.second + (size_t)it * p.rows_cap + en.x + ut) == kind))
                        sx = ld_produced(xrow + (size_t)(pair * T + it) * p.rows_cap);
                    const bool t0 = mbar_test(rawfull + 8 * s, ph), t1 = !reused || mbar_test(empty + 8 * s, ph ^ 1u);
                    bool ok = t0 || mbar_wait(rawfull + 8 * s, ph, p.flag, MM_CODE + 5);
                    if (ok && !t1) ok = mbar_wait(empty + 8 * s, ph ^ 1u, p.flag, MM_CODE + 6);
                    if (!__all_sync(0xFFFFFFFFu, ok)) return false;
                    const uint32_t src = raw_base + (uint32_t)(s * MM_RAW_BYTES) + src0, dst = base + (uint32_t)(s * MM_A_BYTES) + dst0;
                    uint4 w[4];
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[i].x), "=r"(w[i].y), "=r"(w[i].z), "=r"(w[i].w) : "r"(src + i * 2048u) : "memory");
#pragma unroll
                    for (int i = 0; i < 4; i++) { // 32 rows on: four groups of eight
                        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + i * 4096u + c0), "r"(w[i].x), "r"(w[i].y) : "memory");
                        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + i * 4096u + c1), "r"(w[i].z), "r"(w[i].w) : "memory");
                    }
                    const uint32_t sfs = sf_base + (uint32_t)(s * 2 * MM_SF_BYTES);
                    asm volatile("st.shared.b32 [%0], %1;" ::"r"(sfs + sf_at), "r"(sa) : "memory");
                    if (ut < n16) {
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(sfs + MM_SF_BYTES + sf_at), "r"(sx) : "memory");
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(sfs + MM_SF_BYTES + lo_at), "r"(sx - 0x04040404u) : "memory");
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic-proxy stores -> visible to the MMA
                    __syncwarp();
                    if (lane == 0) {
                        mx_arrive(full + 8 * s);
                        mx_arrive(rawempty + 8 * s);
                    }
                }
                if (++turn == MM_TEAMS) turn = 0;
                if (++s == MM_SLOTS) { s = 0; ph ^= 1u; reused = true; }
                return true;
            });
        }
    } else {
        // ---- epilogue: lane = out feature inside this warp's quarter of the accumulator rows ---------------------------------
        const int quad = warp & 3;
        __nv_bfloat16 *outp = reinterpret_cast<__nv_bfloat16 *>(p.out);
        int ul = 0, before = 0; // stages so far
        for (int u = blockIdx.x; u < n_units; u += gridDim.x, ul++) {
            const int tb = u / p.tiles_n, f = u - tb * p.tiles_n;
            const int4 en = ld_produced(p.entries + tb);
            int here = T;
            if (SECOND) mm_second_stages(p, en, [&](int, int) { here++; return true; });
            const int n16 = (en.y + 15) & ~15, buf = ul & 1;
            const int feat = f * MM_ROWS + quad * 32 + lane;
            const bool fv = feat < p.n;
            const float bv = (p.bias && fv) ? load_as_f32(p.bias, p.bias_dtype, (size_t)en.z * p.n + feat) : 0.0f;
            if (!mx_wait(tfull + 8 * buf, ((uint32_t)ul >> 1) & 1u, p.flag, MM_CODE + 4)) break;
            tc_fence_after();
            const uint32_t t0 = tmem_acc + ((uint32_t)(quad * 32) << 16) + (uint32_t)(2 * buf * MM_ACC_COLS);
            const bool two = here > 1; // a single stage leaves one of the accumulators alone
            const uint32_t ta = two || !(before & 1) ? t0 : t0 + MM_ACC_COLS, tb2 = two ? t0 + MM_ACC_COLS : ta;
            before += here;
            for (int c0 = 0; c0 < n16; c0 += 8) {
                uint32_t a[8], b[8], c[8], e[8];
                tmem_ld_x8(ta + c0, a);
                tmem_ld_x8(ta + n16 + c0, b);
                tmem_ld_x8(tb2 + c0, c);
                tmem_ld_x8(tb2 + n16 + c0, e);
                tmem_ld_wait();
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    v[i] = __uint_as_float(a[i]) + __uint_as_float(b[i]);
                    if (two) v[i] += __uint_as_float(c[i]) + __uint_as_float(e[i]);
                    v[i] += bv;
                }
                if (p.epi == 0) {
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        if (fv && c0 + i < en.y) outp[(size_t)(en.x + c0 + i) * p.ldo + feat] = __float2bfloat16_rn(v[i]);
                } else {
                    // even lane = gate feature, odd lane = up feature of the same output column; the even lane takes the even row of
                    // a pair of rows and the odd lane the odd one, so one exchange serves two rows
                    const bool odd = lane & 1;
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        const float other = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[i] : v[i + 1], 1);
                        float gate = odd ? other : v[i], up = odd ? v[i + 1] : other;
                        gate = fminf(gate, p.limit);
                        up = fminf(fmaxf(up, -p.limit), p.limit);
                        const float sig = __fdividef(1.0f, __expf(-1.702f * gate) + 1.0f);
                        const int rowi = c0 + i + (odd ? 1 : 0);
                        if (fv && rowi < en.y)
                            outp[(size_t)(en.x + rowi) * p.ldo + (feat >> 1)] = __float2bfloat16_rn((up + 1.0f) * (gate * sig));
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mx_arrive(tempty + 8 * buf);
        }
    }
}
// Without and with the code for second pairs, whole: in one loop 340 tokens took 248 us a layer, with what they need in a call 192, as
// two kernels of which one returns at once 181 (50 tokens 139), chosen by a vote, which keeps what the loops compute in uniform registers, 180 (137).
__global__ void __launch_bounds__(MM_THREADS, 1)
    moe_mx_kernel(const MoeMxParams p, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap)
{
    extern __shared__ unsigned char smem_raw[];
    pdl_launch_dependents();
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u; // operand slots want 1 KB alignment
    unsigned char *base_ptr = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + MM_BARS;
    const uint32_t rawfull = bars, rawempty = rawfull + 8 * MM_RAW, full = rawempty + 8 * MM_RAW, empty = full + 8 * MM_SLOTS,
                   tfull = empty + 8 * MM_SLOTS, tempty = tfull + 16;
    volatile uint32_t *tail = reinterpret_cast<volatile uint32_t *>(base_ptr + (bars + 8 * MM_NUM_BARS - base));

    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (warp == 0) {
        if (lane < MM_RAW) {
            mbar_init(rawfull + 8 * lane, 1);
            mbar_init(rawempty + 8 * lane, MM_TEAM_WARPS);
        }
        if (lane < MM_SLOTS) {
            mbar_init(full + 8 * lane, MM_TEAM_WARPS + 1); // the team's warps and the rows' producer
            mbar_init(empty + 8 * lane, 1);
        }
        if (lane < 2) {
            mbar_init(tfull + 8 * lane, 2); // both issuers
            mbar_init(tempty + 8 * lane, MM_EPI_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) { // the allocating warp also frees
        tmem_alloc(bars + 8 * MM_NUM_BARS, 512u);
        tmem_relinquish();
    }
    for (uint32_t i = threadIdx.x; i < MM_SLOTS * MM_A_BYTES / 16; i += MM_THREADS) // the unused half of every operand chunk
        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(base + i * 16u), "r"(0u) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tail[0];
    pdl_wait(); // table, rows and their scales come from kernels ahead; their time must not count as this kernel's waits
    const int n_units = ld_produced(p.n_blocks) * p.tiles_n;
    if (__any_sync(0xFFFFFFFFu, ld_produced(p.any) == p.mark)) moe_mx_roles<true>(p, wmap, xmap, base, tmem_base, n_units);
    else moe_mx_roles<false>(p, wmap, xmap, base, tmem_base, n_units);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512u);
    }
}

static thread_local int g_moe_mx_selftest_skip_loads = 0; // set only inside oxq_selftest_moe_mx_wait_expiry

// Rows of a token block.
int moe_mx_block_rows() { return MM_MAX_TOK; }

// Bytes of both pairs of pieces of `rows` rows, of their block scales, and of what says which have a second pair (the call's mark in front).
size_t moe_mx_piece_bytes(int rows, int k) { return (size_t)4 * rows * k; }
size_t moe_mx_scale_bytes(int rows, int k) { return (size_t)8 * rows * moe_mx_stages(k); }
size_t moe_mx_second_bytes(int rows, int k) { return 16 + (size_t)rows * moe_mx_stages(k); } // (read in words of four)

bool moe_mx_supported(int n, int k, const void *blocks, const void *scales)
{
    // k % 32 == 0: whole MXFP4 blocks, and the packed rows (k / 2 bytes) and the pieces' rows keep the 16-byte pitch a tensor map needs
    return n > 0 && n % 2 == 0 && k >= 32 && k % 32 == 0 && scales != nullptr && aligned(blocks, 16);
}

// Row r of the pieces is src[perm[r] / top_k] (perm null: src[r]), for the rows that total_rows[0] counts, at most `most`.
int moe_mx_split(const void *src, const int *perm, int top_k, const int *total_rows, int most, int k, int rows_cap, void *pieces, void *sfx, void *second,
                 unsigned long long mark, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    const long long blocks = (long long)most * moe_mx_stages(k) * 16 / 256 + 1;
    cfg.gridDim = dim3((unsigned)(blocks < 8 * sm_count() ? blocks : 8 * sm_count()), 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    allow_early_start(attr, cfg.numAttrs);
    OXQ_CUDA(cudaLaunchKernelEx(&cfg, moe_mx_split_kernel, (const __nv_bfloat16 *)src, perm, top_k, total_rows,
                                moe_mx_pieces(k, rows_cap, pieces, sfx, second, mark)));
    return OXQ_OK;
}

// out = epilogue(rows . W_e^T + bias_e) for every token block of the table. epi 0: bias; epi 1: clamped SwiGLU.
int moe_mx_grouped(const void *pieces, const void *sfx, const void *second, unsigned long long mark, int rows_cap, const uint8_t *blocks, const uint8_t *scales, int experts, int n, int k,
                   const int4 *entries, const int *n_blocks, const void *bias, int bias_dtype, void *out, int ldo, int epi, float limit,
                   int *flag, cudaStream_t st)
{
    MoeMxParams p = {};
    p.entries = entries; p.n_blocks = n_blocks; p.scales = scales; p.sfx = (const uint32_t *)sfx; p.bias = bias; p.out = out; p.flag = flag;
    p.pieces = (const unsigned char *)pieces; p.any = (const unsigned long long *)second; p.second = (const unsigned char *)second + 8; p.mark = mark;
    p.n = n; p.k = k; p.nkb = k / 32; p.stages = moe_mx_stages(k); p.rows_cap = rows_cap;
    p.scale_bytes = p.nkb % 4 == 0 && aligned(scales, 4) ? 4 : p.nkb % 2 == 0 && aligned(scales, 2) ? 2 : 1;
    p.tiles_n = (n + MM_ROWS - 1) / MM_ROWS;
    p.bias_dtype = bias_dtype; p.ldo = ldo; p.epi = epi; p.limit = limit;
    p.test_skip_loads = g_moe_mx_selftest_skip_loads;
    CUtensorMap wmap, xmap;
    CUresult r = encode_tiled_2d(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, blocks, (uint64_t)k / 2, (uint64_t)experts * n, (uint64_t)k / 2,
                                 MM_BK / 2, MM_ROWS, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (expert blocks) failed with CUresult %d", (int)r);
    r = encode_tiled_2d(&xmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, pieces, (uint64_t)k, (uint64_t)2 * rows_cap, (uint64_t)k, MM_BK, MM_XBOX_ROWS,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (expert rows) failed with CUresult %d", (int)r);
    static size_t configured[64] = {};
    int device = 0;
    OXQ_CUDA(cudaGetDevice(&device));
    if (device >= 64 || configured[device] < MM_SMEM) {
        OXQ_CUDA(cudaFuncSetAttribute(moe_mx_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MM_SMEM));
        if (device < 64) configured[device] = MM_SMEM;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count(), 1, 1);
    cfg.blockDim = dim3(MM_THREADS, 1, 1);
    cfg.dynamicSmemBytes = MM_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    allow_early_start(attr, cfg.numAttrs);
    OXQ_CUDA(cudaLaunchKernelEx(&cfg, moe_mx_kernel, p, wmap, xmap));
    return OXQ_OK;
}

} // namespace oxq

// Self-test of the kernel's abort path: one unit (one expert, 128 out features, 128 in features, 16 rows) whose weights never come. The
// operand team, the issuers, the last waits of the rows' producer and the epilogue warps each give up after their two seconds, side
// by side, the flag word takes the first code, tensor memory is freed and the kernel returns with no copy in flight.
OXQ_EXPORT int oxq_selftest_moe_mx_wait_expiry(void *workspace, size_t workspace_bytes, void *stream)
{
    oxq::clear_error();
    OXQ_REQUIRE(workspace && workspace_bytes >= (1u << 20) && oxq::aligned(workspace, 256), OXQ_ERR_WORKSPACE,
                "oxq_selftest_moe_mx_wait_expiry: 256-byte aligned workspace of at least 1 MiB needed");
    unsigned char *b = reinterpret_cast<unsigned char *>(workspace);
    cudaStream_t st = (cudaStream_t)stream;
    const int n = 128, k = 128, rows = 16, cap = 64;
    // table, no second pairs | pieces [2, 2, 64, 128] | their scales | blocks [128, 64] | scales [128, 4] | out [16, 128] bf16, 64 KB apart
    int4 *entries = reinterpret_cast<int4 *>(b + 4096);
    int *n_blocks = reinterpret_cast<int *>(b + 4096 + 64);
    const int4 en = make_int4(0, rows, 0, 0);
    const int one = 1;
    OXQ_CUDA(cudaMemcpyAsync(entries, &en, sizeof(en), cudaMemcpyHostToDevice, st));
    OXQ_CUDA(cudaMemcpyAsync(n_blocks, &one, sizeof(one), cudaMemcpyHostToDevice, st));
    OXQ_CUDA(cudaStreamSynchronize(st)); // the two host words above live on this stack frame
    oxq::g_moe_mx_selftest_skip_loads = 1;
    const int rc = oxq::moe_mx_grouped(b + (1 << 16), b + (2 << 16), b + 8192, oxq::mx_call_mark(), cap, b + (3 << 16), b + (4 << 16), 1, n, k, entries, n_blocks, nullptr, 0,
                                       b + (5 << 16), n, 0, 0.0f, reinterpret_cast<int *>(workspace), st);
    oxq::g_moe_mx_selftest_skip_loads = 0;
    return rc;
}
