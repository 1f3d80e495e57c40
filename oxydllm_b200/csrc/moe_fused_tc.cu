// Grouped expert matmul of the GPT-OSS MoE layer on MXFP4 weights, with the dequantization inside the
// tensor-core kernel: the packed blocks are read once and no dense copy of the expert weights is written.
// Mirrors the expert half of MoeFeedForward::forward (moe.rs:466-499, dispatch_sparse 563-607) with the
// experts' Mxfp4Linear weights (linear.rs, [experts, out, in / 32, 16] blocks + [experts, out, in / 32] scales).
//
// A unit of work is (token block of one expert: up to 192 or 256 expert-sorted rows) x (128 out features). The grid is
// persistent: CTA b takes units b, b + grid, ... of a device-side table, feature tiles fastest, so that CTAs
// running at the same time share their token block in L2. Stages of 64 input columns are counted over all units of
// a CTA and go round eight slots (blocks of up to 192 rows) or six. Per CTA:
//   warp 0              TMA: boxes of packed nibbles (128 out features x 32 bytes);
//   warp 2              TMA: the stage's tile of the activations ([rows, 64] bf16 in boxes of 64 rows, 128-byte swizzle);
//   warps 4..19         unpack, four teams of four warps taking stages in turn: a thread turns the two 16-byte blocks
//                       (32 weights each; E8M0 scale bytes read through L1/L2) of one out feature into bf16 weights, the bits the
//                       dequantization kernel writes, and stores them as 32 columns of its lane of tensor memory, where the
//                       team has room for one stage;
//   warp 1              tcgen05.mma kind::f16, A = weights [128, 64] from tensor memory, B = activations, D[128, rows] f32 in tensor
//                       memory for the whole of k; the accumulators of successive units follow one another round a ring of six
//                       chunks of 64 columns (two MMAs where one crosses its end); one commit per stage frees its slot and its weights;
//   warps 20..23        epilogue of the previous unit while the next one accumulates: accumulator rows (out
//                       features) -> + bias -> bf16 out[row, feature], or the clamped SwiGLU of GPT-OSS on
//                       interleaved (gate, up) features -> out[row, feature / 2].
// What bounds it: the unpack, about 640 clocks per stage for 350 of MMA at 176 rows. With the weights in shared memory a stage of 256 rows
// moved 104 KB through it at 128 bytes a clock, 812 clocks for 512 of MMA, and a team could not start before its slot was free; now only
// the store waits for that. The weights of four stages take 128 columns of tensor memory, which leaves 384 for accumulators: two of 192
// columns. A stage costs the unpack whatever its rows, so that an expert of 193 to 256 rows wants one block: the epilogue of 256 rows
// takes about 8000 clocks, and hands back its columns a chunk at a time, so that the next block of 256 starts when half of it is done.
// us a layer at 400 / 1024 / 1600 / 1800 / 3300 / 4096 tokens, 32 experts of 2880 x 2880: weights in shared memory, blocks of 256 rows
// 236 / 283 / 338 / 374 / 655 / 784; blocks of 192 only 200 / 242 / 376 / 418 / 669 / 759; now 197 / 246 / 341 / 373 / 628 / 754.
// 16 of 2048 x 1024 at 900 tokens 102 / 104 / 97. Scale bytes a stage ahead and a swizzle against the bank conflicts of the packed rows
// gave nothing more; nor did a ring of 192-row entries of which a larger block takes two, up to 384 rows: with two accumulators at
// once nothing hides the epilogue (4096 tokens 850).
// Every wait is bounded and reports through the workspace flag word.
#include <type_traits>

#include <cuda_bf16.h>

#include "mx_common.cuh"

namespace oxq {

#ifdef OXQ_TUNING
#define MF_DBG(bit) (p.dbg & (bit))
__device__ long long g_mf_trace[10][256]; // clock stamps of CTA 0, per role and stage (tuning builds only)
#define MF_TRACE(role, it) do { if (blockIdx.x == 0 && (it) < 256) g_mf_trace[role][it] = clock64(); } while (0)
#else
#define MF_DBG(bit) 0
#define MF_TRACE(role, it) do { } while (0)
#endif

constexpr int MF_ROWS = 128;                   // out features per unit
constexpr int MF_BK = 64;                      // input columns per stage
constexpr int MF_UNPACK_WARPS = 16, MF_TEAMS = 4, MF_TEAM_WARPS = 4; // four teams: a stage's chain of poll, unpack and arrival overlaps with three others
constexpr int MF_EPI_WARPS = 4;
constexpr int MF_THREADS = (4 + MF_UNPACK_WARPS + MF_EPI_WARPS) * 32;
// Stages on their way (packed weights and activations, barriers) for blocks of at most MAX_TOK rows: as many as shared memory holds.
template <int MAX_TOK> constexpr int MF_SLOTS = MAX_TOK <= 192 ? 8 : 6;
constexpr int MF_CHUNKS = 6, MF_CHUNK = 64;    // accumulator columns are a ring of chunks
constexpr int MF_TMEM_A = MF_CHUNKS * MF_CHUNK, MF_A_COLS = MF_BK / 2; // a team's unpacked weights, two to a column
constexpr int MF_XBOX_ROWS = 64, MF_XBOX_BYTES = MF_XBOX_ROWS * MF_BK * 2; // activation rows travel in boxes of 64
constexpr int MF_RAW_BYTES = MF_ROWS * MF_BK / 2;
static_assert(MF_TMEM_A + MF_TEAMS * MF_A_COLS <= 512, "tensor memory");
static_assert(MF_SLOTS<256> > MF_TEAMS, "the slot of a team's stage before is another one");
constexpr int MF_SMEM_BUDGET = 227 * 1024;

struct MoeFusedParams {
    const int4 *entries;   // token blocks: {first row in the expert-sorted matrix, rows, expert, -}
    const int *n_blocks;   // how many
    const uint8_t *scales; // [experts, n, k / 32]
    const void *bias;      // [experts, n] or null
    void *out;
    int *flag;
    int n, k, nkb, nk2;    // out features per expert, in features, scale bytes per row, stages per unit
    int tiles_n, bias_dtype, ldo, epi;
    float limit;
    int dbg;               // tuning builds: parts of the pipeline switched off for timing
    int test_skip_loads;   // self-test only: the weight producer issues nothing, so the waits of the other roles run out
};

__device__ __forceinline__ uint4 mf_lds128(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
// 32 columns of this warp's quarter of tensor memory.
__device__ __forceinline__ void mf_tmem_st32(uint32_t taddr, const uint32_t (&r)[32])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                 "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
                 "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
                 "r"(r[30]), "r"(r[31])
                 : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc], bf16 x bf16 -> f32; lane i of A's columns is row i, a column two elements of k.
__device__ __forceinline__ void mf_umma(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void mf_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

template <int MAX_TOK>
__global__ void __launch_bounds__(MF_THREADS, 1)
    moe_mxfp4_fused_kernel(const MoeFusedParams p, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap)
{
    constexpr int SLOTS = MF_SLOTS<MAX_TOK>, X_BYTES = MAX_TOK * MF_BK * 2, NUM_BARS = 4 * SLOTS + 2 * MF_CHUNKS;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u; // operand slots want 1 KB alignment
    unsigned char *base_ptr = smem_raw + (base - smem_u32(smem_raw));
    // activation slots | packed slots | barriers | tensor-memory address
    const uint32_t x_base = base, raw_base = base + SLOTS * X_BYTES;
    const uint32_t bars = raw_base + SLOTS * MF_RAW_BYTES;
    auto rawfull_bar = [&](int r) { return bars + 8u * r; };
    auto rawempty_bar = [&](int r) { return bars + 8u * (SLOTS + r); };
    // full: the stage's weights are in tensor memory (one arrival per warp of the team) and its activation tile has landed (the
    // producer's arrival with the byte count); empty: the MMAs that read both have completed (one commit)
    auto full_bar = [&](int s) { return bars + 8u * (2 * SLOTS + s); };
    auto empty_bar = [&](int s) { return bars + 8u * (3 * SLOTS + s); };
    const uint32_t misc = bars + 8u * (4 * SLOTS);
    // per chunk: the accumulator that begins there is complete (one commit); the chunk has been read
    auto tfull_bar = [&](int c) { return misc + 8u * c; };
    auto tempty_bar = [&](int c) { return misc + 8u * (MF_CHUNKS + c); };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(base_ptr + (bars - base) + 8 * NUM_BARS);

    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int n_units = __ldg(p.n_blocks) * p.tiles_n;
    const int nk2 = p.nk2;

    if (threadIdx.x == 0) {
        for (int s = 0; s < SLOTS; s++) {
            mbar_init(rawfull_bar(s), 1);
            mbar_init(rawempty_bar(s), MF_TEAM_WARPS);
            mbar_init(full_bar(s), MF_TEAM_WARPS + 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < MF_CHUNKS; b++) {
            mbar_init(tfull_bar(b), 1);
            mbar_init(tempty_bar(b), MF_EPI_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) { // the allocating warp also frees
        tmem_alloc(smem_u32(tmem_slot), 512u);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // The single-thread roles run as whole warps with one elected lane at the instruction itself: loop counters, addresses and
    // descriptors stay in uniform registers (with the loop inside the elected branch an MMA takes 90 clocks to issue).
    if (warp == 0) {
        // ---- TMA, packed nibbles -----------------------------------------------------------------------
        const bool leader = elect_one();
        int r = 0;
        uint32_t ph = 1; // a fresh barrier passes parity 1
        bool ok = true;
        for (int u = blockIdx.x; ok && u < n_units && !p.test_skip_loads; u += gridDim.x) {
            const int tb = u / p.tiles_n, f = u - tb * p.tiles_n;
            const int rowbase = __ldg(p.entries + tb).z * p.n + f * MF_ROWS;
            for (int it = 0; it < nk2 && ok; it++) {
                ok = mx_wait(rawempty_bar(r), ph, p.flag, 1);
                if (ok && leader) {
                    mbar_arrive_expect_tx(rawfull_bar(r), MF_RAW_BYTES);
                    tma_load_2d(raw_base + r * MF_RAW_BYTES, &wmap, rawfull_bar(r), it * (MF_BK / 2), rowbase);
                }
                __syncwarp();
                if (++r == SLOTS) { r = 0; ph ^= 1u; }
            }
        }
    } else if (warp == 2) {
        // ---- TMA, activation tiles ----------------------------------------------------------------------
        const bool leader = elect_one();
        int xs = 0;
        uint32_t xph = 1;
        bool ok = true;
        for (int u = blockIdx.x; ok && u < n_units; u += gridDim.x) {
            const int4 en = __ldg(p.entries + u / p.tiles_n);
            const int boxes = (en.y + MF_XBOX_ROWS - 1) / MF_XBOX_ROWS;
            for (int it = 0; it < nk2 && ok; it++) {
                ok = mx_wait(empty_bar(xs), xph, p.flag, 5);
                if (ok && leader) {
                    const uint32_t dst = x_base + (uint32_t)xs * X_BYTES;
                    mbar_arrive_expect_tx(full_bar(xs), (uint32_t)boxes * MF_XBOX_BYTES);
#pragma unroll
                    for (int b = 0; b < MAX_TOK / MF_XBOX_ROWS; b++)
                        if (b < boxes)
                            tma_load_2d(dst + (uint32_t)b * MF_XBOX_BYTES, &xmap, full_bar(xs), it * MF_BK, en.x + b * MF_XBOX_ROWS);
                }
                __syncwarp();
                if (++xs == SLOTS) { xs = 0; xph ^= 1u; }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issue ----------------------------------------------------------------------------------
        // One warp issues every MMA of the CTA, so its instruction count per stage is on the critical path: one poll (full) and one
        // commit (empty) per stage.
        const bool leader = elect_one();
        const uint64_t db0 = kmajor_sw128_desc(x_base);
        int s = 0, team = 0, chunk = 0; // slot of a stage, team that unpacks it; first chunk of a unit
        uint32_t ph = 0, cph = ~0u;     // bit c: parity of chunk c's last release (a fresh barrier passes 1)
        bool ok = true;
        for (int u = blockIdx.x; ok && u < n_units; u += gridDim.x) {
            // (shuffled: known to be the same in all lanes, so that what depends on it stays in uniform registers)
            const int mpad = __shfl_sync(0xFFFFFFFFu, (__ldg(p.entries + u / p.tiles_n).y + 15) & ~15, 0);
            const int n1 = min(mpad, (MF_CHUNKS - chunk) * MF_CHUNK), n2 = mpad - n1; // columns up to the ring's end, and from its start on
            const uint32_t idesc = tc_idesc(MF_ROWS, n1), idesc2 = tc_idesc(MF_ROWS, n2 ? n2 : 16), d_tmem = tmem_base + (uint32_t)(chunk * MF_CHUNK);
            const int first = chunk;
            bool free_all = true; // the polls of all chunks are under way together
            for (int c0 = 0; c0 < mpad; c0 += MF_CHUNK) {
                free_all &= mbar_test(tempty_bar(chunk), (cph >> chunk) & 1u);
                cph ^= 1u << chunk;
                if (++chunk == MF_CHUNKS) chunk = 0;
            }
            if (!__all_sync(0xFFFFFFFFu, free_all))
                for (int c0 = 0, c = first; c0 < mpad && ok; c0 += MF_CHUNK, c = c + 1 == MF_CHUNKS ? 0 : c + 1)
                    ok = mx_wait(tempty_bar(c), (~cph >> c) & 1u, p.flag, 8);
            auto stages = [&](auto split_) {
                for (int it = 0; it < nk2 && ok; it++) {
                    ok = mx_wait(full_bar(s), ph, p.flag, 2);
                    if (ok) {
                        tc_fence_after();
                        const uint32_t a_tmem = tmem_base + MF_TMEM_A + (uint32_t)team * MF_A_COLS;
                        const uint64_t db = db0 + (uint64_t)(s * (X_BYTES >> 4));
                        if (leader) {
#pragma unroll
                            for (int kk = 0; kk < MF_BK / 16; kk++) { // 16 input columns: 32 bytes inside a swizzled K-major row
                                mf_umma(d_tmem, a_tmem + 8 * kk, db + 2 * kk, idesc, (it | kk) != 0);
                                if constexpr (decltype(split_)::value)
                                    mf_umma(tmem_base, a_tmem + 8 * kk, db + (uint64_t)(n1 * (MF_BK * 2 >> 4)) + 2 * kk, idesc2, (it | kk) != 0);
                            }
                            umma_commit(empty_bar(s));
                        }
                        __syncwarp();
                    }
                    if (++team == MF_TEAMS) team = 0;
                    if (++s == SLOTS) { s = 0; ph ^= 1u; }
                }
            };
            if (n2) stages(std::true_type{});
            else stages(std::false_type{});
            if (ok && leader) umma_commit(tfull_bar(first)); // the accumulator is complete once the unit's MMAs are
            __syncwarp();
        }
    } else if (warp >= 4 && warp < 4 + MF_UNPACK_WARPS) {
        // ---- unpack ---------------------------------------------------------------------------------------
        const int team = (warp - 4) / MF_TEAM_WARPS;
        const int ut = (threadIdx.x - 128) % (MF_TEAM_WARPS * 32);
        const int row = ut;                                       // this thread: both 16-byte blocks of one out feature per stage
        static_assert(MF_TEAM_WARPS * 32 == MF_ROWS, "a thread per out feature");
        const uint32_t raw_addr = raw_base + (uint32_t)row * 32u;
        const uint32_t a_tmem = tmem_base + ((uint32_t)(warp & 3) << 21) + MF_TMEM_A + (uint32_t)team * MF_A_COLS; // the team's four warps: one quarter each
        int my_units = 0;
        if ((int)blockIdx.x < n_units) my_units = (n_units - 1 - (int)blockIdx.x) / (int)gridDim.x + 1;
        const uint32_t total = (uint32_t)my_units * (uint32_t)nk2;
        // every counter steps along (divisions by the stages of a unit were a third of a stage's instructions)
        int u = (int)blockIdx.x, it = team;
        uint32_t s = (uint32_t)team, ph = 0, prev = 0, prev_ph = 0; // this stage's slot and its parity; those of the team's stage before
        const uint8_t *srow = nullptr;
        auto unit_scales = [&]() { // this thread's row of the scale bytes
            if (u >= n_units) return;
            const int tb = u / p.tiles_n, f = u - tb * p.tiles_n;
            const int e = __ldg(p.entries + tb).z;
            srow = (f * MF_ROWS + row < p.n) ? p.scales + ((size_t)e * p.n + f * MF_ROWS + row) * p.nkb : nullptr;
        };
        while (it >= nk2) { it -= nk2; u += (int)gridDim.x; }
        unit_scales();
        bool ok = true;
        for (uint32_t g = (uint32_t)team; g < total; g += MF_TEAMS) {
            // the scale bytes of the stage's two blocks come straight from L2 (the row's bytes are neighbours, so most loads
            // hit L1); they are asked for before the polls, which hide their latency. Past k (zero-filled boxes) and past the
            // expert's last out feature: 1.0
            const int kb0 = it * 2;
            uint32_t sbv[2];
#pragma unroll
            for (int h = 0; h < 2; h++) sbv[h] = (srow != nullptr && kb0 + h < p.nkb) ? (uint32_t)__ldg(srow + kb0 + h) : 127u;
            // both polls first (they do not depend on each other), the bounded waits only where one failed
            // The team's stage before this one has been multiplied. (The barrier cannot be a phase further: its slot's next stage is
            // multiplied after this one.)
            const uint32_t prev_empty = empty_bar((int)prev);
            const bool tr = mbar_test(rawfull_bar((int)s), ph);
            bool free_a = g < MF_TEAMS || mbar_test(prev_empty, prev_ph);
            free_a = __all_sync(0xFFFFFFFFu, free_a);
            ok = __all_sync(0xFFFFFFFFu, tr) || mx_wait(rawfull_bar((int)s), ph, p.flag, 3);
            if (!ok) break;
            if (ut == 0) MF_TRACE(4, g);
            uint4 rawv[2];
#pragma unroll
            for (int half = 0; half < 2; half++) rawv[half] = mf_lds128(raw_addr + s * MF_RAW_BYTES + 16u * half);
            uint32_t o[MF_A_COLS]; // the row's weights, two to a word
#pragma unroll
            for (int half = 0; half < 2; half++) {
                const uint32_t sb = sbv[half];
                const uint32_t v[4] = {rawv[half].x, rawv[half].y, rawv[half].z, rawv[half].w};
                if (sb >= 4u && sb <= 250u) { // 2^(s-127) as a bf16 pair: the products are exact
                    // The block's eight magnitudes 0, .5, 1, 1.5, 2, 3, 4, 6 times its scale, as bf16 (four multiplies for
                    // 32 weights), split into a table of low bytes and a table of high bytes; the byte permute unit then looks
                    // up four nibbles at a time, and the nibbles' sign bits go into the high bytes, four at a time, before
                    // high and low bytes are paired.
                    const uint32_t s2 = (sb << 7) | (sb << 23);
                    const __nv_bfloat162 sc = *reinterpret_cast<const __nv_bfloat162 *>(&s2);
                    const uint32_t mags[4] = {0x3F000000u, 0x3FC03F80u, 0x40404000u, 0x40C04080u}; // (0, .5) (1, 1.5) (2, 3) (4, 6)
                    uint32_t pm[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const __nv_bfloat162 t = __hmul2(*reinterpret_cast<const __nv_bfloat162 *>(&mags[i]), sc);
                        pm[i] = *reinterpret_cast<const uint32_t *>(&t);
                    }
                    const uint32_t tlo_a = __byte_perm(pm[0], pm[1], 0x6420u), thi_a = __byte_perm(pm[0], pm[1], 0x7531u);
                    const uint32_t tlo_b = __byte_perm(pm[2], pm[3], 0x6420u), thi_b = __byte_perm(pm[2], pm[3], 0x7531u);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const uint32_t w = v[q];
                        const uint32_t sel_l = w & 0x77777777u, sel_h = sel_l >> 16, wl = w << 4;
                        const uint32_t lo_a = __byte_perm(tlo_a, tlo_b, sel_l), lo_b = __byte_perm(tlo_a, tlo_b, sel_h);
                        uint32_t hi_a = __byte_perm(thi_a, thi_b, sel_l), hi_b = __byte_perm(thi_a, thi_b, sel_h);
                        // bit 7 of byte i <- sign of nibble i (4 + i): even nibbles from w << 4, odd ones from w
                        const uint32_t sg_a = __byte_perm(wl, w, 0x5140u), sg_b = __byte_perm(wl, w, 0x7362u);
                        asm("lop3.b32 %0, %1, %2, %0, 0x6A;" : "+r"(hi_a) : "r"(sg_a), "r"(0x80808080u)); // (sg & mask) ^ hi
                        asm("lop3.b32 %0, %1, %2, %0, 0x6A;" : "+r"(hi_b) : "r"(sg_b), "r"(0x80808080u));
                        o[half * 16 + q * 4] = __byte_perm(lo_a, hi_a, 0x5140u);
                        o[half * 16 + q * 4 + 1] = __byte_perm(lo_a, hi_a, 0x7362u);
                        o[half * 16 + q * 4 + 2] = __byte_perm(lo_b, hi_b, 0x5140u);
                        o[half * 16 + q * 4 + 3] = __byte_perm(lo_b, hi_b, 0x7362u);
                    }
                } else { // scales whose products leave the normal range (NaN, 2^-127 among them): f32 product, one rounding
                    const float s = e8m0_to_f32(sb);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
#pragma unroll
                        for (int b = 0; b < 4; b++) {
                            const uint32_t by = (v[q] >> (8 * b)) & 0xFFu;
                            const __nv_bfloat162 hh = __halves2bfloat162(narrow<__nv_bfloat16>(__fmul_rn(e2m1_to_f32(by & 0xFu), s)),
                                                                         narrow<__nv_bfloat16>(__fmul_rn(e2m1_to_f32(by >> 4), s)));
                            o[half * 16 + q * 4 + b] = *reinterpret_cast<const uint32_t *>(&hh);
                        }
                    }
                }
            }
            if (ut == 0) MF_TRACE(5, g);
            __syncwarp();
            if (lane == 0) mf_arrive(rawempty_bar((int)s));
            if (!free_a) ok = mx_wait(prev_empty, prev_ph, p.flag, 7);
            if (!ok) break;
            tc_fence_after();
            mf_tmem_st32(a_tmem, o);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mf_arrive(full_bar((int)s));
            if (ut == 0) MF_TRACE(6, g);
            prev = s;
            prev_ph = ph;
            s += MF_TEAMS;
            if (s >= SLOTS) { s -= SLOTS; ph ^= 1u; }
            it += MF_TEAMS;
            if (it >= nk2) { // the next unit (stages are counted on: slots and teams keep alternating)
                do { it -= nk2; u += (int)gridDim.x; } while (it >= nk2);
                unit_scales();
            }
        }
    } else if (warp >= 4 + MF_UNPACK_WARPS) {
        // ---- epilogue: lane = out feature inside this warp's quarter of the accumulator rows ---------------
        const int quad = warp & 3;
        int chunk = 0;
        uint32_t fph = 0; // bit c: parity of the next accumulator that begins at chunk c
        __nv_bfloat16 *outp = reinterpret_cast<__nv_bfloat16 *>(p.out);
        bool ok = true;
        for (int u = blockIdx.x; ok && u < n_units; u += gridDim.x) {
            const int tb = u / p.tiles_n, f = u - tb * p.tiles_n;
            const int4 en = __ldg(p.entries + tb);
            ok = mbar_wait(tfull_bar(chunk), (fph >> chunk) & 1u, p.flag, 4);
            if (!ok) break;
            fph ^= 1u << chunk;
            tc_fence_after();
            const int feat = f * MF_ROWS + quad * 32 + lane;
            const bool fv = feat < p.n;
            const float bv = (p.bias && fv) ? load_as_f32(p.bias, p.bias_dtype, (size_t)en.z * p.n + feat) : 0.0f;
            for (int c0 = 0; c0 < en.y; c0 += 32) {
                uint32_t rr[32];
                tmem_ld32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(chunk * MF_CHUNK + (c0 & (MF_CHUNK - 1))), rr);
                tmem_ld_wait();
                if (p.epi == 0) {
#pragma unroll
                    for (int c = 0; c < 32; c++)
                        if (fv && c0 + c < en.y)
                            outp[(size_t)(en.x + c0 + c) * p.ldo + feat] = __float2bfloat16_rn(__uint_as_float(rr[c]) + bv);
                } else {
                    // even lane = gate feature, odd lane = up feature of the same output column; the even lane takes the
                    // even row of a pair of rows and the odd lane the odd one, so one exchange serves two rows
                    const bool odd = lane & 1;
#pragma unroll
                    for (int c = 0; c < 32; c += 2) {
                        const float mine0 = __uint_as_float(rr[c]) + bv, mine1 = __uint_as_float(rr[c + 1]) + bv;
                        const float other = __shfl_xor_sync(0xFFFFFFFFu, odd ? mine0 : mine1, 1);
                        float gate = odd ? other : mine0, up = odd ? mine1 : other;
                        gate = fminf(gate, p.limit);
                        up = fminf(fmaxf(up, -p.limit), p.limit);
                        const float sig = __fdividef(1.0f, __expf(-1.702f * gate) + 1.0f);
                        const int rowi = c0 + c + (odd ? 1 : 0);
                        if (fv && rowi < en.y)
                            outp[(size_t)(en.x + rowi) * p.ldo + (feat >> 1)] = __float2bfloat16_rn((up + 1.0f) * (gate * sig));
                    }
                }
                if ((c0 & 32) || c0 + 32 >= en.y) { // the chunk has been read
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mf_arrive(tempty_bar(chunk));
                    if (++chunk == MF_CHUNKS) chunk = 0;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512u);
    }
}

static thread_local int g_moe_selftest_skip_loads = 0; // set only inside oxq_selftest_moe_wait_expiry

// Rows of the largest token block, for `rows` rows an expert on average: the plan cuts an expert's rows into blocks of at most 192, but where
// 256 are allowed and 1 to 64 would be left over it makes one block of more than 192 instead of two. That form has six slots instead
// of eight, so it is for averages at which many experts are there, us with 192 / 256, 32 experts of 2880 x 2880 at 32, 128, 175, 200, 225, 244,
// 256, 300, 375, 412, 437, 475, 512 rows: 197 / 212, 246 / 253, 299 / 298, 374 / 341, 415 / 373, 433 / 413, 448 / 444, 483 / 489, 579 / 568,
// 681 / 628, 701 / 678, 726 / 736, 754 / 760; 16 of 2048 x 1024 at 225, 250: 104 / 97, 110 / 122.
int moe_fused_block_rows(int rows)
{
    const int over = rows % 192;
    return rows >= 176 && (over < 56 || over >= 176) ? 256 : 192;
}

// True when the fused grouped kernel serves these expert weights; otherwise the caller dequantizes expert groups.
bool moe_fused_supported(int n, int k, const void *blocks, const void *scales, const void *a, const void *out, int ldo)
{
    if (const char *env = tuning_env("OXQ_MOE_FUSED"))
        if (env[0] == '0') return false;
    // k % 32 == 0: whole MXFP4 blocks, and the packed rows (k / 2 bytes) keep the 16-byte pitch a tensor map needs
    if (n <= 0 || k <= 0 || k % 32 != 0 || n % 2 != 0 || scales == nullptr) return false;
    return aligned(blocks, 16) && aligned(a, 16) && aligned(out, 2) && ldo > 0;
}

template <int MAX_TOK>
static int moe_fused_launch(const void *a, int a_rows, const uint8_t *blocks, const uint8_t *scales, int experts, int n, int k,
                            const int4 *entries, const int *n_blocks, const void *bias, int bias_dtype, void *out, int ldo, int epi,
                            float limit, int *flag, cudaStream_t st)
{
    auto kern = moe_mxfp4_fused_kernel<MAX_TOK>;
    MoeFusedParams p = {};
    p.entries = entries; p.n_blocks = n_blocks; p.scales = scales; p.bias = bias; p.out = out; p.flag = flag;
    p.n = n; p.k = k; p.nkb = k / 32;
    const int nk = (k + MF_BK - 1) / MF_BK;
    p.nk2 = nk;
    p.tiles_n = (n + MF_ROWS - 1) / MF_ROWS;
    p.bias_dtype = bias_dtype; p.ldo = ldo; p.epi = epi; p.limit = limit;
    p.test_skip_loads = g_moe_selftest_skip_loads;
    if (const char *env = tuning_env("OXQ_MF_DBG")) p.dbg = atoi(env);
    constexpr size_t smem = 1024 + MF_SLOTS<MAX_TOK> * (MAX_TOK * MF_BK * 2 + MF_RAW_BYTES) + 8 * (4 * MF_SLOTS<MAX_TOK> + 2 * MF_CHUNKS) + 16;
    static_assert(smem <= (size_t)MF_SMEM_BUDGET, "the slots must fit one CTA's shared memory");
    CUtensorMap wmap, xmap;
    CUresult r = encode_tiled_2d(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, blocks, (uint64_t)k / 2, (uint64_t)experts * n, (uint64_t)k / 2,
                                 MF_BK / 2, MF_ROWS, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (expert blocks) failed with CUresult %d", (int)r);
    r = encode_tiled_2d(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a, (uint64_t)k, (uint64_t)a_rows, (uint64_t)k * 2, MF_BK, MF_XBOX_ROWS,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (expert rows) failed with CUresult %d", (int)r);
    static size_t configured[64] = {};
    int device = 0;
    OXQ_CUDA(cudaGetDevice(&device));
    if (device >= 64 || configured[device] < smem) {
        OXQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (device < 64) configured[device] = smem;
    }
    kern<<<sm_count(), MF_THREADS, smem, st>>>(p, wmap, xmap);
    OXQ_LAUNCH_CHECK("moe_mxfp4_fused_kernel");
    return OXQ_OK;
}

// out = epilogue(a . W_e^T + bias_e) for every token block of the table: a = expert-sorted activations [a_rows, k] bf16,
// blocks / scales = the MXFP4 weights of all `experts` experts, n out features each. epi 0: bias; epi 1: clamped SwiGLU.
int moe_fused_grouped(const void *a, int a_rows, const uint8_t *blocks, const uint8_t *scales, int experts, int n, int k,
                      const int4 *entries, const int *n_blocks, int block_rows, const void *bias, int bias_dtype, void *out, int ldo,
                      int epi, float limit, int *flag, cudaStream_t st)
{
    return block_rows <= 192 ? moe_fused_launch<192>(a, a_rows, blocks, scales, experts, n, k, entries, n_blocks, bias, bias_dtype, out, ldo, epi, limit, flag, st)
                             : moe_fused_launch<256>(a, a_rows, blocks, scales, experts, n, k, entries, n_blocks, bias, bias_dtype, out, ldo, epi, limit, flag, st);
}

} // namespace oxq

// Self-test of the grouped kernel's abort path: one unit (one expert, 128 out features, 64 in features, 16 rows) whose
// weight producer never loads. The unpack teams, the MMA issuer, the activation producer and the epilogue warps each give
// up on their bounded wait (about two seconds, side by side), the flag word of the workspace takes the first code,
// tensor memory is freed and the kernel returns; oxq_gemm_check(workspace) then reports it. Nothing faults or hangs.
OXQ_EXPORT int oxq_selftest_moe_wait_expiry(void *workspace, size_t workspace_bytes, void *stream)
{
    oxq::clear_error();
    OXQ_REQUIRE(workspace && workspace_bytes >= (1u << 20) && oxq::aligned(workspace, 256), OXQ_ERR_WORKSPACE,
                "oxq_selftest_moe_wait_expiry: 256-byte aligned workspace of at least 1 MiB needed");
    unsigned char *b = reinterpret_cast<unsigned char *>(workspace);
    cudaStream_t st = (cudaStream_t)stream;
    const int n = 128, k = 64, rows = 16;
    // table | rows [256 + 128, 64] bf16 | blocks [128, 32] | scales [128, 2] | out [256, 128] bf16
    int4 *entries = reinterpret_cast<int4 *>(b + 4096);
    int *n_blocks = reinterpret_cast<int *>(b + 4096 + 64);
    void *a = b + 8192;
    uint8_t *blocks = b + 8192 + 384 * 64 * 2, *scales = blocks + 128 * 32;
    void *out = b + 131072;
    const int4 en = make_int4(0, rows, 0, 0);
    const int one = 1;
    OXQ_CUDA(cudaMemcpyAsync(entries, &en, sizeof(en), cudaMemcpyHostToDevice, st));
    OXQ_CUDA(cudaMemcpyAsync(n_blocks, &one, sizeof(one), cudaMemcpyHostToDevice, st));
    OXQ_CUDA(cudaStreamSynchronize(st)); // the two host words above live on this stack frame
    oxq::g_moe_selftest_skip_loads = 1;
    const int rc = oxq::moe_fused_grouped(a, 384, blocks, scales, 1, n, k, entries, n_blocks, 192, nullptr, 0, out, n, 0, 0.0f,
                                          reinterpret_cast<int *>(workspace), st);
    oxq::g_moe_selftest_skip_loads = 0;
    return rc;
}

#ifdef OXQ_TUNING
OXQ_EXPORT int oxq_mf_trace_read(long long *out)
{
    return cudaMemcpyFromSymbol(out, oxq::g_mf_trace, sizeof(oxq::g_mf_trace)) == cudaSuccess ? 0 : 1;
}
#endif
