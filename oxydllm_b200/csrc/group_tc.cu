// AWQ and GPTQ 4-bit matmul with the unpack inside the tensor-core kernel and the quantization scale behind it: what csrc/stream4.cu and csrc/wide4.cu leave, mostly
// wide layers from 97 tokens on and up to 16 tokens of bf16 scales.
//
// The operand that meets the activations is the integer q - z (exact in bf16); a quantization group's product
// leaves tensor memory once, is multiplied by the group's scale in f32 and added to f32 totals in registers:
//   y[t, n] = sum over groups of s[g, n] * (sum over the group's k of (q - z)[k, n] * x[t, k]).
// Nothing is rounded between the packed weight and the f32 total, and a packed word costs 11 to 13
// instructions instead of the 25 of a scaled and rounded bf16 weight.
//
// One CTA per SM walks an equal share of all (tile, unit) pairs (a tile is 128 out features x at most 128 tokens, a unit
// 128 input rows), so every SM works for the whole launch whatever the number of tiles; the pipeline runs on
// across tile borders. Roles:
//   warp 0        TMA: units of packed words (128 out features), the zero points of their groups and the scales of each fold, as
//                 far ahead as the ring allows: this is what is in flight from HBM;
//   warp 2        TMA: the stage's tile of x ([tokens, 64] bf16, 128-byte swizzle);
//   warps 4..11   unpack, four teams of two warps that take the stages (64 input rows) in turn: a packed word becomes one
//                 16-byte chunk of the operand tile (AWQ: eight out features of one input row, MN-major; GPTQ: eight input
//                 rows of one out feature, K-major);
//   warps 1, 3    tcgen05.mma kind::f16, weights [128 x 16] times x [16 x tokens], into one of four tensor-memory buffers;
//   warps 12..19  fold: accumulators -> registers, times scale, into the totals; at the end of a tile -> y, or, where the
//                 tile is shared with other CTAs, -> scratch, and the CTA that arrives last adds the parts in
//                 ascending k (no CTA waits for another, the result does not depend on the order of arrival).
// Every wait is bounded and reports through the workspace flag word.
//
// What bounds it at up to 32 tokens: the unpack, as far as time stamps show (its four teams always at work, about 1250 clocks a
// stage each, 320 a stage together, and the others waiting for them), and behind it most likely shared memory: a stage moves 4 KB
// of packed words in and out and 16 KB of operand in and out, 320 clocks at 128 B, of which ncu's L1 figure (36 %) leaves out the
// MMA's reads; sixteen unpack warps instead of eight were 2 to 5 % slower. Issue slots are 47 %, DRAM 22 % busy (4096 x 28672).
// Beside that about 7 us a launch go into filling the pipeline, which begins when the kernel ahead has finished, and putting shared
// tiles together. Measured in a graph, us at 16 / 77 / 128 tokens (the kernel with scaled bf16 weights before it): 4096 x 4096
// 11.4 / 16.6 / 19.4 (14 / 19 / 22), 4096 x 28672 30.5 / 48 / 54 (55 / 59 / 61), 14336 x 4096 21 / 28 / 32 (28 / 34 / 38). A poll costs
// about 120 clocks even where the phase is complete, so the polls of a stage are under way together (one after the other: 11.8 / 17.0 /
// 19.7, 32.1 / 51 / 56, 21.8 / 30 / 34).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "mx_common.cuh"

namespace oxq {

constexpr int GT_ROWS = 128;                 // out features of a tile
constexpr int GT_BK = 64;                    // input rows of a stage
constexpr int GT_UNIT = 128, GT_UNIT_STAGES = GT_UNIT / GT_BK; // input rows of a unit: what is loaded at a time
constexpr int GT_TEAMS = 4, GT_TEAM_WARPS = 2;
constexpr int GT_UNPACK_WARPS = GT_TEAMS * GT_TEAM_WARPS;
constexpr int GT_FOLD_WARPS = 8;
constexpr int GT_FOLD_WARP0 = 4 + GT_UNPACK_WARPS; // a multiple of four: warp % 4 selects the quarter of the accumulator rows
constexpr int GT_THREADS = (GT_FOLD_WARP0 + GT_FOLD_WARPS) * 32;
constexpr int GT_ROW_BYTES = 64;             // packed words of one input row of the tile (GPTQ: 1 / 8 of a packed row's 512 bytes)
constexpr int GT_ZERO_BYTES = 64;            // zero points of one group of the tile: 16 words
constexpr int GT_RAW_BYTES = GT_UNIT * GT_ROW_BYTES + GT_UNIT / GT_BK * GT_ZERO_BYTES; // a unit holds up to two groups
constexpr int GT_A_BYTES = GT_ROWS * GT_BK * 2;
constexpr int GT_MAX_RAW = 32, GT_MAX_SLOTS = 8, GT_MAX_X = 8;
constexpr int GT_ISSUERS = 2;                // warps that issue MMAs, on alternate units: one warp alone issues one every 90 clocks
constexpr int GT_ACC = 4;                    // accumulator buffers
constexpr int GT_SC = 16, GT_SC_BYTES = 256; // ring of scales: one 128-wide row of 16-bit scales per fold
constexpr int GT_NUM_BARS = 2 * GT_MAX_RAW + 2 * GT_MAX_SLOTS + 2 * GT_MAX_X + 2 * GT_ACC + 2 * GT_SC;
constexpr int GT_MAX_TOKENS = 128;           // per tile
constexpr int GROUP_TC_MAX_M = 256, GT_NARROW_TILES = 74;
constexpr int GT_SMEM_BUDGET = 227 * 1024;
constexpr int GT_CODE = 20;                  // wait codes 21 .. 31: oxq_gemm_check names them beside the other kernels' 1 .. 5
// A parity wait tells a phase from the next one only: whoever waits on a barrier has to see every one of its phases. So a slot
// always meets the same team and the same issuer, and a ring slot the same teams: their counts are multiples of these.
static_assert(GT_MAX_SLOTS % GT_TEAMS == 0 && GT_TEAMS % (GT_UNIT_STAGES * GT_ISSUERS) == 0 &&
                  GT_MAX_RAW % GT_TEAMS == 0 && GT_MAX_X % (GT_UNIT_STAGES * GT_ISSUERS) == 0,
              "slots and who meets them");

template <int V> struct GtInt { static constexpr int value = V; };

struct GroupTcParams {
    const uint32_t *qzeros;
    const void *scales, *bias;
    void *y;
    int scales_f16, bias_dtype, y_dtype;
    int m, n, packed_out;
    int mpad;                       // tokens of a tile, a multiple of 16
    int token_blocks;               // tiles of the same out features: tile = feature tile * token_blocks + token block
    int slots, x_slots, raw_slots;  // operand tiles, x tiles (a stage each), units of packed words in shared memory
    int x_bytes;                    // of an x tile
    int acc_cols;                   // tensor-memory columns of an accumulator buffer, a power of two
    int gshift;                     // log2(group size)
    int fold_rows;                  // min(group size, 128): input rows per accumulator buffer
    int units_per_tile, tiles;
    int sym;                        // GPTQ without stored zero points (zero + 1 = 8)
    int col_base, ldy;
    int split;                      // shares may begin and end inside a tile
    int test_skip_loads;            // self-test: packed words and scales are never loaded
    int *flag;
    float *partials;                // [CTA + tile][mpad][128] f32
    unsigned long long *tickets;    // per tile: this call's mark above, arrivals in the low byte
    unsigned long long mark;
};

__device__ __forceinline__ uint32_t gt_lds32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void gt_sts128(uint32_t addr, const uint4 &v)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint32_t gt_and_or(uint32_t v, uint32_t mask, uint32_t magic) // (v & mask) | magic
{
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(v), "r"(mask), "r"(magic));
    return r;
}
__device__ __forceinline__ uint32_t gt_sub2(uint32_t a, uint32_t b) // bf16 pairs
{
    const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&a), *reinterpret_cast<const __nv_bfloat162 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&d);
}
// MN-major A operand, 128-byte swizzle: an atom is 8 input rows x 64 out features (1 KB); later input rows follow at 1 KB
// (stride byte offset), the second 64 out features at 8 KB (leading byte offset).
__device__ __forceinline__ uint64_t gt_mn_desc(uint32_t smem_addr)
{
    return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)(8192 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// Units [begin, end) of CTA `i`, and the CTA that holds unit u.
__host__ __device__ __forceinline__ long long gt_share(long long total, int ctas, long long i) { return total * i / ctas; }
__host__ __device__ __forceinline__ int gt_owner(long long total, int ctas, long long u) { return (int)(((u + 1) * ctas - 1) / total); }

// NCH: 8-token chunks of a fold warp's half of the tokens (tiles of at most 16 * NCH tokens).
template <bool GPTQ, int NCH>
__global__ void __launch_bounds__(GT_THREADS, 1)
    packed_group_tc_kernel(const GroupTcParams p, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap)
{
    extern __shared__ unsigned char smem_raw[];
    pdl_launch_dependents();
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u; // operand tiles want 1 KB alignment
    unsigned char *base_ptr = smem_raw + (base - smem_u32(smem_raw));
    // operand tiles | x tiles | ring of packed units | ring of scales | barriers | tensor-memory address, ticket
    const int S = p.slots, X = p.x_slots, R = p.raw_slots;
    const uint32_t x_base = base + (uint32_t)(S * GT_A_BYTES), raw_base = x_base + (uint32_t)(X * p.x_bytes);
    const uint32_t sc_base = raw_base + (uint32_t)(R * GT_RAW_BYTES);
    const uint32_t bars = sc_base + GT_SC * GT_SC_BYTES;
    const uint32_t rawfull = bars, rawempty = rawfull + 8 * GT_MAX_RAW, full = rawempty + 8 * GT_MAX_RAW, empty = full + 8 * GT_MAX_SLOTS,
                   xfull = empty + 8 * GT_MAX_SLOTS, xempty = xfull + 8 * GT_MAX_X, accfull = xempty + 8 * GT_MAX_X,
                   accempty = accfull + 8 * GT_ACC, scfull = accempty + 8 * GT_ACC, scempty = scfull + 8 * GT_SC;
    volatile uint32_t *tail = reinterpret_cast<volatile uint32_t *>(base_ptr + (bars + 8 * GT_NUM_BARS - base));

    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int G = p.units_per_tile;
    const long long total = (long long)p.tiles * G;
    long long u0, u1; // this CTA's units
    if (p.split) {
        u0 = gt_share(total, gridDim.x, blockIdx.x);
        u1 = gt_share(total, gridDim.x, blockIdx.x + 1);
    } else {
        u0 = gt_share(p.tiles, gridDim.x, blockIdx.x) * G;
        u1 = gt_share(p.tiles, gridDim.x, blockIdx.x + 1) * G;
    }
    const int nunits = (int)(u1 - u0), nstages = nunits * GT_UNIT_STAGES;
    const int first_tile = (int)(u0 / G), first_unit = (int)(u0 - (long long)first_tile * G);

    if (warp == 0) { // barrier b of each kind is initialised by lane b
        static_assert(GT_MAX_RAW <= 32 && GT_MAX_SLOTS <= 32 && GT_SC <= 32, "one lane per barrier");
        mbar_init(rawfull + 8 * lane, 1);
        mbar_init(rawempty + 8 * lane, GT_UNIT_STAGES * GT_TEAM_WARPS);
        if (lane < GT_MAX_SLOTS) {
            mbar_init(full + 8 * lane, GT_TEAM_WARPS);
            mbar_init(empty + 8 * lane, 1);
        }
        if (lane < GT_MAX_X) {
            mbar_init(xfull + 8 * lane, 1);
            mbar_init(xempty + 8 * lane, 1);
        }
        if (lane < GT_ACC) {
            mbar_init(accfull + 8 * lane, 1);
            mbar_init(accempty + 8 * lane, GT_FOLD_WARPS);
        }
        if (lane < GT_SC) {
            mbar_init(scfull + 8 * lane, 1);
            mbar_init(scempty + 8 * lane, GT_FOLD_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) { // the allocating warp also frees
        tmem_alloc(bars + 8 * GT_NUM_BARS, (uint32_t)(GT_ACC * p.acc_cols));
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tail[0];
    // The kernel ahead may have written anything this one reads, the packed weights included, and its time must not count as this
    // kernel's waits: only what is above overlaps with it.
    pdl_wait();

    // The single-thread roles run as whole warps with one elected lane at the instruction itself: loop counters, addresses
    // and descriptors stay in uniform registers (with the loop inside the elected branch an MMA took 90 clocks to issue
    // and a stage of this kernel 890).
    if (warp == 0) {
        // ---- packed words, zero points and scales, a unit at a time ----------------------------------------------------
        const bool leader = elect_one();
        const int unit_folds = GT_UNIT / p.fold_rows, zgroups = GPTQ && p.sym ? 0 : unit_folds;
        const uint32_t bytes = (uint32_t)(GT_UNIT * GT_ROW_BYTES + zgroups * GT_ZERO_BYTES);
        int n0 = first_tile / p.token_blocks * GT_ROWS, tb = first_tile % p.token_blocks;
        int uk = first_unit, r = 0, c = 0;
        uint32_t ph = 1, cph = 1; // a fresh barrier passes parity 1
        bool ok = true;
        for (int it = 0; it < nunits && ok; it++) {
            const int k0 = uk * GT_UNIT;
            const size_t group = (size_t)(k0 >> p.gshift);
            const uint32_t *zsrc = p.qzeros + group * p.packed_out + n0 / 8;
            const uint16_t *ssrc = reinterpret_cast<const uint16_t *>(p.scales) + group * p.n + n0;
            ok = mx_wait2(rawempty + 8 * r, ph, scempty + 8 * c, cph, p.flag, GT_CODE + 1); // the ring slot, and the first fold's scales
            if (ok && leader && !p.test_skip_loads) {
                const uint32_t dst = raw_base + (uint32_t)(r * GT_RAW_BYTES), bar = rawfull + 8 * r;
                mbar_arrive_expect_tx(bar, bytes);
                if (GPTQ) tma_load_2d(dst, &wmap, bar, n0, k0 / 8);
                else tma_load_2d(dst, &wmap, bar, n0 / 8, k0);
                for (int z = 0; z < zgroups; z++)
                    bulk_copy_g2s(dst + GT_UNIT * GT_ROW_BYTES + z * GT_ZERO_BYTES, zsrc + (size_t)z * p.packed_out, GT_ZERO_BYTES, bar);
            }
            __syncwarp();
            if (++r == R) { r = 0; ph ^= 1u; }
            for (int f = 0; f < unit_folds && ok; f++) { // unit_folds > 1: groups shorter than a unit, one fold each
                if (f > 0) ok = mx_wait(scempty + 8 * c, cph, p.flag, GT_CODE + 8);
                if (ok && leader && !p.test_skip_loads) {
                    mbar_arrive_expect_tx(scfull + 8 * c, GT_SC_BYTES);
                    bulk_copy_g2s(sc_base + c * GT_SC_BYTES, ssrc + (size_t)f * p.n, GT_SC_BYTES, scfull + 8 * c);
                }
                __syncwarp();
                if (++c == GT_SC) { c = 0; cph ^= 1u; }
            }
            if (++uk == G) {
                uk = 0;
                if (++tb == p.token_blocks) { tb = 0; n0 += GT_ROWS; }
            }
        }
    } else if (warp == 2) {
        // ---- x, a stage at a time, as soon as the MMAs that read the slot have completed -----------------------------
        const bool leader = elect_one();
        int tb = first_tile % p.token_blocks, k0 = first_unit * GT_UNIT, x = 0;
        uint32_t ph = 1; // a fresh barrier passes parity 1
        bool ok = true;
        const int step = X == GT_MAX_X ? 2 : 1; // slots per poll; with few of them both would wait for the later one
        for (int it = 0; it < nstages && ok; it += step) {
            ok = mx_wait2(xempty + 8 * x, ph, xempty + 8 * (x + step - 1), ph, p.flag, GT_CODE + 5);
            if (ok && leader) {
                for (int j = 0; j < step; j++) {
                    mbar_arrive_expect_tx(xfull + 8 * (x + j), (uint32_t)p.x_bytes);
                    tma_load_2d(x_base + (uint32_t)((x + j) * p.x_bytes), &xmap, xfull + 8 * (x + j), k0 + j * GT_BK, tb * p.mpad);
                }
            }
            __syncwarp();
            x += step;
            if (x == X) { x = 0; ph ^= 1u; }
            k0 += step * GT_BK;
            if (k0 == G * GT_UNIT) {
                k0 = 0;
                if (++tb == p.token_blocks) tb = 0;
            }
        }
        // The commits of the last stages arrive here asynchronously: the CTA stays until they have.
        for (int left = min(S, nstages), q = nstages - left; left > 0 && ok; left--, q++)
            ok = mx_wait(empty + 8 * (q % S), (uint32_t)(q / S) & 1u, p.flag, GT_CODE + 11);
        for (int left = min(X, nstages), q = nstages - left; left > 0 && ok; left--, q++)
            ok = mx_wait(xempty + 8 * (q % X), (uint32_t)(q / X) & 1u, p.flag, GT_CODE + 11);
    } else if (warp < 4) {
        // ---- MMA issue: warps 1 and 3 take the units in turn -------------------------------------------------------
        const bool leader = elect_one();
        const int me = warp >> 1;
        const uint32_t idesc = tc_idesc(GT_ROWS, p.mpad) | (GPTQ ? 0u : (1u << 15)); // bit 15: A is MN-major
        const uint64_t adesc0 = GPTQ ? kmajor_sw128_desc(base) : gt_mn_desc(base), bdesc0 = kmajor_sw128_desc(x_base);
        const uint32_t x16 = (uint32_t)p.x_bytes >> 4; // 16-byte units
        auto issue = [&](auto fold_mmas) { // MMAs (16 input rows each) per accumulator buffer
            constexpr int FM = decltype(fold_mmas)::value, US = GT_UNIT_STAGES;
            constexpr int UF = US * 4 / FM; // folds of a unit
            int s = me * US, a = me * UF, x = me * US;
            uint32_t ph = 0, xph = 0, aph = 1; // aph: parity of the last release of the buffer (a fresh barrier passes parity 1)
            for (int ui = me; ui < nunits; ui += GT_ISSUERS) {
                bool ok = true;
#pragma unroll
                for (int st = 0; st < US; st++) {
                    const bool first = FM == 4 || st == 0, last = FM == 4 || st == US - 1; // of the buffer's stages
                    if (ok && first) ok = mx_wait3(xfull + 8 * x, xph, full + 8 * s, ph, accempty + 8 * a, aph, p.flag, GT_CODE + 2);
                    else if (ok) ok = mx_wait2(xfull + 8 * x, xph, full + 8 * s, ph, p.flag, GT_CODE + 2);
                    if (ok) {
                        tc_fence_after();
                        const uint32_t d = tmem_base + (uint32_t)(a * p.acc_cols);
                        const uint64_t da = adesc0 + (uint64_t)(s * (GT_A_BYTES >> 4)), db = bdesc0 + (uint64_t)(x * x16);
                        if (leader) {
#pragma unroll
                            for (int kk = 0; kk < 4; kk++) // 16 input rows: two 1 KB atoms of an MN-major A, 32 bytes of a K-major row
                                umma_bf16(d, da + (uint64_t)(kk * (GPTQ ? 2 : (2048 >> 4))), db + 2 * kk, idesc, !(first && kk == 0));
                            if (last) umma_commit(accfull + 8 * a);
                            umma_commit(empty + 8 * s);
                            umma_commit(xempty + 8 * x);
                        }
                        __syncwarp();
                    }
                    if (last) a++;
                    if (++s == S) { s = 0; ph ^= 1u; }
                    if (++x == X) { x = 0; xph ^= 1u; }
                }
                if (!ok) break;
                // on to this warp's next unit
                x += (GT_ISSUERS - 1) * US;
                if (x >= X) { x -= X; xph ^= 1u; }
                s += (GT_ISSUERS - 1) * US;
                if (s >= S) { s -= S; ph ^= 1u; }
                a += (GT_ISSUERS - 1) * UF;
                if (a >= GT_ACC) { a -= GT_ACC; aph ^= 1u; }
            }
        };
        if (p.fold_rows == GT_UNIT) issue(GtInt<8>{});
        else issue(GtInt<4>{});
    } else if (warp < GT_FOLD_WARP0) {
        // ---- unpack ----------------------------------------------------------------------------------------------
        const int team = (warp - 4) / GT_TEAM_WARPS;
        const int ut = threadIdx.x - (4 + team * GT_TEAM_WARPS) * 32; // 0 .. 63
        uint32_t nib_mask, nib_magic; // in registers, opaque to constant propagation: one LOP3 per use
        asm volatile("mov.b32 %0, 0x000F000F;\n\tmov.b32 %1, 0x43004300;" : "=r"(nib_mask), "=r"(nib_magic)); // bf16 128 + nibble
        // AWQ: word column j of rows r0 + 4 i; GPTQ: out features ut and ut + 64, packed rows 0..7
        const int j = ut & 15, r0 = ut >> 4;
        // stage it = half it % 2 of unit it / 2; a team always meets the same half
        constexpr int TEAM_UNITS = GT_TEAMS / GT_UNIT_STAGES;
        int s = team % S, r = team / GT_UNIT_STAGES % R;
        uint32_t ph = 0, rph = 0;
        const uint32_t half_unit = (uint32_t)(team % GT_UNIT_STAGES);
        const uint32_t part = half_unit * (GT_BK * GT_ROW_BYTES);
        // groups of 128 rows and more: one zero point per unit; 64: one per stage
        const uint32_t zeros_at = GT_UNIT * GT_ROW_BYTES + (p.fold_rows == GT_UNIT ? 0u : half_unit * GT_ZERO_BYTES);
        bool ok = true;
        for (int it = team; it < nstages; it += GT_TEAMS) {
            const bool t0 = mbar_test(rawfull + 8 * r, rph);
            const bool t1 = it < S || mbar_test(empty + 8 * s, ph ^ 1u);
            if (!t0) ok = mbar_wait(rawfull + 8 * r, rph, p.flag, GT_CODE + 3);
            if (ok && !t1) ok = mbar_wait(empty + 8 * s, ph ^ 1u, p.flag, GT_CODE + 7);
            if (!ok) break;
            const uint32_t unit = raw_base + (uint32_t)(r * GT_RAW_BYTES), box = unit + part, zeros_addr = unit + zeros_at;
            const uint32_t slot = base + (uint32_t)(s * GT_A_BYTES);
            if constexpr (!GPTQ) {
                const uint32_t src = box + (uint32_t)(r0 * 16 + j) * 4u, zsrc = zeros_addr + 4u * j;
                const uint32_t dst = slot + (uint32_t)(j >> 3) * 8192u;
                uint32_t zp[4];
                const uint32_t zw = gt_lds32(zsrc);
#pragma unroll
                for (int q = 0; q < 4; q++) zp[q] = gt_and_or(zw >> (4 * q), nib_mask, nib_magic);
#pragma unroll
                for (int half = 0; half < 2; half++) {
                    uint32_t w[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) w[i] = gt_lds32(src + (uint32_t)(half * 8 + i) * 256u);
#pragma unroll
                    for (int i = 0; i < 8; i++) { // row r0 + 4 (8 half + i): atom of eight rows, row within it, swizzled chunk
                        const int i4 = 4 * (half * 8 + i);
                        const uint32_t row8 = (uint32_t)(r0 + (i4 & 4));
                        uint4 o;
                        o.x = gt_sub2(gt_and_or(w[i], nib_mask, nib_magic), zp[0]); // nibbles q and q + 4: out features 2q and 2q + 1
                        o.y = gt_sub2(gt_and_or(w[i] >> 4, nib_mask, nib_magic), zp[1]);
                        o.z = gt_sub2(gt_and_or(w[i] >> 8, nib_mask, nib_magic), zp[2]);
                        o.w = gt_sub2(gt_and_or(w[i] >> 12, nib_mask, nib_magic), zp[3]);
                        gt_sts128(dst + (uint32_t)(i4 >> 3) * 1024u + row8 * 128u + ((((uint32_t)j & 7u) ^ row8) << 4), o);
                    }
                }
            } else {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int f = ut + 64 * h; // out feature of the tile
                    uint32_t w[8];
#pragma unroll
                    for (int c = 0; c < 8; c++) w[c] = gt_lds32(box + (uint32_t)(c * 128 + f) * 4u);
                    uint32_t zp = 0x43084308u; // symmetric: zero 7, + 1
                    if (!p.sym) {
                        const uint32_t z1 = ((gt_lds32(zeros_addr + 4u * (f >> 3)) >> (4 * (f & 7))) & 0xFu) + 1u;
                        zp = 0x43004300u | z1 | (z1 << 16); // bf16 pair (128 + z + 1)
                    }
                    const uint32_t dst = slot + (uint32_t)(f >> 3) * 1024u + (uint32_t)(f & 7) * 128u;
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        // byte b of the word: rows 2b (low nibble) and 2b + 1 (high nibble), neighbours in the K-major row
                        const uint32_t w4 = w[c] >> 4;
                        uint4 o;
                        o.x = gt_sub2(gt_and_or(__byte_perm(w[c], w4, 0x4400), nib_mask, nib_magic), zp);
                        o.y = gt_sub2(gt_and_or(__byte_perm(w[c], w4, 0x5511), nib_mask, nib_magic), zp);
                        o.z = gt_sub2(gt_and_or(__byte_perm(w[c], w4, 0x6622), nib_mask, nib_magic), zp);
                        o.w = gt_sub2(gt_and_or(__byte_perm(w[c], w4, 0x7733), nib_mask, nib_magic), zp);
                        gt_sts128(dst + (((uint32_t)c ^ ((uint32_t)f & 7u)) << 4), o);
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic-proxy stores -> visible to the MMA
            __syncwarp();
            if (lane == 0) {
                mx_arrive(full + 8 * s);
                mx_arrive(rawempty + 8 * r);
            }
            s += GT_TEAMS;
            if (s >= S) { s -= S; ph ^= 1u; }
            r += TEAM_UNITS;
            if (r >= R) { r -= R; rph ^= 1u; }
        }
    } else {
        // ---- fold and store: lane = out feature inside the warp's quarter of the accumulator rows ----------------
        const int fw = warp - GT_FOLD_WARP0, quad = warp & 3, half = fw >> 2;
        const int feature = quad * 32 + lane, mh = p.mpad / 2, col0 = half * mh;
        const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)col0;
        const uint32_t sc_lane = sc_base + 2u * feature;
        const int et = threadIdx.x - GT_FOLD_WARP0 * 32; // 0 .. 255
        int a = 0, c = 0;
        uint32_t aph = 0, cph = 0;
        bool ok = true;
        for (long long u = u0; u < u1;) {
            const int tile = (int)(u / G);
            const long long tile_u0 = (long long)tile * G, seg_end = min(u1, tile_u0 + G);
            const int folds = (int)(seg_end - u) * (GT_UNIT / p.fold_rows);
            float tot[NCH * 8];
#pragma unroll
            for (int i = 0; i < NCH * 8; i++) tot[i] = 0.0f;
#pragma unroll 1
            for (int f = 0; f < folds && ok; f++) {
                ok = mx_wait2(scfull + 8 * c, cph, accfull + 8 * a, aph, p.flag, GT_CODE + 4);
                if (!ok) break;
                tc_fence_after();
                uint16_t sraw;
                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sraw) : "r"(sc_lane + (uint32_t)c * GT_SC_BYTES) : "memory");
                const float sc = p.scales_f16 ? __half2float(__ushort_as_half(sraw)) : __uint_as_float((uint32_t)sraw << 16);
                constexpr int B = NCH < 4 ? NCH : NCH < 8 ? 4 : 2; // chunks in flight between tensor memory and the totals
#pragma unroll
                for (int i0 = 0; i0 < NCH; i0 += B) {
                    uint32_t rr[B][8];
#pragma unroll
                    for (int i = 0; i < B; i++)
                        if ((i0 + i) * 8 < mh) tmem_ld_x8(tlane + (uint32_t)(a * p.acc_cols + (i0 + i) * 8), rr[i]);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < B; i++)
                        if ((i0 + i) * 8 < mh) {
#pragma unroll
                            for (int e = 0; e < 8; e++)
                                tot[(i0 + i) * 8 + e] = fmaf(sc, __uint_as_float(rr[i][e]), tot[(i0 + i) * 8 + e]);
                        }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mx_arrive(accempty + 8 * a);
                    mx_arrive(scempty + 8 * c);
                }
                if (++a == GT_ACC) { a = 0; aph ^= 1u; }
                if (++c == GT_SC) { c = 0; cph ^= 1u; }
            }
            const int tok0 = tile % p.token_blocks * p.mpad, n0 = tile / p.token_blocks * GT_ROWS;
            const int mt = min(p.mpad, p.m - tok0); // this tile's tokens
            if (seg_end - u == G) {
                if (ok) {
                    const float bv = p.bias ? load_as_f32(p.bias, p.bias_dtype, (size_t)p.col_base + n0 + feature) : 0.0f;
#pragma unroll
                    for (int i = 0; i < NCH * 8; i++)
                        if (i < mh && col0 + i < mt)
                            store_as(p.y, p.y_dtype, (size_t)(tok0 + col0 + i) * p.ldy + p.col_base + n0 + feature, tot[i] + bv);
                }
            } else {
                // A shared tile. The barriers are among the fold warps, which all get here whether or not a wait gave up
                // (in that case the flag word is set and the output is not to be trusted).
                const size_t part_floats = (size_t)p.mpad * GT_ROWS;
                if (ok) {
                    float *part = p.partials + (size_t)(blockIdx.x + tile) * part_floats + (size_t)col0 * GT_ROWS + feature;
#pragma unroll
                    for (int i = 0; i < NCH * 8; i++)
                        if (i < mh && col0 + i < mt) part[i * GT_ROWS] = tot[i];
                }
                const int i_lo = gt_owner(total, gridDim.x, tile_u0), i_hi = gt_owner(total, gridDim.x, tile_u0 + G - 1);
                asm volatile("bar.sync 1, %0;" ::"n"(GT_FOLD_WARPS * 32) : "memory");
                if (et == 0) {
                    // The scratch area holds anything at first: a ticket without this call's mark counts as no arrival. The last one
                    // leaves the mark with a count of zero (a replayed graph comes back with the same mark).
                    unsigned long long *ticket = p.tickets + tile, old = *reinterpret_cast<volatile unsigned long long *>(ticket), seen;
                    const unsigned last = (unsigned)(i_hi - i_lo);
                    unsigned count;
                    __threadfence(); // the parts of the whole CTA (ordered before this by the barrier) before the ticket
                    for (;;) { // (with a ticket read at the start of the segment the swap mostly failed at first: 4096 x 1024 15 -> 21 us)
                        count = (old >> 8) == p.mark ? (unsigned)(old & 0xFFu) : 0u;
                        seen = atomicCAS(ticket, old, (p.mark << 8) | (count == last ? 0u : count + 1u));
                        if (seen == old) break; // fails only when another of the tile's few CTAs came in between
                        old = seen;
                    }
                    __threadfence(); // the ticket before the others' parts
                    tail[1] = count;
                }
                asm volatile("bar.sync 1, %0;" ::"n"(GT_FOLD_WARPS * 32) : "memory");
                if (tail[1] == (uint32_t)(i_hi - i_lo)) {
                    const float *parts = p.partials + (size_t)(i_lo + tile) * part_floats;
                    // a thread takes four neighbouring features of every eighth token; the loads of four tokens and two parts are in
                    // flight together (one feature per thread and eight loads in flight took 20 us for 128 tokens)
                    const int nn = 4 * (et & 31);
                    float bv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    if (p.bias)
                        for (int e = 0; e < 4; e++) bv[e] = load_as_f32(p.bias, p.bias_dtype, (size_t)p.col_base + n0 + nn + e);
                    constexpr int TOK_STEP = GT_FOLD_WARPS, BATCH = 4;
                    for (int t0 = et >> 5; t0 < mt; t0 += TOK_STEP * BATCH) {
                        float4 sum[BATCH];
#pragma unroll
                        for (int b = 0; b < BATCH; b++) sum[b] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 2
                        for (int sp = 0; sp <= i_hi - i_lo; sp++) { // ascending k
                            float4 v[BATCH];
#pragma unroll
                            for (int b = 0; b < BATCH; b++) {
                                const int tok = min(t0 + b * TOK_STEP, mt - 1);
                                v[b] = __ldcg(reinterpret_cast<const float4 *>(parts + (size_t)sp * part_floats + (size_t)tok * GT_ROWS + nn));
                            }
#pragma unroll
                            for (int b = 0; b < BATCH; b++) { sum[b].x += v[b].x; sum[b].y += v[b].y; sum[b].z += v[b].z; sum[b].w += v[b].w; }
                        }
#pragma unroll
                        for (int b = 0; b < BATCH; b++) {
                            const int tok = t0 + b * TOK_STEP;
                            if (tok < mt) {
                                const size_t at = (size_t)(tok0 + tok) * p.ldy + p.col_base + n0 + nn;
                                store_as(p.y, p.y_dtype, at, sum[b].x + bv[0]);
                                store_as(p.y, p.y_dtype, at + 1, sum[b].y + bv[1]);
                                store_as(p.y, p.y_dtype, at + 2, sum[b].z + bv[2]);
                                store_as(p.y, p.y_dtype, at + 3, sum[b].w + bv[3]);
                            }
                        }
                    }
                }
                asm volatile("bar.sync 1, %0;" ::"n"(GT_FOLD_WARPS * 32) : "memory"); // tail[1] is read by all before it is written again
            }
            u = seg_end;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, (uint32_t)(GT_ACC * p.acc_cols));
    }
}

// Largest batch for this kernel. Above it the kernel of fused_tc.cu, which scales and rounds the weights as it unpacks them and
// folds nothing, is the faster one, us there / here: groups of 64, where every stage is folded, 3072 x 4096 at 32 tokens 14.0 / 12.5,
// 3072 x 14336 26.1 / 21.1, but 3072 x 5120 at 48 tokens 16.6 / 19.3 (when it still began ahead of the wait); one tile per CTA, 4096 x 14336,
// 31.2 / 29.8 at 96 tokens, 31.1 / 31.5 at 128 (likewise). More than 128 tokens are two tiles that unpack the same weights twice: worth it where that fills idle SMs (256 tokens,
// 4096 x 4096: 35 / 23; 4096 x 14336: 41 / 51). Groups of 32 would be folded four times a unit: 4096 x 28672 took 58 us at any batch,
// the GEMV 38 at 8 tokens, and above 32 tokens the dense copy wins.
int group_tc_max_m(int n, int group_size)
{
    const int tiles = n / GT_ROWS;
    if (group_size == 64) return 32;
    return tiles <= GT_NARROW_TILES ? GROUP_TC_MAX_M : tiles <= 148 ? 96 : GT_MAX_TOKENS;
}

// True when this kernel serves the call.
bool group_tc_supported(int m, int k, int n, int group_size, int scales_dtype, const void *x, const void *qweight, const void *qzeros,
                        const void *scales)
{
    return m >= 1 && m <= group_tc_max_m(n, group_size) && n % GT_ROWS == 0 && k % GT_UNIT == 0 && group_size >= 64 &&
           (group_size & (group_size - 1)) == 0 && (scales_dtype == OXQ_F16 || scales_dtype == OXQ_BF16) && aligned(x, 16) &&
           aligned(qweight, 16) && aligned(qzeros, 16) && aligned(scales, 16);
}

static size_t group_tc_ticket_bytes(int tiles) { return ((size_t)tiles * sizeof(unsigned long long) + 255) / 256 * 256; }

// Scratch that lets a call of this size share tiles over all SMs (with less it shares fewer).
size_t group_tc_scratch_bytes(int m, int n)
{
    const int blocks = ceil_div(m, GT_MAX_TOKENS), mpad = ceil_div(ceil_div(m, blocks), 16) * 16, tiles = n / GT_ROWS * blocks;
    return group_tc_ticket_bytes(tiles) + (size_t)(sm_count() + tiles) * mpad * GT_ROWS * sizeof(float);
}

template <bool GPTQ, int NCH>
static int group_tc_launch(const GroupTcParams &p, const CUtensorMap &wmap, const CUtensorMap &xmap, int ctas, size_t smem, cudaStream_t st)
{
    auto kern = packed_group_tc_kernel<GPTQ, NCH>;
    static size_t configured[64] = {};
    int device = 0;
    OXQ_CUDA(cudaGetDevice(&device));
    if (device >= 64 || configured[device] < smem) {
        OXQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (device < 64) configured[device] = smem;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(GT_THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    allow_early_start(attr, cfg.numAttrs);
    OXQ_CUDA(cudaLaunchKernelEx(&cfg, kern, p, wmap, xmap));
    return OXQ_OK;
}

static thread_local int g_group_selftest_skip_loads = 0; // set only inside oxq_selftest_group_wait_expiry

int group_tc_matmul(const void *x, const uint32_t *qweight, const uint32_t *qzeros, const void *scales, int scales_dtype, const void *bias,
                    int bias_dtype, void *y, int y_dtype, int m, int k, int n, int group_size, int col_base, int ldy, int *flag,
                    cudaStream_t st, int gptq, int sym, void *scratch, size_t scratch_bytes)
{
    GroupTcParams p = {};
    p.qzeros = qzeros; p.scales = scales; p.bias = bias; p.y = y;
    p.scales_f16 = scales_dtype == OXQ_F16; p.bias_dtype = bias_dtype; p.y_dtype = y_dtype;
    p.m = m; p.n = n; p.packed_out = n / 8; p.col_base = col_base; p.ldy = ldy; p.flag = flag;
    p.sym = (gptq && (sym || qzeros == nullptr)) ? 1 : 0;
    p.test_skip_loads = g_group_selftest_skip_loads;
    while ((1 << p.gshift) < group_size) p.gshift += 1;
    p.fold_rows = group_size < GT_UNIT ? group_size : GT_UNIT;
    p.token_blocks = ceil_div(m, GT_MAX_TOKENS);
    p.mpad = ceil_div(ceil_div(m, p.token_blocks), 16) * 16;
    p.units_per_tile = k / GT_UNIT;
    p.tiles = n / GT_ROWS * p.token_blocks;
    p.x_bytes = GT_BK * p.mpad * 2;
    // Shared memory: two operand tiles per team (with one, a team waits for the MMAs of its own last stage: 4096 x 28672 at 32
    // tokens 39.6 us against 29.6) while at least four units of packed words, 33 KB, stay in flight.
    const int fixed = 1024 + GT_SC * GT_SC_BYTES + 8 * GT_NUM_BARS + 16;
    p.slots = p.mpad <= 96 ? 2 * GT_TEAMS : GT_TEAMS;
    p.x_slots = p.mpad <= 32 ? GT_MAX_X : GT_MAX_X / 2;
    p.raw_slots = (GT_SMEM_BUDGET - fixed - p.slots * GT_A_BYTES - p.x_slots * p.x_bytes) / GT_RAW_BYTES;
    if (p.raw_slots > GT_MAX_RAW) p.raw_slots = GT_MAX_RAW;
    p.raw_slots -= p.raw_slots % (GT_TEAMS / GT_UNIT_STAGES);
    p.acc_cols = 16;
    while (p.acc_cols < p.mpad) p.acc_cols *= 2;
    const size_t smem = (size_t)p.slots * GT_A_BYTES + (size_t)p.x_slots * p.x_bytes + (size_t)p.raw_slots * GT_RAW_BYTES + fixed;

    // Equal shares of the (tile, unit) list. A unit takes about 0.46 us where it is folded once and 0.67 us where twice (groups of
    // 64), up to 32 tokens; sharing a tile costs its last CTA time that grows with the number of parts and their size. In quarters of
    // the shorter unit that is 10 + (4 + tokens / 10) a part, above 64 tokens (more registers at work) 3 + 7 a part, as long as no share
    // crosses a tile border, and 30 + 3 (1 + tokens / 32) a part where shares do. Measured, us, whole tiles / 2 / 4 / 8 parts: 2048 x
    // 1024 at 16 tokens 10.9 / 9.8 / 9.4 / 11.5, groups of 64 13.2 / 10.7 / 9.8 / 11.8, at 77 tokens 17.1 / 14.1 / 13.7 / 16.6; 1024 x
    // 1024 at 16 tokens 7.1 / 7.8 / 8.5; 4096 x 512 18.1 / 13.3 / 11.2 / 12.1; shares across borders: 2048 x 4096 at 16 tokens 10.0
    // with 128 CTAs, 14.0 with 148. The parts must fit the scratch area.
    const long long total = (long long)p.tiles * p.units_per_tile;
    const size_t part_bytes = (size_t)p.mpad * GT_ROWS * sizeof(float), ticket_bytes = group_tc_ticket_bytes(p.tiles);
    const long long fit = scratch && scratch_bytes > ticket_bytes ? (long long)((scratch_bytes - ticket_bytes) / part_bytes) - p.tiles : 0;
    long long ctas = p.tiles < sm_count() ? p.tiles : sm_count();
    const int unit = p.fold_rows == GT_UNIT ? 4 : 6;
    int best = unit * ceil_div(p.tiles, (int)ctas) * p.units_per_tile;
    p.split = 0;
    for (int c = 2; c <= 16; c++) {
        long long cand = (long long)p.tiles * c;
        if (cand > sm_count()) cand = sm_count();
        if (cand > total / 2) cand = total / 2;
        if (cand > fit) cand = fit;
        if (cand < p.tiles && cand < sm_count()) break; // shares of more than a tile only with every SM at work
        const int parts = ceil_div((int)cand, p.tiles) + (cand % p.tiles ? 1 : 0);
        int share = p.mpad > 64 ? 3 + 7 * parts : (unit == 4 ? 10 : 16) + parts * (40 + p.mpad) / 10;
        if (cand % p.tiles) share = (30 + 3 * parts * (32 + p.mpad) / 32) * (p.mpad > 64 ? 7 : 10) / 10;
        const int cost = unit * ceil_div((int)total, (int)cand) + share;
        if (cost < best) { best = cost; ctas = cand; p.split = 1; }
        if (cand == sm_count()) break;
    }
    p.mark = mx_call_mark();
    p.tickets = reinterpret_cast<unsigned long long *>(scratch);
    p.partials = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(scratch) + ticket_bytes);

    CUtensorMap wmap, xmap;
    CUresult r;
    if (gptq)
        r = encode_tiled_2d(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, qweight, (uint64_t)n, (uint64_t)k / 8, (uint64_t)n * 4, 128, GT_UNIT / 8,
                            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    else
        r = encode_tiled_2d(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, qweight, (uint64_t)p.packed_out, (uint64_t)k, (uint64_t)p.packed_out * 4,
                            16, GT_UNIT, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (weights) failed with CUresult %d", (int)r);
    r = encode_tiled_2d(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x, (uint64_t)k, (uint64_t)m, (uint64_t)k * 2, GT_BK, (uint32_t)p.mpad,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (x) failed with CUresult %d", (int)r);

#define OXQ_GT_LAUNCH(NCH) \
    return gptq ? group_tc_launch<true, NCH>(p, wmap, xmap, (int)ctas, smem, st) : group_tc_launch<false, NCH>(p, wmap, xmap, (int)ctas, smem, st)
    if (p.mpad <= 16) OXQ_GT_LAUNCH(1);
    if (p.mpad <= 32) OXQ_GT_LAUNCH(2);
    if (p.mpad <= 64) OXQ_GT_LAUNCH(4);
    OXQ_GT_LAUNCH(8);
#undef OXQ_GT_LAUNCH
}

} // namespace oxq

// Self-test of the abort path: one tile of one unit (128 x 128, 16 tokens) whose packed words and scales never come. x arrives; the unpack
// teams, the MMA issuers, the x producer's last waits and the fold warps each give up after their two seconds, side by side, the flag
// word takes the first code, tensor memory is freed and the kernel returns with no copy in flight. Nothing faults or hangs.
OXQ_EXPORT int oxq_selftest_group_wait_expiry(void *workspace, size_t workspace_bytes, void *stream)
{
    oxq::clear_error();
    OXQ_REQUIRE(workspace && workspace_bytes >= (1u << 20) && oxq::aligned(workspace, 256), OXQ_ERR_WORKSPACE,
                "oxq_selftest_group_wait_expiry: 256-byte aligned workspace of at least 1 MiB needed");
    unsigned char *b = reinterpret_cast<unsigned char *>(workspace);
    const int m = 16, k = 128, n = 128;
    // x [16, 128] bf16 | words [128, 16] | zero points [1, 16] | scales [1, 128] | y [16, 128] f32, 64 KB apart
    oxq::g_group_selftest_skip_loads = 1;
    const int rc = oxq::group_tc_matmul(b + (1 << 16), reinterpret_cast<uint32_t *>(b + (2 << 16)), reinterpret_cast<uint32_t *>(b + (3 << 16)),
                                        b + (4 << 16), OXQ_F16, nullptr, 0, b + (5 << 16), OXQ_F32, m, k, n, 128, 0, n,
                                        reinterpret_cast<int *>(workspace), (cudaStream_t)stream, 0, 0, nullptr, 0);
    oxq::g_group_selftest_skip_loads = 0;
    return rc;
}
