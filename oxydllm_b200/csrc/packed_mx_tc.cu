// GPTQ 4-bit and E4M3 matmul on the block-scaled 8-bit tensor cores: weights are operands in the bits that they have.
//
// Read as E4M3 a byte 0..16 is that integer times 2^-9 (subnormals and the first binade are evenly spaced), with a sign bit its negative,
// so q - z of 4-bit weights is one byte, looked up in a table of 16 that each out feature has per group; the operand takes half the
// shared memory of a bf16 one. E4M3 weights are not touched at all. Activations are two E4M3 pieces (mx_common.cuh says how exact); a
// small kernel in front writes them with their block scales. Units in which tokens have outliers, infinities or NaN come a second time,
// with a second pair of pieces (64 tokens on 4096 x 14336 20 us, 21 with an outlier in one column, 49 with one in every 32). A group's product leaves tensor memory once and meets the group's scale in f32:
//   y[t, n] = sum over groups of s[g, n] * (sum over the group's k of (q[k, n] - z[g, n]) x[t, k]).
// Nothing is rounded between the packed weight and the f32 total. (With codes 0..15 as operands and z times the sum of x taken off
// afterwards a weight of zero beside a large x left the rounding of two large f32 numbers behind.)
//
// One CTA per SM walks an equal share of all (tile, unit) pairs (a tile is 128 out features x at most 128 tokens, a unit 128 input
// rows), so every SM works for the whole launch whatever the number of tiles; the pipeline runs on across tile borders. Roles:
//   warp 0        TMA: units of weights (8 KB of packed words with their zero points, or 16 KB of E4M3), as far ahead as the ring
//                 allows: this is what is in flight from HBM;
//   warps 1, 3    tcgen05.mma kind::mxf8f6f4 on alternate units, weights [128 x 32] times both pieces of x, and the copies of x's
//                 block scales to tensor memory;
//   warp 2        TMA: the unit's pieces of x ([tokens, 128] bytes each, 128-byte swizzle) with their block scales;
//   warp 4        4-bit weights: the scales of the tile's features, a unit at a time (a warp of its own: with more copies warp 2 took
//                 800 clocks a unit);
//   12 warps      4-bit weights: unpack, three teams of four warps that take the units in turn: two packed words become one 16-byte
//                 chunk of the operand tile (16 input rows of one out feature, K-major); 4096 x 14336 at 6 tokens takes 18.3 us with
//                 two teams, 17.1 with three, 17.3 with four;
//   4 to 16 warps fold: accumulators -> registers, times the scale, into the totals; at the end of a tile -> y, or, where the
//                 tile is shared with other CTAs, -> scratch, and the CTA that arrives last adds the parts in ascending k
//                 (no CTA waits for another, the result does not depend on the order of arrival).
// The pieces of up to 32 tokens are columns of one MMA (the fold adds them); above, two MMAs add into the same column.
#include "mx_common.cuh"

namespace oxq {

#ifdef OXQ_TUNING
__device__ long long g_px_trace[16][128]; // clock stamps of CTA 3, per role and unit (tuning builds only)
#define PX_TRACE(role, it) do { if (blockIdx.x == 3 && (it) < 128 && (threadIdx.x & 31) == 0) g_px_trace[role][it] = clock64(); } while (0)
#else
#define PX_TRACE(role, it) do { } while (0)
#endif

constexpr int PX_ROWS = 128;                 // out features of a tile
constexpr int PX_UNIT = 128;                 // input rows of a unit: what is loaded, unpacked and multiplied at a time
constexpr int PX_TEAMS = 3, PX_TEAM_WARPS = 4, PX_UNPACK_WARPS = PX_TEAMS * PX_TEAM_WARPS;
constexpr int PX_ISSUERS = 2;                // warps that issue MMAs, on alternate units
constexpr int PX_GPTQ = 0, PX_FP8 = 1;       // an AWQ word is eight out features of one row: MN-major, it was no faster than csrc/group_tc.cu
constexpr int PX_UNPACK_WARP0 = 8;           // 4-bit weights; warps 5 to 7 are idle
template <int WT> constexpr int PX_FOLD_WARP0 = WT == PX_FP8 ? 4 : PX_UNPACK_WARP0 + PX_UNPACK_WARPS; // a multiple of four: warp % 4 selects the quarter of the accumulator rows
constexpr int PX_BOX_BYTES = PX_ROWS * PX_UNIT / 2, PX_A_BYTES = PX_ROWS * PX_UNIT;
constexpr int PX_Z_BYTES = PX_ROWS / 2, PX_RAW_BYTES = PX_BOX_BYTES + 128; // ring slot: packed words, zero points of 128 features, pad
constexpr int PX_SF_BYTES = 512;             // block scales of 128 rows of x and 128 k
constexpr int PX_MAX_SLOTS = 8, PX_MAX_X = 4, PX_MAX_RAW = 24, PX_ACC = 4, PX_FR = 8;
constexpr int PX_SC_BYTES = 256;             // a fold's scales of 128 features
constexpr int PX_NUM_BARS = 2 * (PX_MAX_RAW + PX_MAX_SLOTS + PX_MAX_X + PX_ACC + PX_FR);
constexpr int PX_MAX_TOKENS = 128, PX_MERGED_TOKENS = 32; // per tile; both pieces as columns of one MMA up to here
constexpr int PX_SF_COLS = 64;               // tensor-memory columns in front of the accumulators: the scales
constexpr int PX_SMEM_BUDGET = 227 * 1024;
constexpr int PX_CODE = 40;                  // wait codes 41 .. 51: oxq_gemm_check names them
static_assert(2 * PX_TEAMS % PX_ISSUERS == 0 && 2 * PX_TEAMS <= PX_MAX_SLOTS && PX_MAX_RAW % PX_TEAMS == 0 && PX_MAX_X % PX_ISSUERS == 0,
              "a slot always meets the same team and issuer: a parity wait tells a phase from the next one only");
static_assert(8 + 8 * PX_MAX_X <= PX_SF_COLS, "scales of A, then of every x slot");

struct PackedMxParams {
    const uint32_t *qzeros;
    const void *scales, *bias;
    const unsigned char *sf;        // [pair][unit][token block][1 or 2][512] block scales of x's pieces
    const unsigned long long *second; // [unit][token block], a byte per group of 16 tokens, MX_...: whether they have a second pair of pieces there
    const unsigned long long *any;  // this call's mark where some have
    void *y;
    int scales_f16, bias_dtype, y_dtype;
    int m, n, packed_out;
    int mpad;                       // tokens of a tile, a multiple of 16
    int merged;                     // the pieces of x are columns of one MMA
    int token_blocks;               // tiles of the same out features: tile = feature tile * token_blocks + token block
    int slots, x_slots, raw_slots, accs; // operand tiles, x tiles, units of packed words, accumulator buffers
    int issuers;                    // warps that issue MMAs
    int x_bytes, sf_bytes, fr_bytes; // of an x tile, its block scales, a slot of the fold ring
    int acc_cols;                   // tensor-memory columns of an accumulator buffer
    int tmem_cols;
    int gshift;                     // log2(group size)
    int fold_rows;                  // input rows per accumulator buffer: 128, or 64 where E4M3 weights have scale blocks of an odd number of 64s
    int units_per_tile, tiles;
    size_t pair_sf;                 // bytes of a pair's block scales
    const float *scale_inv;         // E4M3: one scale per block_out x block_in weights, s_in blocks a row; null: 1
    int s_in, block_out, block_in;
    int sym;                        // GPTQ without stored zero points (zero 8)
    int col_base, ldy;
    int split;                      // shares may begin and end inside a tile
    int test_skip_loads;            // self-test: weights and scales are never loaded
    int *flag;
    float *partials;                // [CTA + tile][mpad][128] f32
    unsigned long long *tickets;    // per tile: this call's mark above, arrivals in the low byte
    unsigned long long mark;
};

__device__ __forceinline__ uint32_t px_lds32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
// The E4M3 bytes of q - z for q = 0..15. Byte by byte 0x80 + q - z; a negative one is complemented, which makes it 0x80 + |q - z|, a
// positive one loses its top bit.
__device__ __forceinline__ void px_table(uint32_t (&t)[4], uint32_t z)
{
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint32_t v = 0x83828180u + 0x04040404u * j - z * 0x01010101u, neg = (~v >> 7) & 0x01010101u, mask = neg * 0xFFu;
        t[j] = ((v ^ mask) + neg) ^ (~mask & 0x80808080u);
    }
}
__device__ __forceinline__ uint32_t px_prmt(uint32_t a, uint32_t b, uint32_t sel) // a selector's top bit copies the byte's sign over it
{
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
// Eight codes -> their bytes of the table: both halves of it by the low three bits, then one of the two by the fourth.
__device__ __forceinline__ uint2 px_lookup(const uint32_t (&t)[4], uint32_t w)
{
    const uint32_t sel = w & 0x77777777u, up = w << 4, m0 = px_prmt(up, w, 0xD9C8u), m1 = px_prmt(up, w, 0xFBEAu);
    const uint32_t l0 = px_prmt(t[0], t[1], sel), h0 = px_prmt(t[2], t[3], sel);
    const uint32_t l1 = px_prmt(t[0], t[1], sel >> 16), h1 = px_prmt(t[2], t[3], sel >> 16);
    return make_uint2((l0 & ~m0) | (h0 & m0), (l1 & ~m1) | (h1 & m1));
}
__device__ __forceinline__ void px_unpack(uint32_t dst, const uint32_t (&t)[4], uint32_t w0, uint32_t w1)
{
    const uint2 a = px_lookup(t, w0), b = px_lookup(t, w1);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(a.x), "r"(a.y), "r"(b.x), "r"(b.y) : "memory");
}

// Units [begin, end) of CTA `i`, and the CTA that holds unit u.
__host__ __device__ __forceinline__ long long px_share(long long total, int ctas, long long i) { return total * i / ctas; }
__host__ __device__ __forceinline__ int px_owner(long long total, int ctas, long long u) { return (int)(((u + 1) * ctas - 1) / total); }

// Whether any unit of x has a second pair of pieces: a word to load (behind pdl_wait()), and later, when it has come, to look at. The
// vote makes the answer known to be the same in all lanes.
__device__ __forceinline__ unsigned long long px_any_word(const PackedMxParams &p) { return *reinterpret_cast<const volatile unsigned long long *>(p.any); }
__device__ __forceinline__ bool px_any_second(const PackedMxParams &p, unsigned long long word) { return __all_sync(0xFFFFFFFFu, word == p.mark); }
constexpr int PX_GROUP = 16; // tokens that ask for second pairs together
constexpr unsigned long long PX_BYTES = 0x0101010101010101ull;
// The groups' bytes of a unit's second pairs, and those of them that are of a kind.
__device__ __forceinline__ unsigned long long px_second(const PackedMxParams &p, int tb, int u)
{
    return ld_produced(p.second + (size_t)u * p.token_blocks + tb) & (~0ull >> (64 - p.mpad / PX_GROUP * 8));
}
// Units of [from, to) some of whose tokens have a second pair, in order, E4M3 before E5M2: body(unit, MX_...), until it returns false.
template <typename Body> __device__ __forceinline__ bool px_second_units(const PackedMxParams &p, int tb, int from, int to, Body body)
{
    for (int u = from; u < to; u += 32) {
        const int at = u + (int)(threadIdx.x & 31);
        const unsigned long long k = at < to ? px_second(p, tb, at) : 0ull;
        const unsigned e4m3 = __ballot_sync(0xFFFFFFFFu, (k & PX_BYTES * MX_SECOND_E4M3) != 0), e5m2 = __ballot_sync(0xFFFFFFFFu, (k & PX_BYTES * MX_SECOND_E5M2) != 0);
        for (unsigned hit = e4m3 | e5m2; hit; hit &= hit - 1) {
            const int i = __ffs(hit) - 1;
            if ((e4m3 >> i & 1u) && !body(u + i, MX_SECOND_E4M3)) return false;
            if ((e5m2 >> i & 1u) && !body(u + i, MX_SECOND_E5M2)) return false;
        }
    }
    return true;
}
// What a CTA does, in order: its units of a tile, then those of them again some of whose tokens have a second pair of pieces (twice, if
// of both kinds); the next tile.
// All roles walk this list; one that is `first` of `step` that take turns does every step-th of it from the first-th on:
// body(unit of the tile, pair, MX_..., token block, first feature), until it returns false. waited: behind pdl_wait() already. (The usual loop is a plain count, so that
// what it computes stays in uniform registers: with one loop over both pairs a call took 10 to 20 % longer.)
template <typename Body>
__device__ __forceinline__ bool px_walk(const PackedMxParams &p, int tile, int from, int left, int first, int step, bool waited, Body body)
{
    int tb = tile % p.token_blocks, n0 = tile / p.token_blocks * PX_ROWS, skip = first;
    bool ok = true, looked = false, any = false;
    unsigned long long word = 0;
    if (waited) word = px_any_word(p);
    while (left > 0 && ok) {
        const int to = min(p.units_per_tile, from + left);
        int uk = from + skip;
        for (; uk < to && ok; uk += step) ok = body(uk, 0, MX_ONE_PAIR, tb, n0);
        skip = uk - to;
        if (ok && !looked) {
            if (!waited) {
                pdl_wait();
                word = px_any_word(p);
            }
            any = px_any_second(p, word);
            looked = true;
        }
        if (ok && any)
            ok = px_second_units(p, tb, from, to, [&](int u, int kind) {
                if (skip > 0) {
                    skip--;
                    return true;
                }
                skip = step - 1;
                return body(u, 1, kind, tb, n0);
            });
        left -= to - from;
        from = 0;
        if (++tb == p.token_blocks) { tb = 0; n0 += PX_ROWS; }
    }
    return ok;
}

// ---- x -> pieces, block scales ------------------------------------------------------------------------------------------------
// A CTA takes a unit of a group of tokens, sixteen lanes the 128 k of a token. xq: [pair][token block][piece][mpad tokens][k]; sf: a piece's
// rows of a tile in the order tmem_cp_scales wants (merged: both pieces' rows in one 512-byte chunk). The second pair is written for
// all tokens of the group where one of them asks for it, and not at all elsewhere.
__global__ void __launch_bounds__(16 * PX_GROUP)
    packed_mx_split_kernel(const __nv_bfloat16 *x, unsigned char *xq, unsigned char *sf, unsigned char *second, unsigned long long *any,
                           unsigned long long mark, int m, int k, int mpad, int token_blocks, int merged)
{
    // Behind the wait everything ahead of this kernel is complete, so what starts early after the trigger may read the weights at once.
    pdl_wait();
    pdl_launch_dependents();
    const int u = blockIdx.x, units = gridDim.x, tb = blockIdx.y * PX_GROUP / mpad, lane = threadIdx.x & 15;
    const int tok = blockIdx.y * PX_GROUP + (threadIdx.x >> 4), row = tok - tb * mpad;
    const size_t sf_bytes = (merged ? 1 : 2) * PX_SF_BYTES;
    uint4 raw = make_uint4(0u, 0u, 0u, 0u);
    if (tok < m) raw = ld_produced(reinterpret_cast<const uint4 *>(x + (size_t)tok * k + (size_t)u * PX_UNIT) + lane);
    auto store = [&](int pair, uint2 hi, uint2 lo) {
        unsigned char *dst = xq + ((size_t)((pair * token_blocks + tb) * 2) * mpad + row) * k + (size_t)u * PX_UNIT + lane * 8;
        *reinterpret_cast<uint2 *>(dst) = hi;
        *reinterpret_cast<uint2 *>(dst + (size_t)mpad * k) = lo;
    };
    auto store_scale = [&](int pair, uint32_t s) {
        const int j = lane >> 2, lrow = merged ? row + mpad : row; // block of 32 within the unit; lo's row
        unsigned char *c = sf + ((size_t)(pair * units + u) * token_blocks + tb) * sf_bytes;
        c[(row & 31) * 16 + (row >> 5) * 4 + j] = (unsigned char)s;
        if (!merged) c += PX_SF_BYTES;
        c[(lrow & 31) * 16 + (lrow >> 5) * 4 + j] = (unsigned char)(s - 4u);
    };
    const MxBlock b = mx_block(raw);
    float v[8];
    uint2 hi, lo;
    const uint32_t s = mx_first_pair(raw, b, v, hi, lo);
    if (tok < m) store(0, hi, lo);
    if (tok < m && (lane & 3) == 0) store_scale(0, s);
    const int hit = __syncthreads_or(b.second != MX_ONE_PAIR), e5m2 = hit && __syncthreads_or(b.second == MX_SECOND_E5M2);
    if (threadIdx.x == 0) {
        second[((size_t)u * token_blocks + tb) * 8 + row / PX_GROUP] = (unsigned char)(!hit ? MX_ONE_PAIR : e5m2 ? MX_SECOND_E5M2 : MX_SECOND_E4M3);
        if (hit) *any = mark;
    }
    uint32_t s2 = 127; // where other groups of the tile have a second pair this one multiplies zeros, with a scale that is not NaN
    if (hit) {
        s2 = mx_second_pair(raw, v, s, e5m2, hi, lo);
        if (tok < m) store(1, hi, lo);
    }
    if (tok < m && (lane & 3) == 0) store_scale(1, s2);
}

template <int V> struct PxInt { static constexpr int value = V; };

// NCH: 8-token chunks of a fold warp at most, PARTS: fold warps that share an accumulator's columns (tiles of at most 8 * NCH * PARTS
// tokens).
template <int WT, int PARTS> constexpr int PX_THREADS = (PX_FOLD_WARP0<WT> + 4 * PARTS) * 32;
template <int WT, int NCH, int PARTS>
__global__ void __launch_bounds__(PX_THREADS<WT, PARTS>, 1)
    packed_mx_tc_kernel(const PackedMxParams p, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
                        const __grid_constant__ CUtensorMap gmap)
{
    constexpr bool FP8 = WT == PX_FP8;
    constexpr int FOLD_WARP0 = PX_FOLD_WARP0<WT>, FOLD_WARPS = 4 * PARTS;
    constexpr bool MERGED = 8 * NCH * PARTS <= PX_MERGED_TOKENS;
    extern __shared__ unsigned char smem_raw[];
    pdl_launch_dependents();
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u; // operand tiles want 1 KB alignment
    unsigned char *base_ptr = smem_raw + (base - smem_u32(smem_raw));
    // operand tiles | x tiles | ring of packed units | block scales of x | fold ring | barriers | tensor-memory address, ticket
    const int S = p.slots, X = p.x_slots, R = p.raw_slots;
    const uint32_t x_base = base + (uint32_t)(S * PX_A_BYTES), raw_base = x_base + (uint32_t)(X * p.x_bytes);
    const uint32_t sf_base = raw_base + (uint32_t)(R * PX_RAW_BYTES), fr_base = sf_base + (uint32_t)(X * p.sf_bytes);
    const uint32_t bars = fr_base + (uint32_t)(PX_FR * p.fr_bytes);
    const uint32_t rawfull = bars, rawempty = rawfull + 8 * PX_MAX_RAW, full = rawempty + 8 * PX_MAX_RAW, empty = full + 8 * PX_MAX_SLOTS,
                   xfull = empty + 8 * PX_MAX_SLOTS, xempty = xfull + 8 * PX_MAX_X, accfull = xempty + 8 * PX_MAX_X,
                   accempty = accfull + 8 * PX_ACC, frfull = accempty + 8 * PX_ACC, frempty = frfull + 8 * PX_FR;
    volatile uint32_t *tail = reinterpret_cast<volatile uint32_t *>(base_ptr + (bars + 8 * PX_NUM_BARS - base));

    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int G = p.units_per_tile;
    const long long total = (long long)p.tiles * G;
    long long u0, u1; // this CTA's units
    if (p.split) {
        u0 = px_share(total, gridDim.x, blockIdx.x);
        u1 = px_share(total, gridDim.x, blockIdx.x + 1);
    } else {
        u0 = px_share(p.tiles, gridDim.x, blockIdx.x) * G;
        u1 = px_share(p.tiles, gridDim.x, blockIdx.x + 1) * G;
    }
    const int nunits = (int)(u1 - u0);
    const int first_tile = (int)(u0 / G), first_unit = (int)(u0 - (long long)first_tile * G);
    const int unit_folds = FP8 ? PX_UNIT / p.fold_rows : 1;

    if (warp == 0) { // barrier b of each kind is initialised by lane b
        static_assert(PX_MAX_RAW <= 32, "one lane per barrier");
        if (lane < PX_MAX_RAW) {
            mbar_init(rawfull + 8 * lane, 1);
            mbar_init(rawempty + 8 * lane, PX_TEAM_WARPS);
        }
        if (lane < PX_MAX_SLOTS) {
            mbar_init(full + 8 * lane, FP8 ? 1 : PX_TEAM_WARPS);
            mbar_init(empty + 8 * lane, 1);
        }
        if (lane < PX_MAX_X) {
            mbar_init(xfull + 8 * lane, 1);
            mbar_init(xempty + 8 * lane, 1);
        }
        if (lane < PX_ACC) {
            mbar_init(accfull + 8 * lane, 1);
            mbar_init(accempty + 8 * lane, FOLD_WARPS);
        }
        if (lane < PX_FR) {
            mbar_init(frfull + 8 * lane, 1);
            mbar_init(frempty + 8 * lane, FOLD_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) { // the allocating warp also frees
        tmem_alloc(bars + 8 * PX_NUM_BARS, (uint32_t)p.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) PX_TRACE(10, 0);
    const uint32_t tmem_base = tail[0], tmem_acc = tmem_base + PX_SF_COLS;
    // A's scale is the same for every row and block: 1, or 2^9, which makes the integers of the bytes' 2^-9 steps
    if (warp >= FOLD_WARP0 && warp < FOLD_WARP0 + 4)
        tmem_fill4(tmem_base + ((uint32_t)((warp & 3) * 32) << 16), FP8 ? 0x7F7F7F7Fu : 0x88888888u);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // The single-thread roles run as whole warps with one elected lane at the instruction itself: loop counters, addresses
    // and descriptors stay in uniform registers.
    if (warp == 0) {
        // ---- weights: everything ahead of the split kernel had finished when this kernel started -----------------------------
        const bool leader = elect_one();
        const int ring = FP8 ? S : R, zbytes = p.sym ? 0 : PX_Z_BYTES;
        int r = 0, round = 0;
        uint32_t ph = 1;
        px_walk(p, first_tile, first_unit, nunits, 0, 1, false, [&](int uk, int, int, int, int n0) {
            const bool ok = round == 0 || mx_wait((FP8 ? empty : rawempty) + 8 * r, ph, p.flag, PX_CODE + 1); // polls of fresh barriers cost 1 us a call
            if (ok && leader && !p.test_skip_loads) {
                if (FP8) {
                    mbar_arrive_expect_tx(full + 8 * r, PX_A_BYTES);
                    tma_load_2d(base + (uint32_t)(r * PX_A_BYTES), &wmap, full + 8 * r, uk * PX_UNIT, n0);
                } else {
                    const uint32_t dst = raw_base + (uint32_t)(r * PX_RAW_BYTES);
                    mbar_arrive_expect_tx(rawfull + 8 * r, (uint32_t)(PX_BOX_BYTES + zbytes));
                    tma_load_2d(dst, &wmap, rawfull + 8 * r, n0, uk * (PX_UNIT / 8));
                    if (zbytes) // fetched by the unpack warps they would cost a DRAM round trip per unit: 16.7 -> 23 us
                        bulk_copy_g2s(dst + PX_BOX_BYTES, p.qzeros + (size_t)(((long long)uk * PX_UNIT) >> p.gshift) * p.packed_out + n0 / 8,
                                      PX_Z_BYTES, rawfull + 8 * r);
                }
            }
            __syncwarp();
            if (++r == ring) { r = 0; ph ^= 1u; round = 1; }
            return ok;
        });
    } else if (warp == 2) {
        // ---- x with its block scales, as soon as the MMAs that read the slot have completed ----------------------------------
        const bool leader = elect_one();
        int x = 0, done = 0;
        uint32_t xph = 1; // a fresh barrier passes parity 1
        pdl_wait(); // the pieces come from the kernel ahead
        bool ok = px_walk(p, first_tile, first_unit, nunits, 0, 1, true, [&](int uk, int pair, int kind, int tb, int) {
            const bool ok = mx_wait(xempty + 8 * x, xph, p.flag, PX_CODE + 5);
            if (pair && ok) { // group by group: zeros where there is no second pair of this kind
                const unsigned long long k = px_second(p, tb, uk);
                int groups = 0;
                for (int g = 0; g < p.mpad / PX_GROUP; g++) {
                    if ((int)(k >> (8 * g) & 0xFFu) == kind) groups++;
                    else
                        for (int i = lane; i < 2 * PX_GROUP * PX_UNIT / 16; i += 32) { // both pieces
                            const uint32_t half = (uint32_t)(i / (PX_GROUP * PX_UNIT / 16) * p.x_bytes / 2), at = (uint32_t)(i % (PX_GROUP * PX_UNIT / 16) * 16);
                            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(x_base + (uint32_t)(x * p.x_bytes) + half + (uint32_t)(g * PX_GROUP * PX_UNIT) + at), "r"(0u) : "memory");
                        }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic-proxy stores -> visible to the MMA
                __syncwarp();
                if (leader) {
                    mbar_arrive_expect_tx(xfull + 8 * x, (uint32_t)(groups * 2 * PX_GROUP * PX_UNIT + p.sf_bytes));
                    for (int g = 0; g < p.mpad / PX_GROUP; g++)
                        if ((int)(k >> (8 * g) & 0xFFu) == kind)
                            for (int piece = 0; piece < 2; piece++)
                                tma_load_2d(x_base + (uint32_t)(x * p.x_bytes + piece * p.x_bytes / 2 + g * PX_GROUP * PX_UNIT), &gmap, xfull + 8 * x,
                                            uk * PX_UNIT, ((p.token_blocks + tb) * 2 + piece) * p.mpad + g * PX_GROUP);
                    bulk_copy_g2s(sf_base + (uint32_t)(x * p.sf_bytes), p.sf + p.pair_sf + ((size_t)uk * p.token_blocks + tb) * p.sf_bytes,
                                  (uint32_t)p.sf_bytes, xfull + 8 * x);
                }
            } else if (ok && leader) {
                mbar_arrive_expect_tx(xfull + 8 * x, (uint32_t)(p.x_bytes + p.sf_bytes));
                tma_load_2d(x_base + (uint32_t)(x * p.x_bytes), &xmap, xfull + 8 * x, uk * PX_UNIT, tb * 2 * p.mpad);
                bulk_copy_g2s(sf_base + (uint32_t)(x * p.sf_bytes), p.sf + ((size_t)uk * p.token_blocks + tb) * p.sf_bytes,
                              (uint32_t)p.sf_bytes, xfull + 8 * x);
            }
            __syncwarp();
            if (++x == X) { x = 0; xph ^= 1u; }
            done++;
            return ok;
        });
        // The commits of the last units arrive here asynchronously: the CTA stays until they have.
        for (int left = min(S, done), q = done - left; left > 0 && ok; left--, q++)
            ok = mx_wait(empty + 8 * (q % S), (uint32_t)(q / S) & 1u, p.flag, PX_CODE + 11);
        for (int left = min(X, done), q = done - left; left > 0 && ok; left--, q++)
            ok = mx_wait(xempty + 8 * (q % X), (uint32_t)(q / X) & 1u, p.flag, PX_CODE + 11);
    } else if (warp < 4) {
        // ---- MMA issue: warps 1 and 3 take the units in turn (one alone took 900 clocks a unit, most of it polls and commits) -------
        const bool leader = elect_one();
        const uint32_t idesc0 = mx_idesc(MX_E4M3, MERGED ? 2 * p.mpad : p.mpad);
        const uint64_t adesc0 = kmajor_sw128_desc(base), bdesc0 = kmajor_sw128_desc(x_base);
        const uint32_t x16 = (uint32_t)p.x_bytes >> 4, lo16 = x16 / 2; // 16-byte units
        auto issue = [&](auto unit_folds_) {
            constexpr int UF = decltype(unit_folds_)::value, FM = 4 / UF; // folds of a unit, 32-row steps of a fold
            const int step = p.issuers, me = warp >> 1;
            int s = me, a = me * UF, x = me;
            uint32_t ph = 0, xph = 0, aph = 1; // aph: parity of the last release of the buffer (a fresh barrier passes parity 1)
            if (me >= step) return;
            pdl_wait();
            px_walk(p, first_tile, first_unit, nunits, me, step, true, [&](int, int, int kind, int, int) {
                const uint32_t idesc = kind == MX_SECOND_E5M2 ? idesc0 ^ MX_IDESC_B_E5M2 : idesc0;
                bool ok;
                const uint64_t da = adesc0 + (uint64_t)(s * (PX_A_BYTES >> 4)), db = bdesc0 + (uint64_t)(x * x16);
                const uint32_t sfb = tmem_base + 8u + 8u * x;
                ok = mx_wait3(xfull + 8 * x, xph, full + 8 * s, ph, accempty + 8 * a, aph, p.flag, PX_CODE + 2);
#pragma unroll
                for (int f = 0; f < UF; f++) {
                    if (ok && f > 0) ok = mx_wait(accempty + 8 * a, aph, p.flag, PX_CODE + 9);
                    if (ok) {
                        tc_fence_after();
                        const uint32_t d = tmem_acc + (uint32_t)(a * p.acc_cols);
                        if (leader) {
                            if (f == 0) {
                                tmem_cp_scales(sfb, sf_base + (uint32_t)(x * p.sf_bytes));
                                if (!MERGED) tmem_cp_scales(sfb + 4, sf_base + (uint32_t)(x * p.sf_bytes) + PX_SF_BYTES);
                            }
#pragma unroll
                            for (int q = 0; q < FM; q++) { // 32 input rows: 32 bytes of a K-major row
                                const int kk = f * FM + q;
                                const uint64_t dak = da + 2 * kk;
                                umma_mxf8(d, dak, db + 2 * kk, idesc | mx_idesc_blocks(0, kk), tmem_base, sfb, q != 0);
                                if (!MERGED) umma_mxf8(d, dak, db + lo16 + 2 * kk, idesc | mx_idesc_blocks(0, kk), tmem_base, sfb + 4, 1);
                            }
                            umma_commit(accfull + 8 * a);
                            if (f == UF - 1) {
                                umma_commit(empty + 8 * s);
                                umma_commit(xempty + 8 * x);
                            }
                        }
                        __syncwarp();
                    }
                    if (++a == p.accs) { a = 0; aph ^= 1u; }
                }
                // on to this warp's next unit
                s += step;
                if (s >= S) { s -= S; ph ^= 1u; }
                x += step;
                if (x >= X) { x -= X; xph ^= 1u; }
                a += (step - 1) * UF;
                if (a >= p.accs) { a -= p.accs; aph ^= 1u; }
                return ok;
            });
        };
        if (unit_folds == 1) issue(PxInt<1>{});
        else issue(PxInt<2>{});
    } else if (!FP8 && warp == 4) {
        // ---- scales, a unit at a time: weights, as warp 0's ---------------------------------------------------------------
        const bool leader = elect_one();
        int c = 0;
        uint32_t cph = 1;
        px_walk(p, first_tile, first_unit, nunits, 0, 1, false, [&](int uk, int, int, int, int n0) {
            const size_t group = (size_t)(((long long)uk * PX_UNIT) >> p.gshift);
            const bool ok = mx_wait(frempty + 8 * c, cph, p.flag, PX_CODE + 8);
            if (ok && leader && !p.test_skip_loads) {
                mbar_arrive_expect_tx(frfull + 8 * c, PX_SC_BYTES);
                bulk_copy_g2s(fr_base + (uint32_t)(c * p.fr_bytes), reinterpret_cast<const uint16_t *>(p.scales) + group * p.n + n0, PX_SC_BYTES,
                              frfull + 8 * c);
            }
            __syncwarp();
            if (++c == PX_FR) { c = 0; cph ^= 1u; }
            return ok;
        });
    } else if (!FP8 && warp >= PX_UNPACK_WARP0 && warp < FOLD_WARP0) {
        // ---- unpack ----------------------------------------------------------------------------------------------
        const int team = (warp - PX_UNPACK_WARP0) / PX_TEAM_WARPS;
        const int ut = threadIdx.x - (PX_UNPACK_WARP0 + team * PX_TEAM_WARPS) * 32; // 0 .. 127
        const uint32_t src0 = 4u * ut, swz = (uint32_t)ut & 7u, dst0 = ((uint32_t)ut >> 3) * 1024u + swz * 128u; // out feature ut
        int s = team, r = team;
        uint32_t ph = 1, rph = 0; // a fresh barrier passes parity 1
        // px_walk's list, of which only the length matters here: one copy of the loop's body instead of two
        int next = team, end = 0, tile = first_tile, from = first_unit, left = nunits; // this team's next, all so far; what is left of the list
        bool ok = true, any = false, again = false;
        unsigned long long word = 0;
        while (true) {
            while (ok && next >= end && left > 0) { // a tile's units, or those that come a second time, join the list
                const int to = min(G, from + left);
                if (!again) end += to - from;
                else {
                    if (tile == first_tile) {
                        if (next <= team + PX_TEAMS) { // not loaded yet
                            pdl_wait();
                            word = px_any_word(p);
                        }
                        any = px_any_second(p, word);
                    }
                    if (any) px_second_units(p, tile % p.token_blocks, from, to, [&](int, int) { end++; return true; });
                    left -= to - from;
                    from = 0;
                    tile++;
                }
                again = !again;
            }
            if (!ok || next >= end) break;
            if (next == team + PX_TEAMS) { // with a unit done: not before the kernel ahead may have finished, nor when the answer is wanted
                pdl_wait();
                word = px_any_word(p);
            }
            next += PX_TEAMS;
            const bool t0 = mbar_test(rawfull + 8 * r, rph), t1 = mbar_test(empty + 8 * s, ph);
            if (!t0) ok = mbar_wait(rawfull + 8 * r, rph, p.flag, PX_CODE + 3);
            if (ok && !t1) ok = mbar_wait(empty + 8 * s, ph, p.flag, PX_CODE + 7);
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (!ok) break;
            const uint32_t src = raw_base + (uint32_t)(r * PX_RAW_BYTES) + src0, dst = base + (uint32_t)(s * PX_A_BYTES) + dst0;
            uint32_t words[16];
#pragma unroll
            for (int i = 0; i < 16; i++) words[i] = px_lds32(src + i * 512u);
            uint32_t z = 8, table[4];
            if (!p.sym) z = ((px_lds32(raw_base + (uint32_t)(r * PX_RAW_BYTES) + PX_BOX_BYTES + 4u * (ut >> 3)) >> (4 * (ut & 7))) & 0xFu) + 1u; // stored zero + 1
            px_table(table, z);
#pragma unroll
            for (int i = 0; i < 8; i++) px_unpack(dst + (((uint32_t)i ^ swz) << 4), table, words[2 * i], words[2 * i + 1]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic-proxy stores -> visible to the MMA
            __syncwarp();
            if (lane == 0) {
                mx_arrive(full + 8 * s);
                mx_arrive(rawempty + 8 * r);
            }
            s += PX_TEAMS;
            if (s >= S) { s -= S; ph ^= 1u; }
            r += PX_TEAMS;
            if (r >= R) { r -= R; rph ^= 1u; }
        }
    } else if (warp >= FOLD_WARP0) {
        // ---- fold and store: lane = accumulator row inside the warp's quarter -----------------------------------------------
        const int fw = warp - FOLD_WARP0, quad = warp & 3, part_id = fw >> 2;
        const int feature = quad * 32 + lane;
        const int chunks = p.mpad / 8, chunk0 = part_id * chunks / PARTS, col0 = 8 * chunk0;
        const int mh = 8 * ((part_id + 1) * chunks / PARTS - chunk0); // this warp's tokens
        const uint32_t tlane = tmem_acc + ((uint32_t)(quad * 32) << 16) + (uint32_t)col0;
        const int et = threadIdx.x - FOLD_WARP0 * 32;
        int a = 0, c = 0;
        uint32_t aph = 0, cph = 0;
        bool ok = true;
        pdl_wait();
        const bool any = px_any_second(p, px_any_word(p)); // what it waits for comes before x's first tile does
        for (int tile = first_tile, from = first_unit, left = nunits; left > 0; tile++) {
            const int to = min(G, from + left);
            const long long tile_u0 = (long long)tile * G;
            const float *srow = FP8 && p.scale_inv ? p.scale_inv + (size_t)(tile / p.token_blocks * PX_ROWS / p.block_out) * p.s_in : nullptr;
            float s_next = srow ? __ldg(srow + from * PX_UNIT / p.block_in) : 1.0f; // E4M3: the next fold's scale, asked for a fold ahead
            float tot[NCH * 8];
#pragma unroll
            for (int i = 0; i < NCH * 8; i++) tot[i] = 0.0f;
            int more = 0, again = 0; // units of the tile that come a second time; lane i has the i-th, i + 32-nd, ... of them, 32 at a time
            auto list = [&](int skip) {
                more = 0;
                px_second_units(p, tile % p.token_blocks, from, to, [&](int u, int) {
                    if (more >= skip && more < skip + 32 && more - skip == lane) again = u;
                    more++;
                    return true;
                });
            };
            if (any) list(0);
            const int folds = (to - from) * unit_folds, row0 = from * PX_UNIT;
#pragma unroll 1
            for (int f = 0; f < folds + more * unit_folds && ok; f++) {
                float sc = s_next;
                if (FP8 && srow) {
                    if (f + 1 < folds) s_next = __ldg(srow + (row0 + (f + 1) * p.fold_rows) / p.block_in);
                    else if (more) { // the unit of fold f + 1
                        const int nth = (f + 1 - folds) / unit_folds, part = (f + 1 - folds) % unit_folds;
                        if (nth && nth % 32 == 0 && part == 0 && nth < more) list(nth);
                        s_next = __ldg(srow + (__shfl_sync(0xFFFFFFFFu, again, nth & 31) * PX_UNIT + part * p.fold_rows) / p.block_in);
                    }
                }
                if (FP8) ok = mx_wait(accfull + 8 * a, aph, p.flag, PX_CODE + 4);
                else ok = mx_wait2(frfull + 8 * c, cph, accfull + 8 * a, aph, p.flag, PX_CODE + 4);
                if (!ok) break;
                const uint32_t fr = fr_base + (uint32_t)(c * p.fr_bytes);
                if constexpr (!FP8) {
                    uint16_t sraw;
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sraw) : "r"(fr + 2u * feature) : "memory");
                    sc = p.scales_f16 ? __half2float(__ushort_as_half(sraw)) : __uint_as_float((uint32_t)sraw << 16);
                }
                tc_fence_after();
                const uint32_t tacc = tlane + (uint32_t)(a * p.acc_cols);
                constexpr int B = NCH < 2 ? 1 : 2; // chunks in flight between tensor memory and the totals
#pragma unroll
                for (int i0 = 0; i0 < NCH; i0 += B) {
                    uint32_t rr[B][8], rl[MERGED ? B : 1][8];
#pragma unroll
                    for (int i = 0; i < B; i++)
                        if ((i0 + i) * 8 < mh) {
                            tmem_ld_x8(tacc + (uint32_t)((i0 + i) * 8), rr[i]);
                            if constexpr (MERGED) tmem_ld_x8(tacc + (uint32_t)(p.mpad + (i0 + i) * 8), rl[i]);
                        }
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < B; i++)
                        if ((i0 + i) * 8 < mh) {
#pragma unroll
                            for (int e = 0; e < 8; e++) { // two at a time (fma.rn.f32x2) was 3 to 9 % slower from 128 tokens on
                                float v = __uint_as_float(rr[i][e]);
                                if constexpr (MERGED) v += __uint_as_float(rl[i][e]);
                                tot[(i0 + i) * 8 + e] = fmaf(sc, v, tot[(i0 + i) * 8 + e]);
                            }
                        }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mx_arrive(accempty + 8 * a);
                    if (!FP8) mx_arrive(frempty + 8 * c);
                }
                if (++a == p.accs) { a = 0; aph ^= 1u; }
                if (++c == PX_FR) { c = 0; cph ^= 1u; }
            }
            const int tok0 = tile % p.token_blocks * p.mpad, n0 = tile / p.token_blocks * PX_ROWS;
            const int mt = min(p.mpad, p.m - tok0); // this tile's tokens
            if (to - from == G) {
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
                const size_t part_floats = (size_t)p.mpad * PX_ROWS;
                if (ok) {
                    float *part = p.partials + (size_t)(blockIdx.x + tile) * part_floats + (size_t)col0 * PX_ROWS + feature;
#pragma unroll
                    for (int i = 0; i < NCH * 8; i++)
                        if (i < mh && col0 + i < mt) part[i * PX_ROWS] = tot[i];
                }
                const int i_lo = px_owner(total, gridDim.x, tile_u0), i_hi = px_owner(total, gridDim.x, tile_u0 + G - 1);
                asm volatile("bar.sync 1, %0;" ::"n"(FOLD_WARPS * 32) : "memory");
                if (et == 0) {
                    // The scratch area holds anything at first: a ticket without this call's mark counts as no arrival. The last one
                    // leaves the mark with a count of zero (a replayed graph comes back with the same mark).
                    unsigned long long *ticket = p.tickets + tile, old = *reinterpret_cast<volatile unsigned long long *>(ticket), seen;
                    const unsigned last = (unsigned)(i_hi - i_lo);
                    unsigned count;
                    __threadfence(); // the parts of the whole CTA (ordered before this by the barrier) before the ticket
                    for (;;) {
                        count = (old >> 8) == p.mark ? (unsigned)(old & 0xFFu) : 0u;
                        seen = atomicCAS(ticket, old, (p.mark << 8) | (count == last ? 0u : count + 1u));
                        if (seen == old) break; // fails only when another of the tile's few CTAs came in between
                        old = seen;
                    }
                    __threadfence(); // the ticket before the others' parts
                    tail[1] = count;
                }
                asm volatile("bar.sync 1, %0;" ::"n"(FOLD_WARPS * 32) : "memory");
                if (tail[1] == (uint32_t)(i_hi - i_lo)) {
                    const float *parts = p.partials + (size_t)(i_lo + tile) * part_floats;
                    // a thread takes four neighbouring features of some of the tokens; the loads of BATCH tokens and two parts are in
                    // flight together
                    const int nn = 4 * (et & 31);
                    float bv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    if (p.bias)
                        for (int e = 0; e < 4; e++) bv[e] = load_as_f32(p.bias, p.bias_dtype, (size_t)p.col_base + n0 + nn + e);
                    constexpr int TOK_STEP = FOLD_WARPS, BATCH = NCH == 1 ? 4 : 2;
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
                                v[b] = __ldcg(reinterpret_cast<const float4 *>(parts + (size_t)sp * part_floats + (size_t)tok * PX_ROWS + nn));
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
                asm volatile("bar.sync 1, %0;" ::"n"(FOLD_WARPS * 32) : "memory"); // tail[1] is read by all before it is written again
            }
            left -= to - from;
            from = 0;
        }
        if (et == 0) PX_TRACE(10, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        PX_TRACE(10, 2);
        tc_fence_after();
        tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
    }
}

// True when this kernel serves a GPTQ call and is the better one: its unpack is cheaper than that of csrc/group_tc.cu, but the kernel that
// writes x's pieces costs a launch, so the layer has to be large, and the groups at least a unit. us here / there at 6 tokens: 4096 x
// 14336 19.0 / 20.4, 14336 x 4096 21.2 / 22.0; at 16 19.6 / 20.5, 22.2 / 22.2 (17.2, 19.5, 17.9, 20.7 here without second pairs); with two unpack teams and codes
// 0..15 as operands 4096 x 6144 at 16 tokens took 14.1 / 12.7, 2048 x 4096 10.8 / 10.3, 4096 x 14336 at 32 20.7 / 21.7, 14336 x 4096 24.2 / 23.2.
bool packed_mx_supported(int m, int k, int n, int group_size, int scales_dtype, const void *x, const void *qweight, const void *qzeros,
                         const void *scales)
{
    return m >= 1 && m <= 16 && n % PX_ROWS == 0 && k % PX_UNIT == 0 && (long long)n * k >= 40ll << 20 && group_size >= PX_UNIT &&
           (group_size & (group_size - 1)) == 0 && (scales_dtype == OXQ_F16 || scales_dtype == OXQ_BF16) && aligned(x, 16) &&
           aligned(qweight, 16) && aligned(qzeros, 16) && aligned(scales, 16);
}

// Largest batch of E4M3 weights for this kernel, above it the dense copy of the weight and the GEMM on it are the better tool, us
// here / there: 14336 x 4096 at 400 tokens 65 / 81, 600 79 / 104, 700 95 / 110, 800 114 / 118, 1024 129 / 122; 4096 x 4096 at 256 22 / 35,
// 400 24 / 30, 600 36 / 35.
static int fp8_mx_max_m(int n) { return n >= 8192 ? 768 : 512; }
bool fp8_mx_supported(int m, int k, int n, int block_out, int block_in, const void *x, const void *weight, const void *scale_inv)
{
    return m >= 1 && m <= fp8_mx_max_m(n) && n % PX_ROWS == 0 && k % PX_UNIT == 0 && block_out % PX_ROWS == 0 && block_in % 64 == 0 &&
           aligned(x, 16) && aligned(weight, 16) && aligned(scale_inv, 4);
}

// The scratch area: x's two pairs of pieces, their block scales, which units have a second pair; then tickets and parts of shared tiles.
struct PackedMxScratch {
    int token_blocks, mpad, merged, tiles;
    size_t sf, pair_sf, second, tickets, partials, part_bytes; // offsets of the pieces' successors; bytes of a part
};
static PackedMxScratch packed_mx_layout(int m, int k, int n)
{
    PackedMxScratch s;
    s.token_blocks = ceil_div(m, PX_MAX_TOKENS);
    s.mpad = ceil_div(ceil_div(m, s.token_blocks), 16) * 16;
    s.merged = s.mpad <= PX_MERGED_TOKENS;
    s.tiles = n / PX_ROWS * s.token_blocks;
    const size_t rows = (size_t)s.token_blocks * s.mpad, units = (size_t)k / PX_UNIT;
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    s.pair_sf = units * s.token_blocks * (s.merged ? 1 : 2) * PX_SF_BYTES;
    s.sf = up(2 * 2 * rows * k);
    s.second = s.sf + 2 * s.pair_sf;
    s.tickets = s.second + up(8 + 8 * units * s.token_blocks); // the call's mark in front
    s.partials = s.tickets + up((size_t)s.tiles * sizeof(unsigned long long));
    s.part_bytes = (size_t)s.mpad * PX_ROWS * sizeof(float);
    return s;
}

// Scratch that lets a call of this size share tiles over all SMs (with less it shares fewer, below the pieces it is not served).
size_t packed_mx_scratch_bytes(int m, int k, int n)
{
    const PackedMxScratch s = packed_mx_layout(m, k, n);
    return s.partials + (size_t)(sm_count() + s.tiles) * s.part_bytes;
}

template <int WT, int NCH, int PARTS>
static int packed_mx_launch(const PackedMxParams &p, const CUtensorMap (&maps)[3], int ctas, size_t smem, cudaStream_t st)
{
    auto kern = packed_mx_tc_kernel<WT, NCH, PARTS>;
    static size_t configured[64] = {};
    int device = 0;
    OXQ_CUDA(cudaGetDevice(&device));
    if (device >= 64 || configured[device] < smem) {
        OXQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (device < 64) configured[device] = smem;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(PX_THREADS<WT, PARTS>, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    allow_early_start(attr, cfg.numAttrs);
    OXQ_CUDA(cudaLaunchKernelEx(&cfg, kern, p, maps[0], maps[1], maps[2]));
    return OXQ_OK;
}

static thread_local int g_packed_mx_selftest_skip_loads = 0; // set only inside oxq_selftest_packed_mx_wait_expiry

// Shares, tensor maps, the split kernel and the launch, for the parameters that do not depend on the weight's layout.
static int packed_mx_run(PackedMxParams &p, int wt, const void *x, const void *weight, int k, const PackedMxScratch &s, unsigned char *sb,
                         size_t scratch_bytes, cudaStream_t st)
{
    const int m = p.m, n = p.n;
    p.token_blocks = s.token_blocks; p.mpad = s.mpad; p.merged = s.merged; p.tiles = s.tiles;
    p.units_per_tile = k / PX_UNIT;
    p.sf = sb + s.sf; p.pair_sf = s.pair_sf;
    p.any = reinterpret_cast<const unsigned long long *>(sb + s.second); p.second = p.any + 1;
    p.x_bytes = 2 * p.mpad * PX_UNIT;
    p.sf_bytes = (p.merged ? 1 : 2) * PX_SF_BYTES;
    p.fr_bytes = wt == PX_FP8 ? 0 : PX_SC_BYTES;
    const int fixed = 1024 + PX_FR * p.fr_bytes + 8 * PX_NUM_BARS + 16;
    p.x_slots = PX_MAX_X;
    const int room = PX_SMEM_BUDGET - fixed - p.x_slots * (p.x_bytes + p.sf_bytes);
    if (wt == PX_FP8) { // operand tiles straight from memory
        p.slots = room / PX_A_BYTES < PX_MAX_SLOTS ? room / PX_A_BYTES : PX_MAX_SLOTS;
        p.slots -= p.slots % PX_ISSUERS;
    } else {
        p.slots = 2 * PX_TEAMS;
        p.raw_slots = (room - p.slots * PX_A_BYTES) / PX_RAW_BYTES;
        if (p.raw_slots > PX_MAX_RAW) p.raw_slots = PX_MAX_RAW;
        p.raw_slots -= p.raw_slots % PX_TEAMS;
    }
    p.acc_cols = ceil_div(p.merged ? 2 * p.mpad : p.mpad, 32) * 32;
    p.accs = (512 - PX_SF_COLS) / p.acc_cols < PX_ACC ? (512 - PX_SF_COLS) / p.acc_cols : PX_ACC;
    const int unit_folds = PX_UNIT / p.fold_rows;
    p.issuers = PX_ISSUERS;
    // a buffer always meets the same issuer
    if (p.accs >= PX_ISSUERS * unit_folds) p.accs -= p.accs % (PX_ISSUERS * unit_folds);
    else p.issuers = 1;
    p.tmem_cols = 128;
    while (p.tmem_cols < PX_SF_COLS + p.accs * p.acc_cols) p.tmem_cols *= 2;
    const size_t smem = (size_t)fixed + p.x_slots * (p.x_bytes + p.sf_bytes) + (size_t)p.slots * PX_A_BYTES + (size_t)p.raw_slots * PX_RAW_BYTES;

    const long long total = (long long)p.tiles * p.units_per_tile;
    const long long fit = scratch_bytes > s.partials ? (long long)((scratch_bytes - s.partials) / s.part_bytes) - p.tiles : 0;
    long long ctas = p.tiles < sm_count() ? p.tiles : sm_count();
    const int unit = 2;
    int best = unit * ceil_div(p.tiles, (int)ctas) * p.units_per_tile;
    p.split = 0;
    int force = 0;
    if (const char *env = tuning_env("OXQ_PX_C")) force = atoi(env);
    for (int c = 2; c <= 16; c++) {
        long long cand = (long long)p.tiles * c;
        if (cand > sm_count()) cand = sm_count();
        if (cand > total / 2) cand = total / 2;
        if (cand > fit) cand = fit;
        if (cand < p.tiles && cand < sm_count()) break; // shares of more than a tile only with every SM at work
        const int parts = ceil_div((int)cand, p.tiles) + (cand % p.tiles ? 1 : 0);
        int share = p.mpad > 64 ? 3 + 7 * parts : 10 + parts * (40 + p.mpad) / 10;
        if (cand % p.tiles) share = (30 + 3 * parts * (32 + p.mpad) / 32) * (p.mpad > 64 ? 7 : 10) / 10;
        const int cost = unit * ceil_div((int)total, (int)cand) + share;
        if (force ? c <= force : cost < best) { best = cost; ctas = cand; p.split = 1; }
        if (cand == sm_count()) break;
    }
    p.mark = mx_call_mark();
    p.tickets = reinterpret_cast<unsigned long long *>(sb + s.tickets);
    p.partials = reinterpret_cast<float *>(sb + s.partials);

    CUtensorMap maps[3]; // weights, x a token block at a time, x a group at a time
    CUresult r;
    if (wt == PX_FP8)
        r = encode_tiled_2d(&maps[0], CU_TENSOR_MAP_DATA_TYPE_UINT8, weight, (uint64_t)k, (uint64_t)n, (uint64_t)k, PX_UNIT, PX_ROWS,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    else
        r = encode_tiled_2d(&maps[0], CU_TENSOR_MAP_DATA_TYPE_UINT32, weight, (uint64_t)n, (uint64_t)k / 8, (uint64_t)n * 4, PX_ROWS, PX_UNIT / 8,
                            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (weights) failed with CUresult %d", (int)r);
    for (int i = 1; i <= 2; i++) {
        r = encode_tiled_2d(&maps[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, sb, (uint64_t)k, (uint64_t)2 * p.token_blocks * 2 * p.mpad, (uint64_t)k, PX_UNIT,
                            (uint32_t)(i == 1 ? 2 * p.mpad : PX_GROUP), CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
        OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (x) failed with CUresult %d", (int)r);
    }

    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.units_per_tile, p.token_blocks * p.mpad / PX_GROUP, 1);
    cfg.blockDim = dim3(16 * PX_GROUP, 1, 1);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    allow_early_start(attr, cfg.numAttrs);
    OXQ_CUDA(cudaLaunchKernelEx(&cfg, packed_mx_split_kernel, (const __nv_bfloat16 *)x, sb, sb + s.sf, sb + s.second + 8,
                                reinterpret_cast<unsigned long long *>(sb + s.second), p.mark, m, k, p.mpad, p.token_blocks, p.merged));
#define OXQ_PX_LAUNCH(WT, NCH, PARTS) return packed_mx_launch<WT, NCH, PARTS>(p, maps, (int)ctas, smem, st)
    if (wt == PX_FP8) {
        if (p.mpad <= 16) OXQ_PX_LAUNCH(PX_FP8, 1, 2);
        if (p.mpad <= 32) OXQ_PX_LAUNCH(PX_FP8, 2, 2);
        if (p.mpad <= 64) OXQ_PX_LAUNCH(PX_FP8, 2, 4);
        OXQ_PX_LAUNCH(PX_FP8, 4, 4);
    }
    OXQ_PX_LAUNCH(PX_GPTQ, 2, 1);
#undef OXQ_PX_LAUNCH
}

int packed_mx_matmul(const void *x, const uint32_t *qweight, const uint32_t *qzeros, const void *scales, int scales_dtype, const void *bias,
                     int bias_dtype, void *y, int y_dtype, int m, int k, int n, int group_size, int col_base, int ldy, int *flag,
                     cudaStream_t st, int sym, void *scratch, size_t scratch_bytes)
{
    const PackedMxScratch s = packed_mx_layout(m, k, n);
    if (scratch == nullptr || scratch_bytes < s.tickets) return OXQ_ERR_UNSUPPORTED;
    PackedMxParams p = {};
    p.qzeros = qzeros; p.scales = scales; p.bias = bias; p.y = y;
    p.scales_f16 = scales_dtype == OXQ_F16; p.bias_dtype = bias_dtype; p.y_dtype = y_dtype;
    p.m = m; p.n = n; p.packed_out = n / 8; p.col_base = col_base; p.ldy = ldy; p.flag = flag;
    p.sym = sym || qzeros == nullptr;
    p.test_skip_loads = g_packed_mx_selftest_skip_loads;
    while ((1 << p.gshift) < group_size) p.gshift += 1;
    p.fold_rows = PX_UNIT;
    p.block_in = p.block_out = PX_UNIT;
    return packed_mx_run(p, PX_GPTQ, x, qweight, k, s, reinterpret_cast<unsigned char *>(scratch), scratch_bytes, st);
}

// E4M3 weights with one f32 scale per block_out x block_in of them.
int fp8_mx_matmul(const void *x, const uint8_t *weight, const float *scale_inv, int s_in, int block_out, int block_in, const void *bias,
                  int bias_dtype, void *y, int y_dtype, int m, int k, int n, int *flag, cudaStream_t st, void *scratch, size_t scratch_bytes)
{
    const PackedMxScratch s = packed_mx_layout(m, k, n);
    if (scratch == nullptr || scratch_bytes < s.tickets) return OXQ_ERR_UNSUPPORTED;
    PackedMxParams p = {};
    p.bias = bias; p.y = y; p.bias_dtype = bias_dtype; p.y_dtype = y_dtype;
    p.m = m; p.n = n; p.ldy = n; p.flag = flag;
    p.test_skip_loads = g_packed_mx_selftest_skip_loads;
    p.scale_inv = scale_inv; p.s_in = s_in; p.block_out = block_out; p.block_in = block_in;
    p.fold_rows = block_in % PX_UNIT == 0 ? PX_UNIT : 64;
    return packed_mx_run(p, PX_FP8, x, weight, k, s, reinterpret_cast<unsigned char *>(scratch), scratch_bytes, st);
}

} // namespace oxq

// Self-test of the abort path: one tile of one unit (128 x 128, 16 tokens) whose weights never come. x arrives; the MMA issuers, the last
// waits of x's producer and the fold warps each give up after their two seconds, side by side, the flag word takes the first code,
// tensor memory is freed and the kernel returns with no copy in flight. Nothing faults or hangs.
OXQ_EXPORT int oxq_selftest_packed_mx_wait_expiry(void *workspace, size_t workspace_bytes, void *stream)
{
    oxq::clear_error();
    OXQ_REQUIRE(workspace && workspace_bytes >= (1u << 20) && oxq::aligned(workspace, 256), OXQ_ERR_WORKSPACE,
                "oxq_selftest_packed_mx_wait_expiry: 256-byte aligned workspace of at least 1 MiB needed");
    unsigned char *b = reinterpret_cast<unsigned char *>(workspace);
    // x [16, 128] bf16 | weights [128, 128] | y [16, 128] f32 | scratch, 64 KB apart
    oxq::g_packed_mx_selftest_skip_loads = 1;
    const int rc = oxq::fp8_mx_matmul(b + (1 << 16), b + (2 << 16), nullptr, 1, 128, 128, nullptr, 0, b + (3 << 16), OXQ_F32, 16, 128, 128,
                                      reinterpret_cast<int *>(workspace), (cudaStream_t)stream, b + (4 << 16), workspace_bytes - (4 << 16));
    oxq::g_packed_mx_selftest_skip_loads = 0;
    return rc;
}

#ifdef OXQ_TUNING
OXQ_EXPORT int oxq_px_trace(long long *out) { return cudaMemcpyFromSymbol(out, oxq::g_px_trace, sizeof(oxq::g_px_trace)) == cudaSuccess ? 0 : 1; }
#endif
