// What the kernels that stream packed weights through mma.sync share: fragments, and how the CTAs that hold parts of an output
// tile put it together.
#pragma once

#include "mx_common.cuh"

namespace oxq {

constexpr int ST_CODE = 80;           // wait codes 81 .. 83

// D (+)= A B, m16n8k16, bf16 operands, f32 sums.
__device__ __forceinline__ void st_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void st_mma_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) // D = A B
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ void st_ldmatrix(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void st_ldmatrix_t(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// Loads from shared memory, plain ones: the compiler keeps them behind the wait ahead and is free to move them otherwise.
template <typename T> __device__ __forceinline__ T st_lds(const unsigned char *p) { return *reinterpret_cast<const T *>(p); }
__device__ __forceinline__ uint32_t st_and_or(uint32_t v, uint32_t mask, uint32_t magic) // (v & mask) | magic
{
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(v), "r"(mask), "r"(magic));
    return r;
}
__device__ __forceinline__ uint32_t st_sub2(uint32_t a, uint32_t b) // bf16 pairs
{
    const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&a), *reinterpret_cast<const __nv_bfloat162 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&d);
}

__device__ __forceinline__ float2 st_f16x2(uint32_t two) { return __half22float2(*reinterpret_cast<const __half2 *>(&two)); }

__device__ __forceinline__ void st_load_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c1, int c2, int c3)
{
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void st_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c1, int c2)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(c1), "r"(c2) : "memory");
}

// Tensor maps of a 4-bit weight for units of 128 input rows x two blocks of 128 out features, of 16-bit scales and of zero points (null: none) for the
// groups of a unit. For a gated projection dimension 2 of a pair is the gate's block and 3 its partner's, else the two are neighbours in one dimension; a block
// beyond n reads as zeros.
inline int st_packed4_maps(CUtensorMap &words, CUtensorMap &smap, CUtensorMap &zmap, const uint32_t *qweight, const uint32_t *qzeros, const void *scales, int k,
                           int n, int group_size, int gptq, int gate)
{
    const uint64_t blocks = gate ? (uint64_t)n / 256 : (uint64_t)n / 128, pair = gate ? 2 : 1, row4 = (uint64_t)n / 2, row2 = (uint64_t)n * 2;
    const uint32_t box_blocks = gate ? 1 : 2, box_pair = gate ? 2 : 1, groups = group_size >= 128 ? 1 : 128 / group_size;
    CUresult r;
    if (gptq)
        r = encode_tiled_3d(&words, CU_TENSOR_MAP_DATA_TYPE_UINT32, qweight, 32, (uint64_t)k / 8, (uint64_t)n / 32, (uint64_t)n * 4, 128, 32, 16, 8,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    else
        r = encode_tiled_4d(&words, CU_TENSOR_MAP_DATA_TYPE_UINT32, qweight, 16, (uint64_t)k, blocks, pair, row4, 64, gate ? row4 / 2 : row4, 16, 128, box_blocks,
                            box_pair, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (weights) failed with CUresult %d", (int)r);
    r = encode_tiled_4d(&smap, CU_TENSOR_MAP_DATA_TYPE_UINT16, scales, 128, blocks, pair, (uint64_t)k / group_size, 256, gate ? row2 / 2 : 256, row2, 128, box_blocks,
                        box_pair, groups, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (scales) failed with CUresult %d", (int)r);
    zmap = smap;
    if (qzeros) {
        r = encode_tiled_4d(&zmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, qzeros, 16, blocks, pair, (uint64_t)k / group_size, 64, gate ? row4 / 2 : 64, row4, 16, box_blocks,
                            box_pair, groups, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
        OXQ_REQUIRE(r == CUDA_SUCCESS, OXQ_ERR_CUDA, "cuTensorMapEncodeTiled (zero points) failed with CUresult %d", (int)r);
    }
    return OXQ_OK;
}

struct StreamOut {
    const void *bias;
    void *y;
    int bias_dtype, y_dtype;
    int m, n, ldy;               // n: out features of the weight
    int tok_blocks, tok_step;    // tiles of the same out features, and their tokens: tile = feature tile * tok_blocks + token block
    int gate;                    // columns 0 .. 127 of a tile are gates, 128 .. 255 their partners: y = act(gate) * up, 1 SiLU, 2 GeLU-tanh
    int pairs;                   // two neighbouring outputs can be stored at once
    int units_per_tile, total;   // units of k of a tile; of all tiles
    int grain;                   // shares are whole multiples of this many units
    float *partials;             // [CTA + tile][tok_step][out features of a tile] f32
    unsigned long long *flags;   // [CTA + tile]: this call's mark once the CTA's sum of the tile is in scratch
    unsigned long long mark;
};

// Shares of the list of (tile, unit of k) pairs, unit fastest: the first unit of CTA i, and the CTA that holds unit u.
__host__ __device__ __forceinline__ int st_share(const StreamOut &o, int ctas, int i) { return (int)((long long)(o.total / o.grain) * i / ctas) * o.grain; }
__host__ __device__ __forceinline__ int st_owner(const StreamOut &o, int ctas, int u)
{
    return (int)((((long long)(u / o.grain) + 1) * ctas - 1) / (o.total / o.grain));
}

// How many CTAs share the list, and whether they share tiles (o.grain). In hundredths of a microsecond: a unit takes `unit`; a tile in c equal
// parts costs part0 + part1 c to put together, shares that cross tile borders `cross`. Each share says by a mark of its own that its sum is there: counting the
// shares of a tile down with atomics on one word took 0.6 us a share (Q4_0, 2048 x 1024, one token: 7.6 us, with marks 6.4).
inline int st_ctas(StreamOut &o, int unit, int part0, int part1, int cross)
{
    const int sms = sm_count(), tiles = o.total / o.units_per_tile;
    int best = ceil_div(tiles, sms) * o.units_per_tile * unit, ctas = tiles < sms ? tiles : sms;
    o.grain = o.units_per_tile;
    for (int c = 2; tiles * c <= sms && c <= o.units_per_tile; c++) {
        const int cost = ceil_div(o.units_per_tile, c) * unit + part0 + part1 * c;
        if (cost < best) { best = cost; ctas = tiles * c; o.grain = 1; }
    }
    if (o.total >= 2 * sms && tiles % sms != 0) {
        const int cost = ceil_div(o.total, sms) * unit + cross;
        if (cost < best) { best = cost; ctas = sms; o.grain = 1; }
    }
    if (const char *e = tuning_env("ST_CTAS")) { ctas = atoi(e) < o.total ? atoi(e) : o.total; o.grain = 1; }
    return ctas;
}

__device__ __forceinline__ float st_act(float g, float u, int act)
{
    if (act == 1) return g / (1.0f + __expf(-g)) * u;
    const float t = tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g));
    return 0.5f * g * (1.0f + t) * u;
}

__device__ __forceinline__ void st_store_pair(const StreamOut &o, size_t at, float a, float b)
{
    if (o.pairs) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        *reinterpret_cast<__nv_bfloat162 *>(reinterpret_cast<__nv_bfloat16 *>(o.y) + at) = v;
    } else {
        store_as(o.y, o.y_dtype, at, a);
        store_as(o.y, o.y_dtype, at + 1, b);
    }
}

__device__ __forceinline__ int st_tokens(const StreamOut &o, int tile) { return min(o.tok_step, o.m - tile % o.tok_blocks * o.tok_step); }

// Out features 2 i and 2 i + 1 of a tile of COLS (gate: those of the first half) for its token tok, from their sums. mend(sum, token, out
// feature) may put something else in a sum's place.
struct StKeep { __device__ __forceinline__ float operator()(float v, int, int) const { return v; } };
template <int COLS, typename Mend>
__device__ __forceinline__ void st_output(const StreamOut &o, Mend mend, int tile, int tok, int i, float2 v, float2 up)
{
    const int ft = tile / o.tok_blocks;
    tok += tile % o.tok_blocks * o.tok_step;
    if (o.gate) {
        st_store_pair(o, (size_t)tok * o.ldy + ft * (COLS / 2) + 2 * i, st_act(v.x, up.x, o.gate), st_act(v.y, up.y, o.gate));
        return;
    }
    const int col = ft * COLS + 2 * i;
    if (col >= o.n) return;
    v = make_float2(mend(v.x, tok, col), mend(v.y, tok, col + 1));
    if (o.bias) {
        v.x += load_as_f32(o.bias, o.bias_dtype, col);
        v.y += load_as_f32(o.bias, o.bias_dtype, col + 1);
    }
    st_store_pair(o, (size_t)tok * o.ldy + col, v.x, v.y);
}

// The sums of CTAs i_lo .. i_hi for token tok, columns 2 i and 2 i + 1 of a tile, in ascending k; that of CTA i_lo + me is `own`.
template <int COLS>
__device__ __forceinline__ float2 st_total(const StreamOut &o, int tile, int i_lo, int i_hi, int tok, int i, int me = -1, float2 own = make_float2(0.0f, 0.0f))
{
    const size_t pairs = (size_t)o.tok_step * (COLS / 2);
    const float2 *src = reinterpret_cast<const float2 *>(o.partials) + (size_t)(i_lo + tile) * pairs + (size_t)tok * (COLS / 2) + i;
    float2 s = make_float2(0.0f, 0.0f);
    for (int q0 = 0; q0 <= i_hi - i_lo; q0 += 8) { // eight loads under way together
        float2 v[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            v[q] = make_float2(0.0f, 0.0f);
            if (q0 + q <= i_hi - i_lo) v[q] = q0 + q == me ? own : __ldcg(src + (size_t)(q0 + q) * pairs);
        }
#pragma unroll
        for (int q = 0; q < 8; q++) { s.x += v[q].x; s.y += v[q].y; }
    }
    return s;
}
// One warp: whether the sums of CTAs i_lo .. i_hi of a tile, but for this CTA's, are all in scratch. They may be read if so.
__device__ __forceinline__ bool st_others(const StreamOut &o, int tile, int i_lo, int i_hi)
{
    bool all = true;
    for (int i = i_lo + (int)(threadIdx.x & 31); i <= i_hi; i += 32)
        all = all && (i == (int)blockIdx.x || *reinterpret_cast<volatile unsigned long long *>(o.flags + i + tile) == o.mark);
    all = __all_sync(0xFFFFFFFFu, all);
    if (all) __threadfence(); // the flags before the sums
    return all;
}
// One warp sets its CTA's flag, whose sum a barrier has ordered before; true where all flags of the tile are set. Of all that set one the last
// sees them all, and so may another just before it: both then put the same tile together. The flags are cleared for a replayed
// graph, which comes back with the same mark; what the scratch area holds at first is not the mark. (A counter per tile, which has to be swapped in with the
// mark, took 0.6 us for every CTA of the tile: 4096 x 4096 in 8 parts 11.6 us.)
__device__ __forceinline__ bool st_arrive(const StreamOut &o, int tile, int i_lo, int i_hi)
{
    if ((threadIdx.x & 31) == 0) {
        __threadfence(); // the sum before the flag
        *reinterpret_cast<volatile unsigned long long *>(o.flags + blockIdx.x + tile) = o.mark;
        __threadfence(); // this flag before the others' are read
    }
    __syncwarp();
    return st_others(o, tile, i_lo, i_hi);
}
__device__ __forceinline__ void st_clear(const StreamOut &o, int tile, int i_lo, int i_hi)
{
    for (int i = i_lo + (int)(threadIdx.x & 31); i <= i_hi; i += 32) *reinterpret_cast<volatile unsigned long long *>(o.flags + i + tile) = 0ull;
}

// End of this CTA's segment [u, seg_end) of a tile: `planes` partial tiles [token][PLANE] lie `stride` floats apart in `red`, all
// THREADS threads that call this have written theirs. A whole tile goes to y; of a shared one every CTA leaves its sum in scratch, and the
// CTA that arrives last adds the sums in ascending k: no CTA waits for another, and the result does not depend on the order of arrival.
//
// The round trips to L2 that this takes (sums and flag out, flags and sums in) are about 2 us. A CTA whose share goes on (final = false) leaves them
// to a helping warp (st_help). The first CTA of a tile, which comes to it last, mostly knows from before its last box (`others`, the first warp's st_others)
// that all others have arrived: it takes their sums and its own from shared memory.
// `last`: a shared word. `ok`: false after a wait gave up (nothing is stored, the flag word is set).
template <int THREADS, int COLS, int PLANE, typename Mend>
__device__ __forceinline__ void st_finish(const StreamOut &o, Mend mend, const float *red, int planes, int stride, int tile, int u, int seg_end, bool final,
                                          bool others, bool ok, volatile uint32_t *last)
{
    const int et = threadIdx.x;
    const int i_lo = st_owner(o, gridDim.x, tile * o.units_per_tile), i_hi = st_owner(o, gridDim.x, (tile + 1) * o.units_per_tile - 1);
    const unsigned most = (unsigned)(i_hi - i_lo);
    const bool whole = most == 0;
    if (et == 0) *last = !whole && final && others;
    asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
    auto own = [&](int tok, int i) {
        float2 s = make_float2(0.0f, 0.0f);
        for (int q = 0; q < planes; q++) {
            const float2 v = *reinterpret_cast<const float2 *>(red + q * stride + tok * PLANE + 2 * i);
            s.x += v.x;
            s.y += v.y;
        }
        return s;
    };
    const int per = o.gate ? COLS / 4 : COLS / 2, tokens = st_tokens(o, tile); // results of a token, two at a time
    if (whole) {
        if (ok)
            for (int x = et; x < tokens * per; x += THREADS) {
                const int tok = x / per, i = x - tok * per;
                st_output<COLS>(o, mend, tile, tok, i, own(tok, i), o.gate ? own(tok, i + COLS / 4) : make_float2(0.0f, 0.0f));
            }
        return;
    }
    const int me = (int)blockIdx.x - i_lo;
    const bool early = *last; // all others' sums are there
    auto total = [&](int tok, int i) { return early ? st_total<COLS>(o, tile, i_lo, i_hi, tok, i, me, own(tok, i)) : st_total<COLS>(o, tile, i_lo, i_hi, tok, i); };
    auto outputs = [&](int first, int step) {
        for (int x = first; x < tokens * per; x += step) {
            const int tok = x / per, i = x - tok * per;
            st_output<COLS>(o, mend, tile, tok, i, total(tok, i), o.gate ? total(tok, i + COLS / 4) : make_float2(0.0f, 0.0f));
        }
    };
    if (early) {
        if (et < 32) st_clear(o, tile, i_lo, i_hi);
        if (ok) outputs(et, THREADS);
        return;
    }
    if (ok) {
        float2 *part = reinterpret_cast<float2 *>(o.partials) + (size_t)(blockIdx.x + tile) * o.tok_step * (COLS / 2);
        for (int x = et; x < tokens * (COLS / 2); x += THREADS) part[x] = own(x / (COLS / 2), x % (COLS / 2));
    }
    if (!final) { // st_help does the rest
        asm volatile("bar.arrive 2, %0;" ::"n"(THREADS + 32) : "memory");
        return;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
    if (et < 32) {
        const bool all = st_arrive(o, tile, i_lo, i_hi);
        if (all) st_clear(o, tile, i_lo, i_hi);
        if (et == 0) *last = all;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
    if (*last && ok) outputs(et, THREADS);
}

// The helping warp's part of a first segment that does not end the CTA's share: the flag, while the others go on. Where it is the
// tile's last, all THREADS threads put the tile together at the end (st_helped).
template <int THREADS> __device__ __forceinline__ void st_help(const StreamOut &o, int tile, volatile uint32_t *helped)
{
    const int i_lo = st_owner(o, gridDim.x, tile * o.units_per_tile), i_hi = st_owner(o, gridDim.x, (tile + 1) * o.units_per_tile - 1);
    asm volatile("bar.sync 2, %0;" ::"n"(THREADS + 32) : "memory");
    const bool all = st_arrive(o, tile, i_lo, i_hi);
    if (all) st_clear(o, tile, i_lo, i_hi);
    if ((threadIdx.x & 31) == 0) *helped = all;
    __syncwarp();
    asm volatile("bar.arrive 3, %0;" ::"n"(THREADS + 32) : "memory");
}
template <int THREADS, int COLS, typename Mend>
__device__ __forceinline__ void st_helped(const StreamOut &o, Mend mend, int tile, bool ok, volatile uint32_t *helped)
{
    asm volatile("bar.sync 3, %0;" ::"n"(THREADS + 32) : "memory");
    if (!*helped || !ok) return;
    const int i_lo = st_owner(o, gridDim.x, tile * o.units_per_tile), i_hi = st_owner(o, gridDim.x, (tile + 1) * o.units_per_tile - 1);
    const int per = o.gate ? COLS / 4 : COLS / 2;
    for (int x = threadIdx.x; x < st_tokens(o, tile) * per; x += THREADS) {
        const int tok = x / per, i = x - tok * per;
        st_output<COLS>(o, mend, tile, tok, i, st_total<COLS>(o, tile, i_lo, i_hi, tok, i),
                        o.gate ? st_total<COLS>(o, tile, i_lo, i_hi, tok, i + COLS / 4) : make_float2(0.0f, 0.0f));
    }
}
// Whether a CTA's first segment is one for the helping warp.
__device__ __forceinline__ bool st_needs_help(const StreamOut &o, int u0, int u1) { return u0 % o.units_per_tile != 0 && (u0 / o.units_per_tile + 1) * o.units_per_tile < u1; }

} // namespace oxq
