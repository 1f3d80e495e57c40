// GPT-OSS MoE expert layer on MXFP4 weights, device-side end to end (no host round trip):
//   route (softmax, top-k, renormalise) -> count / plan / scatter tokens per expert ->
//   gather rows -> [dequantize expert group -> grouped tcgen05 GEMM + clamped SwiGLU]* ->
//   [dequantize -> grouped GEMM (down)]* -> weighted combine in ascending expert order.
// Mirrors MoeFeedForward::forward + dispatch_sparse + MoeExpert::GptOss (moe.rs:466-499,
// 563-607, 152-173); every reduction has a fixed order, so results are run-to-run identical.
#include "moe_mx_split.cuh"

namespace oxq {

int mxfp4_dequant_rows_bf16(const uint8_t *blocks, const uint8_t *scales, __nv_bfloat16 *out, int k, int n_off,
                            int n_cnt, cudaStream_t st);
int gemm_grouped(const void *a, int a_rows, const void *w, int slab_experts, int e_first, int nw, int k,
                 const int4 *entries, const int *grp_beg, int group, const void *bias, int bias_dtype, void *out,
                 int ldo, int epi, float limit, int *flag, cudaStream_t stream);

int moe_fused_block_rows(int rows);
bool moe_fused_supported(int n, int k, const void *blocks, const void *scales, const void *a, const void *out, int ldo);
int moe_fused_grouped(const void *a, int a_rows, const uint8_t *blocks, const uint8_t *scales, int experts, int n, int k,
                      const int4 *entries, const int *n_blocks, int block_rows, const void *bias, int bias_dtype, void *out, int ldo,
                      int epi, float limit, int *flag, cudaStream_t st);

int moe_mx_block_rows();
size_t moe_mx_piece_bytes(int rows, int k);
size_t moe_mx_scale_bytes(int rows, int k);
size_t moe_mx_second_bytes(int rows, int k);
bool moe_mx_supported(int n, int k, const void *blocks, const void *scales);
int moe_mx_split(const void *src, const int *perm, int top_k, const int *total_rows, int most, int k, int rows_cap, void *pieces, void *sfx, void *second,
                 unsigned long long mark, cudaStream_t st);
int moe_mx_grouped(const void *pieces, const void *sfx, const void *second, unsigned long long mark, int rows_cap, const uint8_t *blocks,
                   const uint8_t *scales, int experts, int n, int k, const int4 *entries, const int *n_blocks, const void *bias, int bias_dtype,
                   void *out, int ldo, int epi, float limit, int *flag, cudaStream_t st);

constexpr int MOE_MAX_EXPERTS = 256;
constexpr int MOE_MAX_TOPK = 8;
// Rows per expert, on average, up to which the block-scaled kernel is the better one: above, most experts take two of its blocks of 48
// rows, and the kernel that unpacks once for up to 192 or 256 is faster. us a layer, this / that, 32 experts of 2880 x 2880 at 13, 50, 200,
// 300, 384, 450 tokens: 124 / 183, 149 / 221, 169 / 228, 186 / 235, 237 / 240, 277 / 245; 16 of 2048 x 1024 at 30, 120, 200: 43 / 64,
// 49 / 67, 70 / 70. Both have come down by about a tenth since (340 tokens 173 here, 400 tokens 197 there). That is for pairs spread evenly.
// The average is all that the host knows; other routings, this / that as it was with blocks of 256 rows: one expert in half of the tokens, 50,
// 200, 340 tokens 135 / 215, 157 / 222, 177 / 235; two experts in all of them, 340 tokens 203 / 256; popularity falling as 1 / rank^1.2, 340
// tokens 217 / 246; the same four experts for all, 50, 100, 200, 340 tokens 64 / 70, 78 / 78, 113 / 93, 155 / 121: only the last one loses,
// from about 100 rows an expert with nothing beside them.
constexpr int MOE_MX_ROWS = 44;
constexpr int MOE_BLOCK_ROWS = 192; // of a token block of the kernel that unpacks, but for one per expert that may be larger

// One warp: f32 softmax over all experts of a token, k rounds of arg-max (ties: lower index) (moe.rs:472-487); PER: experts a
// lane; denom: the sum of the selected probabilities.
template <int PER>
__device__ __forceinline__ void moe_route_token(const void *logits, int dtype, int token, int experts, int top_k, int (&picked_e)[MOE_MAX_TOPK],
                                                float (&picked_w)[MOE_MAX_TOPK], float &denom)
{
    const int lane = threadIdx.x & 31;
    float v[PER];
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int e = lane + 32 * i;
        v[i] = e < experts ? load_as_f32(logits, dtype, (size_t)token * experts + e) : -INFINITY;
        mx = fmaxf(mx, v[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int e = lane + 32 * i;
        v[i] = e < experts ? expf(v[i] - mx) : 0.0f;
        sum += v[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
#pragma unroll
    for (int i = 0; i < PER; i++) v[i] = (lane + 32 * i) < experts ? v[i] / sum : -1.0f;

    denom = 0.0f;
    for (int s = 0; s < top_k; s++) {
        if (PER == 1) { // probabilities order as their bits do; 0 stands for taken ones, and NaN
            const uint32_t key = v[0] >= 0.0f ? __float_as_uint(v[0]) + 1u : 0u, most = __reduce_max_sync(0xFFFFFFFFu, key);
            if (most) {
                picked_e[s] = __ffs(__ballot_sync(0xFFFFFFFFu, key == most)) - 1;
                picked_w[s] = __uint_as_float(most - 1u);
                denom += picked_w[s];
                if (picked_e[s] == lane) v[0] = -1.0f;
                continue;
            }
        }
        float best = -2.0f;
        int best_e = 0x7FFFFFFF;
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const int e = lane + 32 * i;
            if (v[i] > best) { best = v[i]; best_e = e; } // increasing e within a lane: first maximum wins
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xFFFFFFFFu, best, o);
            const int oe = __shfl_xor_sync(0xFFFFFFFFu, best_e, o);
            if (ob > best || (ob == best && oe < best_e)) { best = ob; best_e = oe; }
        }
        picked_w[s] = best;
        picked_e[s] = best_e;
        denom += best;
        if ((best_e & 31) == lane) {
#pragma unroll
            for (int i = 0; i < PER; i++)
                if (lane + 32 * i == best_e) v[i] = -1.0f; // taken
        }
    }
}

// One warp per token; optional renormalisation by the sum of the selected probabilities.
template <int PER>
__global__ void __launch_bounds__(256)
moe_route_kernel(const void *logits, int dtype, int tokens, int experts, int top_k, int norm_topk, int *top_idx, float *top_w)
{
    pdl_wait(); // the logits are the kernel ahead's, and what is written may still be read
    pdl_launch_dependents();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= tokens) return;
    int picked_e[MOE_MAX_TOPK];
    float picked_w[MOE_MAX_TOPK], denom;
    moe_route_token<PER>(logits, dtype, warp, experts, top_k, picked_e, picked_w, denom);
    if (lane == 0)
        for (int s = 0; s < top_k; s++) {
            top_idx[(size_t)warp * top_k + s] = picked_e[s];
            top_w[(size_t)warp * top_k + s] = norm_topk ? picked_w[s] / denom : picked_w[s];
        }
}

// counts[e - e_lo] = number of (token, slot) pairs routed to expert e, for e in [e_lo, e_hi).
__global__ void __launch_bounds__(1024)
moe_count_kernel(const int *__restrict__ top_idx, int pairs, int e_lo, int *__restrict__ counts)
{
    __shared__ int part[32];
    const int e = e_lo + blockIdx.x;
    int c = 0;
    const int quads = pairs / 4; // top_idx sits on a 256-byte boundary of the workspace
    for (int i = threadIdx.x; i < quads; i += blockDim.x) {
        const int4 v = __ldg(reinterpret_cast<const int4 *>(top_idx) + i);
        c += (v.x == e) + (v.y == e) + (v.z == e) + (v.w == e);
    }
    for (int i = quads * 4 + threadIdx.x; i < pairs; i += blockDim.x) c += top_idx[i] == e;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x < 32) {
        int t = part[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
        if (threadIdx.x == 0) counts[blockIdx.x] = t;
    }
}

// offsets = exclusive scan of counts; m-tile table (128 rows each) per expert in ascending order;
// grp_beg[g] = first m tile of expert group g (experts_per_group experts each).
__global__ void moe_plan_kernel(const int *__restrict__ counts, int n_exp, int e_lo, int experts_per_group,
                                int *__restrict__ offsets, int4 *__restrict__ entries, int *__restrict__ grp_beg)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int off = 0, mt = 0, g = 0;
    for (int i = 0; i < n_exp; i++) {
        if (i % experts_per_group == 0) grp_beg[g++] = mt;
        offsets[i] = off;
        const int c = counts[i];
        for (int r = 0; r < c; r += 128) entries[mt++] = make_int4(off + r, min(128, c - r), e_lo + i, 0);
        off += c;
    }
    offsets[n_exp] = off;
    grp_beg[g] = mt;
}

// Inclusive scan over the block's threads (at most 1024) of two values at once; scratch: 64 ints.
__device__ __forceinline__ int2 moe_block_scan(int2 v, int *scratch)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xFFFFFFFFu, v.x, o), y = __shfl_up_sync(0xFFFFFFFFu, v.y, o);
        if (lane >= o) v.x += x, v.y += y;
    }
    if (lane == 31) scratch[warp] = v.x, scratch[32 + warp] = v.y;
    __syncthreads();
    for (int w = 0; w < warp && w < warps; w++) v.x += scratch[w], v.y += scratch[32 + w];
    __syncthreads();
    return v;
}

// Offsets (exclusive scan of counts) and token blocks for the kernel that unpacks MXFP4 inside the tensor-core loop: every
// expert's rows cut into the fewest blocks of at most max_rows rows, of equal size rounded up to 16; above MOE_BLOCK_ROWS that limit holds for
// one block, and only where it saves one (see moe_fused_block_rows). n_blocks[0] = how many. Thread i is expert i (one thread walking 32
// experts took 10 us). Returns the expert's first row.
__device__ __forceinline__ int moe_plan_expert(int c, int n_exp, int e_lo, int max_rows, int *offsets, int4 *entries, int *n_blocks,
                                               int *scratch)
{
    const int i = threadIdx.x;
    int size, first;
    if (c > MOE_BLOCK_ROWS && (c - 1) % MOE_BLOCK_ROWS < max_rows - MOE_BLOCK_ROWS) { // one larger block instead of two smaller ones
        size = MOE_BLOCK_ROWS;
        first = c - (c / MOE_BLOCK_ROWS - 1) * MOE_BLOCK_ROWS;
    } else {
        max_rows = min(max_rows, MOE_BLOCK_ROWS);
        const int parts = (c + max_rows - 1) / max_rows;
        size = parts ? ((c + parts - 1) / parts + 15) / 16 * 16 : 1;
        first = min(size, c);
    }
    const int blocks = c ? 1 + (c - first + size - 1) / size : 0;
    const int2 incl = moe_block_scan(make_int2(c, blocks), scratch);
    const int off = incl.x - c;
    if (i < n_exp) {
        offsets[i] = off;
        for (int q = 0, r = 0; q < blocks; q++) {
            const int rows = q ? min(size, c - r) : first;
            entries[incl.y - blocks + q] = make_int4(off + r, rows, e_lo + i, 0);
            r += rows;
        }
        if (i == n_exp - 1) offsets[n_exp] = incl.x, n_blocks[0] = incl.y;
    }
    return off;
}

__global__ void __launch_bounds__(MOE_MAX_EXPERTS)
moe_plan_blocks_kernel(const int *__restrict__ counts, int n_exp, int e_lo, int max_rows, int *__restrict__ offsets,
                       int4 *__restrict__ entries, int *__restrict__ n_blocks)
{
    __shared__ int scratch[64];
    moe_plan_expert((int)threadIdx.x < n_exp ? counts[threadIdx.x] : 0, n_exp, e_lo, max_rows, offsets, entries, n_blocks, scratch);
}

// Count, plan and scatter of a small batch in one launch of one CTA (a launch each took 16 us for 200 pairs): pairs are taken
// 1024 at a time, a warp's hits of an expert are counted by match, and the warps' counts are scanned per expert, so that
// positions keep the order of the pairs.
constexpr int MOE_SMALL_PAIRS = 2048;
__global__ void __launch_bounds__(1024)
moe_dispatch_small_kernel(const int *top_idx, int pairs, int e_lo, int n_exp, int max_rows, int *counts, int *offsets, int4 *entries,
                          int *n_blocks, int *perm, int *inv)
{
    pdl_launch_dependents();
    constexpr int ROUNDS = MOE_SMALL_PAIRS / 1024, GROUPS = ROUNDS * 32;
    __shared__ unsigned short cnt[GROUPS][MOE_MAX_EXPERTS]; // hits of an expert in a warp of a round, then the hits before it
    __shared__ int base_s[MOE_MAX_EXPERTS], scratch[64];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int groups = (pairs + 31) / 32;
    for (int i = tid; i < groups * MOE_MAX_EXPERTS; i += blockDim.x) (&cnt[0][0])[i] = 0;
    pdl_wait(); // the routing results are the kernel ahead's
    __syncthreads();
    int id[ROUNDS];
    unsigned peers[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int pair = r * 1024 + tid;
        id[r] = pair < pairs ? top_idx[pair] - e_lo : -1;
        if (id[r] >= n_exp || id[r] < 0) id[r] = -1;
        peers[r] = __match_any_sync(0xFFFFFFFFu, id[r]);
        if (id[r] >= 0 && (peers[r] & ((1u << lane) - 1u)) == 0) cnt[r * 32 + warp][id[r]] = (unsigned short)__popc(peers[r]);
    }
    __syncthreads();
    int c = 0;
    if (tid < n_exp)
        for (int q = 0; q < groups; q++) {
            const int h = cnt[q][tid];
            cnt[q][tid] = (unsigned short)c;
            c += h;
        }
    const int off = moe_plan_expert(c, n_exp, e_lo, max_rows, offsets, entries, n_blocks, scratch);
    if (tid < n_exp) counts[tid] = c, base_s[tid] = off;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; r++)
        if (id[r] >= 0) {
            const int pair = r * 1024 + tid, pos = base_s[id[r]] + cnt[r * 32 + warp][id[r]] + __popc(peers[r] & ((1u << lane) - 1u));
            perm[pos] = pair;
            inv[pair] = pos;
        }
}

// All that comes in front of the block-scaled expert kernel for a batch of up to MOE_FRONT_PAIRS pairs in one launch: routing, positions
// by expert, the table of token blocks and the pieces of x. Every CTA routes all tokens for itself and writes its share of the pieces, the last one the
// tables. Bounded by that chain of latencies, about 5 us. us a layer in a graph, 32 experts of 2880 x 2880 at 1 / 2 / 8 tokens: 41.3 / 56.4 / 94 (in three
// launches 44 / 59 / 96; with the loops of the router over 256 experts 44.9 / 59.8 / 96.9). Batches of up to 48 pairs were single-token GEMVs before, one a pair:
// 42.2 / 64 / 188, 12 tokens 267 against 110; 16 of 2048 x 1024, one token, 26.9 against 27.9. A token has the same bits alone and in a batch.
constexpr int MOE_FRONT_PAIRS = 64;
constexpr int MOE_SMALL_MAX_K = 81912; // wider layers keep the dense fallback for blocks off 16 bytes
struct MoeFrontParams {
    const void *logits;
    const int *given; // not null: rows that already carry their expert, weight one
    const __nv_bfloat16 *x;
    int logits_dtype, tokens, experts, top_k, norm_topk, e_lo, n_exp, max_rows;
    int *top_idx, *offsets, *n_blocks, *inv;
    float *top_w;
    int4 *entries;
    MoeMxPieces pieces;
};
__global__ void __launch_bounds__(MOE_MAX_EXPERTS)
moe_front_kernel(const MoeFrontParams p)
{
    __shared__ int ids[MOE_FRONT_PAIRS], perm[MOE_FRONT_PAIRS], scratch[64];
    pdl_wait();
    pdl_launch_dependents(); // the expert kernel behind reads weights ahead of its own wait: whatever wrote them has finished
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, pairs = p.tokens * p.top_k;
    const bool tables = blockIdx.x + 1 == gridDim.x; // the last CTA writes these, the others the pieces
    if (p.given) {
        if (tid < pairs) {
            ids[tid] = ld_produced(p.given + tid);
            if (tables) p.top_idx[tid] = ids[tid], p.top_w[tid] = 1.0f;
        }
    } else {
        for (int t = warp; t < p.tokens; t += MOE_MAX_EXPERTS / 32) {
            int picked_e[MOE_MAX_TOPK];
            float picked_w[MOE_MAX_TOPK], denom;
            if (p.experts <= 32) moe_route_token<1>(p.logits, p.logits_dtype, t, p.experts, p.top_k, picked_e, picked_w, denom);
            else moe_route_token<MOE_MAX_EXPERTS / 32>(p.logits, p.logits_dtype, t, p.experts, p.top_k, picked_e, picked_w, denom);
            if (lane == 0)
                for (int s = 0; s < p.top_k; s++) {
                    ids[t * p.top_k + s] = picked_e[s];
                    if (tables) {
                        p.top_idx[t * p.top_k + s] = picked_e[s];
                        p.top_w[t * p.top_k + s] = p.norm_topk ? picked_w[s] / denom : picked_w[s];
                    }
                }
        }
    }
    __syncthreads();
    auto local = [&](int e) { return e >= p.e_lo && e < p.e_lo + p.n_exp; };
    int pos = 0;
    const bool mine = tid < pairs && local(ids[tid]);
    if (mine) { // ascending experts, pairs of an expert in their order
        for (int j = 0; j < pairs; j++) pos += local(ids[j]) && (ids[j] < ids[tid] || (ids[j] == ids[tid] && j < tid));
        perm[pos] = tid;
        if (tables) p.inv[tid] = pos;
    }
    const int rows = __syncthreads_count(mine);
    if (tables) {
        int c = 0;
        if (tid < p.n_exp)
            for (int j = 0; j < pairs; j++) c += ids[j] == p.e_lo + tid;
        moe_plan_expert(c, p.n_exp, p.e_lo, p.max_rows, p.offsets, p.entries, p.n_blocks, scratch);
    } else moe_mx_split_rows(p.x, rows, p.pieces, gridDim.x - 1, [&](int row) { return perm[row] / p.top_k; });
}

// Stable partition: position of pair i among the pairs of its expert, in pair (= token) order.
// One CTA per expert walks the pairs 4096 at a time (four neighbours per thread); a scan over the threads'
// hit counts keeps the order deterministic.
__global__ void __launch_bounds__(1024)
moe_scatter_kernel(const int *__restrict__ top_idx, int pairs, int e_lo, const int *__restrict__ offsets,
                   int *__restrict__ perm, int *__restrict__ inv)
{
    __shared__ int warp_cnt[32], warp_off[32];
    __shared__ int total_s;
    const int e = e_lo + blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int base = offsets[blockIdx.x];
    for (int start = 0; start < pairs; start += 4096) {
        const int i0 = start + 4 * (int)threadIdx.x;
        int id[4] = {-1, -1, -1, -1};
        if (i0 + 3 < pairs) {
            const int4 v = __ldg(reinterpret_cast<const int4 *>(top_idx + i0)); // top_idx sits on a 256-byte boundary
            id[0] = v.x; id[1] = v.y; id[2] = v.z; id[3] = v.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (i0 + j < pairs) id[j] = top_idx[i0 + j];
        }
        const int cnt = (id[0] == e) + (id[1] == e) + (id[2] == e) + (id[3] == e);
        int incl = cnt; // inclusive scan of the hit counts over the warp
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) warp_cnt[warp] = incl;
        __syncthreads();
        if (warp == 0) { // exclusive scan of the warps' totals
            const int c = warp_cnt[lane];
            int inc2 = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xFFFFFFFFu, inc2, o);
                if (lane >= o) inc2 += t;
            }
            warp_off[lane] = inc2 - c;
            if (lane == 31) total_s = inc2;
        }
        __syncthreads();
        int pos = base + warp_off[warp] + incl - cnt;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (id[j] == e) {
                perm[pos] = i0 + j;
                inv[i0 + j] = pos;
                pos += 1;
            }
        base += total_s;
        __syncthreads(); // warp_cnt, warp_off and total_s are rewritten by the next pass
    }
}

// xs[pos, :] = x[perm[pos] / top_k, :]  (one warp per row, 16-byte copies)
__global__ void __launch_bounds__(256)
moe_gather_kernel(const __nv_bfloat16 *__restrict__ x, const int *__restrict__ perm, const int *__restrict__ total_rows,
                  int top_k, int hidden, __nv_bfloat16 *__restrict__ xs, int rows_by_value = 0)
{
    const int rows = total_rows ? *total_rows : rows_by_value;
    const int lane = threadIdx.x & 31;
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < rows; row += (gridDim.x * blockDim.x) >> 5) {
        const uint4 *src = reinterpret_cast<const uint4 *>(x + (size_t)(perm[row] / top_k) * hidden);
        uint4 *dst = reinterpret_cast<uint4 *>(xs + (size_t)row * hidden);
        for (int c = lane; c < hidden / 8; c += 32) dst[c] = src[c];
    }
}

// out[t, :] = sum over the token's slots whose expert is in [e_lo, e_hi), in ascending expert id,
// of w * yp[inv[pair], :] (f32 accumulation, one rounding). Tokens without such a slot get zeros.
__global__ void __launch_bounds__(256)
moe_combine_kernel(const __nv_bfloat16 *yp, const int *top_idx, const float *top_w, const int *inv, int tokens, int top_k, int hidden, int e_lo, int e_hi, void *out,
                   int out_dtype)
{
    pdl_launch_dependents();
    pdl_wait(); // rows and routing results come from kernels ahead
    // a warp takes part `seg` of a token's 16-byte pieces: the slots are put in order once for all of them (once per piece it took
    // 44 us for 4096 tokens of 2880)
    const int chunks = hidden / 8, lane = threadIdx.x & 31, warps = (int)((gridDim.x * blockDim.x) >> 5);
    const bool out16 = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    const int segs = min((chunks + 31) / 32, (warps + tokens - 1) / tokens);
    for (int job = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); job < tokens * segs; job += warps) {
        const int t = job / segs, seg = job - t * segs;
        int order[MOE_MAX_TOPK], ids[MOE_MAX_TOPK];
#pragma unroll
        for (int s = 0; s < MOE_MAX_TOPK; s++) {
            order[s] = s;
            ids[s] = s < top_k ? ld_produced(top_idx + (size_t)t * top_k + s) : 0x7FFFFFFF;
        }
#pragma unroll
        for (int a = 1; a < MOE_MAX_TOPK; a++) // insertion sort by expert id (k <= 8), in registers
#pragma unroll
            for (int b = a; b > 0; b--)
                if (ids[b] < ids[b - 1]) {
                    const int ti = ids[b]; ids[b] = ids[b - 1]; ids[b - 1] = ti;
                    const int to = order[b]; order[b] = order[b - 1]; order[b - 1] = to;
                }
        // all index loads first, then all row loads, then the sums in ascending expert order: the loads of a token's
        // slots do not wait for one another
        int pos[MOE_MAX_TOPK];
        float wv[MOE_MAX_TOPK];
        bool use[MOE_MAX_TOPK];
#pragma unroll
        for (int s = 0; s < MOE_MAX_TOPK; s++) {
            use[s] = s < top_k && ids[s] >= e_lo && ids[s] < e_hi;
            const size_t pair = (size_t)t * top_k + order[s];
            pos[s] = !use[s] ? 0 : inv ? ld_produced(inv + pair) : (int)pair;
            wv[s] = use[s] ? ld_produced(top_w + pair) : 0.0f;
        }
        for (int c = seg * 32 + lane; c < chunks; c += segs * 32) {
        uint4 rows[MOE_MAX_TOPK];
#pragma unroll
        for (int s = 0; s < MOE_MAX_TOPK; s++)
            rows[s] = use[s] ? reinterpret_cast<const uint4 *>(yp + (size_t)pos[s] * hidden)[c] : make_uint4(0u, 0u, 0u, 0u);
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int s = 0; s < MOE_MAX_TOPK; s++) {
            if (!use[s]) continue;
            const float w = wv[s];
            const uint32_t vv[4] = {rows[s].x, rows[s].y, rows[s].z, rows[s].w};
#pragma unroll
            for (int q = 0; q < 4; q++) {
                acc[2 * q] = fmaf(w, __uint_as_float(vv[q] << 16), acc[2 * q]);
                acc[2 * q + 1] = fmaf(w, __uint_as_float(vv[q] & 0xFFFF0000u), acc[2 * q + 1]);
            }
        }
        if (out_dtype == OXQ_BF16 && out16) {
            uint4 o;
            uint32_t *ov = reinterpret_cast<uint32_t *>(&o);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const __nv_bfloat162 b = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
                ov[q] = *reinterpret_cast<const uint32_t *>(&b);
            }
            reinterpret_cast<uint4 *>(out)[(size_t)t * chunks + c] = o;
        } else {
            for (int q = 0; q < 8; q++) store_as(out, out_dtype, (size_t)t * hidden + c * 8 + q, acc[q]);
        }
        }
    }
}

// offsets = exclusive scan of counts (one warp; at most MOE_MAX_EXPERTS entries).
__global__ void moe_offsets_kernel(const int *__restrict__ counts, int n, int *__restrict__ offsets)
{
    __shared__ int cnt_s[MOE_MAX_EXPERTS];
    for (int i = threadIdx.x; i < n; i += blockDim.x) cnt_s[i] = counts[i];
    __syncthreads();
    if (threadIdx.x != 0) return;
    int off = 0;
    for (int i = 0; i < n; i++) { offsets[i] = off; off += cnt_s[i]; }
    offsets[n] = off;
}

// ids of rows that arrive grouped: group g (source rank g / n_local, local expert g % n_local) holds counts[g] rows of
// expert lo + g % n_local. One CTA: scan of the group sizes in shared memory, then every thread fills whole groups.
__global__ void __launch_bounds__(1024)
moe_expand_ids_kernel(const int *__restrict__ counts, int groups, int n_local, int lo, int *__restrict__ ids)
{
    __shared__ int start_s[2049];
    if (threadIdx.x == 0) {
        int off = 0;
        for (int g = 0; g < groups; g++) { start_s[g] = off; off += counts[g]; }
        start_s[groups] = off;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int g = warp; g < groups; g += 32) {
        const int a = start_s[g], b = start_s[g + 1], e = lo + g % n_local;
        for (int i = a + lane; i < b; i += 32) ids[i] = e;
    }
}

static size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct MoeLayout {
    size_t top_idx, top_w, counts, offsets, grp_beg, entries, perm, inv, xs, h, slab, total;
    size_t h_scales, h_second, x_pieces, x_scales, x_second; // inside the slab
    int group_experts, n_groups, max_mt;
    bool small; // few pairs: no dequantized slab, the block-scaled kernel serves every layer
};

static MoeLayout moe_layout(int tokens, int top_k, int n_exp, int hidden, int inter)
{
    MoeLayout L;
    const size_t pairs = (size_t)tokens * top_k;
    // Experts dequantized at once: as many as fit 1152 MiB of bf16 gate_up weights (all 32 experts of
    // a GPT-OSS-20B layer), at least one. One grouped GEMM over many experts fills whole rounds of
    // the persistent grid; small groups left a third of the SM-rounds idle and paid a launch each.
    const size_t per_expert = (size_t)2 * inter * hidden * 2;
    int ge = (int)(((size_t)1152 << 20) / per_expert);
    if (ge < 1) ge = 1;
    if (ge > n_exp) ge = n_exp;
    L.group_experts = ge;
    L.n_groups = (n_exp + ge - 1) / ge;
    L.max_mt = (int)(pairs / moe_mx_block_rows()) + n_exp + 1;
    size_t off = 256;
    L.top_idx = off; off = align_up(off + pairs * 4, 256);
    L.top_w = off; off = align_up(off + pairs * 4, 256);
    L.counts = off; off = align_up(off + (size_t)n_exp * 4, 256);
    L.offsets = off; off = align_up(off + (size_t)(n_exp + 1) * 4, 256);
    L.grp_beg = off; off = align_up(off + (size_t)(L.n_groups + 1) * 4, 256);
    L.entries = off; off = align_up(off + (size_t)L.max_mt * 16, 256);
    L.perm = off; off = align_up(off + pairs * 4, 256);
    L.inv = off; off = align_up(off + pairs * 4, 256);
    L.xs = off; off = align_up(off + (pairs + 128) * hidden * 2, 256); // also the down-projection output
    L.h = off; off = align_up(off + (pairs + 128) * inter * 2, 256);
    L.small = pairs <= (size_t)MOE_FRONT_PAIRS && hidden <= MOE_SMALL_MAX_K && inter <= MOE_SMALL_MAX_K;
    // dequantized experts; or, for the block-scaled kernel, the pieces of h and of x with their scales and
    // what says which of them have a second pair
    const int cap = (int)pairs + 128;
    L.h_scales = align_up(moe_mx_piece_bytes(cap, inter), 256);
    L.h_second = L.h_scales + align_up(moe_mx_scale_bytes(cap, inter), 256);
    L.x_pieces = L.h_second + align_up(moe_mx_second_bytes(cap, inter), 256);
    L.x_scales = L.x_pieces + align_up(moe_mx_piece_bytes(cap, hidden), 256);
    L.x_second = L.x_scales + align_up(moe_mx_scale_bytes(cap, hidden), 256);
    const size_t mx = L.x_second + moe_mx_second_bytes(cap, hidden);
    const size_t dense = (size_t)ge * per_expert;
    L.slab = off; off = align_up(off + (L.small || dense < mx ? mx : dense), 256);
    L.total = off;
    return L;
}

} // namespace oxq

using namespace oxq;

OXQ_EXPORT size_t oxq_gptoss_moe_workspace_bytes(int tokens, int top_k, int num_local_experts, int hidden, int inter)
{
    if (tokens <= 0 || top_k <= 0 || num_local_experts <= 0 || hidden <= 0 || inter <= 0) return 0;
    return moe_layout(tokens, top_k, num_local_experts, hidden, inter).total;
}

// Rows that already carry their expert: top_idx = the given id, weight one (the owner side of expert parallelism).
__global__ void __launch_bounds__(256) moe_assign_kernel(const int32_t *__restrict__ ids, int rows, int *__restrict__ top_idx,
                                                         float *__restrict__ top_w)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < rows) { top_idx[i] = ids[i]; top_w[i] = 1.0f; }
}

static int moe_forward_impl(const void *x, int x_dtype, const void *router_logits, int logits_dtype, const int32_t *given_ids, int tokens,
                            int num_experts, int top_k, int norm_topk, int hidden, int inter, const uint8_t *gu_blocks,
                            const uint8_t *gu_scales, const void *gu_bias, const uint8_t *dn_blocks,
                            const uint8_t *dn_scales, const void *dn_bias, int bias_dtype, float limit,
                            int expert_lo, int expert_hi, void *out, int out_dtype, void *workspace,
                            size_t workspace_bytes, void *stream)
{
    OXQ_REQUIRE(x && (router_logits || given_ids) && gu_blocks && gu_scales && dn_blocks && dn_scales && out, OXQ_ERR_NULL,
                "oxq_gptoss_moe_forward: null pointer");
    OXQ_REQUIRE(x_dtype == OXQ_BF16, OXQ_ERR_UNSUPPORTED, "oxq_gptoss_moe_forward: activations must be bf16");
    OXQ_REQUIRE(valid_dtype(out_dtype) && (!(gu_bias || dn_bias) || valid_dtype(bias_dtype)), OXQ_ERR_UNSUPPORTED,
                "oxq_gptoss_moe_forward: unsupported dtype");
    OXQ_REQUIRE(tokens > 0 && num_experts > 0 && num_experts <= MOE_MAX_EXPERTS && top_k > 0 && top_k <= MOE_MAX_TOPK &&
                    top_k <= num_experts,
                OXQ_ERR_BAD_SHAPE, "oxq_gptoss_moe_forward: tokens %d, experts %d (max %d), top_k %d (max %d)", tokens,
                num_experts, MOE_MAX_EXPERTS, top_k, MOE_MAX_TOPK);
    OXQ_REQUIRE(hidden % 32 == 0 && inter % 32 == 0, OXQ_ERR_BAD_SHAPE,
                "Mxfp4Linear: in_features (%d, %d) must be a multiple of 32", hidden, inter);
    OXQ_REQUIRE(0 <= expert_lo && expert_lo < expert_hi && expert_hi <= num_experts, OXQ_ERR_BAD_SHAPE,
                "oxq_gptoss_moe_forward: expert range [%d, %d) outside 0..%d", expert_lo, expert_hi, num_experts);
    const int n_exp = expert_hi - expert_lo;
    const MoeLayout L = moe_layout(tokens, top_k, n_exp, hidden, inter);
    OXQ_REQUIRE(workspace && workspace_bytes >= L.total, OXQ_ERR_WORKSPACE,
                "oxq_gptoss_moe_forward: workspace of %zu bytes needed, got %zu", L.total, workspace_bytes);
    OXQ_REQUIRE(aligned(workspace, 256) && aligned(x, 16), OXQ_ERR_BAD_ALIGN,
                "oxq_gptoss_moe_forward: workspace must be 256-byte and x 16-byte aligned");

    cudaStream_t st = (cudaStream_t)stream;
    unsigned char *ws = reinterpret_cast<unsigned char *>(workspace);
    int *flag = reinterpret_cast<int *>(ws);
    int *top_idx = reinterpret_cast<int *>(ws + L.top_idx);
    float *top_w = reinterpret_cast<float *>(ws + L.top_w);
    int *counts = reinterpret_cast<int *>(ws + L.counts), *offsets = reinterpret_cast<int *>(ws + L.offsets);
    int *grp_beg = reinterpret_cast<int *>(ws + L.grp_beg);
    int4 *entries = reinterpret_cast<int4 *>(ws + L.entries);
    int *perm = reinterpret_cast<int *>(ws + L.perm), *inv = reinterpret_cast<int *>(ws + L.inv);
    __nv_bfloat16 *xs = reinterpret_cast<__nv_bfloat16 *>(ws + L.xs), *h = reinterpret_cast<__nv_bfloat16 *>(ws + L.h);
    __nv_bfloat16 *slab = reinterpret_cast<__nv_bfloat16 *>(ws + L.slab);
    const int pairs = tokens * top_k;

    const int a_rows = pairs + 128;
    // Both projections through the kernel that unpacks the MXFP4 blocks inside the tensor-core loop, where it takes the shapes:
    // no dequantized slab, one launch per projection over all experts.
    const bool fused = moe_fused_supported(2 * inter, hidden, gu_blocks, gu_scales, xs, h, inter) &&
                       moe_fused_supported(hidden, inter, dn_blocks, dn_scales, h, xs, hidden);
    // The experts that the pairs are spread over: with router logits all of them, whichever are local; rows that are given with
    // their experts are all local.
    const int spread = given_ids ? n_exp : num_experts;
    // Up to a few dozen rows per expert: the codes as tensor-core operands, nothing unpacked.
    const bool mx = (pairs <= MOE_MX_ROWS * spread || pairs <= MOE_FRONT_PAIRS) && moe_mx_supported(2 * inter, hidden, gu_blocks, gu_scales) &&
                    moe_mx_supported(hidden, inter, dn_blocks, dn_scales);
    const bool front = mx && pairs <= MOE_FRONT_PAIRS; // routing is part of a larger kernel
    OXQ_REQUIRE(!L.small || (aligned(gu_blocks, 16) && aligned(dn_blocks, 16)), OXQ_ERR_BAD_ALIGN,
                "oxq_gptoss_moe_forward: expert blocks must be 16-byte aligned");
    if (given_ids && !front) moe_assign_kernel<<<ceil_div(tokens, 256), 256, 0, st>>>(given_ids, tokens, top_idx, top_w);
    else if (!front && num_experts <= 32)
        OXQ_CUDA(launch_early(moe_route_kernel<1>, ceil_div(tokens * 32, 256), 256, st, router_logits, logits_dtype, tokens, num_experts, top_k,
                              norm_topk, top_idx, top_w));
    else if (!front)
        OXQ_CUDA(launch_early(moe_route_kernel<MOE_MAX_EXPERTS / 32>, ceil_div(tokens * 32, 256), 256, st, router_logits, logits_dtype, tokens,
                              num_experts, top_k, norm_topk, top_idx, top_w));
    // the grouped kernel's table of token blocks goes where the m-tile table of the dense path would (same capacity bound);
    // grp_beg[0] then holds the number of blocks
    const int block_rows = mx ? moe_mx_block_rows() : moe_fused_block_rows(pairs / spread);
    if (front) {
    } else if ((fused || mx) && pairs <= MOE_SMALL_PAIRS) {
        OXQ_CUDA(launch_early(moe_dispatch_small_kernel, 1, 1024, st, top_idx, pairs, expert_lo, n_exp, block_rows, counts, offsets, entries,
                              grp_beg, perm, inv));
    } else {
        moe_count_kernel<<<n_exp, 1024, 0, st>>>(top_idx, pairs, expert_lo, counts);
        if (fused || mx) moe_plan_blocks_kernel<<<1, MOE_MAX_EXPERTS, 0, st>>>(counts, n_exp, expert_lo, block_rows, offsets,
                                                                         entries, grp_beg);
        else moe_plan_kernel<<<1, 32, 0, st>>>(counts, n_exp, expert_lo, L.group_experts, offsets, entries, grp_beg);
        moe_scatter_kernel<<<n_exp, 1024, 0, st>>>(top_idx, pairs, expert_lo, offsets, perm, inv);
    }
    if (mx) {
        unsigned char *sb = reinterpret_cast<unsigned char *>(slab);
        OXQ_LAUNCH_CHECK("moe routing kernels");
        const unsigned long long mark = mx_call_mark();
        int rc = OXQ_OK;
        if (front) {
            MoeFrontParams f = {};
            f.logits = router_logits; f.given = given_ids; f.x = (const __nv_bfloat16 *)x; f.logits_dtype = logits_dtype; f.tokens = tokens;
            f.experts = num_experts; f.top_k = top_k; f.norm_topk = norm_topk; f.e_lo = expert_lo; f.n_exp = n_exp; f.max_rows = block_rows;
            f.top_idx = top_idx; f.offsets = offsets; f.n_blocks = grp_beg; f.inv = inv; f.top_w = top_w; f.entries = entries;
            f.pieces = moe_mx_pieces(hidden, a_rows, sb + L.x_pieces, sb + L.x_scales, sb + L.x_second, mark);
            OXQ_CUDA(launch_early(moe_front_kernel, ceil_div(pairs * f.pieces.stages * 16, MOE_MAX_EXPERTS) + 1, MOE_MAX_EXPERTS, st, f));
        } else rc = moe_mx_split(x, perm, top_k, offsets + n_exp, pairs, hidden, a_rows, sb + L.x_pieces, sb + L.x_scales, sb + L.x_second, mark, st);
        if (rc) return rc;
        rc = moe_mx_grouped(sb + L.x_pieces, sb + L.x_scales, sb + L.x_second, mark, a_rows, gu_blocks, gu_scales, num_experts, 2 * inter, hidden,
                            entries, grp_beg, gu_bias, bias_dtype, h, inter, 1, limit, flag, st);
        if (rc) return rc;
        rc = moe_mx_split(h, nullptr, 1, offsets + n_exp, pairs, inter, a_rows, sb, sb + L.h_scales, sb + L.h_second, mark, st);
        if (rc) return rc;
        rc = moe_mx_grouped(sb, sb + L.h_scales, sb + L.h_second, mark, a_rows, dn_blocks, dn_scales, num_experts, hidden, inter, entries, grp_beg,
                            dn_bias, bias_dtype, xs, hidden, 0, limit, flag, st);
        if (rc) return rc;
        const int warps = tokens * ceil_div(hidden / 8, 32), most = sm_count() * 64; // a warp takes 32 pieces of 16 bytes of a token
        OXQ_CUDA(launch_early(moe_combine_kernel, ceil_div(warps < most ? warps : most, 8), 256, st, xs, top_idx, top_w, inv, tokens, top_k, hidden,
                              expert_lo, expert_hi, out, out_dtype));
        return OXQ_OK;
    }
    moe_gather_kernel<<<sm_count() * 8, 256, 0, st>>>((const __nv_bfloat16 *)x, perm, offsets + n_exp, top_k, hidden, xs);
    OXQ_LAUNCH_CHECK("moe routing kernels");

    if (fused) {
        int rc = moe_fused_grouped(xs, a_rows, gu_blocks, gu_scales, num_experts, 2 * inter, hidden, entries, grp_beg, block_rows,
                                   gu_bias, bias_dtype, h, inter, 1, limit, flag, st);
        if (rc) return rc;
        rc = moe_fused_grouped(h, a_rows, dn_blocks, dn_scales, num_experts, hidden, inter, entries, grp_beg, block_rows, dn_bias,
                               bias_dtype, xs, hidden, 0, limit, flag, st);
        if (rc) return rc;
        moe_combine_kernel<<<sm_count() * 8, 256, 0, st>>>(xs, top_idx, top_w, inv, tokens, top_k, hidden, expert_lo, expert_hi,
                                                         out, out_dtype);
        OXQ_LAUNCH_CHECK("moe_combine_kernel");
        return OXQ_OK;
    }
    const size_t gu_rows = (size_t)2 * inter, nbh = hidden / 32, nbi = inter / 32;
    for (int g = 0; g < L.n_groups; g++) { // gate_up + SwiGLU: h = act(xs . W_gu^T + b_gu)
        const int e0 = expert_lo + g * L.group_experts;
        const int ne = (e0 + L.group_experts <= expert_hi) ? L.group_experts : expert_hi - e0;
        int rc = mxfp4_dequant_rows_bf16(gu_blocks + (size_t)e0 * gu_rows * nbh * 16, gu_scales + (size_t)e0 * gu_rows * nbh,
                                         slab, hidden, 0, (int)(ne * gu_rows), st);
        if (rc) return rc;
        rc = gemm_grouped(xs, a_rows, slab, ne, e0, (int)gu_rows, hidden, entries, grp_beg, g, gu_bias, bias_dtype, h,
                          inter, 1, limit, flag, st);
        if (rc) return rc;
    }
    for (int g = 0; g < L.n_groups; g++) { // down: yp = h . W_dn^T + b_dn (into the xs buffer)
        const int e0 = expert_lo + g * L.group_experts;
        const int ne = (e0 + L.group_experts <= expert_hi) ? L.group_experts : expert_hi - e0;
        int rc = mxfp4_dequant_rows_bf16(dn_blocks + (size_t)e0 * hidden * nbi * 16, dn_scales + (size_t)e0 * hidden * nbi,
                                         slab, inter, 0, ne * hidden, st);
        if (rc) return rc;
        rc = gemm_grouped(h, a_rows, slab, ne, e0, hidden, inter, entries, grp_beg, g, dn_bias, bias_dtype, xs, hidden,
                          0, limit, flag, st);
        if (rc) return rc;
    }
    moe_combine_kernel<<<sm_count() * 8, 256, 0, st>>>(xs, top_idx, top_w, inv, tokens, top_k, hidden, expert_lo, expert_hi, out,
                                                out_dtype);
    OXQ_LAUNCH_CHECK("moe_combine_kernel");
    return OXQ_OK;
}

OXQ_EXPORT int oxq_gptoss_moe_forward(const void *x, int x_dtype, const float *router_logits, int tokens, int num_experts,
                                      int top_k, int norm_topk, int hidden, int inter, const uint8_t *gu_blocks,
                                      const uint8_t *gu_scales, const void *gu_bias, const uint8_t *dn_blocks,
                                      const uint8_t *dn_scales, const void *dn_bias, int bias_dtype, float limit,
                                      int expert_lo, int expert_hi, void *out, int out_dtype, void *workspace,
                                      size_t workspace_bytes, void *stream)
{
    clear_error();
    OXQ_REQUIRE(router_logits != nullptr, OXQ_ERR_NULL, "oxq_gptoss_moe_forward: null pointer");
    return moe_forward_impl(x, x_dtype, router_logits, OXQ_F32, nullptr, tokens, num_experts, top_k, norm_topk, hidden, inter, gu_blocks,
                            gu_scales, gu_bias, dn_blocks, dn_scales, dn_bias, bias_dtype, limit, expert_lo, expert_hi, out,
                            out_dtype, workspace, workspace_bytes, stream);
}

// The same on router logits of any supported dtype, as the router's linear returns them.
OXQ_EXPORT int oxq_gptoss_moe_forward_logits(const void *x, int x_dtype, const void *router_logits, int logits_dtype, int tokens,
                                             int num_experts, int top_k, int norm_topk, int hidden, int inter, const uint8_t *gu_blocks,
                                             const uint8_t *gu_scales, const void *gu_bias, const uint8_t *dn_blocks,
                                             const uint8_t *dn_scales, const void *dn_bias, int bias_dtype, float limit,
                                             int expert_lo, int expert_hi, void *out, int out_dtype, void *workspace,
                                             size_t workspace_bytes, void *stream)
{
    clear_error();
    OXQ_REQUIRE(router_logits != nullptr, OXQ_ERR_NULL, "oxq_gptoss_moe_forward: null pointer");
    OXQ_REQUIRE(valid_dtype(logits_dtype), OXQ_ERR_UNSUPPORTED, "oxq_gptoss_moe_forward: unsupported dtype");
    return moe_forward_impl(x, x_dtype, router_logits, logits_dtype, nullptr, tokens, num_experts, top_k, norm_topk, hidden, inter,
                            gu_blocks, gu_scales, gu_bias, dn_blocks, dn_scales, dn_bias, bias_dtype, limit, expert_lo, expert_hi, out,
                            out_dtype, workspace, workspace_bytes, stream);
}

// Each row through the expert it is already assigned to, weight one: out[r] = expert[ids[r]](rows[r]).
OXQ_EXPORT int oxq_gptoss_experts_forward(const void *rows, int x_dtype, const int32_t *expert_ids, int n_rows, int num_experts,
                                          int hidden, int inter, const uint8_t *gu_blocks, const uint8_t *gu_scales,
                                          const void *gu_bias, const uint8_t *dn_blocks, const uint8_t *dn_scales,
                                          const void *dn_bias, int bias_dtype, float limit, int expert_lo, int expert_hi,
                                          void *out, int out_dtype, void *workspace, size_t workspace_bytes, void *stream)
{
    clear_error();
    OXQ_REQUIRE(expert_ids != nullptr, OXQ_ERR_NULL, "oxq_gptoss_experts_forward: null pointer");
    return moe_forward_impl(rows, x_dtype, nullptr, OXQ_F32, expert_ids, n_rows, num_experts, 1, 0, hidden, inter, gu_blocks, gu_scales,
                            gu_bias, dn_blocks, dn_scales, dn_bias, bias_dtype, limit, expert_lo, expert_hi, out, out_dtype,
                            workspace, workspace_bytes, stream);
}

// Weighted sum of each token's k result rows in ascending expert order (moe.rs:593-605: index_add per expert in order):
// out[t] = sum_s top_w[t, s] * rows[pos[t * k + s]]; f32 accumulation, one rounding. Same bits every run.
OXQ_EXPORT int oxq_moe_combine(const void *rows, const int32_t *top_idx, const float *top_w, const int32_t *pos, int tokens,
                               int top_k, int hidden, int num_experts, void *out, int out_dtype, void *stream)
{
    clear_error();
    OXQ_REQUIRE(rows && top_idx && top_w && pos && out, OXQ_ERR_NULL, "oxq_moe_combine: null pointer");
    OXQ_REQUIRE(valid_dtype(out_dtype), OXQ_ERR_UNSUPPORTED, "oxq_moe_combine: unsupported dtype");
    OXQ_REQUIRE(tokens > 0 && top_k > 0 && top_k <= MOE_MAX_TOPK && hidden > 0 && hidden % 8 == 0, OXQ_ERR_BAD_SHAPE,
                "oxq_moe_combine: tokens %d, top_k %d (max %d), hidden %d (multiple of 8)", tokens, top_k, MOE_MAX_TOPK, hidden);
    OXQ_REQUIRE(aligned(rows, 16), OXQ_ERR_BAD_ALIGN, "oxq_moe_combine: rows must be 16-byte aligned");
    moe_combine_kernel<<<sm_count() * 8, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16 *)rows, top_idx, top_w, pos, tokens,
                                                                          top_k, hidden, 0, num_experts, out, out_dtype);
    OXQ_LAUNCH_CHECK("moe_combine_kernel");
    return OXQ_OK;
}

// Routing alone (moe.rs:472-487): top_idx i32 [tokens, top_k], top_w f32 [tokens, top_k].
OXQ_EXPORT int oxq_moe_route(const float *router_logits, int tokens, int num_experts, int top_k, int norm_topk,
                             int32_t *top_idx, float *top_w, void *stream)
{
    clear_error();
    OXQ_REQUIRE(router_logits && top_idx && top_w, OXQ_ERR_NULL, "oxq_moe_route: null pointer");
    OXQ_REQUIRE(tokens > 0 && num_experts > 0 && num_experts <= MOE_MAX_EXPERTS && top_k > 0 && top_k <= MOE_MAX_TOPK &&
                    top_k <= num_experts,
                OXQ_ERR_BAD_SHAPE, "oxq_moe_route: tokens %d, experts %d (max %d), top_k %d (max %d)", tokens, num_experts,
                MOE_MAX_EXPERTS, top_k, MOE_MAX_TOPK);
    auto kern = num_experts <= 32 ? moe_route_kernel<1> : moe_route_kernel<MOE_MAX_EXPERTS / 32>;
    kern<<<ceil_div(tokens * 32, 256), 256, 0, (cudaStream_t)stream>>>(router_logits, OXQ_F32, tokens, num_experts,
                                                                                    top_k, norm_topk, top_idx, top_w);
    OXQ_LAUNCH_CHECK("moe_route_kernel");
    return OXQ_OK;
}

// Dispatch plan of expert parallelism on the device (the sender side of dispatch_sparse, moe.rs:563-607, when experts live on
// other ranks): pairs (token, slot) sorted by expert id, pair order kept inside an expert. counts [E], offsets [E + 1],
// perm [pairs] (perm[i] = pair sent i-th), inv [pairs] (inv[pair] = its position). No counterpart in the reference.
OXQ_EXPORT int oxq_moe_dispatch_plan(const int32_t *top_idx, int pairs, int num_experts, int32_t *counts, int32_t *offsets,
                                     int32_t *perm, int32_t *inv, void *stream)
{
    clear_error();
    OXQ_REQUIRE(top_idx && counts && offsets && perm && inv, OXQ_ERR_NULL, "oxq_moe_dispatch_plan: null pointer");
    OXQ_REQUIRE(pairs > 0 && num_experts > 0 && num_experts <= MOE_MAX_EXPERTS, OXQ_ERR_BAD_SHAPE,
                "oxq_moe_dispatch_plan: pairs %d, experts %d (max %d)", pairs, num_experts, MOE_MAX_EXPERTS);
    OXQ_REQUIRE(aligned(top_idx, 16), OXQ_ERR_BAD_ALIGN, "oxq_moe_dispatch_plan: top_idx must be 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    moe_count_kernel<<<num_experts, 1024, 0, st>>>(top_idx, pairs, 0, counts);
    moe_offsets_kernel<<<1, 32, 0, st>>>(counts, num_experts, offsets);
    moe_scatter_kernel<<<num_experts, 1024, 0, st>>>(top_idx, pairs, 0, offsets, perm, inv);
    OXQ_LAUNCH_CHECK("moe dispatch plan kernels");
    return OXQ_OK;
}

// out[i, :] = x[perm[i] / top_k, :] for i < rows (bf16 rows, hidden a multiple of 8): the rows of a dispatch in send order.
OXQ_EXPORT int oxq_moe_gather_rows(const void *x, const int32_t *perm, int rows, int top_k, int hidden, void *out, void *stream)
{
    clear_error();
    OXQ_REQUIRE(x && perm && out, OXQ_ERR_NULL, "oxq_moe_gather_rows: null pointer");
    OXQ_REQUIRE(rows > 0 && top_k > 0 && hidden > 0 && hidden % 8 == 0, OXQ_ERR_BAD_SHAPE,
                "oxq_moe_gather_rows: rows %d, top_k %d, hidden %d (multiple of 8)", rows, top_k, hidden);
    OXQ_REQUIRE(aligned(x, 16) && aligned(out, 16), OXQ_ERR_BAD_ALIGN, "oxq_moe_gather_rows: rows must be 16-byte aligned");
    moe_gather_kernel<<<sm_count() * 8, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16 *)x, perm, nullptr, top_k, hidden,
                                                                         (__nv_bfloat16 *)out, rows);
    OXQ_LAUNCH_CHECK("moe_gather_kernel");
    return OXQ_OK;
}

// Expert ids of rows received in groups (source rank major, local expert minor): counts [world * n_local] -> ids [total].
OXQ_EXPORT int oxq_moe_expand_ids(const int32_t *counts, int groups, int n_local, int lo, int32_t *ids, void *stream)
{
    clear_error();
    OXQ_REQUIRE(counts && ids, OXQ_ERR_NULL, "oxq_moe_expand_ids: null pointer");
    OXQ_REQUIRE(groups > 0 && groups <= 2048 && n_local > 0 && groups % n_local == 0, OXQ_ERR_BAD_SHAPE,
                "oxq_moe_expand_ids: groups %d (at most 2048, a multiple of n_local %d)", groups, n_local);
    moe_expand_ids_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(counts, groups, n_local, lo, ids);
    OXQ_LAUNCH_CHECK("moe_expand_ids_kernel");
    return OXQ_OK;
}
