// Router kernels: logits in a pinned fp32 summation order, softmax + top-K selection, pair grouping by expert.
#pragma once
#include "common.cuh"
#include "rows.cuh"

namespace moexb {

__device__ __forceinline__ float4 ld_w4(const float* W, size_t k) { return __ldg(reinterpret_cast<const float4*>(W + k)); }
__device__ __forceinline__ float4 ld_w4(const __half* W, size_t k) {
    const uint2 u = __ldg(reinterpret_cast<const uint2*>(W + k));
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// Asks for a row of weights in L2. Weights that the kernel before this one may still write cannot be loaded before the wait for it, but
// they can be brought this far: what is written meanwhile arrives in L2 too.
template <typename WT>
__device__ __forceinline__ void prefetch_row(const WT* w, int I, int lane) {
    for (int b = 128 * lane; b < I * (int)sizeof(WT); b += 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint8_t*>(w) + b));
}

// y[r][o] = W[o] . x[r]. One warp per (row r, output o): lane j accumulates elements 128c+4j .. 128c+4j+3 for
// c = 0, 1, .. with fused multiply-adds in ascending order, then a xor-butterfly (16, 8, 4, 2, 1) adds the 32 partial
// sums. The CPU oracle follows the same order, so the logits - and with them the selected experts - agree bit for bit.
// Stands behind gemv_f16_k (kernels.cuh:73-91). grid (ceil(O / WARPS), rows).
template <typename WT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) gemv_rows_k(const WT* __restrict__ W, const float* __restrict__ x,
                                                          float* __restrict__ y, int I, int O) {
    const int o = blockIdx.x * WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (o >= O) return;
    const float* xr = x + (size_t)blockIdx.y * I;
    const WT* wr = W + (size_t)o * I;
    float acc = 0.f;
    constexpr int U = 16;  // loads of U steps are in flight before the first multiply-add; the summation order is unchanged
    if (blockIdx.y == 0) prefetch_row(wr, I, lane);
    pdl_wait();
    pdl_trigger();
    for (int c0 = 0; c0 < I / 128; c0 += U) {
        float4 w[U], v[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c0 + u < I / 128) { w[u] = ld_w4(wr, (size_t)128 * (c0 + u) + 4 * lane); v[u] = __ldg(reinterpret_cast<const float4*>(xr + 128 * (c0 + u) + 4 * lane)); }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c0 + u < I / 128) { acc = fmaf(w[u].x, v[u].x, acc); acc = fmaf(w[u].y, v[u].y, acc); acc = fmaf(w[u].z, v[u].z, acc); acc = fmaf(w[u].w, v[u].w, acc); }
    }
    acc = warp_sum(acc);
    if (lane == 0) y[(size_t)blockIdx.y * O + o] = acc;
}

// One tile of the batched rows: a block stages TR activation rows in shared memory and its WARPS warps each own TO outputs, with the
// weights of U steps requested at a time and the next U already in flight; a lane still holds elements 128c+4j..4j+3 of every dot
// product, so every (row, output) sum is formed in exactly the order of gemv_rows_k and the kernels agree bit for bit.
// Waits for the kernel before (pdl_wait); EARLY: only once its first weights, which that kernel must not write, are requested.
// Dynamic shared memory TR * I floats.
template <typename WT, int WARPS, int TO, int TR, int U, bool EARLY>
__device__ __forceinline__ void gemm_tile(const WT* __restrict__ W, const float* __restrict__ x, float* __restrict__ y, int I, int O, int rows) {
    extern __shared__ __align__(16) float xsm[];  // [TR][I]
    const int r0 = blockIdx.y * TR, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int o0 = (blockIdx.x * WARPS + warp) * TO;
    const WT* wr[TO];
#pragma unroll
    for (int i = 0; i < TO; i++) wr[i] = W + (size_t)min(o0 + i, O - 1) * I;
    float4 wn[TO][U];  // the weights of the next U steps
    auto load_w = [&](int c0) {
#pragma unroll
        for (int i = 0; i < TO; i++)
#pragma unroll
            for (int u = 0; u < U; u++)
                if (c0 + u < I / 128) wn[i][u] = ld_w4(wr[i], (size_t)128 * (c0 + u) + 4 * lane);
    };
    if (EARLY) load_w(0);
    else if (blockIdx.y == 0)
#pragma unroll
        for (int i = 0; i < TO; i++) prefetch_row(wr[i], I, lane);
    pdl_wait();
    pdl_trigger();
    if (!EARLY) load_w(0);
    for (int r = 0; r < TR; r++) {   // the tile's token rows: 16-byte asynchronous copies, all in flight at once
        const float* src = x + (size_t)min(r0 + r, rows - 1) * I;
        for (int c = threadIdx.x * 4; c < I; c += WARPS * 128) cp_async16(smem_u32(xsm + r * I + c), src + c);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    float acc[TR][TO];
#pragma unroll
    for (int r = 0; r < TR; r++)
#pragma unroll
        for (int i = 0; i < TO; i++) acc[r][i] = 0.f;
    for (int c0 = 0; c0 < I / 128; c0 += U) {
        float4 w[TO][U];
#pragma unroll
        for (int i = 0; i < TO; i++)
#pragma unroll
            for (int u = 0; u < U; u++) w[i][u] = wn[i][u];
        if (c0 + U < I / 128) load_w(c0 + U);
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (c0 + u >= I / 128) break;
#pragma unroll
            for (int r = 0; r < TR; r++) {
                const float4 v = *reinterpret_cast<const float4*>(xsm + r * I + 128 * (c0 + u) + 4 * lane);
#pragma unroll
                for (int i = 0; i < TO; i++) {
                    float a = acc[r][i];
                    a = fmaf(w[i][u].x, v.x, a); a = fmaf(w[i][u].y, v.y, a); a = fmaf(w[i][u].z, v.z, a); a = fmaf(w[i][u].w, v.w, a);
                    acc[r][i] = a;
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < TR; r++)
#pragma unroll
        for (int i = 0; i < TO; i++) {
            const float sum = warp_sum(acc[r][i]);
            if (lane == 0 && r0 + r < rows && o0 + i < O) y[(size_t)(r0 + r) * O + o0 + i] = sum;
        }
}

// The same result for many rows (a batch or a prefill chunk).
// grid (ceil(O / (WARPS*TO)), ceil(rows / TR)); dynamic shared memory TR * I floats.
template <typename WT, int WARPS, int TO, int TR, int U>
__global__ void __launch_bounds__(WARPS * 32) gemm_rows_k(const WT* __restrict__ W, const float* __restrict__ x,
                                                          float* __restrict__ y, int I, int O, int rows) {
    gemm_tile<WT, WARPS, TO, TR, U, false>(W, x, y, I, O, rows);
}

// Softmax over E logits and the K largest by one warp (kernels.cuh:373-406 does it with a block per token).
// Lane l holds logits l, l+32, ..; each round every lane offers its best remaining value as an order-preserving
// integer key, one warp reduction finds the largest key and a second the lowest index that holds it (ties go to the
// lower index), and the winner is struck from its owner's mask. Selection compares logits (softmax is monotone). NaN
// logits count as -inf. Optional decode outputs: slots_out / wts_out [K+1] = the selected experts' blob pointers and
// weights followed by the shared expert with weight sigmoid(logits[E]); dsubs / dpairs / dnsub = the same K+1 experts as
// one-pair sub-items for the streaming kernels (T = 1).
constexpr int BK_ERR_FULL = 4;
struct TopkOut {
    int* idx; float* w;
    const uint8_t* const* slot_table; const uint8_t** slots_out; float* wts_out;
    moexb_pair_item* dsubs; moexb_pair* dpairs; int* dnsub;
    // expert parallelism (ep.cuh): the warp that selected a token's experts also sends the token to the peers - ids and
    // weights to every rank, the activation row (ep_row_bytes at [token] of the exchange buffer's row area) to the ranks that
    // hold one of the selected experts - and the block then raises the tokens' dispatch flags
    const EpDevice* ep = nullptr; int ep_row_bytes = 0; unsigned ep_phase = 0; const unsigned* ep_step = nullptr;
    // the pairs into the experts' buckets (BucketArgs): experts [e_lo, e_hi) are held here; npairs = T * K
    int* bcnt = nullptr; moexb_pair* bpairs = nullptr; int bstride = 0, e_lo = 0, e_hi = 0, npairs = 0; bool bshared = false; int* err = nullptr;
    int* idx2 = nullptr; float* w2 = nullptr;   // a second copy of ids and weights (the caller's buffers)
};
__device__ __forceinline__ unsigned f2key(float v) { const unsigned u = __float_as_uint(v); return (u & 0x80000000u) ? ~u : (u | 0x80000000u); }
__device__ __forceinline__ float key2f(unsigned k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }

// CG: the logits were written by other blocks of the same launch - read them past L1.
template <int NJ, bool CG>
__device__ __forceinline__ void topk_token(const float* __restrict__ l, int t, int E, int K, int norm, int lane, const TopkOut& o) {
    const int nj = E >> 5;  // <= NJ
    float v[NJ];
    float m = -INFINITY;
#pragma unroll
    for (int j = 0; j < NJ; j++) {
        v[j] = -INFINITY;
        if (j < nj) { const float a = CG ? __ldcg(l + lane + 32 * j) : l[lane + 32 * j]; v[j] = a != a ? -INFINITY : a; }
        m = fmaxf(m, v[j]);
    }
    const float gate_logit = ((o.slots_out || o.bshared) && lane == K) ? (CG ? __ldcg(l + E) : l[E]) : 0.f;
#pragma unroll
    for (int off = 16; off; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    unsigned key[NJ];
#pragma unroll
    for (int j = 0; j < NJ; j++) key[j] = j < nj ? f2key(v[j]) : 0u;  // 0 = not a candidate (below every real key)
    // K rounds, each two warp reductions: the largest remaining key, then the lowest index that holds it. Between them a lane
    // only has to know its own best remaining key, kept by a tree of comparisons that every lane runs without branching (the
    // lower slot wins among equals). The softmax denominator is summed inside the rounds, where the reductions leave issue
    // slots free: one term per round, the rest after the last one.
    int mine_i = 0;
    unsigned mine_key = 0u;
    unsigned bk; int bj;
    auto best = [&] {   // (bk, bj) = the lane's largest key and its lowest slot
        unsigned k2[NJ / 2 > 0 ? NJ / 2 : 1]; int j2[NJ / 2 > 0 ? NJ / 2 : 1];
#pragma unroll
        for (int j = 0; j < NJ / 2; j++) { const bool l = key[2 * j] >= key[2 * j + 1]; k2[j] = l ? key[2 * j] : key[2 * j + 1]; j2[j] = l ? 2 * j : 2 * j + 1; }
#pragma unroll
        for (int w = NJ / 2; w > 1; w >>= 1)
#pragma unroll
            for (int j = 0; j < w / 2; j++) { const bool l = k2[2 * j] >= k2[2 * j + 1]; k2[j] = l ? k2[2 * j] : k2[2 * j + 1]; j2[j] = l ? j2[2 * j] : j2[2 * j + 1]; }
        bk = k2[0]; bj = j2[0];
    };
    best();
    float sum = 0.f;
    for (int k = 0; k < K; k++) {
        const unsigned top = __reduce_max_sync(0xffffffffu, bk);
        const unsigned win = __reduce_min_sync(0xffffffffu, bk == top ? (unsigned)(lane + 32 * bj) : 0x7fffffffu);
        const bool won = (int)(win & 31) == lane;
#pragma unroll
        for (int j = 0; j < NJ; j++) if (won && j == (int)(win >> 5)) key[j] = 0u;
        best();
        if (lane == k) { mine_key = top; mine_i = (int)win; }
#pragma unroll
        for (int j = 0; j < NJ; j++) if (j == k && j < nj) sum += expf(v[j] - m);
    }
#pragma unroll
    for (int j = 0; j < NJ; j++) if (j >= K && j < nj) sum += expf(v[j] - m);
    sum = warp_sum(sum);
    // the K probabilities at once, and their sum in selection order
    float mine = 0.f, total = 0.f;  // lane k keeps the k-th probability
    if (lane < K) mine = expf(key2f(mine_key) - m) / sum;
    for (int k = 0; k < K; k++) total += __shfl_sync(0xffffffffu, mine, k);
    if (lane < K) {
        const float wk = norm ? mine / total : mine;
        o.idx[(size_t)t * K + lane] = mine_i;
        o.w[(size_t)t * K + lane] = wk;
        if (o.bpairs && mine_i >= o.e_lo && mine_i < o.e_hi) {
            const int place = atomicAdd(o.bcnt + mine_i, 1);
            // an expert takes each token once, so a place beyond the bucket means counts that were not zero when the call began
            if (place < o.bstride) o.bpairs[(size_t)mine_i * o.bstride + place] = {t, t * K + lane, wk};
            else atomicExch(o.err, BK_ERR_FULL);
        }
        if (o.idx2) o.idx2[(size_t)t * K + lane] = mine_i;
        if (o.w2) o.w2[(size_t)t * K + lane] = wk;
        if (o.slots_out) { o.slots_out[(size_t)t * (K + 1) + lane] = o.slot_table[mine_i]; o.wts_out[(size_t)t * (K + 1) + lane] = wk; }
        if (o.dsubs) { o.dsubs[lane] = {o.slot_table[mine_i], lane, 1}; o.dpairs[lane] = {0, lane, wk}; }  // one token: expert k = sub-item k
    }
    if (o.bshared && lane == K) o.bpairs[(size_t)E * o.bstride + t] = {t, o.npairs + t, 1.f / (1.f + expf(-gate_logit))};
    if (o.slots_out && lane == K) {
        const float gate = 1.f / (1.f + expf(-gate_logit));
        o.slots_out[(size_t)t * (K + 1) + K] = o.slot_table[E];
        o.wts_out[(size_t)t * (K + 1) + K] = gate;
        if (o.dsubs) { o.dsubs[K] = {o.slot_table[E], K, 1}; o.dpairs[K] = {0, K, gate}; o.dnsub[0] = K + 1; o.dnsub[1] = 0; }
    }
    if (o.ep) {
        const EpDevice& ep = *o.ep;
        const int rank = ep.g.rank, ta = ep.g.tok0[rank] + t;   // t counts from this rank's first token
        unsigned need = 0;
        if (lane < K)
            for (int s = 0; s < ep.g.world; s++) if (mine_i >= ep.g.exp0[s] && mine_i < ep.g.exp0[s + 1]) need = 1u << s;
        need = __reduce_or_sync(0xffffffffu, need);
        const float wk = norm ? mine / total : mine;
        // the row (at most 8 KB = 16 x 16 bytes per lane) is read once, every load in flight before the first store
        const uint4* src = reinterpret_cast<const uint4*>(ep.p.base[rank] + ep.lay.xs + (size_t)ta * o.ep_row_bytes);
        const int n16 = o.ep_row_bytes / 16;
        uint4 v[16];
        if (need & ~(1u << rank)) {
#pragma unroll
            for (int j = 0; j < 16; j++) if (lane + 32 * j < n16) v[j] = src[lane + 32 * j];
        }
        for (int d = 0; d < ep.g.world; d++) {
            if (d == rank) continue;
            uint8_t* db = ep.p.base[d];
            if (lane < K) {
                reinterpret_cast<int*>(db + ep.lay.idx)[(size_t)ta * K + lane] = mine_i;
                reinterpret_cast<float*>(db + ep.lay.w)[(size_t)ta * K + lane] = wk;
            }
            if (need >> d & 1) {
                uint4* out = reinterpret_cast<uint4*>(db + ep.lay.xs + (size_t)ta * o.ep_row_bytes);
#pragma unroll
                for (int j = 0; j < 16; j++) if (lane + 32 * j < n16) out[lane + 32 * j] = v[j];
            }
        }
    }
}

// After the warps of a block have sent tokens [t_first, t_first + n) of this rank (topk_token with o.ep): one system-scope
// fence by one thread behind the block barrier, then the tokens' dispatch flags on every peer.
__device__ __forceinline__ void ep_raise_dispatch_flags(const TopkOut& o, int t_first, int n) {
    if (!o.ep) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        const EpDevice& ep = *o.ep;
        const unsigned value = *o.ep_step * EP_PHASES + o.ep_phase;
        __threadfence_system();
        for (int d = 0; d < ep.g.world; d++) {
            if (d == ep.g.rank) continue;
            unsigned* flags = reinterpret_cast<unsigned*>(ep.p.base[d] + ep.lay.flag_a) + ep.g.tok0[ep.g.rank] + t_first;
            for (int i = 0; i < n; i++) st_relaxed_sys(flags + i, value);
        }
    }
}

// One warp per token.
template <int WARPS, int NJ>
__global__ void __launch_bounds__(WARPS * 32) router_topk_k(const float* __restrict__ logits, int E, int K, int norm, int ld, int T, const TopkOut o) {
    const int t = blockIdx.x * WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    pdl_wait();
    pdl_trigger();
    if (t >= T) return;
    topk_token<NJ, false>(logits + (size_t)t * ld, t, E, K, norm, lane, o);
}

// Whether this block is the last of `expected` blocks to reach this point for counter *cnt (every block calls it once,
// after its global writes); the last one sees the writes of all the others and resets the counter for the next launch.
__device__ __forceinline__ bool last_block_done(int* cnt, int expected) {
    __shared__ int s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();   // one fence per block: the barrier orders the block's writes before it, and it is cumulative
        const int ticket = atomicAdd(cnt, 1);
        s_last = ticket == expected - 1;
        if (s_last) { *cnt = 0; __threadfence(); }
    }
    __syncthreads();
    return s_last;
}

// Router logits and top-K selection of a few tokens in one launch: gemv_rows_k's grid (ceil(O / WARPS) blocks per
// token, O = E + 1), and the last block of a token to finish selects that token's experts - no second launch, no wait:
// the block that comes last simply does the extra work. done[t] must be zero before the first launch.
// x: f32 or bf16 rows. xs (a layer without a norm before it): one block more per token splits the token's row for the experts,
// instead of a launch before this one (mode: ROWS_F16 or ROWS_BF16).
template <typename WT, typename XT, int WARPS, int NJ>
__global__ void __launch_bounds__(WARPS * 32) route_gemv_k(const WT* __restrict__ W, const XT* __restrict__ x, float* __restrict__ y, int I,
                                                           int E, int K, int norm, int* __restrict__ done, const TopkOut o, uint16_t* __restrict__ xs, int mode) {
    static_assert(WARPS == 8, "256 threads split a row");
    const int O = E + 1, t = blockIdx.y;
    const int out = blockIdx.x * WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const XT* xr = x + (size_t)t * I;
    const WT* wr = W + (size_t)min(out, O - 1) * I;
    float acc = 0.f;
    constexpr int U = 16;
    auto steps = [&](int c0, const float4 (&w)[U]) {
        float4 v[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c0 + u < I / 128) v[u] = ld_x4(xr + 128 * (c0 + u) + 4 * lane);
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c0 + u < I / 128) { acc = fmaf(w[u].x, v[u].x, acc); acc = fmaf(w[u].y, v[u].y, acc); acc = fmaf(w[u].z, v[u].z, acc); acc = fmaf(w[u].w, v[u].w, acc); }
    };
    if (xs && blockIdx.x == gridDim.x - 1) {
        pdl_wait();
        pdl_trigger();
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int k0 = 1024 * h + 4 * threadIdx.x;
            const float4 p = ld_x4(xr + k0);
            const float f[4] = {p.x, p.y, p.z, p.w};
            if (mode == ROWS_F16) store_split4<ROWS_F16>(f, k0, xs + (size_t)t * 2 * EH, EH);
            else store_split4<ROWS_BF16>(f, k0, xs + (size_t)t * 2 * EH, EH);
        }
    } else {
        float4 w[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (u < I / 128) w[u] = ld_w4(wr, (size_t)128 * u + 4 * lane);
        pdl_wait();
        pdl_trigger();
        steps(0, w);
    }
    for (int c0 = U; c0 < I / 128; c0 += U) {
        float4 w[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c0 + u < I / 128) w[u] = ld_w4(wr, (size_t)128 * (c0 + u) + 4 * lane);
        steps(c0, w);
    }
    acc = warp_sum(acc);
    if (lane == 0 && out < O) y[(size_t)t * O + out] = acc;
    if (!last_block_done(done + t, gridDim.x)) return;
    if (threadIdx.x < 32) topk_token<NJ, true>(y + (size_t)t * O, t, E, K, norm, lane, o);
    ep_raise_dispatch_flags(o, t, 1);
}

// The same for a batch in gemm_tile's tiles; the last block of a token tile to finish selects the experts of its TR tokens (warp r
// takes tokens r, r + WARPS, ..).
// grid (ceil((E + 1) / (WARPS * TO)), ceil(T / TR)); dynamic shared memory TR * I floats;
// done[tile] zero before the first launch.
template <typename WT, int WARPS, int TO, int TR, int NJ>
__global__ void __launch_bounds__(WARPS * 32) route_gemm_k(const WT* __restrict__ W, const float* __restrict__ x, float* __restrict__ y, int I,
                                                           int E, int K, int norm, int T, int* __restrict__ done, const TopkOut o) {
    const int O = E + 1, r0 = blockIdx.y * TR, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // weights of 8 steps (half of I = 2048) at a time: the first arrive while the kernel before this one still runs (16 would spill)
    gemm_tile<WT, WARPS, TO, TR, 8, true>(W, x, y, I, O, T);
    if (!last_block_done(done + blockIdx.y, gridDim.x)) return;
    for (int r = warp; r < TR && r0 + r < T; r += WARPS) topk_token<NJ, true>(y + (size_t)(r0 + r) * O, r0 + r, E, K, norm, lane, o);
    ep_raise_dispatch_flags(o, r0, min(TR, T - r0));
}

// The sums of n accumulators over the 32 lanes of a warp, n / 32 of them left in each lane (lane l: accumulators l * n / 32 ..): at
// every step a lane keeps half of what it has and hands the other half to its partner. The additions are those of warp_sum's
// butterfly, so every sum has the same bits, with 124 shuffles for 128 accumulators instead of 640.
template <int N, int M = 16>
__device__ __forceinline__ void warp_sums(float* a, int lane) {
    const bool up = lane & M;
#pragma unroll
    for (int k = 0; k < N / 2; k++) {
        const float keep = up ? a[k + N / 2] : a[k], give = up ? a[k] : a[k + N / 2];
        a[k] = keep + __shfl_xor_sync(0xffffffffu, give, M);
    }
    if constexpr (M > 1) warp_sums<N / 2, M / 2>(a, lane);
}

// The logits of a prefill chunk, register-tiled. A block of 8 warps owns 64 tokens x 16 outputs; warp (wm, wn) the 16 tokens
// 16*wm.. and the 8 outputs 8*wn.., every lane the same 4 of each 128 inputs as in gemv_rows_k, so a lane holds 128 partial
// sums and each (token, output) sum is formed in the pinned order. Token and weight rows come through shared memory 128 inputs at a
// time (cp.async, four stages, one block per SM): per 128 inputs a warp reads 24 x 16 bytes per lane for 512 fused multiply-adds, so
// that the shared-memory reads stay below the multiply-adds; with half as many partial sums (32 tokens a block) they were equal.
// 2048 tokens: 77 us (125 with 32 tokens a block, 124 with two outputs per register pair and the two-wide multiply-add).
// The block of the last outputs, when it has only one (E + 1 = 257), takes it warp by warp.
// select (expert parallelism): the last block of a token tile selects the experts of its tokens; otherwise a kernel of its own does,
// with a warp per token on all SMs instead of eight tokens per warp on the last one. grid (ceil((E + 1) / 16), ceil(T / 64)); I = 2048.
constexpr int RG2_TM = 64, RG2_TN = 16, RG2_KC = 128, RG2_ST = 4;
template <typename WT> constexpr int rg2_stage_bytes() { return RG2_TM * RG2_KC * 4 + RG2_TN * RG2_KC * (int)sizeof(WT); }
template <typename WT, int NJ>
__global__ void __launch_bounds__(256, 1) route_gemm2_k(const WT* __restrict__ W, const float* __restrict__ x, float* __restrict__ y, int E, int K,
                                                     int norm, int T, int* __restrict__ done, const TopkOut o, int select) {
    constexpr int I = EH, NCH = I / RG2_KC, STAGE = rg2_stage_bytes<WT>();
    extern __shared__ __align__(16) uint8_t rsm[];   // stages of [64 tokens][128] f32 | [16 outputs][128] WT
    const int O = E + 1, r0 = blockIdx.y * RG2_TM, o0 = blockIdx.x * RG2_TN;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wm = warp >> 1, wn = warp & 1;
    if (O - o0 == 1) {
        pdl_wait();
        pdl_trigger();
        const WT* wr = W + (size_t)o0 * I;
        for (int r = r0 + warp; r < min(r0 + RG2_TM, T); r += 8) {
            float acc = 0.f;
#pragma unroll 8
            for (int c = 0; c < I / 128; c++) {
                const float4 w = ld_w4(wr, (size_t)128 * c + 4 * lane), v = __ldg(reinterpret_cast<const float4*>(x + (size_t)r * I + 128 * c + 4 * lane));
                acc = fmaf(w.x, v.x, acc); acc = fmaf(w.y, v.y, acc); acc = fmaf(w.z, v.z, acc); acc = fmaf(w.w, v.w, acc);
            }
            acc = warp_sum(acc);
            if (lane == 0) y[(size_t)r * O + o0] = acc;
        }
    } else {
        // thread: 16-byte piece tid % 32 of token rows tid / 32 + 8i; for the weights piece and row by PW pieces a row
        constexpr int PW = RG2_KC * (int)sizeof(WT) / 16;
        const float* xp[8]; const WT* wp[RG2_TN * PW / 256];
#pragma unroll
        for (int i = 0; i < 8; i++) xp[i] = x + (size_t)min(r0 + (tid >> 5) + 8 * i, T - 1) * I + 4 * (tid & 31);
#pragma unroll
        for (int i = 0; i < RG2_TN * PW / 256; i++) { const int u = tid + 256 * i; wp[i] = W + (size_t)min(o0 + u / PW, O - 1) * I + (u % PW) * (16 / (int)sizeof(WT)); }
        auto fill_w = [&](int ch) {
            const uint32_t ws = smem_u32(rsm + (ch % RG2_ST) * STAGE + RG2_TM * RG2_KC * 4) + 16 * tid;
#pragma unroll
            for (int i = 0; i < RG2_TN * PW / 256; i++) cp_async16(ws + 4096 * i, wp[i] + ch * RG2_KC);
        };
        auto fill_x = [&](int ch) {
            const uint32_t xs = smem_u32(rsm + (ch % RG2_ST) * STAGE) + 16 * tid;
#pragma unroll
            for (int i = 0; i < 8; i++) cp_async16(xs + 4096 * i, xp[i] + ch * RG2_KC);
        };
        for (int ch = 0; ch < RG2_ST - 1; ch++) fill_w(ch);   // weights do not depend on the kernel before this one
        pdl_wait();
        pdl_trigger();
        for (int ch = 0; ch < RG2_ST - 1; ch++) { fill_x(ch); asm volatile("cp.async.commit_group;" ::: "memory"); }
        float acc[128];
#pragma unroll
        for (int i = 0; i < 128; i++) acc[i] = 0.f;
#pragma unroll 1
        for (int ch = 0; ch < NCH; ch++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(RG2_ST - 2) : "memory");
            __syncthreads();   // chunk ch is in, and every warp is done with the stage that is filled next
            if (ch + RG2_ST - 1 < NCH) { fill_w(ch + RG2_ST - 1); fill_x(ch + RG2_ST - 1); }
            asm volatile("cp.async.commit_group;" ::: "memory");
            const float* xs = reinterpret_cast<const float*>(rsm + (ch % RG2_ST) * STAGE) + (size_t)(16 * wm) * RG2_KC + 4 * lane;
            const WT* ws = reinterpret_cast<const WT*>(rsm + (ch % RG2_ST) * STAGE + RG2_TM * RG2_KC * 4) + (size_t)(8 * wn) * RG2_KC + 4 * lane;
            float4 wv[8], v[2];
            v[0] = *reinterpret_cast<const float4*>(xs);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if constexpr (sizeof(WT) == 4) wv[j] = *reinterpret_cast<const float4*>(ws + (size_t)j * RG2_KC);
                else {
                    const uint2 h = *reinterpret_cast<const uint2*>(ws + (size_t)j * RG2_KC);
                    const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&h.x)), q = __half22float2(*reinterpret_cast<const __half2*>(&h.y));
                    wv[j] = make_float4(p.x, p.y, q.x, q.y);
                }
            }
#pragma unroll
            for (int i = 0; i < 16; i++) {
                if (i + 1 < 16) v[(i + 1) & 1] = *reinterpret_cast<const float4*>(xs + (size_t)(i + 1) * RG2_KC);
                const float4 u = v[i & 1];
#pragma unroll
                for (int j = 0; j < 8; j++) acc[8 * i + j] = fmaf(wv[j].x, u.x, acc[8 * i + j]);
#pragma unroll
                for (int j = 0; j < 8; j++) acc[8 * i + j] = fmaf(wv[j].y, u.y, acc[8 * i + j]);
#pragma unroll
                for (int j = 0; j < 8; j++) acc[8 * i + j] = fmaf(wv[j].z, u.z, acc[8 * i + j]);
#pragma unroll
                for (int j = 0; j < 8; j++) acc[8 * i + j] = fmaf(wv[j].w, u.w, acc[8 * i + j]);
            }
        }
        warp_sums<128>(acc, lane);
        const int r = r0 + 16 * wm + (lane >> 1), oo = o0 + 8 * wn + 4 * (lane & 1);
        if (r < T)
#pragma unroll
            for (int k = 0; k < 4; k++) if (oo + k < O) y[(size_t)r * O + oo + k] = acc[k];
    }
    if (!select || !last_block_done(done + blockIdx.y, gridDim.x)) return;
    for (int r = warp; r < RG2_TM && r0 + r < T; r += 8) topk_token<NJ, true>(y + (size_t)(r0 + r) * O, r0 + r, E, K, norm, lane, o);
    ep_raise_dispatch_flags(o, r0, min(RG2_TM, T - r0));
}

}  // namespace moexb
