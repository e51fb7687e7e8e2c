// Rejection-sampling acceptance over draft and target logits (not in the reference, whose rule
// is "draw the target's token on every row and accept a draft that equals it",
// kernels.metal:1578-1589; this is the textbook speculative-sampling rule, built on the
// reference sampler's conventions so that it can be checked bit for bit).
//
// Per stream, with k drafts x_1..x_k drawn from q_1..q_k and target rows p_0..p_k (bf16 logits):
//   e(x) = 2^((x - max) log2(e) / T) with the sampler's exp2; Z = the sum of e in the sampler's
//   order (thread t of 1024 adds ids t, t + 1024, ...; then tg_scan's association);
//   draft i is accepted iff (u_i * eq(x_i)) * Zp < ep(x_i) * Zq, u_i = uniform01(seed, pos0 + i, 0);
//   at the first rejected i the replacement is drawn from max(0, ep_j Zq - eq_j Zp) by the sampler's
//   inverse CDF at uniform01(seed, pos0 + i, 1); with all accepted, the bonus token from p_k at
//   uniform01(seed, pos0 + k, 0). Outputs: accepted count, that token, rollback = k - accepted.
// Two kernels: statistics for all S (2k + 1) rows at once, a cluster of 8 blocks a row and one read of the logits, then a
// cluster of 8 blocks per stream that decides and draws (its two rows come from L2).
#include <cfloat>
#include <cmath>
#include <mutex>

#include "kernels.h"
#include "sampling.cuh"

namespace vlt {

namespace spec {

constexpr uint32_t THREADS = 1024;
__device__ __forceinline__ uint32_t ex_at(uint32_t t) { return t + t / 32; }

// kernels.metal:1482-1501 `tg_scan` (see k_small.cu).
__device__ void tg_scan(float v, float* ex, float* base, uint32_t tid) {
    ex[ex_at(tid)] = v;
    __syncthreads();
    if (tid < 32) {
        float acc = 0.0f;
        for (uint32_t i = 32 * tid; i < 32 * tid + 32; i++) {
            const float x = ex[ex_at(i)];
            ex[ex_at(i)] = acc;
            acc = __fadd_rn(acc, x);
        }
        base[tid] = acc;
    }
    __syncthreads();
    if (tid == 0) {
        float acc = 0.0f;
        for (uint32_t g = 0; g < 32; g++) {
            const float x = base[g];
            base[g] = acc;
            acc = __fadd_rn(acc, x);
        }
        ex[ex_at(THREADS)] = acc;
    }
    __syncthreads();
    ex[ex_at(tid)] = __fadd_rn(ex[ex_at(tid)], base[tid / 32]);
    __syncthreads();
}

using vlt::SpecRowStats;
typedef SpecRowStats RowStats;
typedef vlt::SpecRowWork RowWork;

__device__ __forceinline__ float e_of(uint16_t x, float mx, float c) { return soft_exp2(__fmul_rn(__fsub_rn(bf16_to_f32(x), mx), c)); }
// e(x) for two logits that are at most mx (or NaN): soft_exp2_scaled_x2 without what only a positive exponent needs, and
// with the exponent's bits shifted straight out of the rounding constant's sum (its own bits fall out at the top). The same
// operations on the value, so the same bits.
__device__ __forceinline__ float2 e_below_x2(float x0, float x1, float minus_mx, float c) {
    const float2 x = __fmul2_rn(__fadd2_rn(make_float2(x0, x1), make_float2(minus_mx, minus_mx)), make_float2(c, c));
    const float2 t = __fadd2_rn(x, make_float2(12582912.0f, 12582912.0f));
    const float2 f = __ffma2_rn(__fadd2_rn(t, make_float2(-12582912.0f, -12582912.0f)), make_float2(-1.0f, -1.0f), x);
    float2 p = make_float2(0.00015403530393381608f, 0.00015403530393381608f);
    p = __ffma2_rn(p, f, make_float2(0.0013333558146428443f, 0.0013333558146428443f));
    p = __ffma2_rn(p, f, make_float2(0.009618129107628477f, 0.009618129107628477f));
    p = __ffma2_rn(p, f, make_float2(0.05550410866482158f, 0.05550410866482158f));
    p = __ffma2_rn(p, f, make_float2(0.2402265069591007f, 0.2402265069591007f));
    p = __ffma2_rn(p, f, make_float2(0.6931471805599453f, 0.6931471805599453f));
    p = __ffma2_rn(p, f, make_float2(1.0f, 1.0f));
    return make_float2(x.x > -125.5f ? __int_as_float(__float_as_int(p.x) + (__float_as_int(t.x) << 23)) : 0.0f,
                       x.y > -125.5f ? __int_as_float(__float_as_int(p.y) + (__float_as_int(t.y) << 23)) : 0.0f);
}
// The larger of two bf16 each (the number where one is a NaN).
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// A block's share of a row -- 128 ids of every 1024: of the 1024 "threads" of the sampler's order the cluster's 8 x 128 -- in
// shared memory: [id / 1024][128]. `vec`: rows start on 16-byte boundaries and hold whole groups of 8 ids, so that the
// share comes by 16-byte asynchronous copies, all in flight at once; else two bytes at a time. N: the block's threads.
constexpr size_t STAGE_MAX = 100 * 1024;  // of one row's share; longer rows are read from global memory at every pass
__host__ __device__ constexpr uint32_t stage_chunks(uint32_t vocab) { return (vocab + THREADS - 1) / THREADS; }
__host__ __device__ constexpr size_t stage_bytes(uint32_t vocab) { return size_t(stage_chunks(vocab)) * SC_THREADS * 2; }
template <uint32_t N>
__device__ __forceinline__ void stage_row(const uint16_t* x, uint32_t vocab, bool vec, uint16_t* sm, uint32_t rank, uint32_t tid) {
    const uint32_t chunks = stage_chunks(vocab);
    if (vec) {
        const uint32_t dst = uint32_t(__cvta_generic_to_shared(sm));
        for (uint32_t g = tid; g < chunks * (SC_THREADS / 8); g += N) {
            const uint32_t id = g / (SC_THREADS / 8) * THREADS + rank * SC_THREADS + g % (SC_THREADS / 8) * 8;
            if (id < vocab) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + g * 16), "l"(x + id) : "memory");
        }
        return;
    }
    for (uint32_t i = tid; i < SC_THREADS; i += N) {
        const uint32_t first = rank * SC_THREADS + i, n = vocab - min(vocab, first);  // ids from this column's first on
        uint32_t ch = 0;
        for (; ch + 7 < chunks && (ch + 7) * THREADS < n; ch += 8) {
            uint16_t v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = x[first + (ch + u) * THREADS];
#pragma unroll
            for (int u = 0; u < 8; u++) sm[(ch + u) * SC_THREADS + i] = v[u];
        }
        for (; ch * THREADS < n; ch++) sm[ch * SC_THREADS + i] = x[first + ch * THREADS];
    }
}
__device__ __forceinline__ void stage_wait() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}

__device__ __forceinline__ float row_max(const RowWork& w) {
    const float4 a = *reinterpret_cast<const float4*>(w.max), b = *reinterpret_cast<const float4*>(w.max + 4);
    return fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w)));
}

// A cluster of 8 blocks per row of logits (p rows first, then q rows): each block's best logit with the lowest id it has
// there, and the sums of e over the row in the sampler's order (thread t of 1024: ids t, t + 1024, ...) as the totals of its
// 32 groups of 32 threads; with a q row its draft id, read here once (an id past the vocabulary as 0, see
// launch_spec_accept_static). The row is read from memory once. A thread stands for two neighbours of the 1024, whose sums
// are the halves of packed registers; the maximum is taken on packed bf16, whoever's ids they are. What the cluster has to
// agree on is the maximum alone: every block stores its own into the others, which a first cluster barrier, under way while the
// row comes in, knows to have started, and a second one says that the maxima are there.
// What bounds it: at 128 256 ids a block takes 33 KB, six fit an SM and 104 rows run at a time; a wave of them loads, finds its
// maxima and adds up one after another, and 288 rows are three waves (43 us alone: issue slots 57 % active, DRAM 21 %). Three
// kernels without clusters that read the row twice (maxima; sums; decision) took 24 / 67 us with the decision for 1 / 32
// streams of k = 4 (9 / 288 rows), one block per row 73 / 122, this 22 / 62.
constexpr uint32_t STATS_THREADS = SC_THREADS / 2;
template <bool STAGED>
__global__ void __cluster_dims__(SC_CTAS, 1, 1) __launch_bounds__(STATS_THREADS) stats_kernel(const uint16_t* __restrict__ p, const uint16_t* __restrict__ q,
                                                                                           const uint32_t* __restrict__ drafts, uint32_t p_rows, uint32_t vocab, bool vec,
                                                                                           float c, RowWork* work) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // "this block is there": waited for before the first store to another one
    extern __shared__ __align__(16) uint16_t row_sm[];
    __shared__ float maxima[SC_CTAS];
    __shared__ uint32_t wbv[STATS_THREADS / 32], first_id;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const uint32_t r = blockIdx.x / SC_CTAS, tid = threadIdx.x, lane = tid % 32, vt = rank * SC_THREADS + 2 * tid;  // and vt + 1
    const uint16_t* x = r < p_rows ? p + size_t(r) * vocab : q + size_t(r - p_rows) * vocab;
    const uint32_t chunks = stage_chunks(vocab);
    uint32_t draft = 0;
    if (tid == 0) {
        first_id = 0xffffffffu;
        if (rank == 0 && r >= p_rows) draft = drafts[r - p_rows];
    }
    if (STAGED) {
        stage_row<STATS_THREADS>(x, vocab, vec, row_sm, rank, tid);
        // What the last 1024 ids lack stands as -inf, whose e is 0.
        for (uint32_t i = tid; i < SC_THREADS; i += STATS_THREADS)
            if ((chunks - 1) * THREADS + rank * SC_THREADS + i >= vocab) row_sm[(chunks - 1) * SC_THREADS + i] = 0xff80u;
        stage_wait();
    }
    auto pair_at = [&](uint32_t ch) {
        if (STAGED) return reinterpret_cast<const uint32_t*>(row_sm)[ch * (SC_THREADS / 2) + tid];
        const uint32_t i = ch * THREADS + vt;
        return (i < vocab ? uint32_t(x[i]) : 0xff80u) | (i + 1 < vocab ? uint32_t(x[i + 1]) << 16 : 0xff800000u);
    };
    uint32_t best = 0xff80ff80u;
#pragma unroll 8
    for (uint32_t ch = 0; ch < chunks; ch++) best = max_bf16x2(best, pair_at(ch));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = max_bf16x2(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (lane == 0) wbv[tid / 32] = best;
    __syncthreads();
#pragma unroll
    for (uint32_t w = 0; w < STATS_THREADS / 32; w++) best = max_bf16x2(best, wbv[w]);
    const float mine = fmaxf(-FLT_MAX, fmaxf(bf16lo(best), bf16hi(best)));
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // (long over, but for a short row: its later blocks have no id to load)
    if (tid < SC_CTAS) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(sc_remote(&maxima[rank], tid)), "f"(mine) : "memory");
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    {  // meanwhile the lowest id of the share's own best
        uint32_t id = 0xffffffffu;
#pragma unroll 8
        for (uint32_t ch = 0; ch < chunks; ch++) {
            const uint32_t v = pair_at(ch), i = ch * THREADS + vt;
            id = min(id, bf16lo(v) == mine ? i : bf16hi(v) == mine ? i + 1 : 0xffffffffu);
        }
        id = __reduce_min_sync(0xffffffffu, id);
        if (lane == 0) atomicMin(&first_id, id);
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // (of the block's threads too; no block touches another's memory after it)
    float mx = maxima[0];
#pragma unroll
    for (uint32_t s = 1; s < SC_CTAS; s++) mx = fmaxf(mx, maxima[s]);
    float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll 8
    for (uint32_t ch = 0; ch < chunks; ch++) {
        const uint32_t v = pair_at(ch);
        sum = __fadd2_rn(sum, e_below_x2(bf16lo(v), bf16hi(v), -mx, c));
    }
    // A group of 32 of the 1024 is half a warp: its sums left to right.
    float group = 0.0f;
#pragma unroll
    for (uint32_t l = 0; l < 16; l++) {
        group = __fadd_rn(group, __shfl_sync(0xffffffffu, sum.x, l, 16));
        group = __fadd_rn(group, __shfl_sync(0xffffffffu, sum.y, l, 16));
    }
    if (lane % 16 == 0) work[r].tot[rank * SC_WARPS + tid / 16] = group;
    __syncthreads();
    if (tid == 0) {
        work[r].max[rank] = mine;
        work[r].argmax[rank] = first_id;
        if (rank == 0) work[r].draft = draft < vocab ? draft : 0u;
    }
}

// The sampler's inverse CDF (kernels.metal:1540-1559) over weights w(i) >= 0; `fallback` if they
// sum to 0 or the target falls past the last term.
template <typename W>
__device__ uint32_t inverse_cdf(uint32_t vocab, W w, float u, uint32_t fallback, float* ex, float* base, uint32_t* pick, uint32_t tid) {
    float a = 0.0f;
    for (uint32_t i = tid; i < vocab; i += THREADS) a = __fadd_rn(a, w(i));
    tg_scan(a, ex, base, tid);
    const float total = ex[ex_at(THREADS)];
    if (!(total > 0.0f)) return fallback;
    const float target = __fmul_rn(u, total);
    if (tid == 0) *pick = 0xffffffffu;
    __syncthreads();
    const float lo = ex[ex_at(tid)];
    // The one thread whose interval holds the target re-adds its terms in order until they pass it; its warp helps:
    // the lanes evaluate 32 of its ids at a time, and only the additions stay in the thread's order.
    const bool mine = lo <= target && target < ex[ex_at(tid + 1)];
    const uint32_t owners = __ballot_sync(0xffffffffu, mine);
    if (owners) {
        const uint32_t lane = tid % 32;
        const int src = __ffs(owners) - 1;
        const uint32_t first = __shfl_sync(0xffffffffu, tid, src);
        const float rest = __fsub_rn(target, __shfl_sync(0xffffffffu, lo, src));
        float acc = 0.0f;
        uint32_t j = 0xffffffffu;
        bool done = false;
        for (uint32_t i0 = first; i0 < vocab && !done; i0 += 32 * THREADS) {
            const uint32_t i = i0 + lane * THREADS;
            walk_32(i < vocab ? w(i) : 0.0f, i0, rest, acc, j, done);
        }
        if (int(lane) == src) *pick = j;
    }
    __syncthreads();
    const uint32_t j = *pick;
    return j == 0xffffffffu ? fallback : j;
}

// The decision, a cluster of 8 blocks per stream: the 1024 "threads" of the sampler's order are the cluster's 8 x 128 (as
// in the sampler's cluster form), so every sum keeps its order and association while a stream's pass over its two rows
// runs on eight SMs. Every block first finishes the rows' sums, a warp a row, and runs the tests, a lane each, so that
// their chains of loads run side by side. Bound by latency; the rows' shares are staged as above, and the pass that adds up
// and the walk to the token read them there (an id at a time from L2, they took 90 us).
constexpr uint32_t MAX_ROWS = 31;  // 2 k + 1 at most
template <bool STAGED>
__global__ void __cluster_dims__(SC_CTAS, 1, 1) __launch_bounds__(SC_THREADS) decide_cluster_kernel(const uint16_t* __restrict__ p, const uint16_t* __restrict__ q,
                                                                                                 const RowWork* __restrict__ work, uint32_t streams, uint32_t k,
                                                                                                 uint32_t vocab, bool vec, float c, const uint64_t* __restrict__ seeds,
                                                                                                 const uint32_t* __restrict__ pos0, uint32_t* accepted, uint32_t* token,
                                                                                                 uint32_t* rollback) {
    pdl_start();
    extern __shared__ __align__(16) uint16_t row_sm[];  // p's share, then q's
    __shared__ ScExchange xc;
    __shared__ float z_s[MAX_ROWS], max_s[MAX_ROWS];  // the k + 1 p rows, then the k q rows
    __shared__ uint32_t first_reject;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const uint32_t s = blockIdx.x / SC_CTAS, tid = threadIdx.x, lane = tid % 32, vt = rank * SC_THREADS + tid;
    const uint64_t seed = seeds[s];
    const uint32_t seed_lo = uint32_t(seed), seed_hi = uint32_t(seed >> 32), first_pos = pos0[s];
    const RowWork* pw = work + size_t(s) * (k + 1);
    const RowWork* qw = work + size_t(streams) * (k + 1) + size_t(s) * k;
    const uint16_t* pp = p + size_t(s) * (k + 1) * vocab;
    const uint16_t* qq = q + size_t(s) * k * vocab;
    uint16_t xp = 0, xq = 0;
    if (tid < k) {
        const uint32_t draft = qw[tid].draft;
        xp = pp[size_t(tid) * vocab + draft];
        xq = qq[size_t(tid) * vocab + draft];
    }
    for (uint32_t r = tid / 32; r < 2 * k + 1; r += SC_WARPS) {
        const RowWork& w = r <= k ? pw[r] : qw[r - k - 1];
        const float tot = w.tot[lane], mx = row_max(w);
        float z;
        lane_prefix(tot, lane, z);
        if (lane == 0) { z_s[r] = z; max_s[r] = mx; }
    }
    if (tid == 0) {
        xc.pick[0] = 0xffffffffu;
        xc.pick[1] = 0xffffffffu;
    }
    __syncthreads();
    if (tid < 32) {  // every block runs the few tests itself: cheaper than sending the result round
        bool fails = false;  // a lane without a test does not fail
        if (tid < k) {
            const float ep = e_of(xp, max_s[tid], c), eq = e_of(xq, max_s[k + 1 + tid], c);
            const float u = uniform01(seed_lo, seed_hi, first_pos + tid, 0);
            const float lhs = __fmul_rn(__fmul_rn(u, eq), z_s[tid]), rhs = __fmul_rn(ep, z_s[k + 1 + tid]);
            fails = !(lhs < rhs);
        }
        const uint32_t failed = __ballot_sync(0xffffffffu, fails);
        if (tid == 0) first_reject = failed ? uint32_t(__ffs(failed) - 1) : k;
    }
    __syncthreads();
    const uint32_t i = first_reject;
    const bool rejected = i < k;
    const uint16_t* pi = pp + size_t(i) * vocab;
    const uint16_t* qi = qq + size_t(rejected ? i : 0) * vocab;
    uint16_t* q_sm = row_sm + stage_chunks(vocab) * SC_THREADS;
    if (STAGED) {
        stage_row<SC_THREADS>(pi, vocab, vec, row_sm, rank, tid);
        if (rejected) stage_row<SC_THREADS>(qi, vocab, vec, q_sm, rank, tid);
    }
    // The token if the weights sum to 0 or the target falls past the last of them: p's best, the lowest id of them.
    float best = -FLT_MAX;
    uint32_t fallback = 0xffffffffu;
#pragma unroll
    for (uint32_t sl = 0; sl < SPEC_SLICES; sl++) better(best, fallback, pw[i].max[sl], pw[i].argmax[sl]);
    if (STAGED) stage_wait();
    auto at = [&](const uint16_t* x, const uint16_t* sm, uint32_t j) { return STAGED ? sm[j / THREADS * SC_THREADS + j % SC_THREADS] : x[j]; };  // ids of this block's share
    constexpr uint32_t B = 8;
    uint32_t tok, i0 = vt;
    float a = 0.0f;
    if (rejected) {
        const float pm = max_s[i], qm = max_s[k + 1 + i], zp = z_s[i], zq = z_s[k + 1 + i];
        auto resid = [&](uint32_t j) {
            const float ea = __fmul_rn(e_of(at(pi, row_sm, j), pm, c), zq), eb = __fmul_rn(e_of(at(qi, q_sm, j), qm, c), zp);
            const float d = __fsub_rn(ea, eb);
            return d > 0.0f ? d : 0.0f;
        };
        for (; i0 + (B - 1) * THREADS < vocab; i0 += B * THREADS) {
            float vp[B], vq[B];
#pragma unroll
            for (uint32_t u = 0; u < B; u++) {
                vp[u] = bf16_to_f32(at(pi, row_sm, i0 + u * THREADS));
                vq[u] = bf16_to_f32(at(qi, q_sm, i0 + u * THREADS));
            }
#pragma unroll
            for (uint32_t u = 0; u < B; u += 2) {
                const float2 ea = __fmul2_rn(e_below_x2(vp[u], vp[u + 1], -pm, c), make_float2(zq, zq));
                const float2 eb = __fmul2_rn(e_below_x2(vq[u], vq[u + 1], -qm, c), make_float2(zp, zp));
                const float d0 = __fsub_rn(ea.x, eb.x), d1 = __fsub_rn(ea.y, eb.y);
                a = __fadd_rn(a, d0 > 0.0f ? d0 : 0.0f);
                a = __fadd_rn(a, d1 > 0.0f ? d1 : 0.0f);
            }
        }
        tok = sc_inverse_cdf_rest(vocab, resid, a, i0, uniform01(seed_lo, seed_hi, first_pos + i, 1), fallback, &xc, 0, 0, rank, tid);
    } else {
        const float pm = max_s[k];
        auto w = [&](uint32_t j) { return e_of(at(pi, row_sm, j), pm, c); };
        for (; i0 + (B - 1) * THREADS < vocab; i0 += B * THREADS) {
            float v[B];
#pragma unroll
            for (uint32_t u = 0; u < B; u++) v[u] = bf16_to_f32(at(pi, row_sm, i0 + u * THREADS));
#pragma unroll
            for (uint32_t u = 0; u < B; u += 2) {
                const float2 e = e_below_x2(v[u], v[u + 1], -pm, c);
                a = __fadd_rn(__fadd_rn(a, e.x), e.y);
            }
        }
        tok = sc_inverse_cdf_rest(vocab, w, a, i0, uniform01(seed_lo, seed_hi, first_pos + k, 0), fallback, &xc, 0, 0, rank, tid);
    }
    if (rank == 0 && tid == 0) {
        accepted[s] = i;
        token[s] = tok;
        rollback[s] = k - i;
    }
    sc_cluster_sync();  // nobody leaves while another block may still read its shared memory
}

}  // namespace spec

// p [S][k+1][V], q [S][k][V] bf16 on the device; work: scratch for S (2k + 1) rows. The first kernel overlaps with nothing
// before it (the caller's stream may hold anything); the second's launch overlaps with it.
// Returns the first error of the launches.
cudaError_t launch_spec_accept(const uint16_t* p, const uint16_t* q, const uint32_t* drafts, uint32_t streams, uint32_t k, uint32_t vocab, float temperature,
                               const uint64_t* seeds, const uint32_t* pos0, SpecRowWork* work, uint32_t* accepted, uint32_t* token, uint32_t* rollback, cudaStream_t s) {
    using namespace spec;
    const float c = LOG2E / temperature;  // the same IEEE division as the device's __fdiv_rn
    const size_t share = stage_bytes(vocab);
    const bool staged = share <= STAGE_MAX, vec = vocab % 8 == 0 && (reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(q)) % 16 == 0;
    static PerDevice configured;
    cudaError_t e = cudaSuccess;
    configured.once([&] {
        e = cudaFuncSetAttribute(stats_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(STAGE_MAX));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(decide_cluster_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(2 * STAGE_MAX));
        return e == cudaSuccess;
    });
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = s;
    cfg.blockDim = dim3(STATS_THREADS);
    cfg.gridDim = dim3(streams * (2 * k + 1) * SC_CTAS);
    cfg.dynamicSmemBytes = staged ? share : 0;
    e = cudaLaunchKernelEx(&cfg, staged ? stats_kernel<true> : stats_kernel<false>, p, q, drafts, streams * (k + 1), vocab, vec, c, work);
    if (e != cudaSuccess) return e;
    launch_counter()++;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.blockDim = dim3(SC_THREADS);
    cfg.gridDim = dim3(streams * SC_CTAS);
    cfg.dynamicSmemBytes = staged ? 2 * share : 0;
    e = cudaLaunchKernelEx(&cfg, staged ? decide_cluster_kernel<true> : decide_cluster_kernel<false>, p, q, static_cast<const RowWork*>(work), streams, k, vocab, vec, c, seeds, pos0,
                           accepted, token, rollback);
    if (e == cudaSuccess) launch_counter()++;
    return e;
}

// ------------------------------------------------ the rule inside the engine's step
// A verify run whose drafts the chain drafter drew (from softmax(q / T), keeping the q rows) in the step before is
// decided by the rule above instead of the reference's sample-then-match. What differs from the stand-alone form:
// the target's rows are the step's fp32 logits over the whole vocabulary; a q row is fp32 over the draft vocabulary
// (v ids, `index_of` maps a target id to its index or NO_TOK), its statistics taken in the sampler's order over
// draft indices, Q being 0 for an id outside it (such a draft is rejected); the uniforms are keyed by the position
// of the token they decide (round 0 the test, round 1 the replacement; the bonus token at the last row's position
// + 1, round 0). The kernels leave the run's candidates -- the accepted drafts, then the drawn token -- in
// out[head0 ..] and their number in spec_e[run]; `accept_kernel` then commits them exactly as it commits a walk
// of the reference's rule (lens, feed, path, on_path, gen, emitted), so rejected rows are rolled back the same
// way: the sequence advances by what was accepted and the K/V past it is overwritten by the next step.
namespace spec {

// Whether run r is decided by this rule: a verify run of a sequence that samples (temperature > 0, no top-p cut),
// whose rows are a plain chain and whose drafts all came with a kept q row. Uniform over a block.
__device__ bool step_applies(const SpecStepArgs& a, uint32_t r) {
    const RunIn ru = a.runs[r];
    if (!ru.verify || ru.count < 2 || ru.nhead != ru.count || ru.count > VERIFY_T) return false;
    const SampleRow sr = a.samples[ru.head0];
    if (!(sr.temperature > 0.0f) || sr.top_p < 1.0f) return false;
    if (a.q_rows[ru.slot] + 1 < ru.count) return false;
    for (uint32_t c = 1; c < ru.count; c++)
        if (a.tree[ru.slot * FEED_W + c] != d_chain_node(c)) return false;
    return true;
}

// One block per row: the step's head rows first, then VERIFY_T - 1 q rows per run. Rows of runs the rule does
// not decide are left alone (and marked for the sampler: row_skip 0); the others get (max, argmax, Z).
__global__ void __launch_bounds__(THREADS) step_stats_kernel(const SpecStepArgs a) {
    pdl_start();
    __shared__ float ex[THREADS + THREADS / 32 + 1];
    __shared__ float base[32];
    __shared__ float bvs[32];
    __shared__ uint32_t bis[32];
    const uint32_t b = blockIdx.x, tid = threadIdx.x, lane = tid % 32;
    const float* x;
    uint32_t n, r;
    RowStats* out;
    if (b < a.n_head) {
        for (r = 0; r < a.n_runs; r++)
            if (b >= a.runs[r].head0 && b < a.runs[r].head0 + a.runs[r].nhead) break;
        const bool on = r < a.n_runs && step_applies(a, r);
        if (tid == 0) a.row_skip[b] = on ? 1u : 0u;
        if (!on) return;
        x = a.logits + size_t(b) * a.vocab;
        n = a.vocab;
        out = a.stats + b;
    } else {
        r = (b - a.n_head) / (VERIFY_T - 1);
        const uint32_t i = (b - a.n_head) % (VERIFY_T - 1) + 1;
        if (!step_applies(a, r) || i >= a.runs[r].count) return;
        x = a.q_keep + (size_t(a.runs[r].slot) * (VERIFY_T - 1) + i - 1) * a.v;
        n = a.v;
        out = a.stats + a.max_head_rows + r * (VERIFY_T - 1) + i - 1;
    }
    const float c = __fdiv_rn(LOG2E, a.samples[a.runs[r].head0].temperature);
    float mx = -FLT_MAX;
    uint32_t am = 0xffffffffu;
    for (uint32_t i = tid; i < n; i += THREADS) better(mx, am, x[i], i);
    warp_best(mx, am);
    if (lane == 0) { bvs[tid / 32] = mx; bis[tid / 32] = am; }
    __syncthreads();
    mx = bvs[0];
    am = bis[0];
    for (uint32_t i = 1; i < 32; i++) better(mx, am, bvs[i], bis[i]);
    float s = 0.0f;
    uint32_t i0 = tid;
    for (; i0 + 7 * THREADS < n; i0 += 8 * THREADS) {  // eight loads in flight, the additions in id order
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = x[i0 + u * THREADS];
#pragma unroll
        for (int u = 0; u < 8; u++) s = __fadd_rn(s, soft_exp2(__fmul_rn(__fsub_rn(v[u], mx), c)));
    }
    for (; i0 < n; i0 += THREADS) s = __fadd_rn(s, soft_exp2(__fmul_rn(__fsub_rn(x[i0], mx), c)));
    tg_scan(s, ex, base, tid);
    if (tid == 0) *out = RowStats{mx, am, ex[ex_at(THREADS)], 0};
}

// A cluster of 8 blocks per run (the sampler's 1024 threads, see decide_cluster_kernel): the tests (a lane each, in
// every block), then the replacement or the bonus token (the cluster).
__global__ void __cluster_dims__(SC_CTAS, 1, 1) __launch_bounds__(SC_THREADS) step_decide_kernel(const SpecStepArgs a) {
    pdl_start();
    __shared__ ScExchange xc;
    __shared__ uint32_t first_reject;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const uint32_t r = blockIdx.x / SC_CTAS, tid = threadIdx.x;
    const RunIn ru = a.runs[r];
    const bool on = step_applies(a, r);
    sc_cluster_sync();  // every thread of the cluster has read q_rows
    if (rank == 0 && tid == 0) {
        a.q_rows[ru.slot] = 0;  // a slot's kept rows serve one step
        if (!on) a.spec_e[r] = 0;
    }
    if (!on) return;  // the whole cluster leaves: no further cluster barrier
    const SampleRow sr = a.samples[ru.head0];
    const float c = __fdiv_rn(LOG2E, sr.temperature);
    const RowStats* ps = a.stats + ru.head0;
    const RowStats* qs = a.stats + a.max_head_rows + r * (VERIFY_T - 1);
    const float* pp = a.logits + size_t(ru.head0) * a.vocab;
    const float* qq = a.q_keep + size_t(ru.slot) * (VERIFY_T - 1) * a.v;
    auto e_of = [&](float x, float mx) { return soft_exp2(__fmul_rn(__fsub_rn(x, mx), c)); };
    // The tests, one lane each (every block of the cluster does them), so that the loads of all of them are in flight at
    // once; the first that fails, or whose draft is outside the draft vocabulary, is where the run stops.
    if (tid < 32) {
        bool fails = false;  // a lane without a test does not fail
        if (tid + 1 < ru.count) {
            const uint32_t i = tid + 1;
            const uint32_t tok = a.tokens[ru.first + i], idx = tok < a.vocab ? a.index_of[tok] : NO_TOK;
            fails = true;
            if (idx != NO_TOK) {
                const float ep = e_of(pp[size_t(i - 1) * a.vocab + tok], ps[i - 1].max), eq = e_of(qq[size_t(i - 1) * a.v + idx], qs[i - 1].max);
                const float u = uniform01(sr.seed_lo, sr.seed_hi, a.meta[2 * (ru.first + i) + 1], 0);
                const float lhs = __fmul_rn(__fmul_rn(u, eq), ps[i - 1].z), rhs = __fmul_rn(ep, qs[i - 1].z);
                fails = !(lhs < rhs);
            }
        }
        const uint32_t failed = __ballot_sync(0xffffffffu, fails);  // lane t holds test t + 1
        if (tid == 0) {
            first_reject = failed ? uint32_t(__ffs(failed)) : ru.count;
            xc.pick[0] = 0xffffffffu;
            xc.pick[1] = 0xffffffffu;
        }
    }
    __syncthreads();
    const uint32_t i = first_reject;
    uint32_t tok;
    if (i < ru.count) {
        const float* pi = pp + size_t(i - 1) * a.vocab;
        const float* qi = qq + size_t(i - 1) * a.v;
        const float pm = ps[i - 1].max, qm = qs[i - 1].max, zp = ps[i - 1].z, zq = qs[i - 1].z;
        const uint32_t* index_of = a.index_of;
        auto resid = [&](uint32_t j) {
            const uint32_t idx = index_of[j];
            const float qv = qi[idx == NO_TOK ? 0u : idx];  // an unconditional load: a batch's loads all go out before the arithmetic
            const float ea = __fmul_rn(e_of(pi[j], pm), zq), eb = idx == NO_TOK ? 0.0f : __fmul_rn(e_of(qv, qm), zp);
            const float d = __fsub_rn(ea, eb);
            return d > 0.0f ? d : 0.0f;
        };
        // A batch in three rounds of loads (draft index and p; q through the index), then the arithmetic.
        constexpr int B = 16;
        auto resid_batch = [&](uint32_t i0, float (&e)[B]) {
            uint32_t idx[B];
            float pv[B], qv[B];
#pragma unroll
            for (int u = 0; u < B; u++) {
                idx[u] = index_of[i0 + u * SAMPLE_THREADS];
                pv[u] = pi[i0 + u * SAMPLE_THREADS];
            }
#pragma unroll
            for (int u = 0; u < B; u++) qv[u] = qi[idx[u] == NO_TOK ? 0u : idx[u]];
#pragma unroll
            for (int u = 0; u < B; u++) {
                const float ea = __fmul_rn(e_of(pv[u], pm), zq), eb = idx[u] == NO_TOK ? 0.0f : __fmul_rn(e_of(qv[u], qm), zp);
                const float d = __fsub_rn(ea, eb);
                e[u] = d > 0.0f ? d : 0.0f;
            }
        };
        tok = sc_inverse_cdf_batched<B>(a.vocab, resid, resid_batch, uniform01(sr.seed_lo, sr.seed_hi, a.meta[2 * (ru.first + i) + 1], 1), ps[i - 1].argmax, &xc, 0, 0,
                                        rank, tid);
    } else {
        const float* pk = pp + size_t(ru.count - 1) * a.vocab;
        const float pm = ps[ru.count - 1].max;
        auto w = [&](uint32_t j) { return e_of(pk[j], pm); };
        tok = sc_inverse_cdf<16>(a.vocab, w, uniform01(sr.seed_lo, sr.seed_hi, a.meta[2 * (ru.first + ru.count - 1) + 1] + 1, 0), ps[ru.count - 1].argmax, &xc, 0, 0, rank, tid);
    }
    if (rank == 0 && tid == 0) {
        for (uint32_t j = 0; j + 1 < i; j++) a.out[ru.head0 + j] = a.tokens[ru.first + j + 1];
        a.out[ru.head0 + i - 1] = tok;
        a.spec_e[r] = i;
    }
    sc_cluster_sync();  // nobody leaves while another block may still read its shared memory
}

// The chain drafter's pick for pass i, one block per run: the draft vocabulary's argmax (ties to the lowest
// index), or -- under the rule, for a sequence that samples -- a draw from softmax(q / T) by the sampler's
// inverse CDF at round 2 of the drafted token's position, the row kept for the next step's test.
__global__ void __launch_bounds__(THREADS) draft_draw_kernel(const float* __restrict__ logits, uint32_t v, const uint32_t* __restrict__ vocab_ids,
                                                             const RunIn* __restrict__ runs, const SampleRow* __restrict__ samples,
                                                             const uint32_t* __restrict__ live, const uint32_t* __restrict__ lens, uint32_t i, uint32_t rule,
                                                             uint32_t* feed, uint32_t* tree, float* q_keep, uint32_t* q_rows) {
    pdl_start();
    __shared__ float ex[THREADS + THREADS / 32 + 1];
    __shared__ float base[32];
    __shared__ float bvs[32];
    __shared__ uint32_t bis[32];
    __shared__ uint32_t pick;
    const uint32_t r = blockIdx.x, tid = threadIdx.x, lane = tid % 32;
    if (!live[r]) return;
    const RunIn ru = runs[r];
    const float* row = logits + size_t(r) * v;
    float mx = -FLT_MAX;
    uint32_t am = 0xffffffffu;
    for (uint32_t j = tid; j < v; j += THREADS) better(mx, am, row[j], j);
    warp_best(mx, am);
    if (lane == 0) { bvs[tid / 32] = mx; bis[tid / 32] = am; }
    __syncthreads();
    mx = bvs[0];
    am = bis[0];
    for (uint32_t j = 1; j < 32; j++) better(mx, am, bvs[j], bis[j]);
    const SampleRow sr = samples[ru.head0];
    const bool draws = rule == 1 && sr.temperature > 0.0f && sr.top_p >= 1.0f;
    uint32_t idx = am;
    if (draws) {
        const float c = __fdiv_rn(LOG2E, sr.temperature);
        auto w = [&](uint32_t j) { return soft_exp2(__fmul_rn(__fsub_rn(row[j], mx), c)); };
        idx = inverse_cdf(v, w, uniform01(sr.seed_lo, sr.seed_hi, lens[ru.slot] + i, 2), am, ex, base, &pick, tid);
        float* keep = q_keep + (size_t(ru.slot) * (VERIFY_T - 1) + i - 1) * v;
        for (uint32_t j = tid; j < v; j += THREADS) keep[j] = row[j];
    }
    if (tid == 0) {
        feed[ru.slot * FEED_W + i] = vocab_ids[idx < v ? idx : 0];
        tree[ru.slot * FEED_W + i] = d_chain_node(i);
        if (draws) q_rows[ru.slot] = i;
        else if (i == 1) q_rows[ru.slot] = 0;
    }
}

}  // namespace spec

void launch_spec_step_stats(const SpecStepArgs& a, cudaStream_t s) {
    launch_pdl(spec::step_stats_kernel, a.n_head + a.n_runs * (VERIFY_T - 1), spec::THREADS, 0, s, a);
}
void launch_spec_step_decide(const SpecStepArgs& a, cudaStream_t s) {
    launch_pdl(spec::step_decide_kernel, a.n_runs * SC_CTAS, SC_THREADS, 0, s, a);
}
void launch_draft_draw(const float* logits, uint32_t v, const uint32_t* vocab_ids, const RunIn* runs, const SampleRow* samples, const uint32_t* live,
                       const uint32_t* lens, uint32_t n_runs, uint32_t i, uint32_t rule, uint32_t* feed, uint32_t* tree, float* q_keep, uint32_t* q_rows,
                       cudaStream_t s) {
    launch_pdl(spec::draft_draw_kernel, n_runs, spec::THREADS, 0, s, logits, v, vocab_ids, runs, samples, live, lens, i, rule, feed, tree, q_keep, q_rows);
}

// ------------------------------------------------ the same, with nothing allocated
// A variant for callers that cannot allocate device memory when they need an acceptance step:
// a serving loop that has handed every byte of the device to its own pools, or one that must not
// pay the device-wide synchronisation an allocation or a free can imply in the middle of decoding.
// Its scratch (the rows' statistics and bounds-checked draft ids) lives in a file-scope device
// array of a fixed size, so a step may cover at most STATIC_MAX_ROWS rows of logits. The array's
// address is looked up once per device, on the first call made with that device current; that
// first call is set-up and belongs before the caller starts any stream capture. All calls on a
// device share the array: nothing in it has to start at zero (the first kernel overwrites every
// word the second reads), but two calls in flight at once on one device race on it.
namespace spec {

constexpr uint32_t STATIC_MAX_ROWS = 2048;  // streams * (2 k + 1) rows of logits a call may cover
static __device__ __align__(256) RowWork static_work[STATIC_MAX_ROWS];

// The array's address on the current device; looked up (cudaGetSymbolAddress) on the first call per device.
static const char* static_scratch(RowWork** out) {
    constexpr int MAX_DEVICES = 64;
    static RowWork* table[MAX_DEVICES] = {};
    static std::mutex mu;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return "spec_accept_static: no usable current device";
    std::lock_guard<std::mutex> lock(mu);
    if (!table[dev]) {
        void* ps = nullptr;
        if (cudaGetSymbolAddress(&ps, static_work) != cudaSuccess || !ps) return "spec_accept_static: cudaGetSymbolAddress failed for the scratch array";
        table[dev] = static_cast<RowWork*>(ps);
    }
    *out = table[dev];
    return nullptr;
}

}  // namespace spec

uint32_t spec_accept_static_max_rows() { return spec::STATIC_MAX_ROWS; }

// Every pointer is device memory of the current device. Returns NULL, or a message (a string literal:
// this path does not allocate on the host either).
const char* launch_spec_accept_static(const uint16_t* p, const uint16_t* q, const uint32_t* drafts, uint32_t streams, uint32_t k, uint32_t vocab,
                                      float temperature, const uint64_t* seeds, const uint32_t* pos0, uint32_t* accepted, uint32_t* token,
                                      uint32_t* rollback, cudaStream_t s) {
    if (!p || !q || !drafts || !seeds || !pos0 || !accepted || !token || !rollback) return "spec_accept_static: null pointer";
    if (streams == 0 || k == 0 || k > 15 || vocab == 0) return "spec_accept_static: needs at least one stream, 1..15 drafts and a vocabulary";
    if (!(std::isnormal(temperature) && temperature > 0.0f)) return "spec_accept_static: needs a normal positive temperature";
    if (uint64_t(streams) * (2 * k + 1) > spec::STATIC_MAX_ROWS)
        return "spec_accept_static: streams * (2 k + 1) exceeds the 2048 rows the static scratch holds; use vlt_spec_accept";
    // The caller's draft ids cannot be checked on the host here; an id past the vocabulary is read as 0 instead of
    // indexing out of the logits (that stream's result then means nothing).
    spec::RowWork* work = nullptr;
    if (const char* e = spec::static_scratch(&work)) return e;
    const cudaError_t e = launch_spec_accept(p, q, drafts, streams, k, vocab, temperature, seeds, pos0, work, accepted, token, rollback, s);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? nullptr : "spec_accept_static: kernel launch failed";
}

}  // namespace vlt
