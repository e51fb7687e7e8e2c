// Chunk (prefill) attention over the paged KV cache: the reference's attn_mma + attn_sum_reduce
// (kernels.metal:1169-1312; engine/src/engine/encode.rs:299-355 runs them whenever a step holds a run longer than
// 8 tokens) for steps that carry prompt chunks.
//
// The decode kernel (k_attn.cu) packs a run's <= 8 rows x G heads into the MMA's narrow side and streams the keys once
// per 8 rows: right when the keys dominate, wasteful for a chunk of hundreds of rows, whose every 8 rows would read the
// context again. Here the queries are the MMA's M side: a block owns 64 rows of one run and one query head (4 warps x
// 16 rows), walks the keys in blocks of 64 (four pages of K and of V by TMA into a three-stage ring of 128-byte-swizzled
// shared memory, shared by the four warps; the G heads of a kv head find the same pages in L2), and keeps the whole
// softmax online in registers: S = Q K^T lands in the accumulator layout that is the A-fragment layout of the next
// product, so P goes into O += P V without leaving the registers. Where it pays (launch_attn_chunk), two such groups of warps
// hold the same rows and take the key blocks in turn, each with a ring of its own, and add up in shared memory at the end: a
// portion of 512 rows is 256 blocks, 1.7 an SM, and with four warps each the dependent chain of a key block is what the SM
// waits on. Three blocks of one group share an SM (168 registers, 49 KB), or two of two groups (128 registers and 20 bytes
// spilled, 97 KB). No partials and no merge kernel: the block writes the normalised rows, fp32 and bf16.
//
// The step's own rows are in the cache already (the qkv projection's epilogue wrote them), so every key is read from
// there; what a row may see is the decode kernel's rule, per row: every cached key below the first position of its
// 8-row tile, and of that tile's keys those its `vis` mask names (causal for a chunk, the tree's for a verify run that
// shares the step). q arrives rotated, scaled by scale * log2(e) and rounded to bf16.
// Every mbarrier wait is bounded and sets the error word on time-out.
#include <cuda.h>

#include "kernels.h"
#include "mma.cuh"

namespace vlt {

namespace prefill {

constexpr uint32_t CQ = 64, CK = 64, HD = 64, PAGE = 16, WARPS = 4, STAGES = 3;
constexpr uint32_t STAGE_BYTES = 2 * CK * HD * 2;  // K block then V block
constexpr uint32_t SPIN_LIMIT = 1u << 24;

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit = SPIN_LIMIT) {
    for (uint32_t i = 0; i < limit; i++) {
        uint32_t ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x),
                 "r"(y), "r"(bar)
                 : "memory");
}
template <uint32_t GROUPS>
__device__ __forceinline__ void group_sync(uint32_t grp) {  // (constant barrier numbers: a variable one would claim all sixteen)
    if (GROUPS == 1) __syncthreads();
    else if (grp == 0) asm volatile("bar.sync 1, %0;" ::"n"(WARPS * 32) : "memory");
    else asm volatile("bar.sync 2, %0;" ::"n"(WARPS * 32) : "memory");
}
constexpr uint32_t blocks_per_sm(uint32_t groups) { return groups == 1 ? 3 : 2; }
// grid (chunk tiles, query heads), GROUPS * 128 threads.
template <uint32_t GROUPS>
__global__ void __launch_bounds__(GROUPS * WARPS * 32, blocks_per_sm(GROUPS)) attn_chunk_kernel(ChunkAttnArgs a, const __grid_constant__ AttnMaps maps) {
    pdl_start();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));  // the swizzle is a function of address bits 4..9
    __shared__ uint64_t bars_all[GROUPS][STAGES];
    __shared__ uint32_t fail[GROUPS];

    const uint32_t tile = blockIdx.x, h = blockIdx.y, kvh = h / (a.n_heads / a.kv.n_kv);
    const uint32_t grp = GROUPS == 1 ? 0 : threadIdx.x / (WARPS * 32), tid = GROUPS == 1 ? threadIdx.x : threadIdx.x % (WARPS * 32), warp = tid / 32, lane = tid % 32, g = lane >> 2, tq = lane & 3;
    uint8_t* ring = smem + grp * STAGES * STAGE_BYTES;
    uint64_t* bars = bars_all[grp];
    const uint32_t t0 = a.ctiles[2 * tile], rows = a.ctiles[2 * tile + 1];
    const uint32_t slot = a.meta[2 * t0];

    // This thread's two rows (g and g + 8 of its warp's 16): the token, the first position of its 8-row tile and its mask.
    uint32_t tok[2], p8[2], vmask[2];
    bool live[2];
    uint32_t my_end = 0;  // one past the last key either row may see
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const uint32_t row = warp * 16 + g + 8 * r;
        live[r] = row < rows;
        tok[r] = t0 + (live[r] ? row : 0);
        const uint32_t in_run = a.tin[2 * tok[r] + 1];
        p8[r] = a.meta[2 * (tok[r] - in_run % 8) + 1];  // that token is the first of the 8-row tile: its position is the tile's
        vmask[r] = live[r] ? a.vis[tok[r]] : 0u;
        if (live[r] && vmask[r]) my_end = max(my_end, p8[r] + 32 - __clz(vmask[r]));
    }
    // The block walks keys [0, block_end): the furthest any of its rows sees.
    uint32_t block_end = my_end;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) block_end = max(block_end, __shfl_xor_sync(0xffffffffu, block_end, o));
    __shared__ uint32_t ends[WARPS];
    if (lane == 0 && grp == 0) ends[warp] = block_end;  // (the groups hold the same rows)
    if (tid == 0) {
        for (uint32_t s = 0; s < STAGES; s++) mbar_init(smem_u32(&bars[s]), 1);
        fail[grp] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    const uint32_t warp_end = ends[warp];
    block_end = max(max(ends[0], ends[1]), max(ends[2], ends[3]));
    const uint32_t n_blocks = (block_end + CK - 1) / CK;
    const uint32_t my_blocks = (n_blocks + GROUPS - 1 - grp) / GROUPS;  // this group's: grp, grp + GROUPS, ...

    const uint32_t* ptab = a.page_table + size_t(slot) * a.kv.max_pages;
    const uint32_t row_base = a.layer * a.kv.n_pages;
    auto issue = [&](uint32_t i) {  // the group's thread 0: its i-th key block into stage i % STAGES
        const uint32_t b = i * GROUPS + grp, st = i % STAGES, bar = smem_u32(&bars[st]), dst = smem_u32(ring + st * STAGE_BYTES);
        mbar_expect_tx(bar, STAGE_BYTES);
        for (uint32_t pi = 0; pi < CK / PAGE; pi++) {
            // Pages past the sequence's last hold nothing this block may see (masked below): any valid page will do.
            const uint32_t idx = min(b * (CK / PAGE) + pi, a.kv.max_pages - 1);
            const uint32_t pg = min(ptab[idx], a.kv.n_pages - 1);
            const int y = int(((row_base + pg) * a.kv.n_kv + kvh) * PAGE);
            tma_load_2d(dst + pi * PAGE * HD * 2, &maps.k, 0, y, bar);
            tma_load_2d(dst + CK * HD * 2 + pi * PAGE * HD * 2, &maps.v, 0, y, bar);
        }
    };
    if (tid == 0)
        for (uint32_t i = 0; i < min(my_blocks, STAGES); i++) issue(i);

    // Q fragments (A operands) straight from global memory: row g / g + 8, dims 16 ks + 2 tq (+ 8).
    uint32_t qa[4][4];
    {
        const uint32_t* q32 = reinterpret_cast<const uint32_t*>(a.q_b);
#pragma unroll
        for (int ks = 0; ks < 4; ks++) {
            const size_t r0 = (size_t(tok[0]) * a.n_heads + h) * (HD / 2) + 8 * ks + tq, r1 = (size_t(tok[1]) * a.n_heads + h) * (HD / 2) + 8 * ks + tq;
            qa[ks][0] = live[0] ? q32[r0] : 0u;
            qa[ks][1] = live[1] ? q32[r1] : 0u;
            qa[ks][2] = live[0] ? q32[r0 + 4] : 0u;
            qa[ks][3] = live[1] ? q32[r1 + 4] : 0u;
        }
    }
    // ldmatrix lane roles: matrix lm = lane / 8, row lr = lane % 8. A page is 16 rows of 128 bytes, 2 KiB (1024-byte aligned
    // halves), so the swizzled 16-byte chunk is (chunk ^ (row & 7)).
    const uint32_t lm = lane >> 3, lr = lane & 7;

    float oacc[8][4];  // O: n-tile jd = dims 8 jd .. 8 jd + 7; [0,1] row g, [2,3] row g + 8
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f};
#pragma unroll
    for (int jd = 0; jd < 8; jd++)
#pragma unroll
        for (int e = 0; e < 4; e++) oacc[jd][e] = 0.0f;

    bool failed = false;
    for (uint32_t i = 0; i < my_blocks; i++) {
        const uint32_t b = i * GROUPS + grp, st = i % STAGES, parity = (i / STAGES) & 1;
        if (!mbar_wait(smem_u32(&bars[st]), parity)) { failed = true; }
        if (__any_sync(0xffffffffu, failed)) { if (lane == 0) fail[grp] = 1; }
        const uint32_t kbase = smem_u32(ring + st * STAGE_BYTES), vbase = kbase + CK * HD * 2, key0 = b * CK;
        if (!failed && key0 < warp_end) {  // (a warp whose rows see nothing of this block skips the arithmetic, not the barriers)
            // S = Q K^T: 16 rows x 64 keys; n-tile j = keys 8 j .. 8 j + 7.
            float sacc[8][4];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                sacc[j][0] = sacc[j][1] = sacc[j][2] = sacc[j][3] = 0.0f;
                const uint32_t krow = 8 * j + lr, kaddr = kbase + (krow / PAGE) * (PAGE * HD * 2) + (krow % PAGE) * 128;
#pragma unroll
                for (int kp = 0; kp < 2; kp++) {  // k steps 2 kp and 2 kp + 1: chunks 4 kp + lm
                    uint32_t kb[4];
                    ldmatrix_x4(kb, kaddr + (((4 * kp + lm) ^ (krow & 7)) << 4));
                    mma16816(sacc[j], qa[2 * kp], kb[0], kb[1]);
                    mma16816(sacc[j], qa[2 * kp + 1], kb[2], kb[3]);
                }
            }
            // What each row may see: keys below its tile's first position, and of the tile's keys those its mask names.
            const uint32_t lo = min(p8[0], p8[1]);
            if (key0 + CK > lo || !live[0] || !live[1]) {
#pragma unroll
                for (int j = 0; j < 8; j++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const uint32_t r = e >> 1, key = key0 + 8 * j + 2 * tq + (e & 1);
                        const bool seen = live[r] && (key < p8[r] || (key - p8[r] < 32 && ((vmask[r] >> (key - p8[r])) & 1u)));
                        if (!seen) sacc[j][e] = -INFINITY;
                    }
            }
            // Online softmax, a row's 64 scores in the four lanes of its quad, with a lazy maximum as in the decode kernel
            // (k_attn.cu): it only has to keep 2^(s - m) in range, so it moves, and the sums so far are rescaled, when a score of
            // the block exceeds it by more than 8 -- one vote in place of the quads' reductions and 32 products a thread.
            float mx[2];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                mx[r] = -INFINITY;
#pragma unroll
                for (int j = 0; j < 8; j++) mx[r] = fmaxf(mx[r], fmaxf(sacc[j][2 * r], sacc[j][2 * r + 1]));
            }
            if (__any_sync(0xffffffffu, mx[0] > m_run[0] + 8.0f || mx[1] > m_run[1] + 8.0f)) {
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
                    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
                    const float m_new = fmaxf(m_run[r], mx[r]), corr = fast_exp2(m_run[r] - (m_new == -INFINITY ? 0.0f : m_new));
                    m_run[r] = m_new;
                    l_run[r] *= corr;
#pragma unroll
                    for (int jd = 0; jd < 8; jd++) {
                        oacc[jd][2 * r] *= corr;
                        oacc[jd][2 * r + 1] *= corr;
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const float m_use = m_run[r] == -INFINITY ? 0.0f : m_run[r];
                float sum = 0.0f;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    sacc[j][2 * r] = fast_exp2(sacc[j][2 * r] - m_use);
                    sacc[j][2 * r + 1] = fast_exp2(sacc[j][2 * r + 1] - m_use);
                    sum += sacc[j][2 * r] + sacc[j][2 * r + 1];
                }
                l_run[r] += sum;  // this lane's share of the row; the quad's shares meet at the end
            }
            // O += P V: key step kk = keys 16 kk .. 16 kk + 15 (one page); P's accumulators are the A fragments.
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {
                uint32_t pa[4];
                pa[0] = pack_bf16(sacc[2 * kk][0], sacc[2 * kk][1]);
                pa[1] = pack_bf16(sacc[2 * kk][2], sacc[2 * kk][3]);
                pa[2] = pack_bf16(sacc[2 * kk + 1][0], sacc[2 * kk + 1][1]);
                pa[3] = pack_bf16(sacc[2 * kk + 1][2], sacc[2 * kk + 1][3]);
                const uint32_t vrow = 8 * (lm & 1) + lr, vaddr = vbase + kk * (PAGE * HD * 2) + vrow * 128;
#pragma unroll
                for (int dp = 0; dp < 4; dp++) {  // dims 16 dp .. 16 dp + 15: n-tiles 2 dp and 2 dp + 1
                    uint32_t vb[4];
                    ldmatrix_x4_trans(vb, vaddr + (((2 * dp + (lm >> 1)) ^ (vrow & 7)) << 4));
                    mma16816(oacc[2 * dp], pa, vb[0], vb[1]);
                    mma16816(oacc[2 * dp + 1], pa, vb[2], vb[3]);
                }
            }
        }
        group_sync<GROUPS>(grp);  // every warp of the group is done with this stage
        if (fail[grp]) break;
        if (tid == 0 && i + STAGES < my_blocks) issue(i + STAGES);
    }
    // The other groups' (m, l, O) to the first through their own rings (their copies have all been read), a float of every
    // thread side by side; the first group adds them up in order and stores.
    constexpr uint32_t ROW = WARPS * 32;
    static_assert(36 * ROW * 4 <= STAGES * STAGE_BYTES, "a group's results must fit in its ring");
    if (grp && !fail[grp]) {
        float* mine = reinterpret_cast<float*>(ring) + tid;
#pragma unroll
        for (int jd = 0; jd < 8; jd++)
#pragma unroll
            for (int e = 0; e < 4; e++) mine[(4 * jd + e) * ROW] = oacc[jd][e];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            mine[(32 + r) * ROW] = m_run[r];
            mine[(34 + r) * ROW] = l_run[r];
        }
    }
    __syncthreads();
    bool any_fail = false;
    for (uint32_t k = 0; k < GROUPS; k++) any_fail = any_fail || fail[k];
    if (any_fail) {
        // A copy never arrived: say so, give the copies in flight a bounded time, and leave.
        if (tid == 0 && fail[grp]) {
            atomicExch(a.err_flag, 3u);
            for (uint32_t s = 0; s < STAGES; s++) mbar_wait(smem_u32(&bars[s]), 0, 1u << 16);
        }
        return;
    }
    if (grp) return;
#pragma unroll
    for (uint32_t k = 1; k < GROUPS; k++) {
        const float* theirs = reinterpret_cast<const float*>(smem + k * STAGES * STAGE_BYTES) + tid;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const float m_other = theirs[(32 + r) * ROW], m_new = fmaxf(m_run[r], m_other), m_use = m_new == -INFINITY ? 0.0f : m_new;
            const float w0 = fast_exp2(m_run[r] - m_use), w1 = fast_exp2(m_other - m_use);
            m_run[r] = m_new;
            l_run[r] = l_run[r] * w0 + theirs[(34 + r) * ROW] * w1;
#pragma unroll
            for (int jd = 0; jd < 8; jd++)
#pragma unroll
                for (int e = 2 * r; e < 2 * r + 2; e++) oacc[jd][e] = oacc[jd][e] * w0 + theirs[(4 * jd + e) * ROW] * w1;
        }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        float l = l_run[r];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        if (!live[r]) continue;
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;
        const size_t at = size_t(tok[r]) * a.n_heads * HD + h * HD;
#pragma unroll
        for (int jd = 0; jd < 8; jd++) {
            const float x = oacc[jd][2 * r] * inv, y = oacc[jd][2 * r + 1] * inv;
            *reinterpret_cast<float2*>(a.out + at + 8 * jd + 2 * tq) = make_float2(x, y);
            if (a.out_b) *reinterpret_cast<uint32_t*>(a.out_b + at + 8 * jd + 2 * tq) = pack_bf16(x, y);
        }
    }
}

}  // namespace prefill

template <uint32_t GROUPS>
static void launch_chunk_groups(const ChunkAttnArgs& a, cudaStream_t s) {
    const size_t smem = size_t(GROUPS) * prefill::STAGES * prefill::STAGE_BYTES + 1024;
    static PerDevice configured;
    configured.once([smem] { VLT_CUDA(cudaFuncSetAttribute(prefill::attn_chunk_kernel<GROUPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem))); });
    launch_pdl(prefill::attn_chunk_kernel<GROUPS>, dim3(a.n_ctiles, a.n_heads), GROUPS * prefill::WARPS * 32, smem, s, a, *a.maps);
}

// key_blocks: the 64-key blocks of all the tiles together. Two groups of warps a block halve a tile's chain of key blocks, and
// cost an exchange and a block less on the SM: they pay from four key blocks a tile on, unless they make a wave of blocks
// more, and where every block has an SM to itself as soon as the second group has something to do (one key block and a
// half a tile). Measured over 1 to 16 tiles of 32 heads and 1 to 40 key blocks a tile (one group / two, us): 1 tile, 1 key block
// 10.3 / 10.4, 32: 51 / 38; 117 rows (2 tiles) 12.2 / 11.3; 8 tiles, 1 key block 11.8 / 13.3, 4: 16.4 / 16.3, 32: 60 / 48;
// 12 tiles (384 blocks: one wave or two), 32 key blocks 68 / 78; 16 tiles (512: two waves either way), 1 key block
// 18.5 / 20.5, 32: 117 / 87; 60 runs of 16 rows, 1 key block 29 / 43. The rule takes the faster one there, or one within 5 %.
void launch_attn_chunk(const ChunkAttnArgs& a, uint32_t key_blocks, uint32_t sm_count, cudaStream_t s) {
    if (!a.n_ctiles) return;
    const uint32_t blocks = a.n_ctiles * a.n_heads;
    auto waves = [&](uint32_t groups) { return (blocks + prefill::blocks_per_sm(groups) * sm_count - 1) / (prefill::blocks_per_sm(groups) * sm_count); };
    if (2 * key_blocks >= (blocks <= sm_count ? 3 : 8) * a.n_ctiles && waves(2) <= waves(1)) launch_chunk_groups<2>(a, s);
    else launch_chunk_groups<1>(a, s);
}

}  // namespace vlt
