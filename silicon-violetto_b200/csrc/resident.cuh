// What the kernels that stay on the SMs for a whole step share: words that carry their own arrival, bounded waits, the ring of
// weights, and the matmul of at most 8 tokens whose activations live in registers.
//
// Words that carry their own arrival. A buffer another block's threads fill is all ones before the launch, and no producer ever
// stores that word: a float result that is not a number is 0x7fffffff and a converted bf16 one 0x7fff, so 0xffffffff is neither
// a float nor a pair of bf16 values that these kernels compute. A reader loads what it needs and loads it again until no word is
// all ones: one trip to L2 behind the producer's store, where a grid-wide barrier takes three (the fence, the count, the poll)
// and the loads follow. Every word is written once per launch; the buffers of one launch are cleared by the next but one
// (two sets take turns), so the end of a kernel orders the clearing against the next use.
#pragma once
#include "kernels.h"
#include "mma.cuh"

namespace vlt {

constexpr uint32_t ABSENT = 0xffffffffu;

__device__ __forceinline__ uint4 ld_word4(const void* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
// 16 bytes as one access (never half of a store): one of its words tells for all, if they were stored as one.
__device__ __forceinline__ uint4 ld_whole(const void* p) {
    uint64_t lo, hi;
    asm volatile("{\n.reg .b128 t;\nld.relaxed.gpu.global.b128 t, [%2];\nmov.b128 {%0, %1}, t;\n}" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    return make_uint4(uint32_t(lo), uint32_t(lo >> 32), uint32_t(hi), uint32_t(hi >> 32));
}
__device__ __forceinline__ void st_whole(void* p, uint4 v) {
    const uint64_t lo = v.x | uint64_t(v.y) << 32, hi = v.z | uint64_t(v.w) << 32;
    asm volatile("{\n.reg .b128 t;\nmov.b128 t, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ uint2 ld_word2(const void* p) {
    uint2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_word(const void* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(void* p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void st_word(void* p, float v) { st_word(p, min(__float_as_uint(v), 0xfffffffeu)); }  // (whatever a NaN's bits may be)
__device__ __forceinline__ bool there(uint4 v) { return v.x != ABSENT && v.y != ABSENT && v.z != ABSENT && v.w != ABSENT; }
__device__ __forceinline__ bool there(uint2 v) { return v.x != ABSENT && v.y != ABSENT; }

// A wait that ends: after some 2^22 polls (seconds) it sets the error word, the launch's own `over` word (all ones before) and the
// block's `dead`, and from then on no wait of the block waits. Another block that finds `over` set gives up as well, so a launch
// ends soon after its first failure. (The error word alone would not do: an earlier kernel may have set it.)
struct Patience {
    uint32_t *err, *over_word;
    volatile uint32_t* dead;  // shared memory
    uint32_t polls = 0;
    __device__ __forceinline__ void give_up() const {
        atomicExch(err, 8u);
        st_word(over_word, 0u);
        *dead = 1u;
    }
    __device__ __forceinline__ bool over() {
        if ((++polls & 31u) != 0) return false;
        if (*dead) return true;
        if (polls > (1u << 22)) give_up();
        else if (ld_word(over_word) != ABSENT) *dead = 1u;
        else return false;
        return true;
    }
};

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar, uint32_t count) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity), "r"(20000u) : "memory");  // (suspended for up to 20 us)
    return ok != 0;
}
// All lanes of a warp, converged. The limit is above every other wait's, so that a block whose data never came still drains its
// copies; what runs out here sets the error word.
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t parity, const Patience& p) {
#pragma unroll 1
    for (uint32_t i = 0; i < (1u << 26); i++)
        if (bar_try(bar, parity)) return;
    p.give_up();
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void tile_load(uint32_t dst, const void* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ void tile_load(uint32_t dst, const void* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}

constexpr uint32_t RES_WARPS = 16, RES_THREADS = RES_WARPS * 32;  // the warps that compute
constexpr uint32_t RES_ASKERS = 128;  // behind them, a warp that asks for weights (and three that make a warpgroup of it, which can give registers away)
constexpr uint32_t RES_SLICE = 2048, RES_PIECE = 128;             // bytes of a weight row in a stage; in pieces, one to a warp
constexpr uint32_t RES_ITEM = 16 * RES_SLICE;                     // [piece][row][128 bytes]
constexpr uint32_t RES_STAGE = RES_ITEM + 1024;                   // the rows' scales behind (and pages of keys land swizzled)
constexpr uint32_t RES_STAGES = 5;
constexpr uint32_t RES_TOK = 20;                                  // floats between two tokens of a warp's sums: 16 rows and room against bank conflicts
constexpr uint32_t RES_SUMS = 8 * RES_TOK;                        // floats of a warp's sums of a 16 x 8 tile
constexpr uint32_t RES_RED = 2 * RES_WARPS * RES_SUMS;            // floats: two buffers of every warp's sums
constexpr uint32_t RES_X = 32 * 1024;                             // bytes: the activations of 8 tokens of 2 KiB weight rows (int8; 4 KiB bf16), as operands
static_assert(RES_STAGE % 1024 == 0, "stages keep the swizzle's alignment");

__device__ __forceinline__ void res_sync() { asm volatile("bar.sync 1, %0;" ::"n"(RES_THREADS) : "memory"); }

// Four int8 (one word) to two fp16 pairs, exactly: byte ^ 0x80 under the exponent byte 0x64 is the half 1024 + 128 + q, and a
// packed subtraction of 1152 leaves q.
__device__ __forceinline__ void i8x4_to_f16(uint32_t w, uint32_t& lo, uint32_t& hi) {
    const uint32_t u = w ^ 0x80808080u;
    const uint32_t a = __byte_perm(u, 0x64646464u, 0x5140), b = __byte_perm(u, 0x64646464u, 0x5342);
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(lo) : "r"(a), "r"(0x64806480u));
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(hi) : "r"(b), "r"(0x64806480u));
}
// The larger of the magnitudes, under a sign.
__device__ __forceinline__ uint32_t max_abs_f16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t max_abs_bf16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ float largest_f16(uint32_t x) {
    float lo, hi;
    asm("{\n.reg .f16 a, b;\nmov.b32 {a, b}, %2;\ncvt.f32.f16 %0, a;\ncvt.f32.f16 %1, b;\n}" : "=f"(lo), "=f"(hi) : "r"(x));
    return fmaxf(fabsf(lo), fabsf(hi));
}
// A pair of bf16 values, each times a power of two, in fp16.
__device__ __forceinline__ uint32_t bf16x2_to_f16x2(uint32_t x, float times) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(bf16hi(x) * times), "f"(bf16lo(x) * times));
    return r;
}
template <bool F16>
__device__ __forceinline__ void mma_16n8k16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if (F16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The ring's stage and its phase for the i-th item.
__device__ __forceinline__ uint32_t ring_stage(uint32_t i) { return i % RES_STAGES; }
__device__ __forceinline__ uint32_t ring_phase(uint32_t i) { return (i / RES_STAGES) & 1u; }

}  // namespace vlt
