// The layers (and the head) of a plain decoder's step of at most 8 tokens as ONE launch that stays on the SMs.
//
// Such a step is a chain: 16 layers of qkv, attention, merge, o, gate_up, down, each needing all of the one before, with 1.2 GB
// of weights that depend on nothing. As a launch each, the chain cost 5 - 16 us a link (dependency gap, pipeline fill, staging of
// the activations, drain) against 9 us of memory time for a layer's 61 MB. Here a block per SM runs through all of them:
//   - a seventeenth warp asks for the block's share of the weights, and of the cached keys and values, in the order the others
//     will want them, a ring of stages ahead of them and across every link: HBM keeps working while the chain waits;
//   - a link is the words themselves (resident.cuh): the activations of the next matmul are polled for in L2 by the warps that
//     multiply by them. No barrier over the grid, no fence;
//   - four warps take a stage of 16 rows x 2 KiB, a quarter of k each; four such groups work on row tiles of their own where a row
//     is a stage wide (the block's activations are then in shared memory, as operands), on a row's parts where it is longer (each
//     warp loads its part's). What is not a product (waits, the sums' meeting, the epilogue) is then 100 instructions of 500 a
//     tile, where 16 warps on every tile together had 200 of 310;
//   - the residual stream stays in shared memory of the block that owns its 16 rows (o and down have the same rows), in fp32,
//     and what the norms need of it, the sum of squares per 16 rows, travels beside the bf16 rows.
// Two things cost more than the work itself until they were seen. Code: an SM holds 32 KB of it, the rest comes from the GPC's cache
// in every layer, 128 bytes in some 50 cycles, so there is one copy of everything and few loops are unrolled. Registers: beside the
// ring, L1 has no room for what 512 threads spill, and each such word is a trip to L2; hence at most 32 registers of operands a warp.
// What bounds it: a link is about 1 us from a store to its reader's registers, six links a layer, and the phases' own chains (copy,
// products, sums, epilogue) between; the rest is the HBM time. One stream over 8 192 keys, int8: 903 us a step with a launch a
// phase, 694 so; one of 5 rows over 3 001 keys, bf16: 1 098 and 843.
// The launch is cooperative: its blocks wait for one another, so all of them must be resident. Every wait is bounded.
#include <algorithm>

#include "resident.cuh"

namespace vlt {

static constexpr uint32_t PAGE = 16, HD = 64;
static constexpr uint32_t ITEM_PAGES = 8, PAGE_BYTES = 2 * PAGE * HD * 2;  // K then V
static_assert(ITEM_PAGES * PAGE_BYTES <= RES_STAGE, "an item of pages fits a stage");
static constexpr uint32_t LISTED = 256;      // of the block's pages, those whose places are kept
static constexpr uint32_t NOT_MINE = 0x7fffffffu;

enum : uint32_t { PH_QKV, PH_ATTN, PH_O, PH_GU, PH_DOWN, PH_HEAD, PH_END };

// An attention unit: a split of a tile's cached keys for one kv head.
struct Unit {
    uint32_t tile, kvh, split, page0, pages;
    uint32_t n_cols, nt, nt_recip, kg;  // query columns, n-tiles of 8 of them (warps side by side), 65536 / nt rounded up, key groups
    uint32_t fresh;                     // the key group that takes the step's own rows (NOT_MINE: another split does)
};

struct DecodeSmem {
    uint64_t full[RES_STAGES], empty[RES_STAGES];
    float2 cs[8][32];           // a token's (cos, sin) per pair of dims
    size_t kvrow[8];            // its row in the first layer's cache for kv head 0
    float resid[DECODE_RESID_TILES][8][16];
    float ssp[RES_WARPS][8];    // a warp's share of a token's sum of squares
    uint32_t mx[2][8];          // a token's largest magnitude (its bits), by turns
    float sc[RES_WARPS / 4][2][16];  // a team's rows' scales, by buffer
    float mw[8][RES_WARPS];     // attention: a warp's maximum per column
    uint32_t tok_tile[8], tok_row[8], vis[8];
    uint32_t t0[8], rows[8], slot[8], p0[8];
    Unit unit[DECODE_UNITS];    // the block's
    uint32_t ids[LISTED];       // the pages of the block's units, as far as there is room
    uint32_t dead, asked;       // asked: items whose stage has come free for them
};

// A block's first row tile; it takes every gridDim.x-th from there. qkv counts from the other end, so that the blocks without a
// tile of o and down have the second ones of qkv.
__device__ __forceinline__ uint32_t first_tile(uint32_t ph) { return ph == PH_QKV ? gridDim.x - 1 - blockIdx.x : blockIdx.x; }
__device__ __forceinline__ uint32_t width_of(const DecodeArgs& a, uint32_t ph) { return ph == PH_O ? a.attn_w : ph == PH_DOWN ? a.ffn : a.d; }
__device__ __forceinline__ uint32_t tiles_of(const DecodeArgs& a, uint32_t ph) {
    return (ph == PH_HEAD ? a.vocab : ph == PH_QKV ? a.qkv_w : ph == PH_GU ? 2 * a.ffn : a.d) / 16;
}

__device__ __forceinline__ Unit unit_of(const DecodeArgs& a, const DecodeSmem& sm, uint32_t u) {
    Unit x;
    const uint32_t su = u / a.kv.n_kv;
    x.kvh = u - su * a.kv.n_kv;
    x.tile = 0;
    while (su >= a.unit0[x.tile + 1]) x.tile++;
    x.split = su - a.unit0[x.tile];
    const uint32_t n_pages = (sm.p0[x.tile] + PAGE - 1) / PAGE, last = a.unit0[x.tile + 1] - a.unit0[x.tile] - 1;
    const uint32_t owner = n_pages ? min((n_pages - 1) / a.split_pages, last) : 0u;
    x.page0 = x.split * a.split_pages;
    x.pages = x.page0 >= n_pages ? 0u : x.split == last ? n_pages - x.page0 : min(a.split_pages, n_pages - x.page0);
    x.n_cols = sm.rows[x.tile] * a.heads_per_kv;
    x.nt = (x.n_cols + 7) / 8;
    x.nt_recip = (65536 + x.nt - 1) / x.nt;
    x.kg = RES_WARPS / x.nt;
    x.fresh = x.split == owner ? x.pages % x.kg : NOT_MINE;
    return x;
}

__device__ __forceinline__ Patience patience(const DecodeArgs& a, DecodeSmem& sm) { return Patience{a.err_flag, reinterpret_cast<uint32_t*>(a.arena + a.ar.over), &sm.dead}; }

// The warp that fills the ring: a copy of 32 KiB a stage (an SM starts no more than one of its copies in some 70 cycles: a copy for
// each of the 16 rows' pieces, 0.6 us a stage, bound everything else). It walks over the block's items -- (row tile, 2 KiB of k) or
// (unit, 8 pages) -- in the order the others want them. Whatever a copy needs is at hand before its turn: the ring is deep in bytes,
// not in time. (Not done: a second warp that has L2 fetch the items 3, 7 or 15 behind the ring's. One stream's step went from 609 to
// 656, 671 and 709 us: the words that the chain waits for queue behind what HBM then delivers.)
__device__ __forceinline__ void ask(const DecodeArgs& a, const AttnMaps& maps, DecodeSmem& sm, uint32_t stages) {
    const uint32_t lane = threadIdx.x % 32;
    uint32_t item = 0;
    auto stage = [&]() -> uint32_t {  // the item's, when it is free
        const uint32_t st = ring_stage(item);
        if (item >= RES_STAGES) bar_wait(smem_u32(&sm.empty[st]), ring_phase(item) ^ 1u, patience(a, sm));
        item++;
        if (lane == 0) *const_cast<volatile uint32_t*>(&sm.asked) = item;
        return st;
    };
    // Lanes 0 .. 3: the layer's scales, fetched while the layer before is asked for (behind the last layer the head's, in lane 0).
    auto fetch = [&](uint32_t layer) -> const uint16_t* {
        const uint32_t i = layer < a.n_layers ? 4 * layer + lane : 4 * a.n_layers;
        if (lane >= (layer < a.n_layers ? 4u : a.n_head ? 1u : 0u)) return nullptr;
        asm volatile("prefetch.tensormap [%0];" ::"l"(&a.maps[i]) : "memory");
        return a.wbytes == 1 ? a.scales[i] : nullptr;
    };
    const uint16_t *at_hand = nullptr, *coming = fetch(a.s0 / PH_HEAD);
    uint32_t layer = a.s0 / PH_HEAD, ph = a.s0 % PH_HEAD;
    bool turned = true;
#pragma unroll 1
    for (uint32_t s = a.s0; s < a.s1 + (a.n_head ? 1u : 0u); s++) {
        if (turned) {
            at_hand = coming;
            coming = fetch(layer + 1);
            turned = false;
        }
        if (s == a.s1) ph = PH_HEAD;
        {
            if (ph == PH_ATTN) {
                uint32_t listed = 0;
#pragma unroll 1
                for (uint32_t u = 0; u * gridDim.x + blockIdx.x < a.n_units; u++) {
                    const Unit& x = sm.unit[u];
#pragma unroll 1
                    for (uint32_t first = 0; first < x.pages; first += ITEM_PAGES, listed += ITEM_PAGES) {
                        const uint32_t count = min(x.pages - first, ITEM_PAGES), st = stage(), bar = smem_u32(&sm.full[st]);
                        if (lane == 0) bar_expect(bar, count * PAGE_BYTES);
                        __syncwarp();
                        if (lane < count) {
                            const uint32_t id = listed + lane < LISTED ? sm.ids[listed + lane] : a.page_table[size_t(sm.slot[x.tile]) * a.kv.max_pages + x.page0 + first + lane];
                            const int y = int(((layer * a.kv.n_pages + id) * a.kv.n_kv + x.kvh) * PAGE);
                            const uint32_t to = stages + st * RES_STAGE + lane * PAGE_BYTES;
                            tile_load(to, &maps.k, 0, y, bar);
                            tile_load(to + PAGE_BYTES / 2, &maps.v, 0, y, bar);
                        }
                    }
                }
                ph++;
                continue;
            }
            const bool head = ph == PH_HEAD;
            const uint32_t which = ph == PH_QKV || head ? 0u : ph - 1;
            const uint16_t* scales = reinterpret_cast<const uint16_t*>(__shfl_sync(0xffffffffu, reinterpret_cast<uint64_t>(at_hand), which));
#pragma unroll 1
            for (uint32_t at = first_tile(ph); at < tiles_of(a, ph); at += gridDim.x)
#pragma unroll 1
                for (uint32_t part = 0; part * RES_SLICE < width_of(a, ph) * a.wbytes; part++) {
                    const uint32_t st = stage(), bar = smem_u32(&sm.full[st]), dst = stages + st * RES_STAGE;
                    const bool with = a.wbytes == 1 && (part + 1) * RES_SLICE >= width_of(a, ph);
                    if (lane == 0) {
                        bar_expect(bar, RES_ITEM + (with ? 32u : 0u));  // (what a box has beyond the matrix counts, and is zero)
                        tile_load(dst, &a.maps[head ? 4 * a.n_layers : 4 * layer + which], 0, int(at * 16), int(part * 16), bar);
                        if (with) bulk_load(dst + RES_ITEM, scales + at * 16, 32, bar);
                    }
                    __syncwarp();
                }
            if (++ph == PH_HEAD) {
                ph = PH_QKV;
                layer++;
                turned = true;
            }
        }
    }
}

// What a warp that computes carries along.
struct Ctx {
    uint32_t warp, lane, g, t;
    uint32_t items;  // of the ring, before the phase
    uint32_t turn;   // of sm.mx
    // Hides from the compiler that these do not change: what it works out from them is worked out again in every phase instead of
    // being kept, in local memory, from one layer to the next (which took longer: L1 has no room beside the ring).
    __device__ __forceinline__ void renew() {
        asm volatile("" : "+r"(warp), "+r"(lane));
        g = lane >> 2;
        t = lane & 3;
    }
};

// Waits for the ring's i-th item; its stage. A warp may want an item before the stage's last one has even come (the groups take
// items of their own), and a barrier only tells odd phases from even ones: so first that the asking warp has come to the item, which
// it does when every reader of the stage's last one is done.
__device__ __forceinline__ uint32_t ring_wait(const DecodeArgs& a, DecodeSmem& sm, uint32_t i) {
    const uint32_t st = ring_stage(i);
#pragma unroll 1
    for (uint32_t n = 0; *const_cast<volatile uint32_t*>(&sm.asked) <= i && n < (1u << 26); n++) __nanosleep(20);
    bar_wait(smem_u32(&sm.full[st]), ring_phase(i), patience(a, sm));
    __syncwarp();
    return st;
}

__device__ __forceinline__ uint8_t* layer_arena(const DecodeArgs& a, uint32_t layer) { return a.arena + size_t(layer - a.l0) * a.ar.layer_bytes; }

// What multiplies int8 weights is fp16 (half the conversion's instructions): the bf16 value, times a power of two by phase. While a
// token's largest, so scaled, lies in [2^-6, 2^15), nothing overflows and what fp16 cannot hold is below 2^-19 of it; else the
// reader goes back to the bf16 words beside (`half` bytes before), scaled as they need it.
__device__ __forceinline__ float scale_of(uint32_t ph) { return ph == PH_O ? 64.0f : ph == PH_DOWN ? 16.0f : 1.0f; }

// A pair of values (bf16 word w) from every `step`-th of the lanes that hold eight values of a token between them, as one 16-byte
// store by the first of them.
template <bool INT8>
__device__ __forceinline__ void publish(uint8_t* words, uint32_t half, uint32_t at, uint32_t w, float times, uint32_t step, bool mine) {
    uint4 v;
    v.x = w;
    v.y = __shfl_down_sync(0xffffffffu, w, step);
    v.z = __shfl_down_sync(0xffffffffu, w, 2 * step);
    v.w = __shfl_down_sync(0xffffffffu, w, 3 * step);
    if (!mine) return;
    words += size_t(at) * 2;
    st_whole(words, v);
    if (INT8) st_whole(words + half, make_uint4(bf16x2_to_f16x2(v.x, times), bf16x2_to_f16x2(v.y, times), bf16x2_to_f16x2(v.z, times), bf16x2_to_f16x2(v.w, times)));
}

// The sum of squares of a tile's 16 rows (row r of token tok to a lane).
__device__ __forceinline__ void tile_squares(const DecodeArgs& a, float* ss, uint32_t tile, uint32_t tok, uint32_t r, float y) {
    float q = y * y;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    if (tok < a.n && r == 0) st_word(ss + tile * 8 + tok, q);
}

// A warp's operands of one 128-byte piece of k: two halves of 64 bytes, a lane 16 bytes of each.
template <bool INT8>
struct Piece {
    static constexpr uint32_t WB = INT8 ? 1 : 2, E = 16 / WB, R = E;  // weights of 16 bytes; words of both halves
    // Loads lane (g, t)'s activations of a piece that begins at x; false while some are not there.
    __device__ static __forceinline__ bool load(uint32_t (&r)[R], const uint16_t* x) {
        bool ok = true;
#pragma unroll
        for (uint32_t q = 0; q < R / 4; q++) {
            const uint4 v = ld_whole(x + (q / (R / 8)) * (64 / WB) + (q % (R / 8)) * 8);
            r[4 * q] = v.x; r[4 * q + 1] = v.y; r[4 * q + 2] = v.z; r[4 * q + 3] = v.w;
            ok = ok && v.x != ABSENT;
        }
        return ok;
    }
};

// The sums of squares of the tokens' rows: this warp's share of the tiles, four lanes to a token (of column lane % 8). The first 128
// tiles' words are asked for before the activations are polled for, and are there when those are.
struct Squares {
    const float* at;
    uint32_t tile, tiles, v0, v1;
    __device__ __forceinline__ void ask() {
        v0 = tile < tiles ? ld_word(at + tile * 8) : 0u;
        v1 = tile + 64 < tiles ? ld_word(at + (tile + 64) * 8) : 0u;
    }
    __device__ __forceinline__ float sum(Patience p) {
        float s = 0.0f;
#pragma unroll 1
        for (;;) {
            while ((v0 == ABSENT || v1 == ABSENT) && !p.over()) ask();
            s += __uint_as_float(v0);
            s += __uint_as_float(v1);
            tile += 128;
            if (tile >= tiles) break;
            ask();
        }
        __syncwarp();
        s += __shfl_xor_sync(0xffffffffu, s, 8);
        return s + __shfl_xor_sync(0xffffffffu, s, 16);
    }
};

// One matmul phase: the block's row tiles of a matrix against the activations x [token][k] (bf16, polled for), the epilogue by phase.
// Columns past the tokens repeat the last one's (nothing reads their sums).
template <bool INT8, bool LIMITE>
__device__ __forceinline__ void matmul_phase(const DecodeArgs& a, DecodeSmem& sm, uint8_t* stages, float* red, uint4* xs, Ctx& c, uint32_t layer, uint32_t ph, const uint8_t* words, const float* ss) {
    using P = Piece<INT8>;
    constexpr uint32_t WB = P::WB, E = P::E, R = P::R, KS = E / 4, PARTS = INT8 ? 1 : 2, CHUNK = 2;  // a group's parts of a row; pieces whose operands a warp holds (at most 32 registers)
    const uint32_t k = width_of(a, ph), tiles = tiles_of(a, ph), first = first_tile(ph);
    if (first >= tiles) return;
    const uint32_t pieces = k * WB / RES_PIECE, parts = (pieces + 15) / 16;
    const uint32_t size = (parts + PARTS - 1) / PARTS, teams = size == 1 ? 4u : size == 2 ? 2u : 1u;  // groups in a team
    const uint32_t group = c.warp / 4, kq = c.warp % 4, team = size == 1 ? group : size == 2 ? group / 2 : group == 3 && size == 3 ? 1u : 0u, mate = group - team * size;
    const uint32_t nx = ph == PH_HEAD ? a.n_head : a.n, col = min(c.g, nx - 1);
    const uint32_t half = ph == PH_O ? a.ar.half_o : ph == PH_DOWN ? a.ar.half_ffn : a.ar.half_d;
    const uint16_t* xrow = reinterpret_cast<const uint16_t*>(words + (INT8 ? half : 0u)) + size_t(ph == PH_HEAD ? a.head_rows[col] : col) * k + c.t * E;
    const bool share = size == 1;  // every group needs all of the activations: a warp polls for a sixteenth

    res_sync();  // (the phase before is done with the buffers)
    Squares sq{nullptr, c.warp + 16 * (c.lane / 8), ss ? a.d / 16 : 0u, 0u, 0u};
    if (ss) {
        const uint32_t tok = min(c.lane % 8, nx - 1);
        sq.at = ss + (ph == PH_HEAD ? a.head_rows[tok] : tok);
        sq.ask();
    }
    if (share) {
#pragma unroll 1
        for (uint32_t i = c.warp * PARTS; i < min((c.warp + 1) * PARTS, pieces); i++) {
            uint32_t xr[R];
            Patience p = patience(a, sm);
            while (!P::load(xr, xrow + i * (RES_PIECE / WB)) && !p.over()) {}
            __syncwarp();
            if (INT8) {
                uint32_t m2 = 0u;
#pragma unroll
                for (uint32_t r = 0; r < R; r++) m2 = max_abs_f16x2(m2, xr[r]);
                uint32_t mx = __float_as_uint(largest_f16(m2));
                mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                if (c.t == 0 && c.g < nx) atomicMax(&sm.mx[c.turn][c.g], mx);
            }
#pragma unroll
            for (uint32_t q = 0; q < R / 4; q++) xs[(i * (R / 4) + q) * 32 + c.lane] = make_uint4(xr[4 * q], xr[4 * q + 1], xr[4 * q + 2], xr[4 * q + 3]);
        }
    }
    if (ss) {
        const float s = sq.sum(patience(a, sm));
        if (c.lane < 8) sm.ssp[c.warp][c.lane] = s;
    }
    if (share || ss) res_sync();
    auto fits = [](float mx) { return mx == 0.0f || (mx >= 0.015625f && mx < 32768.0f); };
    bool direct = !share;  // the operands come from L2 as they are needed (each once, if the block has one row tile)
    if (INT8 && share) {
        direct = __any_sync(0xffffffffu, !fits(__uint_as_float(sm.mx[c.turn][col])));
        c.turn ^= 1u;
        if (threadIdx.x < 8) sm.mx[c.turn][threadIdx.x] = 0u;
    }
    float inv = 1.0f;
    if (ss) {
        float sq = sm.ssp[c.lane % 16][2 * kq + c.lane / 16];
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        inv = rsqrtf(sq * a.inv_d + a.eps);
    }
    const uint32_t mine = (tiles - first + gridDim.x - 1) / gridDim.x;
    // Lane (g, t) reads 16 bytes of MMA row g, and of row g + 8, which are memory rows `row` and `row` + 8: rows four apart side by
    // side in a quarter of a warp, which the 128-byte swizzle keeps in different banks.
    const uint32_t row = c.g / 2 + 4 * (c.g & 1u), at0 = kq * 4 * (16 * RES_PIECE) + row * RES_PIECE + ((c.t ^ row) << 4);
    const uint4* x_lane = xs + kq * 4 * (R / 4 * 32) + col * 4 + c.t;
    uint32_t buf = 0;
#pragma unroll 1
    for (uint32_t i_tile = team < teams ? team : mine; i_tile < mine; i_tile += teams, buf ^= 1u) {
        float tot[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        uint32_t st = 0;
#pragma unroll 1
        for (uint32_t ch = 0; ch < PARTS * (4 / CHUNK); ch++) {  // a part's pieces of this warp, CHUNK at a time
            const uint32_t part = mate * PARTS + ch / (4 / CHUNK), lp = (ch % (4 / CHUNK)) * CHUNK, p0 = part * 16 + kq * 4 + lp;
            if (part >= parts) break;
            uint32_t xr[CHUNK][R];
            float up0 = INT8 ? 1.0f / scale_of(ph) : 1.0f, up1 = up0;  // what the sums of tokens 2 t, 2 t + 1 are multiplied by
            if (!direct) {
#pragma unroll
                for (uint32_t i = 0; i < CHUNK; i++)
#pragma unroll
                    for (uint32_t q = 0; q < R / 4; q++) {  // (a piece past the row's end is whatever was there: it is not multiplied by)
                        const uint4 v = x_lane[((part * 16 + lp + i) * (R / 4) + q) * 32];
                        xr[i][4 * q] = v.x; xr[i][4 * q + 1] = v.y; xr[i][4 * q + 2] = v.z; xr[i][4 * q + 3] = v.w;
                    }
            } else {
                const uint16_t* xp = xrow + p0 * (RES_PIECE / WB);
#pragma unroll 1
                for (bool again = false;; again = true) {
                    bool all = false;
                    Patience p = patience(a, sm);
                    while (!all) {
                        all = true;
#pragma unroll
                        for (uint32_t i = 0; i < CHUNK; i++)
                            if (p0 + i < pieces) all = P::load(xr[i], xp + i * (RES_PIECE / WB)) && all;
                        if (!all && p.over()) break;
                    }
                    __syncwarp();
                    if (!INT8) break;
                    uint32_t m2 = 0u;
#pragma unroll
                    for (uint32_t i = 0; i < CHUNK; i++)
                        if (p0 + i < pieces)
#pragma unroll
                            for (uint32_t r = 0; r < R; r++) m2 = again ? max_abs_bf16x2(m2, xr[i][r]) : max_abs_f16x2(m2, xr[i][r]);
                    float mx = again ? fmaxf(fabsf(bf16lo(m2)), fabsf(bf16hi(m2))) : largest_f16(m2);
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                    if (again) {
                        // (rare) The chunk's bf16 words, a token's times the power of two that puts its largest in [2^14, 2^15).
                        const uint32_t ex = max((__float_as_uint(mx) >> 23) & 0xffu, 15u);  // mx in [2^(ex-127), 2^(ex-126))
                        const float down = __uint_as_float((268u - ex) << 23), up = __uint_as_float((ex - 14u) << 23);
#pragma unroll
                        for (uint32_t i = 0; i < CHUNK; i++)
#pragma unroll
                            for (uint32_t r = 0; r < R; r++) xr[i][r] = bf16x2_to_f16x2(xr[i][r], down);
                        up0 = __shfl_sync(0xffffffffu, up, 8 * c.t);
                        up1 = __shfl_sync(0xffffffffu, up, 8 * c.t + 4);
                        break;
                    }
                    if (!__any_sync(0xffffffffu, !fits(mx))) break;
                    xp -= half / 2;
                }
            }
            if (lp == 0) st = ring_wait(a, sm, c.items + i_tile * parts + part);
            const uint8_t* sw = stages + size_t(st) * RES_STAGE + lp * (16 * RES_PIECE);
            float acc[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
#pragma unroll
            for (uint32_t i = 0; i < CHUNK; i++) {
                if (p0 + i >= pieces) break;  // (the same for the whole warp)
#pragma unroll
                for (uint32_t u = 0; u < 2; u++) {
                    const uint4 wl = *reinterpret_cast<const uint4*>(sw + (at0 ^ (u * 64)) + i * (16 * RES_PIECE));
                    const uint4 wh = *reinterpret_cast<const uint4*>(sw + (at0 ^ (u * 64)) + i * (16 * RES_PIECE) + 8 * RES_PIECE);
                    const uint32_t lo[4] = {wl.x, wl.y, wl.z, wl.w}, hi[4] = {wh.x, wh.y, wh.z, wh.w};
#pragma unroll
                    for (uint32_t ks = 0; ks < KS; ks++) {
                        uint32_t a0, a1, a2, a3;
                        if (INT8) {
                            i8x4_to_f16(lo[ks % 4], a0, a2);
                            i8x4_to_f16(hi[ks % 4], a1, a3);
                        } else {
                            a0 = lo[2 * ks % 4]; a2 = lo[(2 * ks + 1) % 4];
                            a1 = hi[2 * ks % 4]; a3 = hi[(2 * ks + 1) % 4];
                        }
                        mma_16n8k16<INT8>(acc[u], a0, a1, a2, a3, xr[i][u * (R / 2) + 2 * ks], xr[i][u * (R / 2) + 2 * ks + 1]);
                    }
                }
            }
            tot[0] += (acc[0][0] + acc[1][0]) * up0;
            tot[1] += (acc[0][1] + acc[1][1]) * up1;
            tot[2] += (acc[0][2] + acc[1][2]) * up0;
            tot[3] += (acc[0][3] + acc[1][3]) * up1;
            if (lp + CHUNK < 4) continue;
            // The row's last part brought the rows' scales.
            if (INT8 && part + 1 == parts && kq == 0 && c.lane < 16) sm.sc[team][buf][c.lane] = bf16_to_f32(*reinterpret_cast<const uint16_t*>(stages + size_t(st) * RES_STAGE + RES_ITEM + c.lane * 2));
            __syncwarp();
            if (c.lane == 0) bar_arrive(smem_u32(&sm.empty[st]), 4);
        }
        float* rb = red + (buf * RES_WARPS + c.warp) * RES_SUMS + 2 * c.t * RES_TOK + row;  // [token][row]
        rb[0] = tot[0];
        rb[RES_TOK] = tot[1];
        rb[8] = tot[2];
        rb[RES_TOK + 8] = tot[3];
        // The team meets, its first group adds up and stores. A warp may be one tile ahead of the readers, so there are two buffers.
        asm volatile("bar.sync %0, %1;" ::"r"(2 + team), "r"(size * 128) : "memory");
        if (mate) continue;
        const uint32_t r = c.lane & 15u, tok = 2 * kq + c.lane / 16, tile = first + i_tile * gridDim.x;
        const float* sp = red + (buf * RES_WARPS + team * size * 4) * RES_SUMS + tok * RES_TOK + r;
        float sum = 0.0f;
#pragma unroll 1
        for (uint32_t w = 0; w < size; w++, sp += 4 * RES_SUMS) sum += (sp[0] + sp[RES_SUMS]) + (sp[2 * RES_SUMS] + sp[3 * RES_SUMS]);
        if (INT8) sum *= sm.sc[team][buf][r];
        sum *= inv;
        const float other = __shfl_xor_sync(0xffffffffu, sum, 1);  // the pair's other row
        uint8_t* ar = layer_arena(a, layer);
        if (ph == PH_HEAD) {
            const uint32_t at = tile * 16 + r;
            if (tok < a.n_head) a.logits[size_t(tok) * a.vocab + at] = at < a.vocab_real ? sum : -INFINITY;
        } else if (LIMITE && ph == PH_QKV) {  // (the rest of this architecture's qkv work is a kernel of its own)
            if (tok < a.n) {
                a.qkv[tok * a.qkv_w + tile * 16 + r] = sum * a.lim.qkv_scale;
                if (tile == 0 && r == 0) a.inv_out[tok] = inv;
            }
        } else if (ph == PH_QKV) {
            // RoPE on q and k; q scaled for the attention; k and v into the cache and, for this step's attention, beside it.
            const uint32_t head = tile / (HD / 16), pair = (tile % (HD / 16)) * 8 + r / 2;
            if (r % 2 == 0 && tok < a.n) {
                float y0 = sum, y1 = other;
                if (head < a.n_heads + a.kv.n_kv) {
                    const float2 cs = sm.cs[tok][pair];
                    y0 = __fadd_rn(__fmul_rn(cs.x, sum), __fmul_rn(cs.y, other));
                    y1 = __fsub_rn(__fmul_rn(cs.x, other), __fmul_rn(cs.y, sum));
                }
                if (head < a.n_heads) {
                    st_word(ar + a.ar.q + ((tok * a.n_heads + head) * (HD / 2) + pair) * 4, pack_bf16(__fmul_rn(y0, a.scale_log2), __fmul_rn(y1, a.scale_log2)));
                } else {
                    const bool is_v = head >= a.n_heads + a.kv.n_kv;
                    const uint32_t kvh = head - a.n_heads - (is_v ? a.kv.n_kv : 0), word = pack_bf16(y0, y1);
                    st_word(ar + a.ar.kvn + (((tok * 2 + is_v) * a.kv.n_kv + kvh) * (HD / 2) + pair) * 4, word);
                    const size_t at = sm.kvrow[tok] + (size_t(layer) * a.kv.n_pages * a.kv.n_kv + kvh) * PAGE * HD;
                    reinterpret_cast<uint32_t*>((is_v ? a.v_cache : a.k_cache) + at)[pair] = word;
                }
            }
        } else {
            const bool gu = ph == PH_GU;
            float y;
            uint32_t to, at;  // where it goes: rows in the arena, and in them
            if (gu) {
                y = sum * __fdividef(1.0f, 1.0f + __expf(-sum)) * other;  // (of the even rows; the hardware's exponential and quotient: their errors are far below the rounding to bf16)
                to = a.ar.act;
                at = tok * a.ffn + tile * 8 + r / 2;
            } else {
                float& h = sm.resid[i_tile][tok][r];
                if (LIMITE) h = ph == PH_O ? a.lim.ra * h + a.lim.rb * (a.lim.o_scale * sum) : a.lim.ra2 * h + a.lim.rb2 * sum;
                else h += sum;
                y = h;
                to = ph == PH_O ? a.ar.x2 : a.ar.layer_bytes;  // (what down leaves is the next layer's input, or the head's)
                at = tok * a.d + tile * 16 + r;
                if (ph == PH_DOWN && (LIMITE || layer + 1 == a.l1)) {
                    if (tok < a.n) a.out[at] = y;
                    if (layer * PH_HEAD + PH_DOWN + 1 == a.s1 && !a.n_head) continue;  // (nothing follows in this launch)
                }
                tile_squares(a, reinterpret_cast<float*>(ar + to + (ph == PH_O ? a.ar.ss2 - a.ar.x2 : a.ar.ss1)), tile, tok, r, y);
            }
            const uint32_t pair = gu ? 2 : 1;  // lanes from one value to the next
            publish<INT8>(ar + to, gu ? a.ar.half_ffn : a.ar.half_d, at, pack_bf16(y, __shfl_down_sync(0xffffffffu, y, pair)), scale_of(gu ? PH_DOWN : PH_GU), 2 * pair, tok < a.n && r % (8 * pair) == 0);
        }
    }
    c.items += mine * parts;
}

// One unit of the attention: the unit's pages from the ring, a warp per (key group, n-tile of 8 query columns), the step's own rows
// beside them; the key groups meet in shared memory and leave (m, l, o[64]) per column.
__device__ __forceinline__ void attention_unit(const DecodeArgs& a, DecodeSmem& sm, uint8_t* stages, float* red, uint4* xs, Ctx& c, uint32_t layer, const Unit& x) {
    const uint32_t t0 = sm.t0[x.tile], T = sm.rows[x.tile], p0 = sm.p0[x.tile], KG = x.kg, NT = x.nt, pages = x.pages, page0 = x.page0;
    const uint32_t kg = (c.warp * x.nt_recip) >> 16, cw = c.warp - kg * NT;
    auto token_of = [&](uint32_t p) { return (p * a.per_kv_recip) >> 16; };  // of query column p < 32
    uint8_t* ar = layer_arena(a, layer);
    res_sync();  // (the phase before is done with the buffers)

    uint32_t qb[8];
    {
        const uint32_t col = min(8 * cw + c.g, x.n_cols - 1), tok = token_of(col);  // (columns past the last repeat it)
        const uint32_t* qp = reinterpret_cast<const uint32_t*>(ar + a.ar.q) + ((t0 + tok) * a.n_heads + x.kvh * a.heads_per_kv + col - tok * a.heads_per_kv) * (HD / 2) + c.t;
        bool need = true;
        Patience p = patience(a, sm);
        while (need) {
            need = false;
#pragma unroll
            for (int i = 0; i < 8; i++) qb[i] = ld_word(qp + 4 * i);  // dims 8 i + 2 t and + 1
#pragma unroll
            for (int i = 0; i < 8; i++) need = need || qb[i] == ABSENT;
            if (need && p.over()) break;
        }
        __syncwarp();
    }
    float oacc[4][4], m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f};
#pragma unroll
    for (int dm = 0; dm < 4; dm++)
#pragma unroll
        for (int e = 0; e < 4; e++) oacc[dm][e] = 0.0f;

    uint32_t pg = kg < KG ? kg : NOT_MINE, base = 0, have = 0;  // this warp's next page; its stage; items whose stage it holds or has given back
    bool own = x.fresh == kg;
#pragma unroll 1
    for (;;) {
        // On to the item that the page is in; the items before it are given back.
        const uint32_t want = pg < pages ? pg / ITEM_PAGES + 1 : (pages + ITEM_PAGES - 1) / ITEM_PAGES;
#pragma unroll 1
        while (have < want) {
            if (have && c.lane == 0) bar_arrive(smem_u32(&sm.empty[ring_stage(c.items + have - 1)]), 1);
            base = smem_u32(stages + size_t(ring_wait(a, sm, c.items + have)) * RES_STAGE);
            have++;
        }
        const bool fresh = pg >= pages;
        if (fresh && !own) break;
        c.renew();
        const uint32_t lm = c.lane >> 3, lr = c.lane & 7;
        const uint32_t k_off = (8 * (lm & 1) + lr) * 128 + (((lm >> 1) ^ lr) << 4), v_off = (8 * (lm >> 1) + lr) * 128 + (((lm & 1) ^ lr) << 4);
        uint32_t kbase = base + (pg % ITEM_PAGES) * PAGE_BYTES;
        if (fresh) {
            // The step's own rows (at most 8 keys) as a page in shared memory, from the words the qkv phase left: 16 bytes a lane and
            // turn. (The key group's warps each write it, the same.)
            own = false;
            kbase = smem_u32(xs);
            uint4 v[4];
            bool need = true;
            Patience p = patience(a, sm);
            auto from = [&](uint32_t i) -> uint32_t { return (((t0 + i / 16) * 2 + (i >> 3 & 1u)) * a.kv.n_kv + x.kvh) * (HD / 2) + (i & 7u) * 4; };  // row i / 16, K or V, chunk i % 8
            const uint32_t* kn = reinterpret_cast<const uint32_t*>(ar + a.ar.kvn);
            while (need) {
                need = false;
#pragma unroll
                for (uint32_t j = 0; j < 4; j++)
                    if (c.lane + 32 * j < 16 * T) v[j] = ld_word4(kn + from(c.lane + 32 * j));
#pragma unroll
                for (uint32_t j = 0; j < 4; j++) need = need || (c.lane + 32 * j < 16 * T && !there(v[j]));
                if (need && p.over()) break;
            }
#pragma unroll
            for (uint32_t j = 0; j < 8; j++) {
                const uint32_t i = c.lane + 32 * j, r = i / 16, ch = i & 7u;
                const bool is = j < 4 && r < T;  // (values of rows past the step's are zero: nothing there may count)
                if (is || (i >> 3 & 1u)) reinterpret_cast<uint4*>(xs)[(i >> 3 & 1u) * (PAGE * 8) + r * 8 + (ch ^ (r & 7u))] = is ? v[j % 4] : make_uint4(0u, 0u, 0u, 0u);
            }
            __syncwarp();
        }
        float sacc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        uint32_t ka[4][4];
#pragma unroll
        for (int ks = 0; ks < 4; ks++) ldmatrix_x4(ka[ks], (kbase + k_off) ^ (uint32_t(ks) << 5));
#pragma unroll
        for (int ks = 0; ks < 4; ks++) mma16816(sacc, ka[ks], qb[2 * ks], qb[2 * ks + 1]);
        // Every cached key below p0 is seen; of the step's rows those that a column's token names.
        const uint32_t key0 = (page0 + pg) * PAGE;
        const bool edge = !fresh && key0 + PAGE > p0;
        if (edge || fresh) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const uint32_t r = c.g + 8 * (e >> 1);
                if (!(fresh ? r < T && ((sm.vis[t0 + token_of(min(8 * cw + 2 * c.t + (e & 1), x.n_cols - 1))] >> r) & 1u) : key0 + r < p0)) sacc[e] = -INFINITY;
            }
        }
        if (edge) {  // whatever lies past p0 must not count, an infinity not even times zero
            for (uint32_t i = (p0 - key0) * 8 + c.lane; i < PAGE * 8; i += 32) asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(kbase + PAGE_BYTES / 2 + i * 16), "r"(0u) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // (a copy will write there again)
            __syncwarp();
        }
        // The scores become probabilities: a lazy maximum, as in the split kernel (k_attn.cu).
        bool over = false;
#pragma unroll
        for (int e = 0; e < 2; e++) over = over || fmaxf(sacc[e], sacc[e + 2]) > m_run[e] + 8.0f;
        if (__any_sync(0xffffffffu, over)) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                float mx = fmaxf(sacc[e], sacc[e + 2]);
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                const float m_new = fmaxf(m_run[e], mx);
                const float corr = fast_exp2(m_run[e] - (m_new == -INFINITY ? 0.0f : m_new));
                m_run[e] = m_new;
                l_run[e] *= corr;
#pragma unroll
                for (int dm = 0; dm < 4; dm++) {
                    oacc[dm][e] *= corr;
                    oacc[dm][e + 2] *= corr;
                }
            }
        }
        uint32_t pb[2];
        {
            const float m0 = m_run[0] == -INFINITY ? 0.0f : m_run[0], m1 = m_run[1] == -INFINITY ? 0.0f : m_run[1];
            const float p0a = fast_exp2(sacc[0] - m0), p0b = fast_exp2(sacc[1] - m1), p1a = fast_exp2(sacc[2] - m0), p1b = fast_exp2(sacc[3] - m1);
            l_run[0] += p0a + p1a;
            l_run[1] += p0b + p1b;
            pb[0] = movmatrix_trans(pack_bf16(p0a, p0b));
            pb[1] = movmatrix_trans(pack_bf16(p1a, p1b));
        }
#pragma unroll
        for (int dm = 0; dm < 4; dm++) {
            uint32_t va[4];
            ldmatrix_x4_trans(va, (kbase + PAGE_BYTES / 2 + v_off) ^ (uint32_t(dm) << 5));
            mma16816(oacc[dm], va, pb[0], pb[1]);
        }
        __syncwarp();
        if (!fresh) pg += KG;
    }
    if (have && c.lane == 0) bar_arrive(smem_u32(&sm.empty[ring_stage(c.items + have - 1)]), 1);
    c.items += have;
    // The key groups meet: first their maxima, then what each has, scaled to the largest.
    const uint32_t cc = 2 * c.t;
#pragma unroll
    for (int e = 0; e < 2; e++)
        if (c.g == 0) sm.mw[cc + e][c.warp] = kg < KG ? m_run[e] : -INFINITY;
    res_sync();  // (the buffers' readers before are done, too)
    constexpr uint32_t OS = HD + 4;
    static_assert(RES_WARPS * 8 * OS * 4 <= RES_RED * 4 + RES_X, "the warps' sums fit");
    if (kg < KG) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
            float mm = -INFINITY;  // over the warps of this n-tile: cw, cw + NT, ...; every eighth of them a lane
#pragma unroll 1
            for (uint32_t w = cw + c.g * NT; w < KG * NT; w += 8 * NT) mm = fmaxf(mm, sm.mw[cc + e][w]);
            float l = l_run[e];
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
                l += __shfl_xor_sync(0xffffffffu, l, o);
            }
            const float wt = m_run[e] == -INFINITY ? 0.0f : fast_exp2(m_run[e] - mm);
            float* to = red + (c.warp * 8 + cc + e) * OS + c.g;
#pragma unroll
            for (int dm = 0; dm < 4; dm++) {
                to[16 * dm] = oacc[dm][e] * wt;
                to[16 * dm + 8] = oacc[dm][e + 2] * wt;
            }
            if (c.g == 0) {
                to[HD] = mm;
                to[HD + 1] = l * wt;
            }
        }
    }
    res_sync();
    float* part = reinterpret_cast<float*>(ar + a.ar.part);
#pragma unroll 1
    for (uint32_t idx = threadIdx.x; idx < x.n_cols * OS; idx += RES_THREADS) {  // 64 sums, the maximum, l's sum (and two words of nothing)
        const uint32_t p = idx / OS, d = idx % OS, tok = token_of(p);
        const float* from = red + ((p / 8) * 8 + p % 8) * OS + d;
        float sum = 0.0f;
#pragma unroll 4
        for (uint32_t w = 0; w < KG; w++) sum += from[w * NT * 8 * OS];
        if (d == HD) sum = from[0];
        if (d < HD + 2) st_word(part + (((t0 + tok) * a.n_heads + x.kvh * a.heads_per_kv + p - tok * a.heads_per_kv) * a.max_splits + x.split) * ATTN_PART + (d < HD ? 4 + d : d - HD), sum);
    }
    res_sync();  // (before the buffers' next use)
}

// The splits of every (token, head) merged: a block each, half a warp a split, four dims a lane.
template <bool INT8>
__device__ __forceinline__ void merge_phase(const DecodeArgs& a, DecodeSmem& sm, float* red, Ctx& c, uint32_t layer) {
    uint8_t* ar = layer_arena(a, layer);
#pragma unroll 1
    for (uint32_t i = blockIdx.x; i < a.n * a.n_heads; i += gridDim.x) {
        uint32_t tok = 0;
#pragma unroll 1
        for (uint32_t j = i; j >= a.n_heads; j -= a.n_heads) tok++;
        const uint32_t tile = sm.tok_tile[tok], S = a.unit0[tile + 1] - a.unit0[tile];
        const float* pp = reinterpret_cast<const float*>(ar + a.ar.part) + i * a.max_splits * ATTN_PART;
        float m = -INFINITY, l = 0.0f, o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        auto add = [&](float ms, float ls, const float (&x)[4]) {
            const float m_new = fmaxf(m, ms), m0 = m_new == -INFINITY ? 0.0f : m_new;
            const float corr = fast_exp2(m - m0), w = fast_exp2(ms - m0);
            m = m_new;
            l = l * corr + w * ls;
#pragma unroll
            for (int j = 0; j < 4; j++) o[j] = o[j] * corr + w * x[j];
        };
#pragma unroll 1
        for (uint32_t s0 = 0; s0 < S; s0 += 2 * RES_WARPS) {
            const uint32_t s = s0 + 2 * c.warp + c.lane / 16;
            uint2 ml = make_uint2(0xff800000u, 0u);
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (s < S) {
                Patience p = patience(a, sm);
                do {
                    ml = ld_word2(pp + s * ATTN_PART);
                    v = ld_word4(pp + s * ATTN_PART + 4 + 4 * (c.lane % 16));
                } while (!(there(ml) && there(v)) && !p.over());
            }
            const float x[4] = {__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)};
            add(__uint_as_float(ml.x), __uint_as_float(ml.y), x);
        }
        __syncwarp();
        {  // the two halves, then the warps through shared memory
            float x[4];
#pragma unroll
            for (int j = 0; j < 4; j++) x[j] = __shfl_xor_sync(0xffffffffu, o[j], 16);
            add(__shfl_xor_sync(0xffffffffu, m, 16), __shfl_xor_sync(0xffffffffu, l, 16), x);
        }
        res_sync();  // (the buffers' readers before are done)
        float* to = red + c.warp * 68;
        if (c.lane < 16) *reinterpret_cast<float4*>(to + 4 * c.lane) = make_float4(o[0], o[1], o[2], o[3]);
        if (c.lane == 0) *reinterpret_cast<float2*>(to + 64) = make_float2(m, l);
        res_sync();
        if (c.warp == 0) {
            const float2 ml = c.lane < RES_WARPS ? *reinterpret_cast<const float2*>(red + c.lane * 68 + 64) : make_float2(-INFINITY, 0.0f);
            const float w = fast_exp2(ml.x - warp_max(ml.x)), ll = warp_sum(w * ml.y);
            float x0 = 0.0f, x1 = 0.0f;
#pragma unroll 4
            for (uint32_t j = 0; j < RES_WARPS; j++) {
                const float2 v = *reinterpret_cast<const float2*>(red + j * 68 + 2 * c.lane);
                const float wj = __shfl_sync(0xffffffffu, w, j);
                x0 += wj * v.x;
                x1 += wj * v.y;
            }
            publish<INT8>(ar + a.ar.at, a.ar.half_o, i * HD + 2 * c.lane, pack_bf16(x0 / ll, x1 / ll), scale_of(PH_O), 1, c.lane % 4 == 0);
        }
    }
}

// LIMITE: the reference's own architecture, whose attention has kernels of its own: a launch is a qkv phase, or o, gate_up, down and,
// where nothing comes in between, the next layer's qkv; scales and residual lambdas as MatArgs has them.
template <bool INT8, bool LIMITE>
__global__ void __launch_bounds__(RES_THREADS + RES_ASKERS, 1) decode_kernel(const __grid_constant__ DecodeArgs a, const __grid_constant__ AttnMaps maps) {
    extern __shared__ uint8_t decode_smem_raw[];
    uint8_t* stages = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(decode_smem_raw) + 1023) & ~uintptr_t(1023));
    float* red = reinterpret_cast<float*>(stages + RES_STAGES * RES_STAGE);
    uint4* xs = reinterpret_cast<uint4*>(red + RES_RED);
    __shared__ DecodeSmem sm;
    const uint32_t tid = threadIdx.x;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid == 0) {
        for (uint32_t i = 0; i < RES_STAGES; i++) {
            bar_init(smem_u32(&sm.full[i]), 1);
            bar_init(smem_u32(&sm.empty[i]), RES_WARPS);
        }
        sm.dead = 0u;
        sm.asked = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (tid < 16) sm.mx[tid / 8][tid % 8] = 0u;
    if (tid < a.n_tiles) {
        const uint32_t t0 = a.tiles[2 * tid], T = a.tiles[2 * tid + 1];
        sm.t0[tid] = t0;
        sm.rows[tid] = T;
        sm.slot[tid] = a.meta[2 * t0];
        sm.p0[tid] = a.meta[2 * t0 + 1];
        for (uint32_t i = 0; i < T; i++) {
            sm.tok_tile[t0 + i] = tid;
            sm.tok_row[t0 + i] = i;
            sm.vis[t0 + i] = a.vis[t0 + i];
        }
    }
    __syncthreads();
    if (tid < DECODE_UNITS && tid * gridDim.x + blockIdx.x < a.n_units) sm.unit[tid] = unit_of(a, sm, tid * gridDim.x + blockIdx.x);
    __syncthreads();
    if (tid >= RES_THREADS) {
        // (640 threads launch with 96 registers each: 61 440; 128 of 32 and 512 of 112 are as many.)
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (tid >= RES_THREADS + 32) return;
        uint32_t n = 0;
        for (uint32_t u = 0; u * gridDim.x + blockIdx.x < a.n_units && n < LISTED; u++) {
            const Unit& x = sm.unit[u];
            for (uint32_t i = tid - RES_THREADS; i < min(x.pages, LISTED - n); i += 32) sm.ids[n + i] = a.page_table[size_t(sm.slot[x.tile]) * a.kv.max_pages + x.page0 + i];
            n += (x.pages + ITEM_PAGES - 1) / ITEM_PAGES * ITEM_PAGES;
        }
        __syncwarp();
        ask(a, maps, sm, smem_u32(stages));
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    // The set of words that the next launch will use.
    for (size_t i = (size_t(blockIdx.x) * RES_THREADS + tid) * 16; i < a.clear_bytes; i += size_t(gridDim.x) * RES_THREADS * 16)
        *reinterpret_cast<uint4*>(a.clear + i) = make_uint4(ABSENT, ABSENT, ABSENT, ABSENT);
    Ctx c;
    c.warp = tid / 32;
    c.lane = tid % 32;
    c.g = c.lane >> 2;
    c.t = c.lane & 3;
    c.items = 0;
    c.turn = 0;
    if (!LIMITE && tid < 256) {
        const uint32_t tok = tid / 32, pair = tid % 32;
        if (tok < a.n) {
            sm.cs[tok][pair] = reinterpret_cast<const float2*>(a.rope)[size_t(a.meta[2 * tok + 1]) * (HD / 2) + pair];
            if (pair == 0) {
                const uint32_t tile = sm.tok_tile[tok];
                sm.kvrow[tok] = kv_row(a.kv, 0, a.page_table, sm.slot[tile], 0, sm.p0[tile] + sm.tok_row[tok]);
            }
        }
    }
    // The block's rows of the residual stream, and the first layer's input from them.
    {
        const uint32_t q = c.warp & 3u, r = c.lane & 15u, tok = 2 * q + c.lane / 16;
        uint32_t i = c.warp / 4;
#pragma unroll 1
        for (uint32_t at = blockIdx.x + i * gridDim.x; at < a.d / 16; at += 4 * gridDim.x, i += 4) {
            const float y = tok < a.n ? a.h[size_t(tok) * a.d + at * 16 + r] : 0.0f;
            sm.resid[i][tok][r] = y;
            if (LIMITE && a.s0 % PH_HEAD != PH_QKV) continue;
            tile_squares(a, reinterpret_cast<float*>(a.arena + a.ar.ss1), at, tok, r, y);
            publish<INT8>(a.arena, a.ar.half_d, tok * a.d + at * 16 + r, pack_bf16(y, __shfl_down_sync(0xffffffffu, y, 1)), 1.0f, 2, tok < a.n && r % 8 == 0);
        }
    }
    res_sync();
    uint32_t layer = a.s0 / PH_HEAD, ph = a.s0 % PH_HEAD;
#pragma unroll 1
    for (uint32_t s = a.s0; s < a.s1 + (a.n_head ? 1u : 0u); s++) {
        if (s == a.s1) ph = PH_HEAD;
        c.renew();
        if (!LIMITE && ph == PH_ATTN) {
#pragma unroll 1
            for (uint32_t u = 0; u * gridDim.x + blockIdx.x < a.n_units; u++) attention_unit(a, sm, stages, red, xs, c, layer, sm.unit[u]);
            c.renew();
            merge_phase<INT8>(a, sm, red, c, layer);
        } else {
            const uint8_t* ar = layer_arena(a, layer);
            const uint8_t* x = LIMITE && ph == PH_O ? a.attn : ar + (ph == PH_O ? a.ar.at : ph == PH_GU ? a.ar.x2 : ph == PH_DOWN ? a.ar.act : 0u);
            const uint8_t* ss = ph == PH_QKV || ph == PH_HEAD ? ar + a.ar.ss1 : ph == PH_GU ? ar + a.ar.ss2 : nullptr;
            matmul_phase<INT8, LIMITE>(a, sm, stages, red, xs, c, layer, ph, x, reinterpret_cast<const float*>(ss));
        }
        if (++ph == PH_HEAD) {
            ph = PH_QKV;
            layer++;
        }
    }
}

// ---------------------------------------------------------------- host side
constexpr size_t DECODE_SMEM = size_t(RES_STAGES) * RES_STAGE + RES_RED * 4 + RES_X + 1024;
static_assert(DECODE_SMEM + sizeof(DecodeSmem) + 256 <= 227 * 1024, "a block's shared memory");

bool decode_fits(const ModelDesc& md, bool limite, const std::vector<Layer>& layers, uint32_t sm_count) {
    if (layers.empty() || (!limite && (md.hd != HD || md.page != PAGE || md.n_heads % md.n_kv || md.n_heads / md.n_kv > 4))) return false;
    const bool int8 = layers[0].qkv.int8;
    const uint32_t wb = int8 ? 1 : 2, most = 8192, attn_w = md.n_heads * md.hd;  // (a team is at most four groups, a group's parts 2 KiB of int8 and 4 of bf16)
    if (limite && int8) return false;  // (its attention leaves no fp16 words)
    if (md.d > most || md.ffn > most || attn_w > most) return false;
    if (md.d * wb % RES_PIECE || md.ffn * wb % RES_PIECE || attn_w * wb % RES_PIECE || md.d % 16 || md.ffn % 8 || md.qkv_w() % 16) return false;
    if ((md.d / 16 + sm_count - 1) / sm_count > DECODE_RESID_TILES) return false;
    for (const Layer& l : layers)
        for (const Matrix* m : {&l.qkv, &l.o, &l.gate_up, &l.down}) {
            if (m->int8 != int8 || (int8 && m->group != m->k) || m->bias) return false;
            if (reinterpret_cast<uintptr_t>(m->w) % 16 || reinterpret_cast<uintptr_t>(m->scales) % 16) return false;
        }
    return true;
}

DecodeArena decode_arena(const ModelDesc& md, bool int8, uint32_t n, uint32_t max_splits) {
    DecodeArena a{};
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t o = at; at += (bytes + 127) / 128 * 128; return uint32_t(o); };
    auto rows = [&](uint32_t width, uint32_t& half) {  // bf16, and behind them fp16 for int8 weights
        const uint32_t o = take(size_t(n) * width * 2);
        half = uint32_t(at) - o;
        if (int8) take(size_t(n) * width * 2);
        return o;
    };
    rows(md.d, a.half_d);  // x1
    a.over = take(128);    // (the first layer's is used)
    a.ss1 = take(size_t(md.d / 16) * 8 * 4);
    a.q = take(size_t(n) * md.n_heads * HD * 2);
    a.kvn = take(size_t(n) * 2 * md.n_kv * HD * 2);
    a.part = take(size_t(n) * md.n_heads * max_splits * ATTN_PART * 4);
    a.at = rows(md.n_heads * HD, a.half_o);
    a.x2 = rows(md.d, a.half_d);
    a.ss2 = take(size_t(md.d / 16) * 8 * 4);
    a.act = rows(md.ffn, a.half_ffn);
    a.layer_bytes = uint32_t(at);
    return a;
}

// The splits of the cached keys: as many (tile, split, kv head) units as there are blocks, or the least multiple of that, in
// splits of at least 8 pages (an item of the ring). Tiles get splits by their length. The count of splits is bounded by
// n_tiles n_kv splits <= blocks for the longest tile's share, so that the partial sums fit their buffer.
void decode_split(DecodeArgs& a, const uint32_t* cached, uint32_t sm_count) {
    const uint32_t nt = a.n_tiles, nkv = a.kv.n_kv;
    uint32_t pages[8], most = 1;
    for (uint32_t i = 0; i < nt; i++) {
        pages[i] = (cached[i] + PAGE - 1) / PAGE;
        most = std::max(most, pages[i]);
    }
    const uint32_t budget = sm_count * ((nt * nkv + sm_count - 1) / sm_count), cap = decode_max_splits(nkv, sm_count);
    auto units = [&](uint32_t sp) {
        uint32_t u = 0;
        for (uint32_t i = 0; i < nt; i++) u += std::max(1u, (pages[i] + sp - 1) / sp);
        return u * nkv;
    };
    uint32_t lo = std::max(ITEM_PAGES, (most + cap - 1) / cap), hi = std::max(lo, most);
    while (lo < hi) {  // the least split whose units fit the budget
        const uint32_t mid = (lo + hi) / 2;
        if (units(mid) <= budget) hi = mid;
        else lo = mid + 1;
    }
    a.split_pages = lo;
    a.max_splits = 1;
    a.unit0[0] = 0;
    for (uint32_t i = 0; i < nt; i++) {
        const uint32_t s = std::max(1u, (pages[i] + lo - 1) / lo);
        a.max_splits = std::max(a.max_splits, s);
        a.unit0[i + 1] = a.unit0[i] + s;
    }
    for (uint32_t i = nt + 1; i < 9; i++) a.unit0[i] = a.unit0[nt];
    a.n_units = a.unit0[nt] * nkv;
    a.heads_per_kv = a.n_heads / nkv;
    a.per_kv_recip = (65536 + a.heads_per_kv - 1) / a.heads_per_kv;
}

void decode_map(DecodeMap* out, const Matrix& m) { make_tensor_map_rows(out, m.w, m.m, size_t(m.k) * (m.int8 ? 1 : 2), RES_PIECE, 16); }

void launch_decode(DecodeArgs a, const AttnMaps& maps, bool int8, uint32_t sm_count, cudaStream_t s) {
    a.wbytes = int8 ? 1 : 2;
    static PerDevice configured;
    configured.once([] {
        VLT_CUDA(cudaFuncSetAttribute(decode_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(DECODE_SMEM)));
        VLT_CUDA(cudaFuncSetAttribute(decode_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(DECODE_SMEM)));
        VLT_CUDA(cudaFuncSetAttribute(decode_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(DECODE_SMEM)));
    });
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count);
    cfg.blockDim = dim3(RES_THREADS + RES_ASKERS);
    cfg.dynamicSmemBytes = DECODE_SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (a.attn) VLT_CUDA(cudaLaunchKernelEx(&cfg, decode_kernel<false, true>, a, maps));
    else if (int8) VLT_CUDA(cudaLaunchKernelEx(&cfg, decode_kernel<true, false>, a, maps));
    else VLT_CUDA(cudaLaunchKernelEx(&cfg, decode_kernel<false, false>, a, maps));
    launch_counter().fetch_add(1, std::memory_order_relaxed);
}

}  // namespace vlt
