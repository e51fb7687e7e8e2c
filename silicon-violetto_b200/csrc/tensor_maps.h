// The tensor maps of the GEMM's operands, made once and kept by the engine whose buffers they describe.
#pragma once
#include <cstdint>
#include <map>
#include <tuple>

namespace vlt {

void make_tensor_map_2d(void* out_map, const void* base, uint64_t inner, uint64_t rows, uint32_t box_inner, uint32_t box_rows, uint32_t elem_bytes,
                        bool swizzle128, bool swizzle64 = false);

struct GemmMapPair {
    alignas(64) uint8_t a[128];
    alignas(64) uint8_t b[128];
};

// A key holds everything that a map is made from, the weights' type too: a buffer that is freed leaves its address to a later
// one, which may hold the other type.
class GemmMaps {
  public:
    static constexpr uint32_t BM = 128, BK = 64;  // a weight tile's rows, a stage's columns of k

    // Weights [m][k], int8 or bf16, against tokens [n_rows][k] in blocks of n_pad.
    const GemmMapPair& get(const void* w, const void* xb, uint32_t m, uint32_t k, bool int8, uint32_t n_rows, uint32_t n_pad) {
        const auto key = std::make_tuple(w, xb, m, k, int8, n_rows, n_pad);
        auto it = maps_.find(key);
        if (it == maps_.end()) {
            GemmMapPair p;
            if (int8) make_tensor_map_2d(p.a, w, k, m, BK, BM, 1, false, true);
            else make_tensor_map_2d(p.a, w, k, m, BK, BM, 2, true);
            make_tensor_map_2d(p.b, xb, k, n_rows, BK, n_pad, 2, true);  // (a last block's rows past the end read as zeros)
            it = maps_.emplace(key, p).first;
        }
        return it->second;
    }

  private:
    std::map<std::tuple<const void*, const void*, uint32_t, uint32_t, bool, uint32_t, uint32_t>, GemmMapPair> maps_;
};

}  // namespace vlt
