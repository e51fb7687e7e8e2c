// The tensor maps of the GEMM's operands, made once and kept by the engine whose buffers they describe.
#pragma once
#include <cstdint>
#include <map>
#include <tuple>

namespace vlt {

void make_tensor_map_2d(void* out_map, const void* base, uint64_t inner, uint64_t rows, uint32_t box_inner, uint32_t box_rows, uint32_t elem_bytes,
                        bool swizzle128, bool swizzle64 = false);

struct TensorMap {
    alignas(64) uint8_t bytes[128];
};

// A key holds everything that a map is made from, the weights' type too: a buffer that is freed leaves its address to a later
// one, which may hold the other type. The operands are kept apart: a matrix has one map whatever the step's tokens (of which a
// server's portions have some 32 lengths), and the layers share the few buffers of tokens.
class GemmMaps {
  public:
    static constexpr uint32_t BM = 128, BK = 64;  // a weight tile's rows, a stage's columns of k

    // Weights [m][k], int8 or bf16.
    const TensorMap& weights(const void* w, uint32_t m, uint32_t k, bool int8) {
        return find(weights_, std::make_tuple(w, m, k, int8), [&](TensorMap& t) {
            if (int8) make_tensor_map_2d(t.bytes, w, k, m, BK, BM, 1, false, true);
            else make_tensor_map_2d(t.bytes, w, k, m, BK, BM, 2, true);
        });
    }
    // Tokens [n_rows][k] in blocks of n_pad (a last block's rows past the end read as zeros).
    const TensorMap& tokens(const void* xb, uint32_t k, uint32_t n_rows, uint32_t n_pad) {
        return find(tokens_, std::make_tuple(xb, k, n_rows, n_pad), [&](TensorMap& t) { make_tensor_map_2d(t.bytes, xb, k, n_rows, BK, n_pad, 2, true); });
    }

  private:
    template <typename M, typename F>
    static const TensorMap& find(M& maps, const typename M::key_type& key, F make) {
        auto it = maps.find(key);
        if (it == maps.end()) {
            TensorMap t;
            make(t);
            it = maps.emplace(key, t).first;
        }
        return it->second;
    }
    std::map<std::tuple<const void*, uint32_t, uint32_t, bool>, TensorMap> weights_;
    std::map<std::tuple<const void*, uint32_t, uint32_t, uint32_t>, TensorMap> tokens_;
};

}  // namespace vlt
