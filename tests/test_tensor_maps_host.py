"""The GEMM's tensor maps on the host: what is made for an operand, with a stand-in for the driver's encoder that writes its
arguments into the map. A map kept for another operand would have the kernel read past its tiles, so nothing here runs it."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "silicon-violetto_b200" / "csrc"
STUB = r"""
#include <cassert>
#include <cstring>
#include "tensor_maps.h"
static int made = 0;
struct Asked { const void* base; uint64_t inner, rows; uint32_t box_inner, box_rows, elem; bool s128, s64; };
void vlt::make_tensor_map_2d(void* out, const void* base, uint64_t inner, uint64_t rows, uint32_t bi, uint32_t br, uint32_t elem, bool s128, bool s64) {
    made++;
    const Asked a{base, inner, rows, bi, br, elem, s128, s64};
    static_assert(sizeof(a) <= 128);
    std::memcpy(out, &a, sizeof a);
}
static Asked asked(const uint8_t* m) { Asked a; std::memcpy(&a, m, sizeof a); return a; }
int main() {
    char buf[64];
    const void *w = buf, *x = buf + 16;
    vlt::GemmMaps maps;
"""


def run(tmp_path, body):
    src, exe = tmp_path / "maps.cc", tmp_path / "maps"
    src.write_text(STUB + body + "\n}\n")
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True)


@pytest.mark.parametrize("first", ["true", "false"])
def test_weights_of_the_other_type_at_the_same_address_get_a_map_of_their_own(tmp_path, first):
    run(tmp_path, f"""
    const bool first = {first};
    for (int round = 0; round < 2; round++)
        for (const bool int8 : {{first, !first}}) {{
            const Asked a = asked(maps.weights(w, 256, 512, int8).bytes), b = asked(maps.tokens(x, 512, 48, 48).bytes);
            assert(a.base == w && a.inner == 512 && a.rows == 256 && a.box_inner == 64 && a.box_rows == 128);
            assert(a.elem == (int8 ? 1u : 2u) && a.s128 == !int8 && a.s64 == int8);
            assert(b.base == x && b.inner == 512 && b.rows == 48 && b.box_inner == 64 && b.box_rows == 48 && b.elem == 2 && b.s128 && !b.s64);
        }}""")


def test_maps_follow_every_size_of_both_operands(tmp_path):
    run(tmp_path, """
    for (uint32_t m : {128u, 256u})
        for (uint32_t k : {64u, 512u})
            for (uint32_t rows : {16u, 272u, 288u})
                for (uint32_t pad : {16u, 144u}) {
                    const Asked a = asked(maps.weights(w, m, k, true).bytes), b = asked(maps.tokens(x, k, rows, pad).bytes);
                    assert(a.rows == m && a.inner == k && b.inner == k && b.rows == rows && b.box_rows == pad);
                }""")


def test_a_step_of_another_length_makes_one_map_for_each_buffer_of_tokens_and_none_for_the_weights(tmp_path):
    run(tmp_path, """
    for (uint32_t n = 16; n <= 512; n += 16)
        for (int layer = 0; layer < 16; layer++) {
            maps.weights(buf + layer, 256, 512, true);
            maps.tokens(x, 512, n, n <= 256 ? n : (n / 2 + 15) / 16 * 16);
        }
    assert(made == 16 + 32);""")
