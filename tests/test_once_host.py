"""Set-up work done once per device (PerDevice), on the host: a set-up that fails, by a false result or an exception, is tried
again by the next call instead of counting as done."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "silicon-violetto_b200" / "csrc"
SOURCE = r"""
#include <cassert>
#include "common.h"
static int device = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }  // (a stand-in: no GPU is asked)
int main() {
    vlt::PerDevice once;
    int calls = 0;
    auto set_up = [&](bool works) { once.once([&] { calls++; return works; }); };
    set_up(false);
    set_up(false);
    assert(calls == 2);
    set_up(true);
    set_up(true);
    assert(calls == 3);
    device = 5;
    try { once.once([&] { calls++; throw vlt::Error("no"); }); } catch (const vlt::Error&) {}
    once.once([&] { calls++; });
    once.once([&] { calls++; });
    assert(calls == 5);
}
"""


def test_a_failed_set_up_is_tried_again(tmp_path):
    src, exe = tmp_path / "once.cc", tmp_path / "once"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", "-I/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True)
