"""Which host arrays kernels may reach in place of a copy: those that lie whole in one pinned range,
at a float's alignment. (Kernels that follow an array out of its range would fault, so the rule is
tested on the host.)"""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = """
#include "host_array.h"
#include <cstdio>
int main() {
    alignas(16) static char m[256];
    auto in = [&](int at, size_t bytes, int start, size_t size, bool pinned = true, int device = -1) {
        return (int)vfd::kernel_reaches(m + at, bytes, vfd::HostRange{pinned, m + (device < 0 ? at : device), m + start, size});
    };
    printf("%d%d%d%d%d ", in(0, 256, 0, 256), in(64, 192, 0, 256), in(64, 0, 0, 64), in(4, 8, 0, 12), in(252, 4, 0, 256));
    // a tail, or all but the first byte, in another range or in none; before the range; behind it
    printf("%d%d%d%d%d ", in(0, 256, 0, 128), in(0, 256, 0, 255), in(0, 16, 4, 64), in(128, 4, 0, 128), in(132, 0, 0, 128));
    // pageable; mapped at another address; not aligned; a size that wraps
    printf("%d%d%d%d%d", in(0, 16, 0, 256, false), in(0, 16, 0, 256, true, 16), in(1, 16, 0, 256), in(2, 16, 0, 256),
           in(64, ~(size_t)0 - 32, 0, 256));
}
"""


def test_only_whole_aligned_pinned_arrays(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "vfd_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    assert out == "11111 00000 00000"
