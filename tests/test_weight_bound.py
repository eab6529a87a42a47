"""The bound that stops weight-ordered SSSP pulls (sssp_wo_limit), compiled for
the host and compared with 64-bit arithmetic: a weight is left out only where
its sum could not lower the destination, and never on an unreached one, whose
sums past 32 bits have to be noticed."""
import os
import subprocess

from wedge_gb300 import build as B

SOURCE = r"""
#include <cstdio>
#include "engine.cuh"
#include "pull.cuh"
int main()
{
    const unsigned long long top = 0xFFFFFFFFull;
    const unsigned long long near[] = {0, 1, 2, 255, 256, 257, 1ull << 31, top - 512, top - 257, top - 256, top - 255, top - 2, top - 1};
    for (unsigned long long fmin : near)
        for (unsigned long long off = 0; off <= 600; ++off)
            for (int side = 0; side < 2; ++side) {
                const unsigned long long dist = side ? top - off : fmin + off;
                if (dist > top)
                    continue;
                for (unsigned long long w = 0; w < 256; ++w) {
                    const bool read = w < wedge::sssp_wo_limit((uint32_t)dist, (uint32_t)fmin);
                    const bool needed = dist == top || fmin + w < dist;
                    if (read != needed) {
                        printf("dist %llu fmin %llu weight %llu: read %d\n", dist, fmin, w, (int)read);
                        return 1;
                    }
                }
            }
    return 0;
}
"""


def test_bound_against_wide_sums(tmp_path):
    src, exe = tmp_path / "bound.cu", tmp_path / "bound"
    src.write_text(SOURCE)
    r = subprocess.run([B.NVCC, "-std=c++17", "-I" + B.INCLUDE, "-I" + B.CSRC, "-o", str(exe), str(src)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, env=dict(os.environ))
    assert r.returncode == 0, r.stdout
