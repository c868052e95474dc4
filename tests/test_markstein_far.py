"""Markstein's correction (csrc/exact_math.cuh), compiled for the host, for
denominators in [2^24, 2^48) and numerators zero or above 2^-76, against IEEE
division; div_in_double for the smaller numerators there."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

PROGRAM = r'''
#include "exact_math.cuh"
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
using namespace oflow;
static uint32_t bits(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
int main(int argc, char **argv) {
    const long n = atol(argv[1]);
    std::mt19937_64 rng(5);
    long bad = 0, far = 0, small = 0;
    for (long i = 0; i < n; i++) {
        const float g = ldexpf(1.0f + (float)(rng() & 0x7fffff) * 0x1p-23f, 24 + (int)(rng() % 24));
        float p = ldexpf(1.0f + (float)(rng() & 0x7fffff) * 0x1p-23f, (int)(rng() % 200) - 148);
        if (i % 3 == 0) p = (float)((double)ldexpf(1.0f + (float)(rng() & 0x7fffff) * 0x1p-23f, -(int)(rng() % 100)) *
                                    (1.0 + ldexp(1.0, -24)) * g);  // next to a midpoint times g
        if (i % 97 == 0) p = 0.0f;
        if (rng() & 1) p = -p;
        const float y = 1.0f / g, q = p / g;
        if (p == 0.0f || fabsf(p) > 0x1p-76f) {
            far++;
            bad += bits(markstein(p, g, y)) != bits(q);
        }
        if (p != 0.0f) {
            small += fabsf(p) <= 0x1p-76f;
            bad += bits(div_in_double(p, g, y)) != bits(q);
        }
    }
    printf("%ld %ld %ld\n", bad, far, small);
    return 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_equal_ieee_division(tmp_path):
    src, exe = tmp_path / "far.cpp", tmp_path / "far"
    src.write_text(PROGRAM)
    cuda_inc = os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I", os.path.join(PKG, "csrc"),
                           "-I", cuda_inc, str(src), "-o", str(exe), "-lm"])
    out = subprocess.run([str(exe), "3000000"], capture_output=True, text=True, check=True)
    bad, far, small = map(int, out.stdout.split())
    assert far > 1000000 and small > 300000
    assert bad == 0
