"""div_in_double (csrc/exact_math.cuh), compiled for the host, against IEEE
single-precision division: numerators of every exponent, subnormal ones and
subnormal quotients among them, and pairs whose quotient lies next to a rounding
midpoint of single precision."""
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
    std::mt19937_64 rng(7);
    long bad = 0, sub = 0, near = 0;
    auto check = [&](float p, float g) {
        if (p == 0.0f || !rcp_in_range(g)) return;
        const float q = p / g;
        if (std::isinf(q)) return;
        sub += fabsf(q) < 0x1p-126f;
        bad += bits(div_in_double(p, g, 1.0f / g)) != bits(q);
    };
    for (long i = 0; i < n; i++) {
        const float g = ldexpf(1.0f + (float)(rng() & 0x7fffff) * 0x1p-23f, (int)(rng() % 64) - 40);
        uint32_t u = (uint32_t)rng();                      // any exponent
        if ((u & 0x7f800000u) == 0x7f800000u) u &= 0x3fffffffu;
        if (i & 1) u = (u & 0x807fffffu) | ((uint32_t)(rng() % 40) << 23);  // below 2^-87, subnormal too
        float p;
        memcpy(&p, &u, 4);
        check(p, g);
        // q0 + half a unit of the last place of a quotient, times g, rounded both ways
        const float q0 = ldexpf(1.0f + (float)(rng() & 0x7fffff) * 0x1p-23f, -(int)(rng() % 149));
        const double mid = (double)q0 + 0.5 * ((double)nextafterf(q0, 2.0f) - (double)q0);
        for (float x : {(float)(mid * g), nextafterf((float)(mid * g), 0.0f), nextafterf((float)(mid * g), 1e30f)}) {
            near++;
            check(x, g);
        }
    }
    printf("%ld %ld %ld\n", bad, sub, near);
    return 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_equals_ieee_division(tmp_path):
    src, exe = tmp_path / "div.cpp", tmp_path / "div"
    src.write_text(PROGRAM)
    cuda_inc = os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I", os.path.join(PKG, "csrc"),
                           "-I", cuda_inc, str(src), "-o", str(exe), "-lm"])
    out = subprocess.run([str(exe), "2000000"], capture_output=True, text=True, check=True)
    bad, sub, near = map(int, out.stdout.split())
    assert sub > 100000 and near > 1000000
    assert bad == 0
