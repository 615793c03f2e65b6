"""div_by of plane_rx.cuh (division by a constant through its reciprocal and
one residual correction) against the exact division, compiled for the host."""
import os
import shutil
import subprocess

import pytest

from pscf_b200.build import CSRC, nvcc

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include "pscf_gpu.h"
#include "plane_rx.cuh"
using pscfg::div_by;

template <typename T> static bool same(T a, T b) { return a == b || (std::isnan(a) && std::isnan(b)); }

template <typename T> static int run(const char *name)
{
    using L = std::numeric_limits<T>;
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> m(-2.0, 2.0);
    std::uniform_int_distribution<int> e(L::min_exponent + 60, L::max_exponent - 2);
    int bad = 0;
    // the divisors of the kernels: 3, 2 N and 6 N
    const double divs[] = {3, 2, 6, 8, 30, 54, 128, 750, 2 * 64 * 64, 2 * 27 * 25, 6 * 27. * 40 * 50, 6. * 64 * 128 * 224};
    for (double dd : divs) {
        const T d = (T)dd, r = (T)(1.0 / dd);
        const T edge[] = {(T)0, (T)1, L::max(), -L::max(), L::quiet_NaN()};
        for (T x : edge) bad += !same(div_by(x, d, r), x / d);
        for (int i = 0; i < 200000; i++) {
            const T x = std::ldexp((T)m(g), e(g));
            bad += !same(div_by(x, d, r), x / d);
        }
    }
    std::printf("%s %d\n", name, bad);
    return bad;
}

int main() { return run<double>("double") + run<float>("float") ? 1 : 0; }
"""


@pytest.mark.skipif(not shutil.which(nvcc()) and not os.path.exists(nvcc()), reason="needs nvcc")
def test_div_by_is_the_division(tmp_path):
    """Bit for bit (quotients below the normal range are not drawn)."""
    src, exe = tmp_path / "div.cu", tmp_path / "div"
    src.write_text(SOURCE)
    subprocess.run([nvcc(), "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", CSRC, "-I", os.path.join(CSRC, "..", "..", "include"),
                    "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
