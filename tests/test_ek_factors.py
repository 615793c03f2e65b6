"""The k-space filter as a product of 1-D factors (ek_xy and ek_value of
plane_rx.cuh), compiled for the host, against the filter in long double."""
import os
import shutil
import subprocess

import pytest

from pscf_b200.build import CSRC, nvcc

SOURCE = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include "pscf_gpu.h"
#include "plane_rx.cuh"

template <typename T> static T rest(long double v) { return sizeof(T) == 4 ? (T)(v - (long double)(T)v) : (T)0; }

// largest error in units of the last place of the exact value
template <typename T> static double worst()
{
    std::mt19937_64 g(11);
    std::uniform_real_distribution<double> u(0.0, 6.0);
    double w = 0.0;
    for (int i = 0; i < 1000000; i++) {
        long double f[3], x = 1.0L;
        for (auto &v : f) x *= v = expl(-(long double)u(g));
        pscfg::EkFactor<T> x3[3];
        for (int j = 0; j < 3; j++) x3[j] = {(T)f[j], rest<T>(f[j])};
        const T e = pscfg::ek_value<T>(pscfg::ek_xy<T>(x3[0], x3[1]), x3[2]);
        const long double ulp = ldexpl(1.0L, ilogbl(x) - (sizeof(T) == 4 ? 23 : 52));
        w = std::max(w, (double)(fabsl((long double)e - x) / ulp));
    }
    return w;
}

int main()
{
    const double f = worst<float>(), d = worst<double>();
    std::printf("float %.4f double %.4f\n", f, d);
    return f <= 0.51 && d <= 4.0 ? 0 : 1;
}
"""


@pytest.mark.skipif(not shutil.which(nvcc()) and not os.path.exists(nvcc()), reason="needs nvcc")
def test_the_product_is_rounded_once_in_fp32(tmp_path):
    """FP32: half an ulp and the remainders' own rounding (some 2^-22 of it).
    FP64: three rounded factors and two products, 2.5 ulp of the larger of two
    binades: below 4 here, where a table's exp alone allows 1."""
    src, exe = tmp_path / "ek.cu", tmp_path / "ek"
    src.write_text(SOURCE)
    subprocess.run([nvcc(), "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", CSRC, "-I", os.path.join(CSRC, "..", "..", "include"),
                    "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
