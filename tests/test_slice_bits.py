"""The balanced digits of csrc/slice_bits.cuh on the host: they sum to the element rounded
to its row's fixed-point scale, and each lies in the range the exact FP32 accumulation
rests on."""
import os
import shutil
import subprocess

import pytest

SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "slice_bits.cuh"
using namespace hfgpu;
template <int N> int check()
{
    const int F = SliceFmt<N>::F, top = N == 6 ? 128 : 64;
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> u(1.0, 2.0);
    for (int it = 0; it < 400000; ++it) {
        const int e = (int)(g() % 200) - 100;
        double x = std::ldexp(u(g), e - 1 - (int)(g() % 75));
        if (it % 7 == 0) x = std::ldexp(1.0 - std::ldexp(1.0, -53), e);  // rounds up to 2^F
        if (it % 11 == 0) x = std::ldexp(1.0, e - F - 1);                // half a unit
        if (it % 13 == 0) x = it % 2 ? 0.0 : 4e-310;                     // zero, subnormal
        if (g() & 1) x = -x;
        uint64_t b;
        std::memcpy(&b, &x, 8);
        const uint64_t U = biased_digits<N>(b, e);
        __int128 sum = 0;
        for (int t = 0; t < N; ++t) {
            const int bias = t == 0 ? top : 64;
            const int d = (int)digit_field<N>(U, t) - bias;
            if (t == 0 ? std::abs(d) > top : (d < -64 || d > 63)) return std::printf("range N %d t %d d %d\n", N, t, d), 1;
            sum = sum * 128 + d;
        }
        // round half away from zero of |x| 2^(F - e), exactly: |x| = m 2^q
        int q;
        const __int128 m = (__int128)std::ldexp(std::frexp(std::fabs(x), &q), 53);
        const int sh = q - 53 + F - e;
        __int128 want = std::fabs(x) < 1e-307 ? 0 : sh >= 0 ? m << sh : sh < -100 ? 0 : (m + ((__int128)1 << (-sh - 1))) >> -sh;
        if (x < 0) want = -want;
        if (sum != want) return std::printf("sum N %d x %.17g e %d\n", N, x, e), 1;
    }
    return 0;
}
int main() { return check<6>() || check<9>(); }
"""


def test_balanced_digits(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    src = tmp_path / "digits.cpp"
    src.write_text(SRC)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hfsolver_gb300", "csrc")
    exe = tmp_path / "digits"
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", csrc, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
