"""The quotient and the root by residual correction (octopus.jl_b200/csrc/residual.h) against the division and the square
root, on the CPU: the header is compiled with the host compiler, whose division, square root and fused multiply-add round
as IEEE 754 says, as the device's do.  Random operands over all exponents with the reciprocal up to three units off, as
its callers' are: one unit from the exact operation where the residual cannot underflow, seven below (the product alone);
and zeros, infinities, NaN, subnormals and the largest numbers in every combination but a subnormal divisor, with the
reciprocal the division gives: the same, but for a zero's sign."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER_DIR = os.path.join(ROOT, "octopus.jl_b200", "csrc")

DRIVER = r"""
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include "residual.h"

static int64_t bits(double v) { int64_t b; std::memcpy(&b, &v, 8); return b < 0 ? INT64_MIN - b : b; }
static double value(uint64_t b) { double v; std::memcpy(&v, &b, 8); return v; }

int main() {
    std::mt19937_64 rng(7);
    for (int t = 0; t < 4000000; ++t) {
        const double x = value(rng()), d = value(rng());
        if (!std::isfinite(x) || !std::isfinite(d) || std::fpclassify(d) != FP_NORMAL) continue;
        const double want = x / d;
        double rd = 1.0 / d;
        const int off = (int)(rng() % 7) - 3;
        for (int k = 0; k < (off < 0 ? -off : off); ++k) rd = std::nextafter(rd, off < 0 ? -INFINITY : INFINITY);
        const double got = octo::quotient(x, d, rd);
        if (std::isinf(want) && std::isinf(got) && (want > 0) == (got > 0)) continue;
        const int64_t away = bits(got) - bits(want), limit = std::fabs(x) >= 0x1p-960 && std::fabs(want) >= 0x1p-1021 ? 1 : 7;
        if (away > limit || away < -limit) {
            std::printf("%a / %a (%d off): %a, division %a\n", x, d, off, got, want);
            return 1;
        }
    }
    // sizes that a kernel meets, the reciprocal as the division gives it: always the division's result
    for (int t = 0; t < 4000000; ++t) {
        std::uniform_real_distribution<double> u(-1.0, 1.0);
        const double x = std::ldexp(u(rng), (int)(rng() % 200) - 100), d = std::ldexp(u(rng), (int)(rng() % 200) - 100);
        if (d == 0.0) continue;
        if (octo::quotient(x, d, 1.0 / d) != x / d || octo::quotient_in_range(x, d, 1.0 / d) != x / d) {
            std::printf("%a / %a: %a\n", x, d, octo::quotient(x, d, 1.0 / d));
            return 1;
        }
    }
    const double top = std::numeric_limits<double>::max(), low = std::numeric_limits<double>::min(),
                 sub = std::numeric_limits<double>::denorm_min();
    const double odd[] = {0.0, 1.0, 3.0, 0.5, 1e308, top, low, 7 * low, sub, 5 * sub, 1e-310, INFINITY, NAN, 1e153, 1e-153};
    for (double x : odd)
        for (double d : odd)
            for (int s = 0; s < 4; ++s) {
                if (std::fpclassify(d) == FP_SUBNORMAL) continue;
                const double a = s & 1 ? -x : x, b = s & 2 ? -d : d, want = a / b, got = octo::quotient(a, b, 1.0 / b);
                if (std::isnan(want) ? !std::isnan(got) : !(got == want || std::llabs(bits(got) - bits(want)) <= 1)) {
                    std::printf("%a / %a: %a, division %a\n", a, b, got, want);
                    return 1;
                }
            }
    for (int t = 0; t < 4000000; ++t) {
        const double v = std::fabs(value(rng()));
        if (std::fpclassify(v) != FP_NORMAL) continue;
        const double want = std::sqrt(v);
        double rs = 1.0 / want;
        const int off = (int)(rng() % 7) - 3;
        for (int k = 0; k < (off < 0 ? -off : off); ++k) rs = std::nextafter(rs, off < 0 ? -INFINITY : INFINITY);
        const double got = octo::root(v, rs);
        const int64_t away = bits(got) - bits(want), limit = v >= 0x1p-960 ? 1 : 7;
        if (away > limit || away < -limit) {
            std::printf("root of %a (%d off): %a, sqrt %a\n", v, off, got, want);
            return 1;
        }
    }
    std::puts("ok");
    return 0;
}
"""


def test_quotient_and_root_against_the_exact_operations(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "residual.cpp", tmp_path / "residual"
    src.write_text(DRIVER.replace("#include <cstdint>", "#include <cmath>\n#include <cstdint>\n#include <cstdlib>"))
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", HEADER_DIR, "-o", str(exe), str(src)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stdout
