"""Double-precision sines, cosines, logarithm, square root and reciprocal of the step kernels
(csrc/sp_fp64.cuh), compiled for the host, against 113-bit arithmetic.

Bounds in units of the last place, from the methods.  Sine and cosine: half an ulp from the
last addition, up to half an ulp of the reduced angle, and at most half an ulp of the
polynomial terms: 1.5.  Logarithm: half an ulp from the last addition and at most a quarter
from the table interval's part: 0.75.  Square root and reciprocal: half an ulp and 2^-20 of
their residual correction: 0.51.  The host build's first approximations are single precision
(2^-24), the device's 2^-19, whose squares and cubes leave the same digits."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "stochasticphysics_b200" / "csrc"

PROGRAM = r"""
#include <quadmath.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include "sp_fp64.cuh"
using namespace sp;
typedef __float128 Q;
static const double kRows[kLogRows][3] = {SP_LOG_TABLE};
static double worst = 0;
static void see(double got, Q want) {
    int e;
    frexp((double)want, &e);
    const double u = (double)fabsq(((Q)got - want) / scalbnq(1, e - 53));
    if (!(u <= worst)) worst = u;
}
static void see_angle(double x) {
    Q s, c;
    sincosq((Q)x, &s, &c);
    const SinCosD o = sincos_reduced(x);
    see(o.s, s);
    see(o.c, c);
}
static void see_turn(uint32_t b) {
    Q s, c;
    sincosq(2 * M_PIq * ((Q)b + 0.5Q) * scalbnq(1, -32), &s, &c);
    const SinCosD o = sincos_turn(b);
    see(o.s, s);
    see(o.c, c);
}
int main(int argc, char** argv) {
    std::mt19937_64 g(7);
    auto unit = [&] { return (double)(g() >> 11) * 0x1p-53; };
    const char* what = argv[1];
    if (!strcmp(what, "angle")) {  // a step's angles, and the neighbours of every multiple of pi/4
        for (int i = 0; i < 200000; ++i) see_angle((2 * unit() - 1) * 4 * M_PI);
        for (int k = -64; k <= 64; ++k)
            for (int d = -40; d <= 40; ++d) see_angle(k * (M_PI / 4) * (1 + d * 0x1p-52));
        for (int e = -300; e < 0; ++e) see_angle(ldexp(1 + unit(), e));
    } else if (!strcmp(what, "range")) {  // up to the bound the kernels check
        for (int i = 0; i < 200000; ++i) see_angle((2 * unit() - 1) * 8192);
    } else if (!strcmp(what, "turn")) {
        for (int i = 0; i < 200000; ++i) see_turn((uint32_t)g());
        for (uint32_t k = 0; k < 16; ++k)
            for (int d = -300; d <= 300; ++d) see_turn((k << 28) + (uint32_t)d);
    } else if (!strcmp(what, "log")) {
        LogTab t;
        for (int i = 0; i < kLogRows; ++i) { t.c[i] = kRows[i][0]; t.l[i][0] = kRows[i][1]; t.l[i][1] = kRows[i][2]; }
        auto one = [&](uint32_t a) { see(log_unit(a, t), logq(((Q)a + 0.5Q) * scalbnq(1, -32))); };
        for (int i = 0; i < 300000; ++i) one((uint32_t)g());
        for (uint32_t d = 0; d < 3000; ++d) { one(d); one(0xffffffffu - d); one(0x80000000u + d); one(0x80000000u - d); one(0xc0000000u + d); one(0xc0000000u - d); }
        for (uint32_t i = 0; i < 256; ++i)  // both sides of every table interval's edge
            for (int d = -2; d <= 2; ++d) for (int s = 0; s < 20; s += 5) one(((0x80000000u + (i << 23)) >> s) + (uint32_t)d);
    } else if (!strcmp(what, "sqrt")) {
        for (int i = 0; i < 300000; ++i) { const double x = ldexp(1 + unit(), (int)(g() % 120) - 90); see(sqrt_normal(x), sqrtq((Q)x)); }
    } else if (!strcmp(what, "quotient")) {  // the correctly rounded quotient, bit for bit
        for (int i = 0; i < 300000; ++i) {
            const double b = (2 * unit() - 1) * ldexp(1, (int)(g() % 20) - 10), a = (2 * unit() - 1) * ldexp(1, (int)(g() % 80) - 70);
            if (b != 0 && quotient(a, b, rcp_normal(b)) != a / b) worst = 1e9;
        }
        if (quotient(0.0, 3.0, rcp_normal(3.0)) != 0.0) worst = 1e9;
    } else {
        for (int i = 0; i < 300000; ++i) { const double x = (2 * unit() - 1) * ldexp(1, -(int)(g() % 60)); if (x != 0) see(rcp_or_zero(x), 1 / (Q)x); }
        if (rcp_or_zero(0.0) != 0.0 || rcp_or_zero(-0.0) != 0.0) worst = 1e9;
    }
    printf("%.4f\n", worst);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("fp64")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-O2", "-std=gnu++17", "-mfma", "-ffp-contract=off", "-I", str(CSRC), "-o", str(d / "t"),
                    str(d / "t.cpp"), "-lquadmath"], check=True)
    return d / "t"


@pytest.mark.parametrize("what, bound", [("angle", 1.5), ("range", 1.5), ("turn", 1.5), ("log", 0.75), ("sqrt", 0.51),
                                         ("quotient", 0.0), ("reciprocal", 0.51)])
def test_error_in_ulp(program, what, bound):
    worst = float(subprocess.run([str(program), what], check=True, capture_output=True, text=True).stdout)
    assert worst <= bound, f"{what}: {worst} ulp"
