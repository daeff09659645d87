"""The step kernels' double-precision sines, reciprocals and quotients (csrc/sp_fp64.cuh) on the
device, beside CUDA's own results and 64-bit-mantissa arithmetic.

Bounds.  Reciprocal: the exact one rounded once, 2^-23 ulp apart at most, plus the 2^-11 ulp of
the wide arithmetic: 0.501 ulp.  Quotient: the correctly rounded one, which is what CUDA's
division returns.  Sine and cosine: no less accurate than CUDA's sincos over a step's angles; the
root mean square error of 2^19 samples is known to 0.2 %, so five times that, 1.01."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parents[1] / "stochasticphysics_b200" / "csrc"
N = 1 << 19

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "sp_fp64.cuh"
__global__ void rows(const double* x, const double* a, double* o, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s, c;
    sincos(x[i], &s, &c);
    const sp::SinCosD t = sp::sincos_reduced(x[i]);
    const double y = sp::rcp_normal(x[i]);
    const double r[8] = {s, c, t.s, t.c, 1.0 / x[i], y, a[i] / x[i], sp::quotient(a[i], x[i], y)};
    for (int k = 0; k < 8; ++k) o[k * n + i] = r[k];
}
int main(int, char** argv) {
    const int n = 1 << 19;
    std::vector<double> in(2 * n), out(8 * n);
    FILE* f = fopen(argv[1], "rb");
    if (!f || fread(in.data(), 8, in.size(), f) != in.size()) return 1;
    fclose(f);
    double *x, *o;
    if (cudaMalloc(&x, in.size() * 8) || cudaMalloc(&o, out.size() * 8)) return 2;
    if (cudaMemcpy(x, in.data(), in.size() * 8, cudaMemcpyHostToDevice)) return 3;
    rows<<<n / 256, 256>>>(x, x + n, o, n);
    if (cudaGetLastError() || cudaMemcpy(out.data(), o, out.size() * 8, cudaMemcpyDeviceToHost)) return 4;
    f = fopen(argv[2], "wb");
    return fwrite(out.data(), 8, out.size(), f) != out.size() || fclose(f);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("fp64")
    (d / "t.cu").write_text(PROGRAM)
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC), "-o",
                    str(d / "t"), str(d / "t.cu")], check=True)
    return d


def ulp(got, want):
    exponent = np.frexp(want.astype(np.float64))[1]
    return np.abs((got.astype(np.longdouble) - want) * np.ldexp(np.longdouble(1), 53 - exponent)).astype(np.float64)


@pytest.mark.parametrize("kind", ["angles", "exponents"])
def test_against_cuda(program, kind):
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no wide long double")
    rng = np.random.default_rng(3)
    x = rng.uniform(-2 * np.pi, 2 * np.pi, N)
    if kind == "exponents":  # sines near zero, Newton pivots
        x = np.ldexp(x, rng.integers(-60, 20, N))
    a = rng.uniform(-1, 1, N) * np.ldexp(1.0, rng.integers(-40, 40, N))
    np.concatenate([x, a]).tofile(program / "in")
    subprocess.run([str(program / "t"), str(program / "in"), str(program / "out")], check=True, timeout=120)
    out = np.fromfile(program / "out").reshape(8, N)
    assert np.all(np.isfinite(out))
    wide = x.astype(np.longdouble)
    assert np.max(ulp(out[5], 1 / wide)) <= 0.501
    np.testing.assert_array_equal(out[7], out[6])
    if kind == "angles":
        for k, want in enumerate((np.sin(wide), np.cos(wide))):
            theirs, ours = (np.sqrt(np.mean(ulp(out[j], want) ** 2)) for j in (k, k + 2))
            assert ours <= 1.01 * theirs
