"""Which particle a lane past the ensemble's end loads (csrc/sp_types.h, source_particle): one
that its own warp holds, whatever the tile, the particles per thread and the remainder.  Another
warp may store its particles while this one still loads."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "stochasticphysics_b200" / "csrc"
CUDA_INCLUDE = Path("/usr/local/cuda/include")

PROGRAM = r"""
#include <cstdio>
#include <cuda_runtime.h>
#include "sp_types.h"
int main() {
    long checked = 0;
    for (unsigned block : {32u, 64u, 128u, 256u})
        for (int ppt = 1; ppt <= (block >= 64 ? 2 : 1); ++ppt)
            for (unsigned long long n = 1; n <= 2 * block + 1; ++n)
                for (unsigned long long first = 0; first < n; first += block) {
                    const unsigned threads = block / ppt;
                    for (unsigned t = 0; t < threads; ++t) {
                        const unsigned warp = t & ~31u;
                        if (first + warp >= n) continue;  // the warp holds no particle: it leaves
                        for (int k = 0; k < ppt; ++k) {
                            const unsigned long long own = first + (unsigned long long)k * threads + t;
                            const unsigned long long at = sp::source_particle(first, threads, t, k, n);
                            bool held = false;
                            for (int j = 0; j < ppt; ++j) {
                                const unsigned long long lane0 = first + (unsigned long long)j * threads + warp;
                                held = held || (at >= lane0 && at < lane0 + 32);
                            }
                            if (at >= n || !held || (own < n && at != own)) {
                                std::printf("block %u ppt %d n %llu first %llu thread %u k %d: %llu\n", block, ppt, n, first, t, k, at);
                                return 1;
                            }
                            ++checked;
                        }
                    }
                }
    std::printf("%ld\n", checked);
}
"""


def test_lanes_past_the_end_load_from_their_own_warp(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists():
        pytest.skip("no g++ or no CUDA headers")
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", str(CUDA_INCLUDE), "-I", str(CSRC), "-o", str(tmp_path / "t"),
                    str(tmp_path / "t.cpp")], check=True)
    run = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
    assert int(run.stdout) > 100000
