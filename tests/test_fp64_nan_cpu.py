"""No routine of csrc/sp_fp64.cuh returns NaN or infinity where its ulp test looks.

The error accumulator of test_fp64_math_cpu.py, `if (!(u <= worst)) worst = u;`, takes a NaN in
and lets the next finite error replace it.  The same program is run here with one that keeps
it; a NaN planted before the samples shows the difference."""
import shutil
import subprocess

import pytest

from test_fp64_math_cpu import CSRC, PROGRAM

FORGETS = "if (!(u <= worst)) worst = u;"
KEEPS = "if (!(u < 1e9)) worst = 1e9; else if (u > worst) worst = u;"
START = "const char* what = argv[1];"
PLANT = START + " if (argc > 2) see(NAN, 1);"


@pytest.fixture(scope="module")
def programs(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    assert PROGRAM.count(FORGETS) == 1 and PROGRAM.count(START) == 1
    d = tmp_path_factory.mktemp("fp64")
    for name, rule in (("forgets", FORGETS), ("keeps", KEEPS)):
        (d / f"{name}.cpp").write_text(PROGRAM.replace(FORGETS, rule).replace(START, PLANT))
        subprocess.run([cxx, "-O2", "-std=gnu++17", "-mfma", "-ffp-contract=off", "-I", str(CSRC), "-o", str(d / name),
                        str(d / f"{name}.cpp"), "-lquadmath"], check=True)
    return d


def worst(program, *args):
    return float(subprocess.run([str(program), *args], check=True, capture_output=True, text=True).stdout)


@pytest.mark.parametrize("what, bound", [("angle", 1.5), ("range", 1.5), ("turn", 1.5), ("log", 0.75), ("sqrt", 0.51),
                                         ("quotient", 0.0), ("reciprocal", 0.51)])
def test_every_sample_is_finite_and_within_its_bound(programs, what, bound):
    assert worst(programs / "keeps", what) <= bound


def test_a_planted_nan_is_kept(programs):
    assert worst(programs / "forgets", "sqrt", "plant") <= 0.51
    assert worst(programs / "keeps", "sqrt", "plant") >= 1e9
