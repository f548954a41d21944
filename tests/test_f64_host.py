"""The FP64 functions of the pair integrals (vp_f64.cuh), compiled for the host, against the library's in long double: the
bounds are the ones the header states (2 ulp for the reciprocal, the reciprocal square root and the square root,
2^-52 max(1, |log x|) for the logarithm, 2 ulp of the angle for atan2), and arguments outside the normal range give
the library's values."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("f64") / "check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I/usr/local/cuda/include",
                    "-I" + os.path.join(ROOT, "vortexpanel.jl_gb300", "csrc"), "-o", exe,
                    os.path.join(HERE, "f64_check.cpp")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {k: float(v) for k, v in (ln.split() for ln in out.splitlines())}


@pytest.mark.parametrize("name,bound", [("rcp", 2.0), ("rsqrt", 2.0), ("sqrt", 2.0), ("log", 1.0), ("atan2", 1.0),
                                        ("special", 0.0)])
def test_errors(errors, name, bound):
    assert errors[name] <= bound, errors
