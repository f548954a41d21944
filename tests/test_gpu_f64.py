"""The FP64 functions of the pair integrals (vp_f64.cuh) as the device computes them, against the library's in long
double, within the bounds that the header states and the host's test uses: 2 ulp for the reciprocal, the square root and
its reciprocal, 2^-52 max(1, |log x|) for the logarithm, 2 ulp of the angle for atan2. Arguments outside the normal range
give CUDA's values (4 ulp of each other for atan2, 2 for each side)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    from vortexpanel_gpu import _build
    exe = str(tmp_path_factory.mktemp("f64") / "check")
    subprocess.run([_build.nvcc(), *_build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-I", _build.CSRC,
                    "-o", exe, os.path.join(HERE, "f64_device_check.cu")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout
    return {k: float(v) for k, v in (ln.split() for ln in out.splitlines())}


@pytest.mark.parametrize("name,bound", [("rcp", 2.0), ("rsqrt", 2.0), ("sqrt", 2.0), ("sqrt_inv", 2.0), ("log", 1.0),
                                        ("log_half", 1.0), ("atan2", 1.0), ("special", 0.0)])
def test_errors(errors, name, bound):
    assert errors[name] <= bound, errors
