"""The FP64 LU with its trailing updates on the tensor cores (exact products of 7-bit digits, nine digits an operand)
against the same LU on cuBLAS DGEMM: both are backward stable, so their solutions and condition estimates agree to the
bound n u cond of each, u = 2^-53, and the residual of the first is within three times that of the second plus n u.
Orders 643 (the first that reach the
digits' products: 320 x 320 x 320), 945 and 1,900 (updates, triangular solves and k slices above 448)."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import sys, numpy as np
sys.path[:0] = [%r, %r]
import vortexpanel_gpu as vp
kind, m1, m2 = sys.argv[2], int(sys.argv[3]), int(sys.argv[4])
V = np.array([1.0, 0.0, 0.1]); V /= np.linalg.norm(V)
if kind == "sphere":
    g, dm = vp.meshes.sphere_case(m1); W = None; wake = None
else:
    w = vp.meshes.wing(m1, m2, aspect=6.0); g, dm = w.g, w.dm
    wake = vp.meshes.build_wake(g, dm, (1.0, 0.0, 0.0), length=1.0); W = vp.meshes.wake_rows(dm, wake.te)
els = vp.build_elements(g)
A, b, _ = vp.assemble(g, dm, els, vp.source_strengths(els, V), V, wake=wake, opts=vp.AssemblyOptions(precision="mixed"))
s = vp.solve_galerkin(dm, A, b, W=W, precision="fp64")
np.savez(sys.argv[1], q=s["q"], cond=s["cond"], residual=s["residual"])
""" % (os.path.join(ROOT, "vortexpanel.jl_gb300"), ROOT)


@pytest.mark.parametrize("kind,a,b", [("sphere", 3, 0), ("wing", 30, 16), ("wing", 44, 22)])
def test_fp64_lu_on_tensor_cores(vp, tmp_path, kind, a, b):
    out = {}
    for flag in ("1", "0"):
        path = str(tmp_path / f"s{flag}.npz")
        subprocess.run([sys.executable, "-c", CODE, path, kind, str(a), str(b)], check=True,
                       env=dict(os.environ, VP_LU_TENSOR_CORES=flag), timeout=600)
        out[flag] = dict(np.load(path))
    t, c = out["1"], out["0"]
    n, u = len(t["q"]), 2.0 ** -53
    assert abs(t["cond"] / c["cond"] - 1) < n * u * float(c["cond"])
    assert np.abs(t["q"] - c["q"]).max() <= 2 * n * u * float(c["cond"]) * np.abs(c["q"]).max()
    assert float(t["residual"]) <= 3 * float(c["residual"]) + n * u
