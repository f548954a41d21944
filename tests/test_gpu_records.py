"""The pair-parallel kernels' evaluation by records against the evaluation piece by piece: pairs whose rules outgrow a
lane's records (deep quadtrees: near_depth 9 on triangle pairs in contact) fall back to the latter, and the two must give
the oracle's entries alike; the adjoint's gradients of such pairs against central differences of the forward."""
import math

import numpy as np
import pytest
import wingcase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 5e-5)])
@pytest.mark.parametrize("near_depth,near_ratio", [(0, 1.5), (3, 1.5), (5, 3.0), (9, 2.0)])
def test_forward_against_oracle(vp, oracle, precision, tol, near_depth, near_ratio):
    # the bars are the assembly's (FP64 1e-10, mixed 5e-5 of a row's largest entry)
    w = vp.meshes.wing(6, 4, aspect=4.0)
    wake = vp.meshes.build_wake(w.g, w.dm, (1.0, 0.0, 0.0), length=0.5)
    V = np.array([1.0, 0.0, 0.1])
    els = vp.build_elements(w.g)
    sig = vp.source_strengths(els, V)
    A, b, st = vp.assemble(w.g, w.dm, els, sig, V, wake=wake,
                           opts=vp.AssemblyOptions(precision=precision, near_depth=near_depth, near_ratio=near_ratio))
    Ao, bo, so = oracle.assemble(w.g, w.dm, sig, V, wake=wake, near_depth=near_depth, near_ratio=near_ratio)
    assert st["pairs"] == so["pairs"] and st["points"] == so["points"]
    scale = np.abs(Ao).max(axis=1, keepdims=True)
    assert (np.abs(A.download() - Ao) / scale).max() < tol
    assert np.abs(b - bo).max() < tol * np.abs(bo).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_gradient_at_depth(vp, precision):
    # depth 7 puts contact and touching pairs on both sides of what the records hold; central differences of the FP64
    # forward with the same rules, step and bar of test_gpu_adjoint.py (1e-6 chord, 1e-5 of the largest entry)
    from vortexpanel_gpu.adjoint import wing_gradients

    w = wingcase.jittered(vp.meshes.wing(6, 4, aspect=4.0))
    wake = vp.meshes.build_wake(w.g, w.dm, (1.0, 0.0, 0.0), length=0.5)
    W = vp.meshes.wake_rows(w.dm, wake.te)

    def run(ww, wk, prec):
        return wing_gradients(ww, wk, W, math.radians(5.0), precision=prec,
                              opts=vp.AssemblyOptions(precision=prec, near_depth=7, near_ratio=3.0))

    out = run(w, wake, precision)
    h = 1e-6 * w.chord
    for n in (int(w.dm.wake_te.node[2]), 9):
        for c in range(3):
            J = []
            for sgn in (1, -1):
                x = w.g.x.copy()
                x[n, c] += sgn * h
                ww, wk = wingcase.moved(w, wake, x)
                J.append(run(ww, wk, "fp64"))
            for name in ("CL", "CDi"):
                g = out[f"d{name}_dx"]
                fd = (J[0][name] - J[1][name]) / (2 * h)
                assert abs(g[n, c] - fd) <= 1e-5 * np.abs(g).max(), (name, n, c, g[n, c], fd)
