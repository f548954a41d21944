"""The non-far tiers' blocks and their adding to A, where the path depends on sizes: test triangles whose list of
non-far sources exceeds what the adding kernel stages (2,048), lists shorter than and around a chunk of 32 pairs, and
closed bodies without a wake next to wings with filaments."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(vp, oracle, g, dm, V, opts, tol, wake=None):
    els = vp.build_elements(g)
    sig = vp.source_strengths(els, V)
    A, b, st = vp.assemble(g, dm, els, sig, V, opts=opts, wake=wake)
    Ao, bo, so = oracle.assemble(g, dm, sig, V, wake=wake, far_ratio=opts.far_ratio)
    assert st["pairs"] == so["pairs"] and st["points"] == so["points"]
    scale = np.abs(Ao).max(axis=1, keepdims=True)
    assert (np.abs(A.download() - Ao) / scale).max() < tol
    assert np.abs(b - bo).max() < tol * np.abs(bo).max()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 5e-5)])
def test_long_lists(vp, oracle, precision, tol):
    # every pair non-far: 2,352 sources per test triangle. The bars are the assembly's own (FP64 1e-10 and mixed 5e-5 of
    # a row's largest entry), which no count of pairs enters
    g, dm = vp.meshes.ellipsoid_case(14)
    V = np.array([1.0, 0.2, -0.1])
    _check(vp, oracle, g, dm, V, vp.AssemblyOptions(precision=precision, far_ratio=1e3), tol)


@pytest.mark.parametrize("far_ratio", [0.6, 1.5, 3.0])
@pytest.mark.parametrize("nc,ns", [(3, 3), (9, 5)])
def test_short_lists(vp, oracle, nc, ns, far_ratio):
    w = vp.meshes.wing(nc, ns, aspect=4.0)
    wake = vp.meshes.build_wake(w.g, w.dm, (1.0, 0.0, 0.0), length=1.0)
    _check(vp, oracle, w.g, w.dm, np.array([1.0, 0.0, 0.1]), vp.AssemblyOptions(far_ratio=far_ratio), 1e-10, wake=wake)
