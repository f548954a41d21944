"""The FP64 self pairs, a CTA a test triangle: A and b of meshes whose self pairs weigh most (an icosahedron of 20 triangles,
an 80- and a 320-triangle sphere) and of a small wing with a wake, against the oracle; the counts of self pairs and their
points; and a batch of the same systems bit for bit. Tolerance: sums of n < 5,000 products in another order, n 2^-53 <
6e-13 of the largest entry, 1e-11 with the functions' own rounding, as the other assembly tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
V = np.array([0.9, 0.2, 0.3])


def _case(vp, name):
    if name.startswith("sphere"):
        g, dm = vp.meshes.sphere_case(int(name[-1]))
        return g, dm, None
    w = vp.meshes.wing(5, 4, aspect=4.0)
    return w.g, w.dm, vp.meshes.build_wake(w.g, w.dm, (1.0, 0.0, 0.0), length=1.0)


@pytest.mark.parametrize("test", ["hat", "onering", "dual"])
def test_self_pairs(vp, oracle, test):
    opts = vp.AssemblyOptions(test=test)
    cases = []
    for name in ("sphere0", "sphere1", "sphere2", "wing"):
        g, dm, wake = _case(vp, name)
        els = vp.build_elements(g)
        cases.append((g, dm, els, vp.source_strengths(els, V), wake))
    batch = vp.assemble_batch([(g, dm, sig, V, wake) for g, dm, _, sig, wake in cases], opts)
    for (g, dm, els, sig, wake), (A1, b1, st1) in zip(cases, batch):
        A, b, st = vp.assemble(g, dm, els, sig, V, opts, wake=wake)
        Ao, bo, so = oracle.assemble(g, dm, sig, V, wake=wake, test=test)
        got = A.download()
        assert np.abs(got - Ao).max() < 1e-11 * np.abs(Ao).max()
        assert np.abs(b - bo).max() < 1e-11 * max(np.abs(bo).max(), np.abs(Ao).max())
        assert st["pairs"]["self"] == g.ntri and st["pairs"] == st1["pairs"] and st["points"] == st1["points"]
        assert np.array_equal(got, A1.download()) and np.array_equal(b, b1)
