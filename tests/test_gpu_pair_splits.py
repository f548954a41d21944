"""FP64 self, touching and contact pairs of small meshes, whose points go to several warps a pair while there are few pairs
(parts added in order): an icosahedron of 20 triangles and an 80-triangle sphere (8 warps a pair), a 320-triangle sphere
(fewer), a small wing with contact pairs at its trailing edge and a wake, and a depth beyond the records' room (a pair
walked piece by piece). A and b against the oracle, and the counts of pairs and points equal to those of a batch of one,
which does not split. Tolerance: sums of n <= 5,000 products in another order, n 2^-53 < 6e-13, of the largest entry;
1e-11 with the functions' own rounding, as the other assembly tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(vp, name):
    if name.startswith("sphere"):
        g, dm = vp.meshes.sphere_case(int(name[-1]))
        return g, dm, None
    w = vp.meshes.wing(5, 4, aspect=4.0)
    return w.g, w.dm, vp.meshes.build_wake(w.g, w.dm, (1.0, 0.0, 0.0), length=1.0)


@pytest.mark.parametrize("name,depth", [("sphere0", 3), ("sphere1", 3), ("sphere2", 3), ("wing", 3), ("wing", 6)])
def test_split_pairs(vp, oracle, name, depth):
    g, dm, wake = _case(vp, name)
    V = np.array([0.9, 0.2, 0.3])
    els = vp.build_elements(g)
    sig = vp.source_strengths(els, V)
    opts = vp.AssemblyOptions(near_depth=depth)
    A, b, st = vp.assemble(g, dm, els, sig, V, opts, wake=wake)
    Ao, bo, _ = oracle.assemble(g, dm, sig, V, wake=wake, near_depth=depth)
    got = A.download()
    assert np.abs(got - Ao).max() < 1e-11 * np.abs(Ao).max()
    assert np.abs(b - bo).max() < 1e-11 * max(np.abs(bo).max(), np.abs(Ao).max())
    (A1, _, st1), = vp.assemble_batch([(g, dm, sig, V, wake)], opts)
    assert np.abs(got - A1.download()).max() < 1e-12 * np.abs(Ao).max()
    assert st["pairs"] == st1["pairs"] and st["points"] == st1["points"]
