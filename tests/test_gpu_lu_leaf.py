"""The LU's panels (leaves of 16 columns in the registers of one CTA, or of a cluster of 8 or 16, and the swaps and updates
inside a panel of 64 columns) at the row counts where the cluster's size changes. A factorization passes through every
panel height below its order: orders 643 and 2,563 cross 256, 1,024 and 2,048 rows, 10,243 crosses 8,192 and takes the
FP64 leaf of 8 columns. The unknowns are mixed (C R, R = I + 2 S with S from one half of the unknowns to the other), so
that partial pivoting swaps rows: the diagonal is not the largest of its column. Solutions against LAPACK's within the
bound n u cond of each (u = 2^-53), the largest order by its residual."""
import dataclasses

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _system(vp, k):
    g, dm = vp.meshes.sphere_case(k)
    V = np.array([1.0, 0.3, -0.2]) / np.linalg.norm([1.0, 0.3, -0.2])
    els = vp.build_elements(g)
    A, b, _ = vp.assemble(g, dm, els, vp.source_strengths(els, V), V, opts=vp.AssemblyOptions(precision="mixed"))
    rng = np.random.default_rng(k)
    n, h = dm.nq, dm.nq // 2
    rows, cols = rng.integers(0, h, 2 * (n - h)), np.tile(np.arange(h, n), 2)
    R = sp.identity(n, format="csr") + 2.0 * sp.csr_matrix((np.ones(len(rows)), (rows, cols)), shape=(n, n))
    return dataclasses.replace(dm, C=(dm.C @ R).tocsr()), A, b


@pytest.mark.parametrize("k", [3, 4])
def test_lu_panels_against_lapack(vp, oracle, k):
    dm, A, b = _system(vp, k)
    ref = oracle.solve_galerkin(dm, A.download(), b)
    n = dm.nq + 1
    assert np.mean(ref["F"].lu[1][:n] != np.arange(n)) > 0.1  # the pivots do leave the diagonal
    for precision in ("fp64", "mixed"):
        s = vp.solve_galerkin(dm, A, b, precision=precision)
        assert np.abs(s["q"] - ref["q"]).max() <= 2 * n * U * ref["cond"] * np.abs(ref["q"]).max(), precision
        assert abs(s["cond"] / ref["cond"] - 1) < 0.05


def test_lu_panels_of_16_ctas(vp):
    dm, A, b = _system(vp, 5)
    s = {p: vp.solve_galerkin(dm, A, b, precision=p) for p in ("fp64", "mixed")}
    n, cond = dm.nq + 1, s["fp64"]["cond"]
    for p in s:
        assert s[p]["residual"] <= n * U * cond
    assert np.abs(s["fp64"]["q"] - s["mixed"]["q"]).max() <= 2 * n * U * cond * np.abs(s["fp64"]["q"]).max()
