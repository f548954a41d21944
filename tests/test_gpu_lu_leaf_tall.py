"""The LU leaf that keeps the panel in shared memory: above 16,384 rows, and wherever clusters of 16 CTAs are not to be had
(vp_set_lu_cluster 8: from 2,049 rows in FP64 and 8,193 in FP32, so order 2,563 passes from one leaf to the other in
FP64; 0: at every height, so orders 643 and 2,563 end in the smallest panels). Solutions against LAPACK's within the
bound n u cond of each (u = 2^-53), as for the leaf in registers; order 10,243 (leaves of 8 columns in FP64, FP32 panels
above 8,192 rows) by its residual."""
import numpy as np
import pytest
from test_gpu_lu_leaf import U, _system

pytestmark = pytest.mark.gpu


@pytest.fixture
def cluster(vp):
    ctx, lib = vp.api.default_context(), vp._lib.load()
    yield lambda n: vp._lib.check(ctx.h, lib.vp_set_lu_cluster(ctx.h, n))
    vp._lib.check(ctx.h, lib.vp_set_lu_cluster(ctx.h, 16))


@pytest.mark.parametrize("k", [3, 4])
def test_tall_leaf_against_lapack(vp, oracle, cluster, k):
    dm, A, b = _system(vp, k)
    ref = oracle.solve_galerkin(dm, A.download(), b)
    n = dm.nq + 1
    for ctas in (0, 8):
        cluster(ctas)
        for precision in ("fp64", "mixed"):
            s = vp.solve_galerkin(dm, A, b, precision=precision)
            assert np.abs(s["q"] - ref["q"]).max() <= 2 * n * U * ref["cond"] * np.abs(ref["q"]).max(), (ctas, precision)
            assert abs(s["cond"] / ref["cond"] - 1) < 0.05


def test_tall_leaf_of_8_columns(vp, cluster):
    dm, A, b = _system(vp, 5)
    cluster(8)
    for precision in ("fp64", "mixed"):
        s = vp.solve_galerkin(dm, A, b, precision=precision)
        assert s["residual"] <= (dm.nq + 1) * U * s["cond"], precision


def test_cluster_sizes(vp, cluster):
    for n in (-1, 1, 4, 32):
        with pytest.raises(ValueError):
            cluster(n)
