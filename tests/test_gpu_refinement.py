"""Refined solves (mixed precision) whose numbers are not finite, below and above the number of right hand sides from
which the residual is one product on the tensor cores (24, order 1,024). A finite right hand side beyond FP32's range
overflows in the FP32 solve: refused, as no refinement brings it back (FP64 solves it). A right hand side that is not
finite itself gives a solution that is not, as in FP64, and leaves the other columns' solutions as they are without it:
within the bound n u cond of two solutions of one system, u = 2^-53."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.fixture(scope="module")
def sphere(vp):
    g, dm = vp.meshes.sphere_case(4)
    V = np.array([1.0, 0.3, -0.2]) / np.linalg.norm([1.0, 0.3, -0.2])
    els = vp.build_elements(g)
    A, b, _ = vp.assemble(g, dm, els, vp.source_strengths(els, V), V, opts=vp.AssemblyOptions(precision="mixed"))
    F = {p: vp.factorize_galerkin(dm, A, precision=p) for p in ("mixed", "fp64")}
    return dm, b, F


@pytest.mark.parametrize("nrhs", [1, 3, 32])
def test_overflow_of_fp32_is_refused(vp, sphere, nrhs):
    dm, b, F = sphere
    B = np.outer(b, np.linspace(1.0, 2.0, nrhs))
    B[:, nrhs // 2] *= 1e60
    with pytest.raises(vp._lib.VPError) as e:
        vp.solve_galerkin(F["mixed"], B)
    assert e.value.code == vp._lib.VP_ERR_NOCONV
    assert np.isfinite(vp.solve_galerkin(F["fp64"], B)["q"]).all()


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("nrhs", [3, 32])
def test_a_column_that_is_not_finite_stays_alone(vp, sphere, nrhs, value):
    dm, b, F = sphere
    B = np.outer(b, np.linspace(1.0, 2.0, nrhs))
    k = nrhs // 2
    C = B.copy()
    C[len(b) // 3, k] = value
    rest = np.arange(nrhs) != k
    ref = vp.solve_galerkin(F["mixed"], B)["q"]
    q = vp.solve_galerkin(F["mixed"], C)["q"]
    assert not np.isfinite(q[:, k]).all()
    assert np.abs(q[:, rest] - ref[:, rest]).max() <= 2 * dm.nq * U * F["mixed"].cond * np.abs(ref).max()
