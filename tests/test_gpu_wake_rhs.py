"""The free wake's right hand side by chunks of sources with the close sheets, filaments and particles by their points, over
the forms that take it different ways: test functions (the dual test's pairs go to the warp), near depths up to and beyond
the leaf codes' three levels, a far rule of more than three points, a wing with more sheets than a warp's list of 32.
Against the oracle's simulation; FP64 to 1e-9 of each record as the other free wake tests, mixed within FP32's class
(2^-24 times a few hundred near points' rounding and the system's condition: 2e-4 of each record)."""
import freewake_oracle as OF
import numpy as np
import pytest

from vortexpanel_gpu import api, freewake as fw, meshes

pytestmark = pytest.mark.gpu
V = np.array([np.cos(0.12), 0.0, np.sin(0.12)])

FORMS = [dict(), dict(test="onering"), dict(test="dual"), dict(near_depth=4), dict(near_depth=1, near_ratio=2.5),
         dict(far_points=7, near_points=6)]


@pytest.mark.parametrize("form", FORMS, ids=lambda f: "-".join(f"{k}{v}" for k, v in f.items()) or "default")
def test_wake_right_hand_side_forms(vp, oracle, form):
    w = meshes.wing(5, 7, aspect=3.0)
    dt = 0.6 * meshes.te_panel_size(w.g, w.dm)
    kw = dict(dt=dt, max_rows=6, core=0.05)
    ref = OF.FreeWakeSim(w.g, w.dm, V, OF.FreeWakeOptions(**kw), **form)
    sims = {p: fw.FreeWakeSim(w.g, w.dm, V, fw.FreeWakeOptions(**kw), capacity=64,
                              assembly=api.AssemblyOptions(precision=p, **form)) for p in ("fp64", "mixed")}
    for _ in range(9):
        b = ref.step()
        for p, tol in (("fp64", 1e-9), ("mixed", 2e-4)):
            a = sims[p].step()
            assert (a["n"], a["rows"], a["particles"]) == (b["n"], b["rows"], b["particles"])
            for k in ("F_pressure", "M_pressure", "F_kj", "mu_w"):
                assert np.abs(a[k] - b[k]).max() < tol * max(np.abs(b[k]).max(), 1e-3), (p, a["n"], k)
    assert b["particles"] > 0
