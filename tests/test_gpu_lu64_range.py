"""The FP64 LU over the range of FP64: a system whose matrix is a power of two of another's has the same factors and the
same solution to the power of two, bit for bit: entries down to 2^-942 here, their cancelled remainders 2^-56 below that, and
all products stay normal numbers. Order 643 has products of digits (320 x 320 x 320), order 43 has none."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [-466, -300, 250, 440])
@pytest.mark.parametrize("k", [1, 3])
def test_scaled_system(vp, k, power):
    g, dm = vp.meshes.sphere_case(k)
    V = np.array([1.0, 0.3, -0.2]) / np.linalg.norm([1.0, 0.3, -0.2])
    els = vp.build_elements(g)
    A, b, _ = vp.assemble(g, dm, els, vp.source_strengths(els, V), V)
    # C' A C of unknowns 2^power as large: M, its border and the right hand side scale by 2^(2 power) and 2^power
    scaled = dataclasses.replace(dm, C=dm.C * 2.0 ** power)
    q = vp.solve_galerkin(dm, A, b, precision="fp64")["q"]
    s = vp.solve_galerkin(scaled, A, b, precision="fp64")["q"]
    assert np.array_equal(s * 2.0 ** power, q)
