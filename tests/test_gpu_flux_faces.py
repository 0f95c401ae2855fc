"""The flux at the face of two elements, as each of them forms it in flux form: the same bits,
so that what leaves one element enters the other exactly. The surface terms B f* of the two
sides are then each other's negatives on a mesh of equal elements."""
import numpy as np
import pytest

import p2de
from p2de import abi, problems
from p2de import solver as S

from helpers import setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed-acc64"])
@pytest.mark.parametrize("N", [1, 2, 3, 4, 5])
def test_both_sides_of_a_face_form_the_same_flux(N, precision):
    # equal elements, sizes a power of two: every rxJ and syJ has the same bits
    param, md, bc, desc, U0 = setup(problems.kelvin_helmholtz, N=N, Kx=16, Ky=8, precision=precision)
    assert len(np.unique(md.geom, axis=0)) == 1
    rng = np.random.default_rng(N)
    U = np.empty_like(U0)
    rho, p = 0.1 + rng.random(U.shape[:-1]), 0.01 + rng.random(U.shape[:-1])
    u, v = 4.0 * rng.standard_normal((2, *rho.shape))
    U[..., 0], U[..., 1], U[..., 2] = rho, rho * u, rho * v
    U[..., 3] = p / (param.equation.gamma - 1.0) + 0.5 * rho * (u * u + v * v)
    g = S.Solver(param, md, desc)
    g.set_Uq(U)
    S.rhs_bang(None, g, None, p2de.TimeParam(0.0, 1e-4, 2))
    partner = np.asarray(bc.mapP).reshape(-1) - 1
    assert (partner != np.arange(partner.size)).all()  # periodic: no face is its own partner
    for field in (abi.FIELD_BF_L, abi.FIELD_BF_H):
        f = g.get_field(field).reshape(partner.size, 8)
        assert np.abs(f).max() > 0.0
        np.testing.assert_array_equal(f, -f[partner])
    g.close()
