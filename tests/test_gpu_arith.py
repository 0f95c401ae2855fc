"""The stage kernels' reciprocal, square root and two-point flux over the range of doubles:
elements with a constant state at rest, from 1e-100 to 1e100 in density and pressure
(exponents of both parities, mantissas next to powers of two).

Tolerances: the CFL time step is a quotient of sums of a dozen operations, held to the 1e-13
of the other parity tests against the oracle; the right-hand sides of a constant state are 0
(the oracle's entropy variables overflow at the far ends, so it is no reference there) but
for the rounding of the momentum fluxes p, held to 1e-12 of one flux's contribution
p / (h w / 2).
"""
import numpy as np
import pytest

import p2de
from p2de import abi, problems
from p2de import solver as S

from helpers import setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rho", [1.0, 1.0 + 2.0**-52, 2.0 - 2.0**-52, 0.5 + 2.0**-53, 3.0, 1e-100, 7e99])
@pytest.mark.parametrize("p", [1.0, 2.0 - 2.0**-52, 1.0 / 3.0, 1e-12, 1e100])
def test_constant_state_over_the_range(rho, p):
    from oracle.binding import Oracle

    param, md, bc, desc, U0 = setup(problems.kelvin_helmholtz, N=3, Kx=2, Ky=2)
    U = np.zeros_like(U0)
    U[..., 0] = rho
    U[..., 3] = p / 0.4
    ts = param.timestepping_param
    o = Oracle(desc)
    o.set_Uq(U)
    want = o.rhs(0.0, ts.CFL * ts.dt0, 1)
    g = S.Solver(param, md, desc)
    g.set_Uq(U)
    dt = S.rhs_bang(None, g, None, p2de.TimeParam(0.0, ts.CFL * ts.dt0, 1))
    assert abs(dt - want) <= 1e-13 * want
    flux = p / (0.5 * 0.5 / 6)  # p / (h w / 2): h = 1/2, the end node's w = 1/6
    for f in (abi.FIELD_RHSU, abi.FIELD_RHSL, abi.FIELD_RHSH):
        assert np.abs(g.get_field(f)).max() <= 1e-12 * flux, f
    g.close()
    o.close()
