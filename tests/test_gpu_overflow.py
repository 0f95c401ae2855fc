"""Subcell fluxes that overflow: a limited flux f_L + l (f_H - f_L) with either one infinite or
NaN is not finite, whatever the factor l (0 x Inf is NaN), so the step ends with an error and
the right-hand side shows where. FP32 two-point fluxes overflow from 2^128 on."""
from dataclasses import replace

import numpy as np
import pytest

import p2de
from p2de import abi, problems
from p2de import solver as S
from p2de.types import PositivityAndCellEntropyBound, PositivityAndMinEntropyBound, PositivityBound, TVDBound

from helpers import setup

pytestmark = pytest.mark.gpu

NOT_POSITIVE = 5
BOUNDS = {"pos": PositivityBound(), "cell": PositivityAndCellEntropyBound(), "tvd": TVDBound(),
          "min": PositivityAndMinEntropyBound()}


def solver_with(problem, N, bound, reference, precision, energy):
    param, md, bc, desc, U0 = setup(problem, N=N, Kx=6, Ky=4, bound=BOUNDS[bound], precision=precision,
                                    reference_semantics=reference)
    U = U0.copy()
    U[9, 1, 3] = energy
    g = S.Solver(param, md, desc)
    g.set_Uq(U)
    return g


@pytest.mark.parametrize("precision,energy", [("fp64", np.inf), ("mixed", 1e60), ("mixed-acc64", 1e60)])
@pytest.mark.parametrize("reference", [True, False])
@pytest.mark.parametrize("bound", list(BOUNDS))
@pytest.mark.parametrize("N", [1, 3])
def test_overflowed_fluxes_reach_the_right_hand_side(N, bound, reference, precision, energy):
    g = solver_with(problems.riemann2d, N, bound, reference, precision, energy)
    S.rhs_bang(None, g, None, p2de.TimeParam(0.0, 1e-6, 2))
    n, K = N + 1, 24
    bad = ~np.isfinite(g.get_field(abi.FIELD_F_BAR_H)) | ~np.isfinite(g.get_field(abi.FIELD_F_BAR_L))
    bad = bad.reshape(2, K, n * (n + 1), 4)
    fx = bad[0].reshape(K, n, n + 1, 4)  # [line][face]
    fy = bad[1].reshape(K, n + 1, n, 4)  # [face][line]
    want = fx[:, :, 1:] | fx[:, :, :-1] | fy[:, 1:] | fy[:, :-1]
    assert want.any()
    np.testing.assert_array_equal(~np.isfinite(g.get_field(abi.FIELD_RHSU)).reshape(want.shape), want)
    L = g.get_field(abi.FIELD_L_LOCAL, 2)
    assert not np.signbit(L).any() and (L <= 1).all()
    g.close()


@pytest.mark.parametrize("precision", ["mixed", "mixed-acc64"])
@pytest.mark.parametrize("bound", list(BOUNDS))
@pytest.mark.parametrize("N", [1, 3])
def test_a_step_with_overflowed_fluxes_fails(N, bound, precision):
    g = solver_with(problems.riemann2d, N, bound, True, precision, 1e60)
    with pytest.raises(abi.P2deError) as ei:
        S.ssp33_step(g, 0.0)
    assert ei.value.status == NOT_POSITIVE
    g.close()


@pytest.mark.parametrize("rho", [1.0, 20.0])
def test_large_boundary_fluxes_with_a_finite_difference_stay_finite(rho):
    """At an inflow face the low-order flux and the dissipation it has on top of the high-order
    one reach 2^1023 here; the high-order flux is 0 in the energy, so nothing overflows (the
    nodal form scales its fluxes in another order and overflows)."""
    param, md, bc, _, U0 = setup(problems.double_mach_reflection, N=1, Kx=8, Ky=2)
    geom = md.geom.copy()
    geom[:, 0] *= 2.0**16  # the right-hand side is the flux over J
    U = np.zeros_like(U0)
    U[..., 0] = rho
    # half the wavespeed times E: 1.06 x 2^1023 and 1.08 x 2^1023
    U[..., 3] = 2.0**683 * (1.0 if rho == 1.0 else 2.75)
    g = S.Solver(param, md, S.make_descriptor(param, replace(md, geom=geom), bc))
    g.set_Uq(U)
    S.rhs_bang(None, g, None, p2de.TimeParam(0.0, 2.0**-700, 2))
    assert np.isfinite(g.get_field(abi.FIELD_F_BAR_L)).all() and np.isfinite(g.get_field(abi.FIELD_F_BAR_H)).all()
    assert np.isfinite(g.get_field(abi.FIELD_RHSU)).all()
    g.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed-acc64"])
@pytest.mark.parametrize("N", [1, 2, 3, 4, 5])
def test_states_from_which_fluxes_may_overflow_give_the_same_bits(N, precision):
    """Blocks with a density outside [2^-24, 2^24), a pressure outside [2^-40, 2^30) or an energy
    from 2^30 on combine all their faces. Under the reference's reading the factors are 0, so
    rhsU is the low-order one, which scales exactly with powers of two from states inside the
    ranges: density by 2^a, velocity by 2^c."""
    param, md, bc, desc, U0 = setup(problems.riemann2d, N=N, Kx=5, Ky=4, bound=PositivityBound(), precision=precision)
    rng = np.random.default_rng(N)
    shape = U0.shape[:-1]
    rho, p = 0.5 + rng.random(shape), 0.5 + rng.random(shape)
    u, v = rng.standard_normal((2, *shape))
    U = np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], axis=-1)

    def rhs(a, c):
        g = S.Solver(param, md, desc)
        g.set_Uq(U * np.exp2([a, a + c, a + c, a + 2 * c]))
        S.rhs_bang(None, g, None, p2de.TimeParam(0.0, 2.0 ** (-14 - c), 2))
        out = g.get_field(abi.FIELD_RHSU).reshape(U.shape)
        g.close()
        return out * np.exp2(-np.array([a + c, a + 2.0 * c, a + 2 * c, a + 3 * c]))

    want = rhs(0, 0)
    assert np.isfinite(want).all()
    for a, c in ((25, 0), (-26, 0), (0, 16), (0, -22), (10, 5)):  # the last one inside the ranges
        np.testing.assert_array_equal(rhs(a, c), want, err_msg=f"{a} {c}")
