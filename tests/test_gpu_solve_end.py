"""A solve whose time step grows ends after fewer steps than its first step sizes let expect:
p2de_ssp33 looks at the time every 64 steps, so that it replays at most 63 steps that do
nothing."""
import numpy as np
import pytest

from p2de import problems
from p2de import solver as S

from helpers import setup

pytestmark = pytest.mark.gpu


def test_growing_time_step_leaves_few_launches_after_the_end():
    # one element at 1e5 times the others' pressure: dt grows from 6.6e-5 to 4e-4
    param, md, bc, desc, U0 = setup(problems.kelvin_helmholtz, N=1, Kx=8, Ky=8, T=0.05)
    U = np.zeros_like(U0)
    U[..., 0] = 1.0
    U[..., 3] = 0.1 / 0.4
    U[0, :, 3] = 1e4 / 0.4
    g = S.Solver(param, md, desc)
    g.set_Uq(U)
    before = g.launch_count()
    t, dt = S.ssp33_step(g, 0.0)
    per_step = g.launch_count() - before
    assert (param.timestepping_param.T - t) / dt > 600
    g.set_Uq(U)
    before = g.launch_count()
    t, steps, _ = S.ssp33(g)
    assert t == param.timestepping_param.T and steps < 250
    assert g.launch_count() - before <= per_step * (steps + 63)
    g.close()
