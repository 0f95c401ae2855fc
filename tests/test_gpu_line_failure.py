"""A Line solve whose steps fail ends with the failure's code: its step does not read the
status word, so p2de_ssp33 has to look at it between batches of steps."""
from dataclasses import replace

import pytest

from p2de import abi, problems
from p2de import solver as S

from helpers import setup

pytestmark = pytest.mark.gpu

BAD_DT = 6


@pytest.mark.parametrize("N", [1, 3])
def test_solve_with_zero_time_steps_ends(N):
    param, md, bc, _, U0 = setup(problems.shu_osher, N=N, K=8, T=0.1)
    p = replace(param, timestepping_param=replace(param.timestepping_param, CFL=0.0))
    g = S.Solver(p, md, S.make_descriptor(p, md, bc))
    g.set_Uq(U0)
    with pytest.raises(abi.P2deError) as ei:
        S.ssp33(g)
    assert ei.value.status == BAD_DT
    g.close()
