"""The elements per block that a batch reports are those that its members run at: members in
nodal form (FP32 sums, rotated elements) and in flux form have defaults of their own."""
from dataclasses import replace

import numpy as np
import pytest

from p2de import problems
from p2de import solver as S
from p2de.batch import Batch

from helpers import setup

pytestmark = pytest.mark.gpu

NODAL = {1: 16, 2: 7, 3: 4, 4: 2, 5: 1}
FLUX = {1: 16, 2: 5, 3: 4, 4: 3, 5: 2}


@pytest.mark.parametrize("precision,want", [("mixed", NODAL), ("fp64", FLUX), ("mixed-acc64", FLUX)])
@pytest.mark.parametrize("N", [1, 2, 3, 4, 5])
def test_reported_elements_per_block(N, precision, want):
    param, md, bc, desc, U0 = setup(problems.riemann2d, N=N, Kx=5, Ky=3, precision=precision)
    b = Batch(pool_bytes=64 << 20, max_solves=2, precision=precision)
    assert b.elements_per_block(N)[0] == want[N]
    b.add(desc, U0)
    assert b.elements_per_block(N)[0] == want[N]
    b.close()


def test_tuning_of_nodal_and_flux_members_together():
    """The tuned choice may be the two forms' own defaults; the members keep their bits and the
    reported value is in range, and is the one set from then on."""
    flux = setup(problems.riemann2d, N=2, Kx=9, Ky=5, reference_semantics=False)
    param, md, bc, _, U0 = flux
    geom = md.geom.copy()
    geom[-1, 2] = np.finfo(np.float64).tiny
    nodal = S.make_descriptor(param, replace(md, geom=geom), bc)
    runs = []
    for tune in (False, True):
        b = Batch(pool_bytes=64 << 20, max_solves=2)
        slots = [b.add(flux[3], U0), b.add(nodal, U0)]
        assert b.elements_per_block(2)[0] == FLUX[2]
        if tune:
            best = b.autotune()
            assert best == {2: b.elements_per_block(2)[0]} and 1 <= best[2] <= b.elements_per_block(2)[1]
        b.step(3)
        runs.append([b.Uq(s) for s in slots])
        b.remove(slots[0])
        if not tune:
            assert b.elements_per_block(2)[0] == NODAL[2]
        b.set_elements_per_block(2, 6)
        assert b.elements_per_block(2)[0] == 6
        b.close()
    for a, c in zip(*runs):
        np.testing.assert_array_equal(a, c)
