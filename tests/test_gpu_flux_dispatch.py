"""Which solves run in flux form and in which layout of its lines. The default launch shape of
a solve tells its form; a batch always splits the lines of a member without extended bounds
over its blocks, and a solve of its own does so only below 65,536 nodes (110,000 from N = 4
on), so a mesh above that runs both layouts of the same kernel body."""
from dataclasses import replace

import numpy as np
import pytest

import p2de
from p2de import abi, problems
from p2de import solver as S
from p2de.batch import Batch
from p2de.types import PositivityAndMinEntropyBound, PositivityBound, TVDBound

from helpers import setup
from test_gpu_flux_form import both_forms

pytestmark = pytest.mark.gpu


def shapes(**kw):
    """(default elements per block, the largest) of a solve that is nodal by one metric term,
    and of the solve itself."""
    param, md, bc, desc, U0 = setup(problems.riemann2d, Kx=7, Ky=3, **kw)
    desc.bc = bc
    pair = both_forms(param, md, desc, U0)
    out = [s.elements_per_block() for s in pair]
    for s in pair:
        s.close()
    return out


# at N = 1 and 2 the limits of both forms are 32 and the extended bounds' defaults are alike
@pytest.mark.parametrize("precision", ["fp64", "mixed-acc64"])
@pytest.mark.parametrize("N,bound", [(N, PositivityBound()) for N in (1, 2, 3, 4, 5)] +
                         [(3, TVDBound()), (3, PositivityAndMinEntropyBound()), (5, PositivityAndMinEntropyBound())])
def test_axis_aligned_solves_run_in_flux_form(N, bound, precision):
    nodal, flux = shapes(N=N, bound=bound, precision=precision)
    assert nodal != flux


def test_fp32_sums_run_in_nodal_form():
    for N in (1, 2, 3, 4, 5):
        nodal, mixed = shapes(N=N, precision="mixed")
        assert nodal == mixed


def test_dropped_low_order_pairs_run_in_nodal_form():
    param, md, bc, _, U0 = setup(problems.kelvin_helmholtz, N=3, Kx=4, Ky=4)
    param = replace(param, global_constants=p2de.GlobalConstant(POSTOL=1e-14, ZEROTOL=0.2))
    desc = S.make_descriptor(param, md, bc)
    desc.bc = bc
    nodal, flux = both_forms(param, md, desc, U0)
    assert nodal.elements_per_block() == flux.elements_per_block()
    nodal.close()
    flux.close()


# the smallest ragged meshes above the threshold: 65,564 nodes at N = 1, 65,619 at N = 2,
# 65,584 at N = 3, 110,075 at N = 4, 110,088 at N = 5
LARGE = {1: (37, 443), 2: (23, 317), 3: (4099, 1), 4: (37, 119), 5: (22, 139)}


@pytest.mark.parametrize("reference", [True, False])
@pytest.mark.parametrize("precision", ["fp64", "mixed-acc64"])
@pytest.mark.parametrize("N", [1, 2, 3, 4, 5])
def test_both_layouts_of_the_lines_give_the_same_bits(N, precision, reference):
    Kx, Ky = LARGE[N]
    assert Kx * Ky * (N + 1) ** 2 >= (110000 if N >= 4 else 65536)
    param, md, bc, desc, U0 = setup(problems.double_mach_reflection, N=N, Kx=Kx, Ky=Ky, bound=PositivityBound(),
                                    precision=precision, reference_semantics=reference)
    b = Batch(pool_bytes=1 << 30, max_solves=1, precision=precision)
    slot = b.add(desc, U0)
    b.step(2)
    want, t = b.Uq(slot), b.states()[slot, 0]
    b.close()
    assert np.abs(want - np.ravel(U0)).max() > 0.0
    for threads in (64, 128):
        g = S.Solver(param, md, desc)
        default = g.elements_per_block()[0]
        # the split layout's defaults are 8, 3, 2, 3, 2 elements a block
        assert default > {1: 8, 2: 3, 3: 2, 4: 3, 5: 2}[N]
        g.set_threads_per_block(threads)
        g.set_Uq(U0)
        tg = 0.0
        for _ in range(2):
            tg, _ = S.ssp33_step(g, tg)
        assert tg == t
        np.testing.assert_array_equal(g.get_field(abi.FIELD_UQ), want)
        g.close()
