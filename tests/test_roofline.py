"""The work that the benchmark's roofline figures divide by time: FP64 operations only, and no
byte that the kernels of a form do not move."""
import pytest

from p2de import roofline

K = 57600  # double Mach reflection 480x120


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5])
def test_fp32_operations_are_not_counted(N):
    n = N + 1
    pairs = n * n * (n - 1)
    a = {p: roofline.stage_a_flops(N, 1, 0, p) for p in ("fp64", "mixed", "mixed-acc64")}
    assert a["fp64"] - a["mixed-acc64"] == 52 * pairs + 2 * n * n
    assert a["mixed-acc64"] - a["mixed"] == 16 * pairs + 24 * n * n + 64 * n
    f = [roofline.flux_form_flops(N, 1, 0, fp32) for fp32 in (False, True)]
    assert f[0] - f[1] == 34 * pairs + 3 * n * n


def test_settled_bounds_are_not_counted():
    # the reference's reading: only the solves evaluate a density bound, 10 operations each
    full = roofline.stage_a_flops(3, K, 0)
    assert roofline.stage_a_flops(3, K, 0, "fp64", True) == full - 640 * K
    assert roofline.stage_a_flops(3, K, 100, "fp64", True) == full - 640 * K + 6100


def test_flux_form_bytes():
    # N = 3, 16 nodes and 2 x 20 faces an element: factors 320, state 512, neighbours 64 + 16
    b = roofline.stage_bytes(3, K, flux=True)
    assert b["stage_a"] == K * (512 + 80 + 40 + 512 + 320)
    assert b["stage_b"] == K * (320 + 64 + 3 * 512 + 512 + 320)
    nodal = roofline.stage_bytes(3, K)
    assert b["stage_b"] < 0.5 * nodal["stage_b"]
    # kernel B took 42.8 us: below the 6.77 TB/s of a copy
    assert b["stage_b"] / 42.8e-6 < 6.77e12


def test_step_is_larger_than_the_cache():
    # state, copy, rhs, 4 x factors, subcell fluxes, metrics, neighbours
    assert roofline.step_bytes(3, K) == K * (3 * 512 + 4 * 320 + 2560 + 40 + 80) > 129e6
