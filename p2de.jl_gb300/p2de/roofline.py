"""Algorithmic work of the stage kernels, for the roofline figures.

Stage kernel A is bound by the FP64 pipe (GB300 runs FP64 at 1/58 of its FP32 rate),
so its roofline is in FP64 TFLOP/s. The work below counts one operation per IEEE
operation written in the kernel source (+, -, *, /, sqrt, log, fabs, min/max,
compare), an FMA-contractible a*b+c as two; a division, square root or logarithm
counts as ONE operation although the FP64 pipe spends several instructions on it,
so the fraction of peak understates how busy the pipe is. The data-dependent part
(the quadratic internal-energy solves that the exact l == 0 shortcut skips) is
counted from the kernel's own counter of solves evaluated.

Per element and stage, with n = N+1, Nq = n^2, Nfp = 4n, low-order pairs
NPL = 2n(n-1), high-order pairs NPH = n^2(n-1), subcell faces NSF = n(n+1):
  nodes: primitives, fluxes, two wavespeeds, two logs          50 Nq
  low-order pairs: lambda, averaged flux, viscosity             31 NPL
  gather of the low-order pairs (8 adds + lambda per side)       8 Nq + 18 NPL
  surface (neighbour wavespeed, fluxes, LF, B f*)               74 Nfp
  low-order finish (face terms, 1/(wq J), CFL)                  17 Nq + 9 Nfp
  high-order pairs: Chandrashekar flux with two log-means       52 NPH
  gather and lift of the high-order pairs                       24 Nq + 16 NPH + 16 Nfp
  subcell prefix sums and the low-order update                  55 Nq
  bound evaluations (P[0], density bound): with the intended
  bounds all of them; the reference's reading settles the
  others by integer comparisons                                 10 * 4 Nq, or 10 a solve
  quadratic solves evaluated (P vector, a, b, c, roots)         51 each
With FP32 pairs (mixed precision) the pair fluxes, their logarithms, gather and lift are
FP32 operations and not counted; with FP64 accumulation of them (mixed-acc64) the gather
and lift are.

In flux form (csrc/p2de_flux.cuh), with the interior faces NI = 2n(n-1):
  nodes: primitives and two logs                               15 Nq
  node fluxes and wavespeeds along both lines                  22 Nq
  boundary faces: exterior values, flux, dissipation           37 Nfp
  interior faces: flux and dissipation                         17 NI
  high-order pairs: flux, suffix and face sums                 42 NPH
  low-order rhs and update                                     29 Nq
  faces listed for a solve: energy bounds, quadratics, blend   70 each
With FP32 pairs (mixed-acc64) only the 8 additions a pair and 12 operations a node of the
first and fifth line are FP64.
"""
from __future__ import annotations


def stage_a_flops_per_elem(N: int, precision: str = "fp64", reference: bool = False) -> int:
    n = N + 1
    Nq, Nfp = n * n, 4 * n
    NPL, NPH = 2 * n * (n - 1), n * n * (n - 1)
    return (
        (50 if precision == "fp64" else 48) * Nq
        + 31 * NPL
        + 8 * Nq + 18 * NPL
        + 74 * Nfp
        + 17 * Nq + 9 * Nfp
        + (52 * NPH if precision == "fp64" else 0)
        + (0 if precision == "mixed" else 24 * Nq + 16 * NPH + 16 * Nfp)
        + 55 * Nq
        + (0 if reference else 10 * 4 * Nq)
    )


FLOPS_PER_BOUND = 10
FLOPS_PER_QUAD_SOLVE = 51


def stage_a_flops(N: int, K: int, quad_solves: float, precision: str = "fp64", reference: bool = False) -> float:
    """FP64 operations of one launch of stage kernel A over K elements."""
    per_solve = FLOPS_PER_QUAD_SOLVE + (FLOPS_PER_BOUND if reference else 0)
    return stage_a_flops_per_elem(N, precision, reference) * K + per_solve * quad_solves


def stage_bytes(N: int, K: int, flux: bool = False) -> dict:
    """Compulsory bytes per launch (each input read once, each output written once). Flux form:
    kernel A writes rhsU and, at the last stage of a step only, the subcell fluxes (not
    counted), and kernel B reads rhsU instead of them."""
    n = N + 1
    Nq, Nfp, NSF = n * n, 4 * n, n * (n + 1)
    factors, state, subcell = 8 * 2 * NSF, 32 * Nq, 8 * 16 * NSF
    if flux:
        a = K * (state + 5 * Nfp + 40 + state + factors)  # state, neighbours, metrics; rhsU, factors
        b = K * (factors + 4 * Nfp + 3 * state + state + factors)  # rhsU, U and W; U (W at stage 1); factors
    else:
        a = K * (state + 32 * Nfp + 40 + subcell + factors)
        b = K * (factors + 8 * 4 * n + subcell + 3 * state + 2 * state + factors + 8)
    return {"stage_a": a, "stage_b": b}


def step_bytes(N: int, K: int) -> int:
    """Bytes of the arrays that a whole step touches: state, its copy and right-hand side, the
    factors before and after symmetrization (three stages of those), subcell fluxes, metrics and
    neighbours."""
    n = N + 1
    Nq, Nfp, NSF = n * n, 4 * n, n * (n + 1)
    return K * (3 * 32 * Nq + 4 * 8 * 2 * NSF + 8 * 16 * NSF + 40 + 5 * Nfp)


def flux_form_flops_per_elem(N: int, fp32_pairs: bool = False) -> int:
    n = N + 1
    nodes, pairs = (12, 8) if fp32_pairs else (15, 42)
    return (nodes + 22 + 29) * n * n + 37 * 4 * n + 17 * 2 * n * (n - 1) + pairs * n * n * (n - 1)


FLOPS_PER_LISTED_FACE = 70


def flux_form_flops(N: int, K: int, listed_faces: float, fp32_pairs: bool = False) -> float:
    """FP64 operations of one launch of stage kernel A in flux form over K elements."""
    return flux_form_flops_per_elem(N, fp32_pairs) * K + FLOPS_PER_LISTED_FACE * listed_faces
