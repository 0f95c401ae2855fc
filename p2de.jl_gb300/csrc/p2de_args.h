// Launch arguments shared by the host code and the stage kernels.
#pragma once

#include <cmath>

#include <stdint.h>

#include "p2de_tables.h"

namespace p2de {

// flag bits of StageArgs::flags
enum : int {
  F_DO_LOW = 1 << 0,        // low-order graph-viscosity RHS
  F_DO_HIGH = 1 << 1,       // high-order ES flux differencing RHS
  F_DO_LIMIT = 1 << 2,      // subcell limiter
  F_WRITE_DEBUG = 1 << 3,   // write rhsxyL/H, BF_L/H, rhsL, rhsH to global
  F_AXIS_ALIGNED = 1 << 4,  // all elements have sxJ = ryJ = 0
  F_REF_SEM = 1 << 5,       // reference 4-name destructuring of the 5-tuple bound
  F_CELL_ENTROPY = 1 << 6,  // PositivityAndCellEntropyBound
  F_UPDATE = 1 << 7,        // stage kernel B applies the SSP-RK3 stage update
  F_RHSU_FROM_L = 1 << 8,   // rhsU = rhsL (LowOrderPositivity)
  F_RHSU_FROM_H = 1 << 9,   // rhsU = rhsH (FluxDiffRHS)
  F_CFL = 1 << 10,          // stage 1: low-order positivity CFL reduction
  F_ACC64 = 1 << 11,        // FP32 kernel: pair fluxes gathered and lifted in FP64
  F_TVD = 1 << 12,          // TVD density bounds from the low-order densities in rhoL
  F_LOW_ONLY = 1 << 13,     // kernel A stops after the low-order RHS and stores rhoL
  F_SHOCK = 1 << 14,        // HennemannShockCapture blending factor caps the subcell factors
  F_ZHANG_SHU = 1 << 15,    // ZhangShuLimiter: one factor per element, rhsU written by kernel A
  F_MIN_ENTROPY = 1 << 16,  // min-entropy bounds: bisection for phi >= Lphi - POSTOL
  F_RELAXED = 1 << 17,      // relaxed bounds: smoothness factor from the modal energies
  F_GAUSS = 1 << 18,        // GaussCollocation: projected face states, face pairs, Vf lift
  F_EPROJ = 1 << 19,        // NodewiseScaledExtrapolation: theta per face node
  F_KPP = 1 << 20,          // KPP{Dim2}: the scalar in component 0, the others 0
  F_LFPROJ = 1 << 21,       // LaxFriedrichsOnProjectedVal low-order flux: its CFL term
  F_FLUX = 1 << 22          // stage kernels in flux form (flux_form, p2de_flux.cuh)
};
// the modes whose branches only the EXT instantiation of stage kernel A compiles
constexpr int kExtFlags = F_ZHANG_SHU | F_MIN_ENTROPY | F_RELAXED | F_GAUSS | F_EPROJ | F_KPP | F_LFPROJ;

// boundary codes per face node
enum : int8_t { BC_INTERIOR = 0, BC_INFLOW = 1, BC_OUTFLOW = 2, BC_WALL = 3, BC_SHOCK = 4 };

// device scalar slots
enum : int { S_T = 0, S_DT_LIM = 1, S_DT = 2, S_DONE = 3, S_STEPS = 4, S_NSCAL = 8 };

// status bits
enum : int { ST_NOT_POSITIVE = 1, ST_BAD_DT = 2, ST_NAN = 4 };

struct StageArgs {
  int K;
  int nstage;  // 1..3
  int flags;
  int epb;  // elements per block (<= the degree's maximum, Cfg::E_MAX)
  // thread layout of the high-order pair and gather phases (p2de_layout): 0 flat (element,
  // pair) and (element, node) loops; 1 whole lines per warp on axis-aligned LGL elements
  int layout;
  // threads per block of stage kernel A (a multiple of 32 up to Cfg::THREADS; 0: Cfg::THREADS)
  int threads;
  int split;  // flux form: lines spread over the block (flux_shape)
  const OpTable* ops;
  double* Uq;
  double* resW;
  const double* geom;     // K x 5: J, rxJ, sxJ, ryJ, syJ
  const int32_t* nbr;     // Nfp x K: 0-based exterior face-node linear index (mapP - 1)
  const int8_t* bc;       // Nfp x K boundary code
  const int32_t* bcidx;   // Nfp x K index into Ival / xyS
  const double* Ival;     // nI x 4
  const double* xyS;      // nS x 2
  double shock_x0, shock_inv_slope, shock_speed;
  double shock_post[4], shock_pre[4];
  double gamma, gm1, CFL, dt0, T, zeta, ZEROTOL;
  double* rhsL;
  double* rhsH;
  double* rhsU;
  double* rhsxyL;
  double* rhsxyH;
  double* BFL;
  double* BFH;
  double* fbar;  // K x (2 dirs x 2 (H, L) x NSF x 4)
  double* Lpre;  // K x 2 x (Nq+N1D), before symmetrization (nodal form: a set sign bit marks
                 // a face whose fluxes overflow)
  double* Lfin;  // 3 stages x K x 2 x (Nq+N1D)
  double* scal;  // S_* slots
  unsigned long long* dtmin_bits;
  long long* minrec;  // 3 stages x {min rho, min rhoe} as ordered keys
  int* status;
  unsigned long long* counters;  // [0] quadratic rhoe solves evaluated by the bound phase
  double* rhoL;  // K x Nq low-order densities U + dt rhsL (TVD bounds only)
  const double* geomx;  // K x 16 geometry factors (geom_factor), or null: computed per launch
  double sc_TN, sc_q;   // HennemannShockCapture: TN and -log((1-1e-4)/1e-4) / TN
  double* Lelem;        // 3 stages x K: ZhangShuLimiter factors (F_ZHANG_SHU)
  double* phimin;       // [0]: min of phi = rhoe rho^-gamma over the state at t0, stage 1
  double t0, POSTOL;
  double s0;            // log10(N^-4), the centre of the smoothness ramp (subcell.jl:944)
  double beta;          // relaxed cell-entropy bounds: target scale 1 - beta eps_k
  double* ufproj;       // K x Nfp x 4: entropy-projected face states (GaussCollocation)
  double* theta;        // 3 stages x K x Nfp: entropy-projection limiting factors
  double eta;           // LimitingParameter eta (bounds of the projected face states)
  // constants of the gas, formed once (set_gas): 1/(gamma-1), (gamma-1)/2, gamma (gamma-1)/4,
  // and FP32 gamma, gamma-1, 2 (gamma-1)
  double rgm1, hgm1, cws;
  float gasf[3];
  // floor(log2((1 - zeta)/zeta)) (set_zeta): the quadratics' constant term is at least
  // rho (zeta rhoe) 2^kzeta; very negative when zeta is not in (0, 1)
  int kzeta;
};

inline void set_zeta(StageArgs& a, double zeta) {
  a.zeta = zeta;
  a.kzeta = zeta > 0.0 && zeta < 1.0 ? std::ilogb((1.0 - zeta) / zeta) : -100000;
}

inline void set_gas(StageArgs& a, double gamma) {
  a.gamma = gamma;
  a.gm1 = gamma - 1.0;
  a.rgm1 = 1.0 / a.gm1;
  a.hgm1 = 0.5 * a.gm1;
  a.cws = 0.25 * (gamma * a.gm1);
  a.gasf[0] = (float)a.gamma;
  a.gasf[1] = (float)a.gm1;
  a.gasf[2] = (float)(2.0 * a.gm1);
}

// Whether every face node of a boundary list (1-based, as mapI, mapO, mapW, mapS) is its own
// exterior face.
inline bool own_faces(const int64_t* list, int64_t count, const int64_t* mapP) {
  for (int64_t i = 0; i < count; ++i)
    if (mapP[list[i] - 1] != list[i]) return false;
  return true;
}

// Whether a solve's stage kernels run in flux form (p2de_flux.cuh): subcell-limited Euler on
// axis-aligned LGL elements with the nodal low-order flux. own_boundaries: every face with a
// boundary code is its own exterior face (mapP), as uniform meshes have it; the limited flux
// there then needs no neighbour's factor. No low-order pair may have been dropped by ZEROTOL
// (its entry is half the tangential weight, at least 1/(N (N+1))), since the form divides
// the lines' common weight out. acc32: the FP32 two-point sums of mixed precision do not
// telescope, and whether the difference they leave at an element face blends is decided by
// the sign of FP64 rounding, so those solves keep the nodal form and its bits. Under the reference's reading of the bounds every interior
// factor is 0, so a shock-capture cap acts only on the rounding of f_bar_H - f_bar_L at
// element faces, which the flux form makes exactly 0: those solves keep the nodal form.
inline bool flux_form(int flags, int N, double zerotol, bool own_boundaries, bool acc32) {
  return (flags & F_AXIS_ALIGNED) && (flags & F_DO_LIMIT) && !(flags & (F_GAUSS | F_KPP | F_LFPROJ | F_ZHANG_SHU)) &&
         !((flags & F_SHOCK) && (flags & F_REF_SEM)) && !acc32 && own_boundaries && zerotol < 0.999999 / ((double)N * (N + 1));
}

// Steps to launch before looking at the device's time again: enough to reach T at the last
// step size, so that a run which ends (or fails) earlier than nsteps does not replay the step
// as no-ops, seven launches each (the 5x5 vortex solve takes 8 steps of the 64 that
// p2de_ssp33 asked for: 680 us with the other 56 replayed, 210 without). dt: the last step of
// this run, 0 at its start.
inline int64_t steps_ahead(double t, double T, double dt, int64_t left) {
  const int64_t first = 4, most = 4096;
  if (!(dt > 0.0)) return left < first ? left : first;
  const double need = (T - t) / dt;
  const int64_t n = need < 1.0 ? 1 : need < (double)most ? (int64_t)need + 1 : most;
  return left < n ? left : n;
}

// StageArgs shock-capture constants of update_blending_factor! (shock_capture.jl:123-126)
inline void set_shock_capture(StageArgs& a, int N, double sc_a, double sc_c) {
  const double TN = sc_a * std::pow(10.0, -sc_c * std::pow((double)(N + 1), 0.25));
  const double alphaE0 = 0.0001;
  const double s_factor = std::log((1 - alphaE0) / alphaE0);
  a.sc_TN = TN;
  a.sc_q = -s_factor / TN;
}

// flag bits of a SubcellLimiter bound type (p2de_bound_type, Solver.jl:47-62)
inline int bound_flags(int bound_type) {
  switch (bound_type) {
    case 1: return F_CELL_ENTROPY;                            // PositivityAndCellEntropyBound
    case 2: return F_TVD;                                     // TVDBound
    case 3: return F_TVD | F_CELL_ENTROPY;                    // TVDAndCellEntropyBound
    case 4: return F_MIN_ENTROPY;                             // PositivityAndMinEntropyBound
    case 5: return F_MIN_ENTROPY | F_RELAXED;                 // PositivityAndRelaxedMinEntropyBound
    case 6: return F_CELL_ENTROPY | F_RELAXED;                // PositivityAndRelaxedCellEntropyBound
    case 7: return F_TVD | F_MIN_ENTROPY;                     // TVDAndMinEntropyBound
    case 8: return F_TVD | F_MIN_ENTROPY | F_RELAXED;         // TVDAndRelaxedMinEntropyBound
    case 9: return F_TVD | F_CELL_ENTROPY | F_RELAXED;        // TVDAndRelaxedCellEntropyBound
    default: return 0;                                        // PositivityBound
  }
}

// StageArgs constants of the min-entropy and relaxed bounds: t0 (the stage at which the
// initial minimum of phi is taken), POSTOL, s0 = log10(N^-4) (subcell.jl:944, with N^-4
// as Float64(N)^-4) and the relaxed cell-entropy beta
inline void set_bound_constants(StageArgs& a, int N, double t0, double POSTOL, double beta) {
  a.t0 = t0;
  a.POSTOL = POSTOL;
  a.s0 = std::log(1.0 / ((double)N * N * N * N)) / std::log(10.0);
  a.beta = beta;
}

}  // namespace p2de
