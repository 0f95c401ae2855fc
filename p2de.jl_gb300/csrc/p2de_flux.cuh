// Stage kernel A in flux form: subcell-limited Euler solves on axis-aligned LGL elements.
//
// On such elements every term of the right-hand side is a difference of fluxes along the
// lines of the tensor-product grid. A line (element, direction, tangential node) with nodes
// 0..n-1 has n+1 subcell faces; face t lies between nodes t-1 and t, faces 0 and n on the
// element boundary. In units of -g w (g the element's rxJ or syJ, w the line's tangential
// weight) the subcell fluxes f_bar of subcell.jl:163-206 are
//   low order   phi_t = (F_{t-1} + F_t)/2 - ws/2 (U_t - U_{t-1})
//               (the pair terms of low_order_graph_viscosity.jl:139-173 and the surface terms
//               of :175-204; the prefix sums of accumulate_f_bar! telescope to them),
//   high order  phi_t = sum_{j < t <= i} c_ij fS(i, j),   c_ij = -hp_S[ij] / w
//               (the prefix sums of the two-point terms of flux_differencing.jl:164-361;
//               on the element boundary the surface flux of :223-272),
// and the right-hand sides are their differences, rhs = cx dphi_x + cy dphi_y with
// cx = -rxJ / (J w_r), cy = -syJ / (J w_s). So the kernel forms the faces' fluxes once and
// takes one difference per node, where the nodal form gathers pair terms at nodes, scales
// them by the mass and sums the scaled values back to faces: 24 multiply-adds per node and
// component there, 4 here, and the boundary faces carry f_bar_H = f_bar_L exactly.
//
// What bounds it: FP64 instruction issue, as everywhere here (2 FMA/clk/SM; a warp
// instruction holds the pipe 17-20 clocks, measured). One thread per line holds the line's
// wavespeeds, fluxes and high-order sums in registers: neither pair terms nor nodal fluxes
// nor wavespeeds go through shared memory, and a node's flux and wavespeed along a line are
// formed by the one thread that uses them. DMR 480x120 N=3 FP64, per stage: kernel A 1103 us
// in the nodal form, 590 us here; kernel B 123 us there, 42 us here (it no longer blends).
//
// Every operation is an explicitly rounded one (dadd, dmul, dfma ...): nothing is left for
// the compiler to contract, so the batch kernels give a member the bits it has alone.
#pragma once

#include "p2de_stage.cuh"

namespace p2de {

__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dfma(double a, double b, double c) { return __fma_rn(a, b, c); }

__device__ __forceinline__ bool negative(double x) { return __double2hiint(x) < 0; }
// > 0 and not NaN, by the bits
__device__ __forceinline__ bool positive_bits(double x) {
  const long long b = __double_as_longlong(x);
  return b > 0 && b <= 0x7ff0000000000000LL;
}
template <int N1D>
struct FluxCfg {
  static constexpr int n = N1D;
  static constexpr int Nq = n * n;
  static constexpr int Nfp = 4 * n;
  static constexpr int NL = 2 * n;         // lines per element
  static constexpr int NSF = n * (n + 1);  // subcell faces per direction
  static constexpr int NF = 2 * NSF;
  static constexpr int NI = 2 * n * (n - 1);  // interior subcell faces
  static constexpr int PPL = n * (n - 1) / 2;
  static constexpr int THREADS = 128;
  // default elements per block: lines and nodes in (nearly) full warps
  static constexpr int E = n == 2 ? 16 : n == 3 ? 10 : n == 4 ? 4 : n == 5 ? 6 : 5;
  // and in the batched kernel (split lines, 128 threads)
  static constexpr int E_BATCH = n == 2 ? 16 : n == 3 ? 5 : n == 4 ? 4 : n == 5 ? 3 : 2;
  // shared-memory doubles per element; arrays over nodes and faces are component-major
  static constexpr int O_C = 0;                 // 6n: cx, cy; s = 4 dt c of both; 1/s of both
  static constexpr int O_U = O_C + 6 * n;       // 4 Nq: state
  static constexpr int O_W = O_U + 4 * Nq;      // 12 Nq (14 Nq EXT): node data, see W_*
  // W before the line phase: u/2, v/2, u, v, rho/p, log rho, log(rho/p), p/2, gamma gm1/(4 rho)
  // (FP32 pairs: planes 4-5, W_F32, hold rho, u, v, beta as floats); indicator and modal
  // energies 9, 10.
  // After it: uL (0-3), zeta rhoe, Lrho, Urho, phi threshold, the quadratics' c; EXT: bound
  // evaluations 10-13.
  // In the cell-entropy phase: its scratch.
  static constexpr int W_HU = 0, W_HV = 1, W_U = 2, W_V = 3, W_BETA = 4, W_LR = 5, W_LB = 6, W_PH = 7, W_CRR = 8,
                       W_IND = 9, W_EN = 10, W_F32 = 4;
  static constexpr int W_UL = 0, W_LRHOE = 4, W_LRHO = 5, W_URHO = 6, W_THR = 7, W_QC = 8, W_EV = 10;
  static constexpr int NPH = NL * PPL;
  template <bool EXT, bool SPLIT = false>
  struct Lay {
    static constexpr int O_R = O_W + (EXT ? 14 : 12) * Nq;  // 4 Nq: rhsL; before that CFL sums (0, 1)
    static constexpr int O_PH = O_R + 4 * Nq;               // 4 NF: low-order (then limited) fluxes
    // 4 NF: high-order minus low-order fluxes; under upper0, where one comparison settles most
    // interior faces, those hold the high-order flux until a bound asks for the difference
    // (factor -0 marks those that never did)
    static constexpr int O_DF = O_PH + 4 * NF;
    static constexpr int O_L = O_DF + 4 * NF;               // NF: factors
    // smoothness factor of the relaxed bounds, 2 flags of the entropy phase, blending factor
    static constexpr int O_X = O_L + NF;
    // SPLIT: pair fluxes, along-axis node values (normal, tangential and energy half flux, half
    // wavespeed; per direction), half wavespeeds of the faces
    static constexpr int O_SF = O_X + 4;
    static constexpr int O_SN = O_SF + 4 * NPH;
    static constexpr int O_SW = O_SN + 8 * Nq;
    static constexpr int PE = SPLIT ? O_SW + NF : O_X + 4;
  };
  // plus the list of faces whose bounds need solves (and, EXT, the list of bisections)
  template <bool EXT, bool SPLIT = false>
  static constexpr size_t smem(int e) {
    return sizeof(double) * Lay<EXT, SPLIT>::PE * e + sizeof(int) * ((size_t)NF * e + 4 + (EXT ? 2 * (size_t)NF * e : 0));
  }
  static constexpr int E_MAX_RAW =
      (int)((224 * 1024 - 64) / (sizeof(double) * Lay<true>::PE + sizeof(int) * 3 * NF));
  static constexpr int E_MAX = E_MAX_RAW < 32 ? E_MAX_RAW : 32;
  static constexpr int E_SPLIT_RAW =
      (int)((224 * 1024 - 64) / (sizeof(double) * Lay<false, true>::PE + sizeof(int) * NF));
  static constexpr int E_SPLIT_MAX = E_SPLIT_RAW < 32 ? E_SPLIT_RAW : 32;
  static_assert(E <= E_MAX && E_BATCH <= E_SPLIT_MAX && E_SPLIT_MAX <= E_MAX, "flux layout");
};

// fS(Dim2) (compressible_Navier_Stokes.jl:220-249) along axis ax for line nodes a and b, in
// FP64: one reciprocal gives 1/(beta_a + beta_b) and the two quotients of the log means.
// The log mean's branch test |da/aavg| < 1e-4 is decided from the exponents of da and of the
// sum where they settle it (all but two of them), else as written. In its series branch
// x = da/aavg has x^2 < 1e-8, so the x^4 and x^6 terms of the series (and of its reciprocal,
// for betalog) are below 2^-53 and are not formed.
struct PairState {
  double rho, vn, vt, hn, ht, beta, lr, lb;  // velocities normal and tangential to the axis, and halves
};
__device__ __forceinline__ void fS_line(double ig, const PairState& a, const PairState& b, double* F0, double* Ft,
                                        double* Fn, double* F3) {
  const double sr = dadd(a.rho, b.rho), dr = dsub(b.rho, a.rho);
  const double sb = dadd(a.beta, b.beta), db = dsub(b.beta, a.beta);
  const bool ser_r = series_branch(dr, sr), ser_b = series_branch(db, sb);
  const double den_r = ser_r ? sr : dsub(a.lr, b.lr);
  const double den_b = ser_b ? sb : db;
  const double t = dmul(den_r, den_b), D = dmul(t, sb);
  double isb, idr, idb;  // 1/sb, 1/den_r, 1/den_b
  if (mid_exponent(t) && mid_exponent(D)) {
    const double r = rcp(D), q = dmul(sb, r);
    isb = dmul(t, r);
    idr = dmul(den_b, q);
    idb = dmul(den_r, q);
  } else {  // the products leave the range of doubles
    isb = rcp(sb);
    idr = rcp(den_r);
    idb = rcp(den_b);
  }
  const double x = dmul(dr, idr);
  double rl = -x;                  // rho log mean
  double nb = dsub(b.lb, a.lb);    // numerator of 1/beta log mean
  if (ser_r) rl = dmul(sr, dfma(dmul(x, x), -0.4, 0.5));
  if (ser_b) {
    const double y = dmul(db, isb);
    nb = dfma(dmul(y, y), 1.6, 2.0);
  }
  const double ilb = dmul(nb, idb);
  const double pa = dmul(sr, isb);
  const double un = dadd(a.hn, b.hn), ut = dadd(a.ht, b.ht);
  const double w = dfma(a.vt, b.ht, dmul(a.vn, b.hn));
  const double f4 = dfma(dmul(rl, ilb), ig, dfma(rl, w, pa));
  *F0 = dmul(rl, un);
  *Ft = dmul(*F0, ut);
  *Fn = dfma(*F0, un, pa);
  *F3 = dmul(f4, un);
}

// Whether a node's density factor is 0 for P0 = s dF0 >= +0 under upper0 (Urho = 0, the Lphi
// slot of the reference's destructuring): U0 >= Lrho > 0 gives U0 + P0 >= Lrho and > 0 = Urho,
// so the factor max((0 - U0)/P0, 0) is 0.
__device__ __forceinline__ bool zero_factor(double U0, double s, double Lrho) {
  const long long u = __double_as_longlong(U0), l = __double_as_longlong(Lrho);
  return u > 0 && u < 0x7ff0000000000000LL && l <= u &&
         (__double_as_longlong(s) & 0x7ff0000000000000LL) != 0x7ff0000000000000LL;
}

// rhoe_quadratic_solve (limiter_utils.jl:108-146) for P = s dF (s the node's 4 dt cx): the
// quadratic is solved in l' = s l, whose coefficient a = A(dF) serves both nodes of the face
// (r2a = 1/(2a)); is = 1/s. Comparisons of the roots with +-ZEROTOL on l itself.
__device__ __forceinline__ double rhoe_root(const double* U, const double* dF, double a4, double r2a, double c,
                                            double Lrhoe, double s, double is, double ZEROTOL) {
  double b = dmul(dsub(U[3], Lrhoe), dF[0]);
  b = dfma(U[0], dF[3], b);
  b = dfma(-U[1], dF[1], b);
  b = dfma(-U[2], dF[2], b);
  // |a| + |b| < c/2 on l in [0, 1]: no root there, the factor is 1
  const double t = dmul(dfma(0.25 * fabs(a4), fabs(s), fabs(b)), fabs(s));
  if (t < 0.5 * c) return 1.0;
  const double disc = dfma(b, b, -dmul(a4, c));
  double l = 1.0;
  if (disc >= 0.0) {
    const double sq = sqrt_rn(disc);
    const double k = dmul(r2a, is);
    const double r1 = dmul(dsub(sq, b), k), r2 = dmul(dsub(-b, sq), k);
    if (r1 > ZEROTOL && r2 > ZEROTOL)
      l = fmin(r1, r2);
    else if (r1 > ZEROTOL && r2 < -ZEROTOL)
      l = r1;
    else if (r2 > ZEROTOL && r1 < -ZEROTOL)
      l = r2;
  }
  return l;
}

// zeta rhoe_ufun(uL) and c of the quadratics (limiter_utils.jl:141-146)
__device__ __forceinline__ void energy_bound(const double* uL, double zeta, double& Lrhoe, double& c) {
  const double ke2 = dfma(uL[1], uL[1], dmul(uL[2], uL[2]));
  Lrhoe = dmul(zeta, dfma(-0.5, dmul(ke2, rcp(uL[0])), uL[3]));
  c = dfma(uL[0], dsub(uL[3], Lrhoe), dmul(-0.5, ke2));
}

// phi = rhoe rho^-gamma (s_modified_ufun) of U + l P, explicitly rounded
__device__ __forceinline__ double phi_at(const double* U, const double* P, double l, double gamma,
                                         const OpTable& op) {
  const double r = dfma(l, P[0], U[0]), m1 = dfma(l, P[1], U[1]), m2 = dfma(l, P[2], U[2]), E = dfma(l, P[3], U[3]);
  const double rhoe = dfma(-0.5, dmul(dfma(m1, m1, dmul(m2, m2)), rcp(r)), E);
  return dmul(rhoe, pow_fast(r, -gamma, op));
}

// Along-axis values of one line node: the state (rho, normal and tangential momentum, E) and
// its half flux (normal, tangential and energy components; the mass flux is the normal
// momentum) and half wavespeed (compressible_Navier_Stokes.jl:48-62, 175-194).
struct LineNode {
  double U[4], fn, ft, fe, wh;
};
// from hn, ht = half velocities, ph = p/2, crr = gamma gm1/(4 rho); U filled
__device__ __forceinline__ void line_node(LineNode& q, double hn, double ht, double ph, double crr) {
  q.fn = dfma(q.U[1], hn, ph);
  q.ft = dmul(q.U[1], ht);
  q.fe = dmul(hn, dfma(2.0, ph, q.U[3]));
  const double pe = dfma(-q.U[1], hn, q.U[3]);
  q.wh = dadd(fabs(hn), sqrt_rn(dmul(pe, crr)));
}

// One line of an element: its places in the element's shared memory and the pieces of its
// fluxes. Components of states and fluxes here are (rho, normal, tangential, E).
//
// Two layouts call them, with the same operations per value and so the same bits. On large
// meshes one thread takes a whole line: the fewest FP64 instructions, all lanes busy. An SM
// quarter issues one FP64 warp instruction per 64 clocks and holds no second one in flight
// (measured: 64 clocks a dependent chain, with 1 to 8 chains in a warp), so on small meshes,
// where an SM has few warps, a line's chain of ~300 instructions is the stage's duration;
// SPLIT spreads the pairs, boundary faces, node values and sums over the block's warps.
template <int N1D, class Y>
struct FluxLine {
  using C = FluxCfg<N1D>;
  static constexpr int n = C::n, Nq = C::Nq, Nfp = C::Nfp, NSF = C::NSF, NF = C::NF;
  const StageArgs& a;
  const OpTable& op;
  double* base;
  const int k, ax, l;
  const double t_now, gd;
  const int sg;     // the sign of f_bar's unit
  const bool visc;  // the reference adds the viscosity of an x pair only when |S0x| > 1e-10 (:156-163)
  const int q0, qs;  // nodes q0 + qs i
  const int f0, fs;  // faces f0 + fs t
  double *PH, *DF;

  __device__ __forceinline__ FluxLine(const StageArgs& a_, const OpTable& op_, double* base_, int k_, int ax_, int l_,
                                      double t_)
      : a(a_), op(op_), base(base_), k(k_), ax(ax_), l(l_), t_now(t_), gd(a_.geom[5 * (size_t)k_ + (ax_ ? 4 : 1)]),
        sg(negative(gd) ? -1 : 1),
        visc(ax_ == 1 || magnitude_above(dmul(gd, op_.lp_S[l_ * (n - 1)]), 1e-10)),
        q0(ax_ ? l_ : n * l_), qs(ax_ ? n : 1), f0(ax_ ? NSF + l_ : (n + 1) * l_), fs(ax_ ? n : 1),
        PH(base_ + Y::O_PH), DF(base_ + Y::O_DF) {}

  // the array component of line component q
  __device__ __forceinline__ int comp(int q) const { return q == 1 ? 1 + ax : q == 2 ? 2 - ax : q; }

  __device__ __forceinline__ void load(int i, LineNode& q) const {
    const double* U = base + C::O_U + q0 + qs * i;
    const double* W = base + C::O_W + q0 + qs * i;
    q.U[0] = U[0];
    q.U[1] = U[(1 + ax) * Nq];
    q.U[2] = U[(2 - ax) * Nq];
    q.U[3] = U[3 * Nq];
    line_node(q, W[ax * Nq], W[(1 - ax) * Nq], W[C::W_PH * Nq], W[C::W_CRR * Nq]);
  }

  // the exterior state at boundary face `side` of the line (0 low, 1 high) and its values; off:
  // the high-order flux has no dissipation there
  __device__ __forceinline__ void exterior(int side, const LineNode& own, LineNode& P, bool& off) const {
    const size_t fk = (size_t)k * Nfp + (2 * ax + side) * n + l;
    const int lin = a.nbr[fk], code = a.bc[fk];
    double S[4];
    if (code == BC_INTERIOR) {
      const int kP = lin / Nfp, iP = lin % Nfp, sP = iP / n, tP = iP % n;
      const int qP = sP == 0 ? n * tP : sP == 1 ? (n - 1) + n * tP : sP == 2 ? tP : tP + n * (n - 1);
      const double* s = a.Uq + ((size_t)kP * Nq + qP) * 4;
#pragma unroll
      for (int c = 0; c < 4; ++c) S[c] = __ldg(s + c);
    } else if (code == BC_INFLOW) {
      const double* iv = a.Ival + 4 * (size_t)a.bcidx[fk];
#pragma unroll
      for (int c = 0; c < 4; ++c) S[c] = iv[c];
    } else if (code == BC_SHOCK) {
      const double* xy = a.xyS + 2 * (size_t)a.bcidx[fk];
      const bool post = xy[0] < a.shock_x0 + (xy[1] + a.shock_speed * t_now) * a.shock_inv_slope;
#pragma unroll
      for (int c = 0; c < 4; ++c) S[c] = post ? a.shock_post[c] : a.shock_pre[c];
    } else {  // outflow: the own state; wall: the own state reflected along the axis
      const double mn = code == BC_WALL ? -own.U[1] : own.U[1];
      S[0] = own.U[0];
      S[1] = ax ? own.U[2] : mn;
      S[2] = ax ? mn : own.U[2];
      S[3] = own.U[3];
    }
    P.U[0] = S[0];
    P.U[1] = ax ? S[2] : S[1];
    P.U[2] = ax ? S[1] : S[2];
    P.U[3] = S[3];
    const double rr = rcp(P.U[0]), hr = half(rr);
    const double hn = dmul(P.U[1], hr), ht = dmul(P.U[2], hr);
    // p/2 as the node phase forms it, so that the two elements at a face form the same flux bits
    // (times gm1/2, not half of times gm1: 595 us a stage against 605 on DMR 480x120)
    const double ph = dmul(a.hgm1, dfma(-0.5, dmul(dfma(S[1], S[1], dmul(S[2], S[2])), rr), S[3]));
    line_node(P, hn, ht, ph, dmul(a.cws, rr));
    // a boundary face's wavespeed is the own one (its mapP is itself)
    if (code != BC_INTERIOR) P.wh = own.wh;
    off = code == BC_INFLOW || code == BC_OUTFLOW || code == BC_SHOCK;
  }

  // phi of face t between A (lower) and B with half wavespeed w
  __device__ __forceinline__ void face(const LineNode& A, const LineNode& B, double w, int t) const {
    const double wv = visc || t == 0 || t == n ? signed_by(w, sg) : 0.0;
    double* ph = PH + f0 + fs * t;
    ph[0] = dfma(-wv, dsub(B.U[0], A.U[0]), half(dadd(A.U[1], B.U[1])));
    ph[(1 + ax) * NF] = dfma(-wv, dsub(B.U[1], A.U[1]), dadd(A.fn, B.fn));
    ph[(2 - ax) * NF] = dfma(-wv, dsub(B.U[2], A.U[2]), dadd(A.ft, B.ft));
    ph[3 * NF] = dfma(-wv, dsub(B.U[3], A.U[3]), dadd(A.fe, B.fe));
  }
  // high minus low order at a boundary face: the dissipation where the high-order flux has none
  __device__ __forceinline__ void face_diff(const LineNode& A, const LineNode& B, double w, bool off, int t) const {
    const double wv = signed_by(w, sg);
    double* df = DF + f0 + fs * t;
#pragma unroll
    for (int q = 0; q < 4; ++q) df[comp(q) * NF] = off ? dmul(wv, dsub(B.U[q], A.U[q])) : 0.0;
  }
  // the surface terms B f* of boundary face `side` for p2de_get_field, from phi and dF
  __device__ __forceinline__ void debug_surface(int side) const {
    const int f = f0 + fs * (side ? n : 0);
    const double gw = gd * op.w1D[l] * (side ? 1.0 : -1.0);
    const size_t g = ((size_t)k * Nfp + (2 * ax + side) * n + l) * 8;
    for (int c = 0; c < 4; ++c) {
      a.BFL[g + 4 * ax + c] = gw * PH[c * NF + f];
      a.BFH[g + 4 * ax + c] = gw * (PH[c * NF + f] + DF[c * NF + f]);
      a.BFL[g + 4 - 4 * ax + c] = a.BFH[g + 4 - 4 * ax + c] = 0.0;
    }
  }
  // node i's share of the CFL sum along this line: the half wavespeeds of its two faces
  __device__ __forceinline__ void cfl_sum(int i, double wl, double wr) const {
    base[Y::O_R + ax * Nq + q0 + qs * i] = dadd(wl, wr);
  }

  // the two-point flux of line nodes i > j; in FP32 (TH = float) already times its coefficient
  // and converted
  template <typename TH>
  __device__ __forceinline__ void pair(const Gas<float>& gf, int i, int j, double* F) const {
    const int mi = q0 + qs * i, mj = q0 + qs * j;
    if constexpr (sizeof(TH) == 8) {
      PairState qi, qj;
      pstate(mi, qi);
      pstate(mj, qj);
      fS_line(a.rgm1, qj, qi, &F[0], &F[2], &F[1], &F[3]);
    } else {
      const float* Wf = reinterpret_cast<const float*>(base + C::O_W + C::W_F32 * Nq);
      const float UJ[4] = {Wf[mj], Wf[Nq + mj], Wf[2 * Nq + mj], Wf[3 * Nq + mj]};
      const float UI[4] = {Wf[mi], Wf[Nq + mi], Wf[2 * Nq + mi], Wf[3 * Nq + mi]};
      const float c = op.hpcf[(ax * n + l) * C::PPL + i * (i - 1) / 2 + j];
      float G[4];
      fS_f32_axis(gf, UI, UJ, ax, G);
      F[0] = (double)__fmul_rn(c, G[0]);
      F[1] = (double)__fmul_rn(c, ax ? G[2] : G[1]);
      F[2] = (double)__fmul_rn(c, ax ? G[1] : G[2]);
      F[3] = (double)__fmul_rn(c, G[3]);
    }
  }
  // suffix sum s over the pairs (i.., j) of one component, started at i = n - 1
  template <typename TH>
  __device__ __forceinline__ double suffix(int i, int j, double F, double s) const {
    if constexpr (sizeof(TH) == 8) {
      const double c = op.hpc[(ax * n + l) * C::PPL + i * (i - 1) / 2 + j];
      return i == n - 1 ? dmul(c, F) : dfma(c, F, s);
    } else {
      return i == n - 1 ? F : dadd(s, F);
    }
  }
  __device__ __forceinline__ void pstate(int m, PairState& q) const {
    const double* W = base + C::O_W + m;
    q.rho = base[C::O_U + m];
    q.vn = W[(C::W_U + ax) * Nq];
    q.vt = W[(C::W_V - ax) * Nq];
    q.hn = W[ax * Nq];
    q.ht = W[(1 - ax) * Nq];
    q.beta = W[C::W_BETA * Nq];
    q.lr = W[C::W_LR * Nq];
    q.lb = W[C::W_LB * Nq];
  }
};

// The body for the elements k0 .. k0 + epb - 1 of the solve `a`; early returns are uniform
// over the block.
template <int N1D, typename TH, bool EXT, bool SPLIT = false>
__device__ __forceinline__ void flux_a_body(const StageArgs& a, int k0, double* sm) {
  using C = FluxCfg<N1D>;
  using Y = typename C::template Lay<EXT, SPLIT>;
  constexpr int n = C::n, Nq = C::Nq, Nfp = C::Nfp, NL = C::NL, NSF = C::NSF, NF = C::NF, NI = C::NI, PE = Y::PE;
  constexpr bool F32 = sizeof(TH) == 4;
  if (a.scal[S_DONE] != 0.0) return;
  const int E = a.epb;
  const int Ke = min(E, a.K - k0);
  if (Ke <= 0) return;
  int* s_cnt = reinterpret_cast<int*>(sm + PE * E);  // [0] faces, [1] bisections
  int* s_list = s_cnt + 4;
  int* s_bis = s_list + NF * E;
  const OpTable& op = *a.ops;
  const int tid = threadIdx.x, bs = blockDim.x;
  const int flags = EXT ? a.flags : (a.flags & ~kExtFlags);
  const double dt_lim = a.scal[S_DT_LIM];
  const double t_now = a.scal[S_T];
  const bool upper0 = flags & F_REF_SEM;

  // ---- node phase: the state and its primitives (calculate_primitive_variables!); per
  //      element and line position the coefficients c, s = 4 dt c and 1/s
  if (tid < 2) s_cnt[tid] = 0;
  for (int w = tid; w < Ke * NL; w += bs) {
    const int e = w / NL, r = w % NL, d = r / n, i = r % n;
    const double* gg = a.geom + 5 * (size_t)(k0 + e);
    const double rJ = a.geomx ? a.geomx[(size_t)(k0 + e) * kGeomStride + 11] : rcp(gg[0]);
    double* c = sm + e * PE + C::O_C + r;
    const double cd = dmul(-dmul(gg[d ? 4 : 1], rJ), op.rw1D[i]);
    const double s = dmul(4.0 * dt_lim, cd);
    c[0] = cd;
    c[2 * n] = s;
    if (!upper0) c[4 * n] = rcp(s);
  }
  // SPLIT deals a node's logarithms to other warps (part 1: log rho; part 2: beta, from its own
  // copy of p, and log beta), each part in whole warps
  constexpr int parts = SPLIT && !F32 ? 3 : 1;
  bool far = false;  // some state from which a flux may overflow
  const int n32 = parts == 1 ? Ke * Nq : (Ke * Nq + 31) & ~31;
  for (int v = tid; v < parts * n32; v += bs) {
    const int part = v / n32, w = v % n32;
    if (w >= Ke * Nq) continue;
    const int e = w / Nq, m = w % Nq;
    double* base = sm + e * PE;
    const double2* src = reinterpret_cast<const double2*>(a.Uq + ((size_t)k0 * Nq + w) * 4);
    const double2 v01 = src[0], v23 = src[1];
    const double rho = v01.x, m1 = v01.y, m2 = v23.x, En = v23.y;
    if (parts == 3 && part == 1) {
      base[C::O_W + C::W_LR * Nq + m] = log_fast(rho, op);
      continue;
    }
    double* U = base + C::O_U + m;
    double* W = base + C::O_W + m;
    const double rr = rcp(rho);
    // p to the bits of the nodal form: log means of nearly equal states amplify its last bit
    const double p = dmul(a.gm1, dfma(-0.5, dmul(dfma(m1, m1, dmul(m2, m2)), rr), En));
    if (parts == 3 && part == 2) {
      const double beta = dmul(rho, rcp(p));
      W[C::W_BETA * Nq] = beta;
      W[C::W_LB * Nq] = log_fast<true>(beta, op);
      continue;
    }
    U[0] = rho;
    U[Nq] = m1;
    U[2 * Nq] = m2;
    U[3 * Nq] = En;
    const double hr = half(rr);
    const double hu = dmul(m1, hr), hv = dmul(m2, hr);
    // rho in [2^-24, 2^24), p in [2^-40, 2^30), E < 2^30: no two-point flux of such states
    // overflows, in FP32 either (beta in [2^-55, 2^63], |u| <= 2^27.5, so the terms of the energy
    // flux stay below 2^108 / (gamma - 1))
    if (!((unsigned)(__double2hiint(rho) - (999 << 20)) < (48u << 20) &&
          (unsigned)(__double2hiint(p) - (983 << 20)) < (70u << 20) && __double2hiint(En) < (1053 << 20))) {
      far = true;
      // a state the reference would stop on (DomainError from log or sqrt of a negative,
      // flux_differencing.jl:49-50): density or pressure -0, negative or NaN
      if (!positive_bits(rho) || !positive_bits(p)) atomicOr(a.status, ST_NOT_POSITIVE);
    }
    W[C::W_HU * Nq] = hu;
    W[C::W_HV * Nq] = hv;
    W[C::W_PH * Nq] = half(p);
    W[C::W_CRR * Nq] = dmul(a.cws, rr);
    if (EXT && (flags & F_RELAXED) || (flags & F_SHOCK)) W[C::W_IND * Nq] = dmul(rho, p);  // shock_capture.jl:92-103
    if (F32) {
      // FP32 (rho, u, v, beta), converted once per node
      float* Wf = reinterpret_cast<float*>(base + C::O_W + C::W_F32 * Nq) + m;
      const float rf = (float)rho;
      Wf[0] = rf;
      Wf[Nq] = 2.0f * (float)hu;
      Wf[2 * Nq] = 2.0f * (float)hv;
      Wf[3 * Nq] = rf / (2.0f * (float)p);
    } else {
      W[C::W_U * Nq] = twice(hu);
      W[C::W_V * Nq] = twice(hv);
      if (parts == 1) {
        const double beta = dmul(rho, rcp(p));  // 2 beta of the reference
        W[C::W_BETA * Nq] = beta;
        W[C::W_LR * Nq] = log_fast(rho, op);
        W[C::W_LB * Nq] = log_fast<true>(beta, op);  // log of the reference's beta
      }
    }
  }
  const bool overflow = __syncthreads_or(far);

  // ---- smoothness indicator (shock_capture.jl:49-81): modal energies through inv(VDM), the
  //      Hennemann blending factor (:118-137) and the relaxed bounds' smoothness factor
  //      (subcell.jl:937-956)
  if (flags & (F_SHOCK | F_RELAXED)) {
    for (int w = tid; w < Ke * Nq; w += bs) {
      const int e = w / Nq, i = w % Nq;
      double* W = sm + e * PE + C::O_W;
      const double* Vi = op.VDMinv + i * Nq;
      double sum = 0.0;
      for (int j = 0; j < Nq; ++j) sum = dfma(Vi[j], W[C::W_IND * Nq + j], sum);
      W[C::W_EN * Nq + i] = dmul(sum, sum);
    }
    __syncthreads();
    for (int e = tid; e < Ke; e += bs) {
      double* base = sm + e * PE;
      double modeN = 0.0, modeNm1 = 0.0, total = 0.0;
      for (int j = 0; j < n; ++j)
        for (int i = 0; i < n; ++i) {
          const double energy = base[C::O_W + C::W_EN * Nq + i + n * j];
          if (i == n - 1 || j == n - 1) modeN = dadd(modeN, energy);
          if (i == n - 2 || j == n - 2) modeNm1 = dadd(modeNm1, energy);
          total = dadd(total, energy);
        }
      const double smooth = fmax(__ddiv_rn(modeN, total), __ddiv_rn(modeNm1, total));
      if (flags & F_SHOCK) {
        const double alpha = __ddiv_rn(1.0, dadd(1.0, exp(dmul(a.sc_q, dsub(smooth, a.sc_TN)))));
        base[Y::O_X + 3] = fmax(fmin(dsub(1.0, alpha), 1.0), 0.5);
      }
      if (flags & F_RELAXED) {
        // kappa = 1; log(10, x) = log(x) / log(10)
        const double sk = __ddiv_rn(log(smooth), 2.302585092994046);
        double eps;
        if (sk < a.s0 - 1.0)
          eps = 0.0;
        else if (sk > a.s0 + 1.0)
          eps = 1.0;
        else
          eps = dfma(-0.5, sin(dmul(3.141592653589793, dmul(dsub(sk, a.s0), 0.5))), 0.5);
        base[Y::O_X] = eps;
      }
    }
    __syncthreads();
  }

  // ---- lines: one thread per (element, direction, tangential node), or SPLIT (FluxLine)
  const bool low_only = flags & F_LOW_ONLY;
  const bool cfl = flags & F_CFL;
  const Gas<float> gf{a.gasf[0], a.gasf[1], a.gasf[2]};
  if constexpr (!SPLIT) {
    for (int w = tid; w < Ke * NL; w += bs) {
      const int e = w / NL, r = w % NL;
      FluxLine<N1D, Y> ln(a, op, sm + e * PE, k0 + e, r / n, r % n, t_now);
      {
        LineNode A, B, P;
        bool off;
        ln.load(0, A);
        ln.exterior(0, A, P, off);
        double wl = max_nonneg_bits(P.wh, A.wh);
        ln.face(P, A, wl, 0);
        ln.face_diff(P, A, wl, off, 0);
#pragma unroll
        for (int i = 1; i < n; ++i) {
          ln.load(i, B);
          const double wr = max_nonneg_bits(A.wh, B.wh);
          ln.face(A, B, wr, i);
          if (cfl) ln.cfl_sum(i - 1, wl, wr);
          wl = wr;
          A = B;
        }
        ln.exterior(1, A, P, off);
        const double wr = max_nonneg_bits(P.wh, A.wh);
        ln.face(A, P, wr, n);
        ln.face_diff(A, P, wr, off, n);
        if (cfl) ln.cfl_sum(n - 1, wl, wr);
      }
      if (low_only) continue;
      if (flags & F_WRITE_DEBUG) {
        ln.debug_surface(0);
        ln.debug_surface(1);
      }
      // high order: for j ascending, the suffix sums over i of c_ij fS(i, j), added to face i
      double acc[4][n];
#pragma unroll
      for (int j = 0; j < n - 1; ++j) {
        double s[4];
#pragma unroll
        for (int i = n - 1; i > j; --i) {
          double F[4];
          ln.template pair<TH>(gf, i, j, F);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            s[q] = ln.template suffix<TH>(i, j, F[q], s[q]);
            acc[q][i] = j == 0 ? s[q] : dadd(acc[q][i], s[q]);
          }
        }
      }
#pragma unroll
      for (int t = 1; t < n; ++t)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int f = ln.comp(q) * NF + ln.f0 + ln.fs * t;
          ln.DF[f] = upper0 ? acc[q][t] : dsub(acc[q][t], ln.PH[f]);
        }
    }
    __syncthreads();
  } else {
    // the same operations spread over more threads: (element, pair) fluxes, boundary faces and
    // along-axis node values, each in whole warps; then (element, line, component) sums
    const int np = low_only ? 0 : Ke * NL * C::PPL, nb = Ke * Nfp, nn = Ke * 2 * Nq;
    const int p32 = (np + 31) & ~31, b32 = (nb + 31) & ~31;
    for (int w = tid; w < p32 + b32 + nn; w += bs) {
      if (w < p32) {
        if (w >= np) continue;
        const int e = w / (NL * C::PPL), r = w % (NL * C::PPL), lr = r / C::PPL, pp = r % C::PPL;
        double* base = sm + e * PE;
        FluxLine<N1D, Y> ln(a, op, base, k0 + e, lr / n, lr % n, t_now);
        int i = 1;  // pair pp = i (i - 1) / 2 + j
        while (i * (i + 1) / 2 <= pp) ++i;
        double F[4];
        ln.template pair<TH>(gf, i, pp - i * (i - 1) / 2, F);
#pragma unroll
        for (int q = 0; q < 4; ++q) base[Y::O_SF + q * C::NPH + r] = F[q];
      } else if (w < p32 + b32) {
        const int v = w - p32;
        if (v >= nb) continue;
        const int e = v / Nfp, side = (v % Nfp) / NL, lr = v % NL;
        double* base = sm + e * PE;
        FluxLine<N1D, Y> ln(a, op, base, k0 + e, lr / n, lr % n, t_now);
        LineNode A, P;
        bool off;
        ln.load(side ? n - 1 : 0, A);
        ln.exterior(side, A, P, off);
        const double wv = max_nonneg_bits(P.wh, A.wh);
        const int t = side ? n : 0;
        ln.face(side ? A : P, side ? P : A, wv, t);
        ln.face_diff(side ? A : P, side ? P : A, wv, off, t);
        if (cfl) base[Y::O_SW + ln.f0 + ln.fs * t] = wv;
        if (!low_only && (flags & F_WRITE_DEBUG)) ln.debug_surface(side);
      } else {
        const int v = w - p32 - b32, e = v / (2 * Nq), r = v % (2 * Nq), ax = r / Nq, m = r % Nq;
        double* base = sm + e * PE;
        const double* W = base + C::O_W;
        LineNode A;
        A.U[1] = base[C::O_U + (1 + ax) * Nq + m];
        A.U[3] = base[C::O_U + 3 * Nq + m];
        line_node(A, W[ax * Nq + m], W[(1 - ax) * Nq + m], W[C::W_PH * Nq + m], W[C::W_CRR * Nq + m]);
        double* N = base + Y::O_SN + ax * 4 * Nq + m;
        N[0] = A.fn;
        N[Nq] = A.ft;
        N[2 * Nq] = A.fe;
        N[3 * Nq] = A.wh;
      }
    }
    __syncthreads();
    for (int w = tid; w < Ke * NL * 4; w += bs) {
      const int e = w / (NL * 4), lr = w % (NL * 4) / 4, q = w % 4;
      double* base = sm + e * PE;
      FluxLine<N1D, Y> ln(a, op, base, k0 + e, lr / n, lr % n, t_now);
      // the interior faces' low-order fluxes of component q (FluxLine::face, one component)
      const double* N = base + Y::O_SN + ln.ax * 4 * Nq;
      const double* Uq = base + C::O_U + ln.comp(q) * Nq;
      const double* Fq = q == 0 ? base + C::O_U + (1 + ln.ax) * Nq : N + (q - 1) * Nq;
      double* PH = ln.PH + ln.comp(q) * NF + ln.f0;
      double* DF = ln.DF + ln.comp(q) * NF + ln.f0;
      double uA = Uq[ln.q0], fA = Fq[ln.q0], wA = N[3 * Nq + ln.q0];
#pragma unroll
      for (int t = 1; t < n; ++t) {
        const int m = ln.q0 + ln.qs * t;
        const double uB = Uq[m], fB = Fq[m], wB = N[3 * Nq + m];
        const double wv = max_nonneg_bits(wA, wB);
        const double sum = dadd(fA, fB);
        PH[ln.fs * t] = dfma(-(ln.visc ? signed_by(wv, ln.sg) : 0.0), dsub(uB, uA), q == 0 ? half(sum) : sum);
        if (cfl && q == 0) base[Y::O_SW + ln.f0 + ln.fs * t] = wv;
        uA = uB;
        fA = fB;
        wA = wB;
      }
      if (low_only) continue;
      const double* F = base + Y::O_SF + q * C::NPH + lr * C::PPL;
      double acc[n];
#pragma unroll
      for (int j = 0; j < n - 1; ++j) {
        double s = 0.0;
#pragma unroll
        for (int i = n - 1; i > j; --i) {
          s = ln.template suffix<TH>(i, j, F[i * (i - 1) / 2 + j], s);
          acc[i] = j == 0 ? s : dadd(acc[i], s);
        }
      }
#pragma unroll
      for (int t = 1; t < n; ++t) DF[ln.fs * t] = upper0 ? acc[t] : dsub(acc[t], PH[ln.fs * t]);
    }
    __syncthreads();
  }

  // ---- node phase: low-order rhs (:139-243) and update, bounds' data, CFL
  double dt_loc = __longlong_as_double(0x7ff0000000000000LL);
  bool nan_seen = false;
  // the node's difference of the fluxes in A (PH or DF) along both lines
  auto divergence = [&](const double* base, const double* A, int m, int c) {
    const int ir = m % n, is = m / n;
    const double* fx = A + c * NF + (n + 1) * is + ir;
    const double* fy = A + c * NF + NSF + ir + n * is;
    return dfma(base[C::O_C + n + is], dsub(fy[n], fy[0]), dmul(base[C::O_C + ir], dsub(fx[1], fx[0])));
  };
  if constexpr (SPLIT) {  // one component per thread first
    for (int w = tid; w < Ke * Nq * 4; w += bs) {
      const int e = w / (Nq * 4), c = w % (Nq * 4) / Nq, m = w % Nq;
      double* base = sm + e * PE;
      const double rl = divergence(base, base + Y::O_PH, m, c);
      base[Y::O_R + c * Nq + m] = rl;
      base[C::O_W + (C::W_UL + c) * Nq + m] = dfma(dt_lim, rl, base[C::O_U + c * Nq + m]);
    }
    __syncthreads();
  }
  for (int w = tid; w < Ke * Nq; w += bs) {
    const int e = w / Nq, m = w % Nq, k = k0 + e;
    const int ir = m % n, is = m / n;
    double* base = sm + e * PE;
    const double* U = base + C::O_U + m;
    double* R = base + Y::O_R + m;
    double* W = base + C::O_W + m;
    if (flags & F_CFL) {
      double lx, ly;
      if constexpr (SPLIT) {
        const double* wx = base + Y::O_SW + (n + 1) * is + ir;
        const double* wy = base + Y::O_SW + NSF + ir + n * is;
        lx = dadd(wx[0], wx[1]);
        ly = dadd(wy[0], wy[n]);
      } else {
        lx = R[0];
        ly = R[Nq];
      }
      const double lam = dfma(fabs(base[C::O_C + n + is]), ly, dmul(fabs(base[C::O_C + ir]), lx));
      const double d = dmul(a.CFL * 0.5, rcp(lam));
      if (isnan(d)) nan_seen = true;
      dt_loc = fmin(dt_loc, d);
    }
    double uL[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if constexpr (SPLIT) {
        uL[c] = W[(C::W_UL + c) * Nq];
      } else {
        const double rl = divergence(base, base + Y::O_PH, m, c);
        R[c * Nq] = rl;
        uL[c] = dfma(dt_lim, rl, U[c * Nq]);
        W[(C::W_UL + c) * Nq] = uL[c];
      }
    }
    if (low_only) {  // the low-order densities for the TVD bounds (subcell.jl:112-125)
      a.rhoL[(size_t)k * Nq + m] = uL[0];
      continue;
    }
    // the internal-energy bound; under upper0 few faces ask for it, and the list forms it
    if (!upper0) energy_bound(uL, a.zeta, W[C::W_LRHOE * Nq], W[C::W_QC * Nq]);
    // global node index of stencil member t of low_order_stencil (limiter_utils.jl:222-231):
    // r-neighbours, then s-neighbours, across a face through mapP
    auto stencil = [&](int t) -> size_t {
      const int dir = t >> 1, up = t & 1;
      const int c = dir == 0 ? ir : is;
      if (up ? c < n - 1 : c > 0) return (size_t)k * Nq + m + (dir == 0 ? 1 : n) * (up ? 1 : -1);
      const int f = (2 * dir + up) * n + (dir == 0 ? is : ir);
      const int lin = a.nbr[(size_t)k * Nfp + f];
      const int kP = lin / Nfp, iP = lin % Nfp, sP = iP / n, tP = iP % n;
      const int qP = sP == 0 ? n * tP : sP == 1 ? (n - 1) + n * tP : sP == 2 ? tP : tP + n * (n - 1);
      return (size_t)kP * Nq + qP;
    };
    double lo = dmul(a.zeta, uL[0]), hi = __longlong_as_double(0x7ff0000000000000LL);
    if (flags & F_TVD) {
      // min/max of the low-order density over the node and its stencil (subcell.jl:112-141)
      lo = hi = a.rhoL[(size_t)k * Nq + m];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const double v = a.rhoL[stencil(t)];
        lo = fmin(lo, v);
        hi = fmax(hi, v);
      }
    }
    W[C::W_LRHO * Nq] = lo;
    W[C::W_URHO * Nq] = hi;
    if (flags & F_MIN_ENTROPY) {
      // initialize_lower_bound!(::Dim2) (subcell.jl:53-72): Lphi = eps_k min(phi over the
      // node and its stencil) + (1 - eps_k) phi_min; eps_k = 1 unless relaxed
      const double z[4] = {0.0, 0.0, 0.0, 0.0};
      const double Uo[4] = {U[0], U[Nq], U[2 * Nq], U[3 * Nq]};
      double lb = phi_at(Uo, z, 0.0, a.gamma, op);
#pragma unroll 1
      for (int t = 0; t < 4; ++t) lb = fmin(lb, phi_at(a.Uq + 4 * stencil(t), z, 0.0, a.gamma, op));
      if (flags & F_RELAXED) {
        const double eps = base[Y::O_X];
        lb = dfma(eps, lb, dmul(dsub(1.0, eps), a.phimin[0]));
      }
      W[C::W_THR * Nq] = dsub(lb, a.POSTOL);
    }
  }
  if (flags & F_CFL) {
    for (int o = 16; o > 0; o >>= 1) dt_loc = fmin(dt_loc, __shfl_xor_sync(0xffffffffu, dt_loc, o));
    if ((tid & 31) == 0) {
      if (dt_loc > 0.0) atomicMin(a.dtmin_bits, (unsigned long long)__double_as_longlong(dt_loc));
      else if (dt_loc <= 0.0) atomicOr(a.status, ST_BAD_DT);
    }
    if (nan_seen) atomicOr(a.status, ST_NAN);
  }
  if (low_only) return;
  __syncthreads();

  // ---- f_bar for p2de_get_field (after p2de_rhs, and the last stage of a step): per element
  //      [d][DF, phi_L][face][c], DF as O_DF has it here (under upper0 phi_H on interior faces);
  //      the debug fields of p2de_rhs
  const bool dbg = flags & F_WRITE_DEBUG, keep_fbar = dbg || ((flags & F_UPDATE) && a.nstage == 3);
  if (keep_fbar) {
    for (int w = tid; w < Ke * 16 * NSF; w += bs) {
      const int e = w / (16 * NSF), r = w % (16 * NSF);
      const int dh = r / (4 * NSF), f = (dh >> 1) * NSF + (r / 4) % NSF, c = r % 4;
      a.fbar[(size_t)k0 * 16 * NSF + w] = sm[e * PE + (dh & 1 ? Y::O_PH : Y::O_DF) + c * NF + f];
    }
  }
  if (dbg) {
    for (int w = tid; w < Ke * Nq * 4; w += bs) {
      const int e = w / (Nq * 4), m = (w / 4) % Nq, c = w % 4, ir = m % n, is = m / n;
      const double* base = sm + e * PE;
      const double* px = base + Y::O_PH + c * NF + (n + 1) * is + ir;
      const double* py = base + Y::O_PH + c * NF + NSF + ir + n * is;
      const double* dx = px + (Y::O_DF - Y::O_PH);
      const double* dy = py + (Y::O_DF - Y::O_PH);
      const double cx = base[C::O_C + ir], cy = base[C::O_C + n + is];
      const double lx = cx * (px[1] - px[0]), ly = cy * (py[n] - py[0]);
      // phi_H at the node's four faces
      const double x0 = !upper0 || ir == 0 ? px[0] + dx[0] : dx[0], x1 = !upper0 || ir == n - 1 ? px[1] + dx[1] : dx[1];
      const double y0 = !upper0 || is == 0 ? py[0] + dy[0] : dy[0], y1 = !upper0 || is == n - 1 ? py[n] + dy[n] : dy[n];
      const double hx = cx * (x1 - x0), hy = cy * (y1 - y0);
      const size_t g = ((size_t)k0 * Nq) * 8 + (w / 4) * 8 + c;
      a.rhsxyL[g] = lx;
      a.rhsxyL[g + 4] = ly;
      a.rhsxyH[g] = hx;
      a.rhsxyH[g + 4] = hy;
      a.rhsL[(size_t)k0 * Nq * 4 + w] = lx + ly;
      a.rhsH[(size_t)k0 * Nq * 4 + w] = hx + hy;
    }
  }

  if (keep_fbar && upper0) __syncthreads();  // the bounds turn DF into differences in place

  // ---- bounds (subcell_bound_limiter!(::Dim2), subcell.jl:288-345). A face's factor is the
  //      min over its one or two nodes: the lower node with P = s dF, the upper with -s dF.
  //      First the density bounds; only faces where neither is 0 go to the list, whose
  //      internal-energy quadratics (and min-entropy tests) run with all lanes busy.
  const bool minent = flags & F_MIN_ENTROPY;
  // face of item r: the interior faces first, then the boundary faces; its line position t
  auto face_of = [&](int r, int& d, int& t, int& l) {
    if (r < NI) {
      d = r / (NI / 2);
      const int q = r % (NI / 2);
      t = d == 0 ? q % (n - 1) + 1 : q / n + 1;
      l = d == 0 ? q / (n - 1) : q % n;
    } else {
      const int q = r - NI;
      d = q / (2 * n);
      t = (q / n) % 2 ? n : 0;
      l = q % n;
    }
    return d == 0 ? t + (n + 1) * l : NSF + l + n * t;
  };
  // node on side h of the face (0: below it, whose upper face it is), or -1
  auto node_of = [&](int d, int t, int l, int h) {
    const int i = t - 1 + h;
    if (i < 0 || i >= n) return -1;
    return d == 0 ? i + n * l : l + n * i;
  };
  for (int w = tid; w < Ke * NF; w += bs) {
    // items of all elements' interior faces, then of all their boundary faces
    const int e = w < Ke * NI ? w / NI : (w - Ke * NI) / (NF - NI);
    const int r = w < Ke * NI ? w % NI : NI + (w - Ke * NI) % (NF - NI);
    int d, t, l;
    const int f = face_of(r, d, t, l);
    double* base = sm + e * PE;
    double* DF = base + Y::O_DF + f;
    const double blend = (flags & F_SHOCK) ? base[Y::O_X + 3] : 1.0;
    double L = blend;
    double* PHf = base + Y::O_PH + f;
    const bool inner = r < NI;
    // the sign of P0 = +-s dF0 settles the bound of one of an interior face's two nodes under
    // upper0; dF0 = phi_H0 - phi_L0 is negative where its terms compare so
    bool zero = false;
    if (upper0) {
      const long long hb = __double_as_longlong(DF[0]), lb = inner ? __double_as_longlong(PHf[0]) : 0;
      const bool finite = (hb & 0x7ff0000000000000LL) != 0x7ff0000000000000LL &&
                          (lb & 0x7ff0000000000000LL) != 0x7ff0000000000000LL;
      const bool neg = inner ? order_key(DF[0]) < order_key(PHf[0]) : hb < 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = node_of(d, t, l, h);
        if (m < 0 || !finite) continue;
        const double s = base[C::O_C + 2 * n + d * n + t - 1 + h];
        const bool down = neg != (negative(s) != (h == 1));  // P0 has its sign bit set
        zero = zero || (!down && zero_factor(base[C::O_W + C::W_UL * Nq + m], s, base[C::O_W + C::W_LRHO * Nq + m]));
      }
    }
    if (upper0 && !zero && inner) {
#pragma unroll
      for (int c = 0; c < 4; ++c) DF[c * NF] = dsub(DF[c * NF], PHf[c * NF]);
    }
    if (!zero) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = node_of(d, t, l, h);
        if (m < 0) continue;
        const double* W = base + C::O_W + m;
        const double s = base[C::O_C + 2 * n + d * n + t - 1 + h];
        const double P0 = dmul(h ? -s : s, DF[0]);
        const double lm = density_bound(W[C::W_UL * Nq], P0, W[C::W_LRHO * Nq], upper0 ? 0.0 : W[C::W_URHO * Nq], upper0,
                                        dmul(0.5, W[C::W_UL * Nq]));
        L = min_nonneg_bits(L, fmin(lm, 1.0));
      }
    }
    if (zero) L = -0.0;  // DF still the high-order flux
    base[Y::O_L + f] = L;
    if (is_zero_bits(L)) continue;
    // dF = 0 (most boundary faces): P = 0 leaves the quadratics' factor 1
    if (!minent && is_zero_bits(DF[0]) && is_zero_bits(DF[NF]) && is_zero_bits(DF[2 * NF]) && is_zero_bits(DF[3 * NF]))
      continue;
    s_list[atomicAdd(&s_cnt[0], 1)] = e * NF + r;
  }
  __syncthreads();
  const int nlist = s_cnt[0];
  for (int w = tid; w < nlist; w += bs) {
    const int e = s_list[w] / NF;
    int d, t, l;
    const int f = face_of(s_list[w] % NF, d, t, l);
    double* base = sm + e * PE;
    const double* DFp = base + Y::O_DF + f;
    const double dF[4] = {DFp[0], DFp[NF], DFp[2 * NF], DFp[3 * NF]};
    const double A = dfma(dF[0], dF[3], dmul(-0.5, dfma(dF[1], dF[1], dmul(dF[2], dF[2]))));
    const double a4 = dmul(4.0, A), r2a = rcp(dmul(2.0, A));
    double L = base[Y::O_L + f];
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      const int m = node_of(d, t, l, h);
      if (m < 0) continue;
      const double* W = base + C::O_W + m;
      const double uL[4] = {W[0], W[Nq], W[2 * Nq], W[3 * Nq]};
      double s = base[C::O_C + 2 * n + d * n + t - 1 + h];
      double is = upper0 ? rcp(s) : base[C::O_C + 4 * n + d * n + t - 1 + h];
      if (h) s = -s, is = -is;
      double Lrhoe, qc;
      if (upper0) {
        energy_bound(uL, a.zeta, Lrhoe, qc);
      } else {
        Lrhoe = W[C::W_LRHOE * Nq];
        qc = W[C::W_QC * Nq];
      }
      double lm = rhoe_root(uL, dF, a4, r2a, qc, Lrhoe, s, is, a.ZEROTOL);
      // the second solve of limiting_param_bound_rho_rhoe: Urhoe = Urho_i (the TVD upper
      // density bound) under the reference semantics, else Inf, for which it returns 1.0
      if (upper0 && (flags & F_TVD)) {
        const double ub = W[C::W_URHO * Nq];
        const double c = dfma(uL[0], dsub(uL[3], ub), dmul(-0.5, dfma(uL[1], uL[1], dmul(uL[2], uL[2]))));
        lm = fmin(lm, rhoe_root(uL, dF, a4, r2a, c, ub, s, is, a.ZEROTOL));
      }
      if (minent) {
        // min-entropy bounds (limiter_utils.jl:19-50): the factor so far is lpos; a node that
        // fails phi >= Lphi - POSTOL there goes to the list of bisections
        const double P[4] = {dmul(s, dF[0]), dmul(s, dF[1]), dmul(s, dF[2]), dmul(s, dF[3])};
        const double lden = density_bound(uL[0], P[0], W[C::W_LRHO * Nq], W[C::W_URHO * Nq], false, 0.0);
        lm = fmin(fmin(lden, lm), 1.0);
        if (!(phi_at(uL, P, lm, a.gamma, op) >= W[C::W_THR * Nq])) {
          const int id = 2 * s_list[w] + h;
          base[C::O_W + (C::W_EV + 2 * d + h) * Nq + m] = lm;
          s_bis[atomicAdd(&s_cnt[1], 1)] = id;
          continue;
        }
      }
      L = min_nonneg_bits(L, fmin(lm, 1.0));
    }
    base[Y::O_L + f] = L;
  }
  if (a.counters && tid == 0 && nlist) atomicAdd(&a.counters[0], (unsigned long long)nlist);
  __syncthreads();
  if (EXT && minent) {
    // bisection (nonlinear_solvers.jl:3-20) on the grid of 21 halvings of [0, lpos]
    const int nbis = s_cnt[1];
    for (int w = tid; w < nbis; w += bs) {
      const int h = s_bis[w] & 1, e = (s_bis[w] >> 1) / NF;
      int d, t, l;
      const int f = face_of((s_bis[w] >> 1) % NF, d, t, l);
      double* base = sm + e * PE;
      const int m = node_of(d, t, l, h);
      const double* W = base + C::O_W + m;
      const double uL[4] = {W[0], W[Nq], W[2 * Nq], W[3 * Nq]};
      const double* DFp = base + Y::O_DF + f;
      double s = base[C::O_C + 2 * n + d * n + t - 1 + h];
      if (h) s = -s;
      const double P[4] = {dmul(s, DFp[0]), dmul(s, DFp[NF]), dmul(s, DFp[2 * NF]), dmul(s, DFp[3 * NF])};
      double* ev = base + C::O_W + (C::W_EV + 2 * d + h) * Nq + m;
      const double thr = W[C::W_THR * Nq];
      double good = 0.0, bad = *ev;
      for (int it = 0; it <= 20; ++it) {
        const double mid = dmul(0.5, dadd(good, bad));
        if (phi_at(uL, P, mid, a.gamma, op) >= thr)
          good = mid;
        else
          bad = mid;
      }
      *ev = good;
    }
    __syncthreads();
    for (int w = tid; w < nbis; w += bs) {  // the face's min, over its one or two bisections
      const int h = s_bis[w] & 1, e = (s_bis[w] >> 1) / NF;
      int d, t, l;
      const int f = face_of((s_bis[w] >> 1) % NF, d, t, l);
      double* base = sm + e * PE;
      const double ev = base[C::O_W + (C::W_EV + 2 * d + h) * Nq + node_of(d, t, l, h)];
      atomicMin(reinterpret_cast<long long*>(base + Y::O_L + f), __double_as_longlong(ev));
    }
    __syncthreads();
  }

  // ---- cell entropy bound (enforce_ES_subcell!, subcell.jl:462-744), in the oracle's order
  //      of sums; the per-face products on all lanes, the greedy per element and direction
  if (flags & F_CELL_ENTROPY) {
    constexpr int M = Nq - n;  // interior subcell faces per direction
    constexpr int O_DV = C::O_W + 4 * Nq, O_DL = O_DV + 2 * M, O_BP = O_DL + 2 * M, O_KEY = O_BP + 4 * n,
                  O_ORD = O_KEY + 2 * M;
    static_assert(4 * Nq + 7 * M + 4 * n <= 12 * Nq, "cell-entropy scratch fits the node data");
    // an element-direction whose interior factors are all zero has sum(L dvdf) = 0 (or NaN)
    // and the check of subcell.jl:676-677 is false: nothing to do
    for (int w = tid; w < Ke * 2; w += bs) {
      const int e = w / 2, d = w % 2;
      double* base = sm + e * PE;
      bool any = false;
      for (int q = 0; q < M; ++q) {
        int dd, t, l;
        const int f = face_of(d * M + q, dd, t, l);
        if (!is_zero_bits(base[Y::O_L + f])) any = true;
      }
      base[Y::O_X + 1 + d] = any ? 1.0 : 0.0;
    }
    __syncthreads();
    // entropy variables v_ufun (compressible_Navier_Stokes.jl:134-144); s = log(p) - gamma log(rho)
    for (int w = tid; w < Ke * Nq; w += bs) {
      const int e = w / Nq, m = w % Nq;
      double* base = sm + e * PE;
      if (is_zero_bits(base[Y::O_X + 1]) && is_zero_bits(base[Y::O_X + 2])) continue;
      const double* U = base + C::O_U + m;
      const double ke = dadd(dmul(U[Nq], U[Nq]), dmul(U[2 * Nq], U[2 * Nq]));
      const double p = dmul(a.gm1, dsub(U[3 * Nq], __ddiv_rn(dmul(0.5, ke), U[0])));
      const double s = dsub(log_fast(p, op), dmul(a.gamma, log_fast(U[0], op)));
      const double rp = rcp(p);
      double* vq = base + C::O_W + m;
      vq[0] = dsub(dsub(dadd(a.gamma, 1.0), s), dmul(dmul(a.gm1, U[3 * Nq]), rp));
      vq[Nq] = dmul(dmul(U[Nq], a.gm1), rp);
      vq[2 * Nq] = dmul(dmul(U[2 * Nq], a.gm1), rp);
      vq[3 * Nq] = dmul(dmul(-U[0], a.gm1), rp);
    }
    __syncthreads();
    // per interior face dvdf, its sort key (Julia's isless order: NaN above everything) and
    // dv . f_bar_L (subcell.jl:540-562); per boundary face node of the direction, B psi
    // (:521-529). dvdf index of a face: x, (si-1) + (n-1) sj; y, si + n (sj-1).
    for (int w = tid; w < Ke * 2 * (M + 2 * n); w += bs) {
      const int e = w / (2 * (M + 2 * n)), r = w % (2 * (M + 2 * n));
      const int d = r / (M + 2 * n), j = r % (M + 2 * n);
      double* base = sm + e * PE;
      if (is_zero_bits(base[Y::O_X + 1 + d])) continue;
      const double gd = a.geom[5 * (size_t)(k0 + e) + (d ? 4 : 1)];
      if (j < M) {
        int dd, t, l;
        const int f = face_of(d * M + j, dd, t, l);
        const double gw = -dmul(gd, op.w1D[l]);
        const double* vm = base + C::O_W + node_of(d, t, l, 0);
        const double* vp = base + C::O_W + node_of(d, t, l, 1);
        const double* DF = base + Y::O_DF + f;
        const double* PH = base + Y::O_PH + f;
        const bool raw = negative(base[Y::O_L + f]);
        double sd = 0.0, sl = 0.0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const double dv = dsub(vm[c * Nq], vp[c * Nq]);
          const double df = raw ? dsub(DF[c * NF], PH[c * NF]) : DF[c * NF];
          sd = c ? dfma(dv, df, sd) : dmul(dv, df);
          sl = c ? dfma(dv, PH[c * NF], sl) : dmul(dv, PH[0]);
        }
        const double dvdf = dmul(gw, sd);
        base[O_DV + d * M + j] = dvdf;
        base[O_DL + d * M + j] = dmul(gw, sl);
        const long long bits = __double_as_longlong(dvdf);
        reinterpret_cast<long long*>(base + O_KEY)[d * M + j] =
            (bits & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL ? 0x7fffffffffffffffLL : order_key(dvdf);
      } else {
        const int q = j - M, side = q / n, l = q % n;  // side 0 low, 1 high
        const int m = d == 0 ? (side ? n - 1 : 0) + n * l : l + (side ? n * (n - 1) : 0);
        const double B = dmul(gd, side ? op.w1D[l] : -op.w1D[l]);
        base[O_BP + d * 2 * n + q] = dmul(B, dmul(a.gm1, base[C::O_U + (1 + d) * Nq + m]));
      }
    }
    __syncthreads();
    // the descending sort of (dvdf, index) (sort!(rev = true), subcell.jl:676-741) as ranks
    for (int w = tid; w < Ke * 2 * M; w += bs) {
      const int e = w / (2 * M), r = w % (2 * M), d = r / M, i = r % M;
      double* base = sm + e * PE;
      if (is_zero_bits(base[Y::O_X + 1 + d])) continue;
      const long long* key = reinterpret_cast<const long long*>(base + O_KEY) + d * M;
      const long long ki = key[i];
      int rank = 0;
#pragma unroll
      for (int j = 0; j < M; ++j) rank += (key[j] > ki || (key[j] == ki && j > i)) ? 1 : 0;
      reinterpret_cast<int*>(base + O_ORD)[d * M + rank] = i;
    }
    __syncthreads();
    for (int w = tid; w < Ke * 2; w += bs) {
      const int e = w / 2, d = w % 2;
      double* base = sm + e * PE;
      if (is_zero_bits(base[Y::O_X + 1 + d])) continue;
      double sB = 0.0;
      for (int q = 0; q < 2 * n; ++q) sB = dadd(sB, base[O_BP + d * 2 * n + q]);
      const double* dvdf = base + O_DV + d * M;
      double* L = base + Y::O_L;
      auto face_of_idx = [&](int idx) {
        int dd, t, l;
        return face_of(d * M + idx, dd, t, l);
      };
      // sum_dvfbarL and sum of L dvdf (subcell.jl:540-562, 654-670) in the reference's order:
      // x: line outer, face inner; y: line outer, face inner
      double sdl = 0.0, sumLd = 0.0;
      for (int a2 = 0; a2 < n; ++a2)
        for (int b2 = 1; b2 < n; ++b2) {
          const int idx = d == 0 ? (b2 - 1) + (n - 1) * a2 : a2 + n * (b2 - 1);
          sdl = dadd(sdl, base[O_DL + d * M + idx]);
          sumLd = dadd(sumLd, dmul(L[face_of_idx(idx)], dvdf[idx]));
        }
      double rhs = dsub(sB, sdl);
      // rhs_es of the relaxed bounds (subcell.jl:750-753)
      if (flags & F_RELAXED) rhs = dmul(dsub(1.0, dmul(a.beta, base[Y::O_X])), rhs);
      const double est = dsub(sumLd, rhs);
      const double tol = jmax(0.0, dsub(sdl, sB));
      if (est > tol) {
        const int* ord = reinterpret_cast<const int*>(base + O_ORD) + d * M;
        int curr = 0;
        double lhs = sumLd;
        const double target = dadd(rhs, tol);
        while (lhs > target && curr < M) {
          const int idx = ord[curr];
          if (dvdf[idx] < a.ZEROTOL) break;
          lhs = dsub(lhs, dmul(L[face_of_idx(idx)], dvdf[idx]));
          ++curr;
        }
        for (int i2 = 0; i2 < curr; ++i2) {
          const int idx = ord[i2], f = face_of_idx(idx);
          const double l_new = (i2 == curr - 1) ? jmax(__ddiv_rn(dsub(target, lhs), dvdf[idx]), 0.0) : 0.0;
          L[f] = jmin(L[f], l_new);
        }
      }
    }
    __syncthreads();
  }

  // ---- limited fluxes (accumulate_f_bar_limited!, subcell.jl:841-876): phi + l dF where the
  //      face blends anything. A boundary face with dF != 0 is its own neighbour, so its
  //      factor is final here; the others' factors multiply 0. Where a flux may overflow, all
  //      faces: 0 x Inf = NaN ends the step. (DMR 480x120, FP64: 595 us a stage with the lines
  //      looking at their high-order fluxes, 589 with the node phase looking at the states,
  //      590 with neither.)
  for (int w = tid; w < Ke * NF; w += bs) {
    const int e = w < Ke * NI ? w / NI : (w - Ke * NI) / (NF - NI);
    const int r = w < Ke * NI ? w % NI : NI + (w - Ke * NI) % (NF - NI);
    int d, t, l;
    const int f = face_of(r, d, t, l);
    double* base = sm + e * PE;
    const double L = base[Y::O_L + f];
    double* PH = base + Y::O_PH + f;
    const double* DF = base + Y::O_DF + f;
    const bool on = overflow || (!is_zero_bits(L) && (r < NI || !(is_zero_bits(DF[0]) && is_zero_bits(DF[NF]) &&
                                                                  is_zero_bits(DF[2 * NF]) && is_zero_bits(DF[3 * NF]))));
    if (on) {
#pragma unroll
      for (int c = 0; c < 4; ++c) PH[c * NF] = dfma(L, DF[c * NF], PH[c * NF]);
    }
    a.Lpre[(size_t)(k0 + e) * NF + f] = fabs(L);
    // the face's mark for the node phase below (dF is no longer needed)
    base[Y::O_DF + f] = on ? 1.0 : 0.0;
  }
  __syncthreads();
  // ---- rhsU (apply_subcell_limiter!, subcell.jl:894-924): the low-order rhs where none of the
  //      node's faces blends, else the difference of the limited fluxes
  for (int w = tid; w < Ke * Nq; w += bs) {
    const int e = w / Nq, m = w % Nq, ir = m % n, is = m / n;
    const double* base = sm + e * PE;
    const double* fx = base + Y::O_DF + (n + 1) * is + ir;
    const double* fy = base + Y::O_DF + NSF + ir + n * is;
    const bool on = !(is_zero_bits(fx[0]) && is_zero_bits(fx[1]) && is_zero_bits(fy[0]) && is_zero_bits(fy[n]));
    double ru[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) ru[c] = on ? divergence(base, base + Y::O_PH, m, c) : base[Y::O_R + c * Nq + m];
    double2* dst = reinterpret_cast<double2*>(a.rhsU + ((size_t)k0 * Nq + w) * 4);
    dst[0] = make_double2(ru[0], ru[1]);
    dst[1] = make_double2(ru[2], ru[3]);
  }
}

template <int N1D, typename TH, bool EXT, bool SPLIT = false>
__global__ void __launch_bounds__(FluxCfg<N1D>::THREADS) k_flux_a(StageArgs a) {
  extern __shared__ __align__(16) double sm[];
  flux_a_body<N1D, TH, EXT, SPLIT>(a, blockIdx.x * a.epb, sm);
}

// =====================================================================================
// Kernel B after it: SSP-RK3 stage combination (SSPRK33.jl:127-135), the symmetrized factors
// and the stage's positivity record, for the elements k0 .. k0 + epb - 1
// =====================================================================================
template <int N1D>
__device__ __forceinline__ void flux_b_body(const StageArgs& a, int k0) {
  using C = FluxCfg<N1D>;
  constexpr int n = C::n, Nq = C::Nq, Nfp = C::Nfp, NSF = C::NSF, NF = C::NF;
  if (a.scal[S_DONE] != 0.0) return;
  const int tid = threadIdx.x, bs = blockDim.x;
  const int Ke = min(a.epb, a.K - k0);
  if (Ke <= 0) return;
  const int s = a.nstage - 1;
  const double dt = a.nstage == 1 ? __longlong_as_double((long long)*a.dtmin_bits) : a.scal[S_DT];
  // symmetrize_limiting_parameters!(::Dim2) with subcell_index_P_x/y (limiter_utils.jl:179-237)
  for (int w = tid; w < Ke * NF; w += bs) {
    const int e = w / NF, r = w % NF, d = r / NSF, fi = r % NSF, k = k0 + e;
    const int t = d == 0 ? fi % (n + 1) : fi / n, l = d == 0 ? fi / (n + 1) : fi % n;
    double L = a.Lpre[(size_t)k0 * NF + w];
    if (t == 0 || t == n) {
      const int lin = a.nbr[(size_t)k * Nfp + (2 * d + (t == n)) * n + l];
      const int kP = lin / Nfp, iP = lin % Nfp, lP = iP % n;
      const int idxP = d == 0 ? (iP / n == 0 ? 0 : n) + (n + 1) * lP : lP + n * (iP / n == 2 ? 0 : n);
      L = fmin(L, a.Lpre[(size_t)kP * NF + d * NSF + idxP]);
    }
    a.Lfin[((size_t)s * a.K + k0) * NF + w] = L;
  }
  if (!(a.flags & F_UPDATE)) return;
  long long rmin = order_key(__longlong_as_double(0x7ff0000000000000LL)), emin = rmin;
  for (int w = tid; w < Ke * Nq; w += bs) {
    const size_t g = ((size_t)k0 * Nq + w) * 4;
    double2* Up = reinterpret_cast<double2*>(a.Uq + g);
    double2* Wp = reinterpret_cast<double2*>(a.resW + g);
    const double2* Rp = reinterpret_cast<const double2*>(a.rhsU + g);
    const double2 u0 = Up[0], u1 = Up[1], r0 = Rp[0], r1 = Rp[1];
    double U[4] = {u0.x, u0.y, u1.x, u1.y};
    const double R[4] = {r0.x, r0.y, r1.x, r1.y};
    if (a.nstage == 1) {
      Wp[0] = u0;
      Wp[1] = u1;
#pragma unroll
      for (int c = 0; c < 4; ++c) U[c] = dfma(dt, R[c], U[c]);
    } else {
      const double2 w0 = Wp[0], w1 = Wp[1];
      const double W0[4] = {w0.x, w0.y, w1.x, w1.y};
      const double cw = a.nstage == 2 ? 3.0 / 4.0 : 1.0 / 3.0, cz = a.nstage == 2 ? 1.0 / 4.0 : 2.0 / 3.0;
#pragma unroll
      for (int c = 0; c < 4; ++c) U[c] = dfma(cw, W0[c], dmul(cz, dfma(dt, R[c], U[c])));
    }
    Up[0] = make_double2(U[0], U[1]);
    Up[1] = make_double2(U[2], U[3]);
    const double re = dfma(-0.5, dmul(dfma(U[1], U[1], dmul(U[2], U[2])), rcp(U[0])), U[3]);  // rhoe_ufun(U)
    const long long kr = order_key(U[0]), ke = order_key(re);
    rmin = kr < rmin ? kr : rmin;
    emin = ke < emin ? ke : emin;
    if (!positive_bits(U[0]) || !positive_bits(re)) atomicOr(a.status, ST_NOT_POSITIVE);
  }
  for (int o = 16; o > 0; o >>= 1) {
    const long long x = __shfl_xor_sync(0xffffffffu, rmin, o), y = __shfl_xor_sync(0xffffffffu, emin, o);
    rmin = x < rmin ? x : rmin;
    emin = y < emin ? y : emin;
  }
  if ((tid & 31) == 0) {
    // most warps do not lower the minima: look before the atomic (they only ever fall)
    if (rmin < *(volatile long long*)&a.minrec[2 * s]) atomicMin(&a.minrec[2 * s], rmin);
    if (emin < *(volatile long long*)&a.minrec[2 * s + 1]) atomicMin(&a.minrec[2 * s + 1], emin);
  }
  if (k0 == 0 && tid == 0) {
    if (a.nstage == 1) {
      a.scal[S_DT] = dt;
      a.scal[S_DT_LIM] = dt;
    }
    if (a.nstage == 3) {
      a.scal[S_T] = a.scal[S_T] + dt;
      a.scal[S_STEPS] = a.scal[S_STEPS] + 1.0;
    }
  }
}

template <int N1D>
__global__ void __launch_bounds__(256) k_flux_b(StageArgs a) {
  flux_b_body<N1D>(a, blockIdx.x * a.epb);
}

}  // namespace p2de
