// The fused passes: one right-hand side and Runge-Kutta stage of the general
// gas (one to twelve species, calorically or thermally perfect, any flux
// function and reconstruction, inviscid or viscous, coupled chemistry) in
// four to seven launches over every block instead of the per-block path's
// fourteen:
//
//   k_rcell   per interior cell: fromQ (the eos's Newton from the cell's last
//             T), then the transport properties and species enthalpies (the
//             per-block path's k_fromQ then k_transport, one thread doing both
//             on the state it just formed)
//             (peregrine/simulator/euler/kernels/state/fromQ.mako:5-19,
//              peregrine/simulator/navstokes/kernels/transport.mako:5-35);
//   k_halo_fields  Q's halo and every field's, in one pass over the halo's
//             boxes (uniface.cuh); a shard, whose traded halo cells get Q
//             alone, fills Q's first and forms the cells over the halo too;
//   k_source  the coupled chemistry source beginning dQ, as on the per-block
//             path (peregrine/simulator/chemint/kernels/source.mako:3-10);
//   k_ufaces  uniform blocks: the faces of all three axes, without gradient
//             arrays (uniface.cuh);
//   k_grads, k_rface  the other blocks: the cell gradients and their first
//             halo layer, then one face a thread, the advective flux and the
//             diffusive rows in the same thread, stored once (the per-block
//             path stores the advective flux, then reads and stores it again
//             with the diffusive rows added);
//   k_rapply  per cell: the divergence added to the source and the stage's
//             combines, with dQ kept in the thread and never stored
//             (peregrine/simulator/advec/kernels/applyflux.mako:2-11,
//              peregrine/integrators/kernels/combine.mako:1-13).
//
// The cells and the general faces run the per-block kernels' own device
// functions in the same order, the uniform faces the same arithmetic without
// its zeros; the two paths' results agree to rounding.
//
// Measured and set aside: (a) the chemistry source in the cell kernel, the
// rate state then spilling to local memory, 0.80 ms a pass at 96^3 against
// 0.52 ms for the three passes apart; (b) one tile kernel of every face of a
// plane marching up k with the face fluxes in shared memory and the cell
// records read through L1: at 252 registers a face, one CTA of eight warps
// an SM could not hide the face's two hundred global loads, 4.6 ms a stage
// against 1.0 ms for the three face passes; (c) the three axes' faces in one
// launch ordered slab by slab, so a slab's cell records are read by all its
// faces while in L2: 5.3 to 5.8 ms an RK3 step over slabs of 2 to 96 planes
// against 5.4 ms for the passes per axis (the face passes wait on load
// latency, not on DRAM bandwidth); the plain axis-after-axis launch kept here
// saves the two tails, which small cases feel.
#pragma once
#include "chem.cuh"
#include "layout.cuh"
#include "physics.cuh"
#include "plain.cuh"
#include "plain_api.h"
#include "uniface.cuh"

namespace pgb {

// fromQ and the transport of one cell (k_fromQ then k_transport); t over the
// block's full extents, or, with INNER, over its interior cells (a halo
// cell's values are then its source's, copied after)
template <int NS, bool VISC, bool INNER = false>
__global__ void __launch_bounds__(256) k_rcell(const BlockDev *__restrict__ blks, int b,
                                               const double *__restrict__ Qall, double *__restrict__ stall,
                                               double *__restrict__ trall, double *__restrict__ hall,
                                               const int uvel, const int2 *__restrict__ ctab = nullptr) {
  constexpr int NE = 4 + NS;
  PGB_WHERE(B, tt);
  long long t = tt;
  if (INNER) {
    if (tt >= (long long)B.nx * B.ny * B.nz) return;
    t = inner_cell(B, tt);
  } else if (t >= B.vol) {
    return;
  }
  const long long v = B.vol;
  const double *Q = Qall + NE * B.cv + t;
  double *st = stall + SW * B.cv + t;
  auto Qf = [&](int c) { return Q[c * v]; };
  const State s = fromQ<NS>(Qf, st[1 * v]);
  st[0 * v] = s.p, st[1 * v] = s.T, st[2 * v] = s.rhoinv, st[3 * v] = s.rho;
  st[4 * v] = s.e, st[5 * v] = s.cp, st[6 * v] = s.gamma, st[7 * v] = s.c;
  if (uvel) {
    // the velocity the uniform faces read (uniface.cuh)
#pragma unroll
    for (int m = 0; m < 3; m++) st[(ST_U + m) * v] = Qf(1 + m) * s.rhoinv;
  }
  if (VISC) {
    double tr[2 + NS], h[NS];
    transport<NS, decltype(Qf), false>(Qf, s, tr, h, 0.0);
    double *trp = trall + (2 + NS) * B.cv + t;
    double *hp = hall + NS * B.cv + t;
#pragma unroll
    for (int n = 0; n < 2 + NS; n++) trp[n * v] = tr[n];
#pragma unroll
    for (int n = 0; n < NS; n++) hp[n * v] = h[n];
  }
}

// what the divergence-and-combine pass reads: dQ (the coupled source on the
// way in, and dQ out when write_dq), the step size and the stage's combines
struct RApplyArgs {
  double *dQ;
  const double *dt;
  int chem;      // 1: dQ holds the source the divergence adds to
  int write_dq;  // 1: store dQ (the right-hand side alone)
  int ncomb;
  RCombine comb[2];
};

// the face of axis A whose high-side cell is R: the advective flux (kepaec on
// the cells as they are, or a Riemann solver FN on the cells or MUSCL's
// sides), then with VISC the diffusive rows added, into F[NE]
template <int NS, int A, int FN, bool VISC>
__device__ __forceinline__ void rface(const BlockDev &B, const double *Q, const double *st, const double *tr,
                                      const double *hs, const double *gr, const double *M, const int lim,
                                      const long long R, double *F) {
  if (FN == 0) advflux_face<NS, A>(B, Q, st, M, R, F);
  else riemann_face<NS, A, FN, false, false>(B, Q, st, M, lim, R, F);
  if (VISC) {
    // the diffusive rows' loads (two cells' gradients, transport and
    // enthalpies) are not hoisted above the advective flux: in flight all at
    // once they would hold twice the registers
    asm volatile("" ::: "memory");
    diffflux_face<NS, A>(B, Q, st, tr, hs, gr, M, R, F);
  }
}

// One face a thread: the advective flux and, with VISC, the diffusive rows in
// the same thread, stored once (the per-block path's k_riemann then
// k_diffflux, without the flux's round trip between them).  All three axes'
// faces in one launch, the CTAs of an axis together: no axis waits for the
// last CTAs of the one before, which on small cases is most of a pass
template <int NS, int FN, bool KOREN, bool VISC>
__global__ void __launch_bounds__(RF_TH, 4) k_rface(const BlockDev *__restrict__ blks, const double *__restrict__ Qall,
                                                  const double *__restrict__ stall, const double *__restrict__ trall,
                                                  const double *__restrict__ hall, const double *__restrict__ gall,
                                                  const double *__restrict__ met, double *F0, double *F1, double *F2,
                                                  const int limiter, const int skipu, const unsigned n0, const unsigned n1,
                                                  const int2 *__restrict__ ctab) {
  constexpr int NE = 4 + NS, NGRAD = NE - 1;
  const int lim = KOREN ? LIM_KOREN : limiter;
  unsigned t;
  int row;
  const int axis = face_work(n0, n1, ctab, row, t);
  const BlockDev &B = blks[row];
  // the uniform blocks' faces are k_ufaces'
  if (skipu && B.uniform) return;
  long long R;
  int pos;
  if (!face_cell(B, axis, t, R, pos)) return;
  double F[NE];
  const double *Q = Qall + NE * B.cv, *st = stall + SW * B.cv, *M = met + M_NCOMP * B.cv;
  const double *tr = VISC ? trall + (2 + NS) * B.cv : nullptr, *hs = VISC ? hall + NS * B.cv : nullptr;
  const double *gr = VISC ? gall + 3 * NGRAD * B.cv : nullptr;
  if (axis == 0) rface<NS, 0, FN, VISC>(B, Q, st, tr, hs, gr, M, lim, R, F);
  else if (axis == 1) rface<NS, 1, FN, VISC>(B, Q, st, tr, hs, gr, M, lim, R, F);
  else rface<NS, 2, FN, VISC>(B, Q, st, tr, hs, gr, M, lim, R, F);
  double *Fo = (axis == 0 ? F0 : axis == 1 ? F1 : F2) + NE * B.cv + R;
#pragma unroll
  for (int l = 0; l < NE; l++) Fo[l * B.vol] = F[l];
}

// The divergence added to the source (the per-block applyflux's order) and the
// stage's combines, RA_COMPS components of a cell a thread (the grid's plane
// the group).  A cell a thread walked its components one after another, the
// loads of each behind the stores of the last: 65 us for 64^3 of nine species
// and 18 for 53 x 45 x 61 of two; a component a thread spent most of its
// instructions finding its cell, 42 and 14.7; a group, 40 and 12.5, the first
// near the 25 its bytes take.
constexpr int RA_COMPS = 4;
template <int NS>
__global__ void __launch_bounds__(256) k_rapply(const BlockDev *__restrict__ blks, int b, const double *__restrict__ Fi,
                                                const double *__restrict__ Fj, const double *__restrict__ Fk,
                                                const double *__restrict__ met, const RApplyArgs a,
                                                const int2 *__restrict__ ctab = nullptr) {
  constexpr int NE = 4 + NS;
  PGB_WHERE(B, t);
  if (t >= (long long)B.nx * B.ny * B.nz) return;
  const long long c = inner_cell(B, t), v = B.vol;
  const long long sJ = B.X, sK = (long long)B.X * B.Y;
  const int l0 = (int)blockIdx.z * RA_COMPS;
  const double detJinv = met[M_NCOMP * B.cv + M_DETJINV * v + c];
  const double dt = *a.dt;
  const long long at0 = NE * B.cv + l0 * v + c;
  double dq[RA_COMPS], first[RA_COMPS];
#pragma unroll
  for (int l = 0; l < RA_COMPS; l++) {
    if (l0 + l >= NE) break;
    const long long at = at0 + l * v;
    const double *fi = Fi + at, *fj = Fj + at, *fk = Fk + at;
    const double f = fi[0] + fj[0] + fk[0] - fi[1] - fj[sJ] - fk[sK];
    dq[l] = a.chem ? div_onto(a.dQ[at], f, detJinv) : div_begin(f, detJinv);
  }
  if (a.write_dq) {
#pragma unroll
    for (int l = 0; l < RA_COMPS; l++)
      if (l0 + l < NE) a.dQ[at0 + l * v] = dq[l];
  }
  for (int m = 0; m < a.ncomb; m++) {
    const RCombine &cb = a.comb[m];
    double acc[RA_COMPS];
    for (int n = 0; n < cb.nterms; n++) {
      const double w = term_weight(cb.w[n], cb.step && n == cb.nterms - 1, dt);
      const int src = cb.src[n];
      const double *X = cb.X[n];
#pragma unroll
      for (int l = 0; l < RA_COMPS; l++) {
        if (l0 + l >= NE) break;
        const double x = src == -1 ? dq[l] : src == -2 ? first[l] : X[at0 + l * v];
        acc[l] = n == 0 ? term_first(w, x) : term_next(acc[l], w, x);
      }
    }
#pragma unroll
    for (int l = 0; l < RA_COMPS; l++) {
      if (l0 + l >= NE) break;
      if (m == 0) first[l] = acc[l];
      if (cb.write) cb.out[at0 + l * v] = acc[l];
    }
  }
}

// What a double-flux face reads of a cell: velocity, pressure, density and its
// reciprocal, the carried mass fractions and the frozen plane
template <int NS>
struct DFCell {
  double u, v, w, p, rho, ri, th, ep, ka;
  double Y[NS > 1 ? NS - 1 : 1], ze[NS > 1 ? NS - 1 : 1];
};

// the cell at c (an index into the block's arrays Q and st, component stride
// v), its pressure in the state's field pf
template <int NS>
__device__ __forceinline__ DFCell<NS> df_cell(const double *__restrict__ Q, const double *__restrict__ st,
                                              const long long v, const long long c, const int pf) {
  DFCell<NS> x;
  const double q0 = Q[c], q1 = Q[v + c], q2 = Q[2 * v + c], q3 = Q[3 * v + c];
  x.p = st[pf * v + c];
  x.th = st[ST_THETA * v + c], x.ep = st[ST_EPS * v + c], x.ka = st[ST_KAPPA * v + c];
#pragma unroll
  for (int n = 0; n < NS - 1; n++) x.Y[n] = Q[(5 + n) * v + c], x.ze[n] = st[(ST_ZETA + n) * v + c];
  x.rho = q0;
  x.ri = 1.0 / q0;
  x.u = q1 * x.ri, x.v = q2 * x.ri, x.w = q3 * x.ri;
#pragma unroll
  for (int n = 0; n < NS - 1; n++) x.Y[n] *= x.ri;
  return x;
}

// the double flux's kepaec of the face between L and R (advflux_df_face,
// plain.cuh), the energy row in R's frozen plane with RPLANE, else in L's
template <int NS, bool RPLANE>
__device__ __forceinline__ void df_face(const DFCell<NS> &L, const DFCell<NS> &R, const double S0, const double S1,
                                        const double S2, double *F) {
  const double uf = 0.5 * (R.u + L.u), vf = 0.5 * (R.v + L.v), wf = 0.5 * (R.w + L.w);
  const double U = S0 * uf + S1 * vf + S2 * wf;
  const double pf = 0.5 * (R.p + L.p);
  const double C = 0.5 * (R.rho + L.rho) * U;
  F[0] = C;
  F[1] = C * uf + pf * S0;
  F[2] = C * vf + pf * S1;
  F[3] = C * wf + pf * S2;
  const double Kj = C * 0.5 * (R.u * L.u + R.v * L.v + R.w * L.w);
  const double Pj = 0.5 * (L.p * (R.u * S0 + R.v * S1 + R.w * S2) + R.p * (L.u * S0 + L.v * S1 + L.w * S2));
  const DFCell<NS> &P = RPLANE ? R : L;
  double comp = 0.0;
#pragma unroll
  for (int n = 0; n < NS - 1; n++) {
    const double Ys = R.Y[n] + L.Y[n];
    F[5 + n] = 0.5 * Ys * C;
    comp += P.ze[n] * Ys;
  }
  const double tL = (P.th * L.p + P.ka) * L.ri, tR = (P.th * R.p + P.ka) * R.ri;
  F[4] = (P.ep + 0.5 * comp + 2.0 * tL * tR / (tL + tR)) * C + Kj + Pj;
}

// The double flux's stage for an inviscid gas with kepaec, a cell a thread:
// its six faces' two-point fluxes (each face formed by both cells it joins;
// kepaec reads the two cells alone), the divergence in the per-block
// applyflux_df's order (the energy row takes the second energy row on the
// cell's low faces, where it is the right cell, the first on its high
// faces), and the stage's combines
// (peregrine/simulator/eulerdf/kernels/flux/function/kepaec.mako:1-21,
//  peregrine/simulator/eulerdf/kernels/applyflux.mako:2-14).
//
// The cell is read once and kept for its six faces, a neighbour's velocity is
// its momentum times one reciprocal, and a face's energy is formed in this
// cell's plane alone: 7 cells' loads and 19 divisions where each face reading
// its two cells took 12 and 72.  A face reads no thermodynamics but p (field
// pf of the state), which comes off the frozen plane, so with pto >= 0 the
// cell's p for the next stage is formed here from combine pm's new Q, into
// field pto: that stage then needs no state pass.
template <int NS>
__global__ void __launch_bounds__(128) k_rcellflux_df(const BlockDev *__restrict__ blks, int b,
                                                      const double *__restrict__ Qall, double *__restrict__ stall,
                                                      const double *__restrict__ met, const RApplyArgs a,
                                                      const int pf, const int pto, const int pm) {
  constexpr int NE = 4 + NS;
  const BlockDev &B = blks[b + (int)blockIdx.y];
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)B.nx * B.ny * B.nz) return;
  const long long c = inner_cell(B, t), v = B.vol;
  const double *Q = Qall + NE * B.cv, *M = met + M_NCOMP * B.cv;
  double *st = stall + SW * B.cv;
  const DFCell<NS> me = df_cell<NS>(Q, st, v, c, pf);
  // the faces one after another, each summed in as it is formed, in the
  // divergence's order (low i, j, k faces added, high ones taken off)
  double acc[NE];
#pragma unroll
  for (int l = 0; l < NE; l++) acc[l] = 0.0;
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int A = f % 3;
    const bool low = f < 3;
    const long long d = A == 0 ? 1 : A == 1 ? B.X : (long long)B.X * B.Y;
    const long long at = low ? c : c + d;
    double S[3] = {0.0, 0.0, 0.0};
    // on a uniform block the component along the axis is all of the area
    if (B.uniform) {
      S[A] = M[(M_S + 4 * A) * v + at];
    } else {
#pragma unroll
      for (int e = 0; e < 3; e++) S[e] = M[(M_S + 3 * A + e) * v + at];
    }
    const DFCell<NS> nb = df_cell<NS>(Q, st, v, low ? c - d : c + d, pf);
    double F[NE];
    if (low) df_face<NS, true>(nb, me, S[0], S[1], S[2], F);
    else df_face<NS, false>(me, nb, S[0], S[1], S[2], F);
#pragma unroll
    for (int l = 0; l < NE; l++) acc[l] = f == 0 ? F[l] : low ? acc[l] + F[l] : acc[l] - F[l];
  }
  const double detJinv = M[M_DETJINV * v + c];
  const long long at = NE * B.cv + c;
  const double dt = *a.dt;
  double first[NE], qn[NE];
#pragma unroll
  for (int l = 0; l < NE; l++) {
    const double dq = div_begin(acc[l], detJinv);
    if (a.write_dq) a.dQ[at + l * v] = dq;
    for (int m = 0; m < a.ncomb; m++) {
      const RCombine &cb = a.comb[m];
      auto val = [&](int n) {
        const int s = cb.src[n];
        return s == -1 ? dq : s == -2 ? first[l] : cb.X[n][at + l * v];
      };
      auto weight = [&](int n) { return term_weight(cb.w[n], cb.step && n == cb.nterms - 1, dt); };
      double acc = term_first(weight(0), val(0));
      for (int n = 1; n < cb.nterms; n++) acc = term_next(acc, weight(n), val(n));
      if (m == 0) first[l] = acc;
      if (m == pm) qn[l] = acc;
      if (cb.write) cb.out[at + l * v] = acc;
    }
  }
  if (pto >= 0) {
    // pplane (peregrine/simulator/mixture/eos/realgasdf/kernels/eos.mako:50-56)
    double comp = 0.0;
#pragma unroll
    for (int n = 0; n < NS - 1; n++) comp += me.ze[n] * qn[5 + n];
    st[pto * v + c] = (qn[4] - 0.5 * (qn[1] * qn[1] + qn[2] * qn[2] + qn[3] * qn[3]) / qn[0] - me.ep * qn[0] - comp -
                       me.ka) / me.th;
  }
}

// Closed constant-volume reactors, a cell each, for the serving pool: a
// uniform closed box has no flux divergence, so a reactor's stage is fromQ
// (the Newton from its last T), the finite-rate source and the stage's
// combines, in one thread (the reference's auto-ignition case, a closed
// box of Euler and chemistry, examples/autoIgnition.py:33-56; the coupled
// source, peregrine/simulator/chemint/kernels/source.mako:3-10).  A
// reactor's registers hold it at row r of a [component][capacity] table.
template <int NS>
__global__ void __launch_bounds__(256) k_reactors(const ReactorStage a) {
  constexpr int NE = 4 + NS;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n) return;
  const long long r = a.rows[t], cap = a.cap;
  auto Qf = [&](int c) { return a.Q[c * cap + r]; };
  const State s = fromQ<NS>(Qf, a.T[r]);
  a.T[r] = s.T;
  double omega[NS];
  cellrates<NS>(Qf, s.T, omega);
  const double dt = *a.dt;
  double first[NE];
#pragma unroll
  for (int l = 0; l < NE; l++) {
    const double dq = l < 5 ? 0.0 : omega[l - 5];
    const long long at = l * cap + r;
    for (int m = 0; m < a.ncomb; m++) {
      const RCombine &cb = a.comb[m];
      auto val = [&](int n) {
        const int src = cb.src[n];
        return src == -1 ? dq : src == -2 ? first[l] : cb.X[n][at];
      };
      auto weight = [&](int n) { return term_weight(cb.w[n], cb.step && n == cb.nterms - 1, dt); };
      double acc = term_first(weight(0), val(0));
      for (int n = 1; n < cb.nterms; n++) acc = term_next(acc, weight(n), val(n));
      if (m == 0) first[l] = acc;
      if (cb.write) cb.out[at] = acc;
    }
  }
}

// A warp per reactor: every lane forms the same clipped mass fractions, state
// and rate state; the lanes take the reactions' rates of progress k, k + 32,
// ... (the mechanism's global copy, lanes reading different reactions),
// staged in shared memory; then every lane sums the fold in reaction order,
// as cellrates' fold does (the same products and sums in the same order: the
// same bits), and lane l writes component l's combines.
template <int NS>
__global__ void __launch_bounds__(256) k_reactors_warp(const ReactorStage a) {
  constexpr int NE = 4 + NS;
  __shared__ double sh[8][MAXRXN];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 8 + w;
  if (t >= a.n) return;  // a warp's lanes alike
  const long long r = a.rows[t], cap = a.cap;
  auto Qf = [&](int c) { return a.Q[c * cap + r]; };
  const State st = fromQ<NS>(Qf, a.T[r]);
  // cellrates: the clipped mass fractions and the rate state
  const double rho = Qf(0), rhoinv = 1.0 / rho;
  double Ylast = 1.0, Ysum = 0.0;
#pragma unroll
  for (int n = 0; n < NS - 1; n++) {
    const double Yn = fmax(fmin(Qf(5 + n) * rhoinv, 1.0), 0.0);
    Ylast -= Yn;
    Ysum += Yn;
  }
  const double Yscale = 1.0 / fmax(Ysum, 1.0);
  Ylast = fmax(Ylast, 0.0);
  auto Y = [&](int n) { return n < NS - 1 ? fmax(fmin(Qf(5 + n) * rhoinv, 1.0), 0.0) * Yscale : Ylast; };
  RateState<NS> s;
  ratestate<NS>(s, rho, Y, st.T);
  const int nr = kMech.nr;
  for (int k = lane; k < nr; k += 32) {
    const Rxn &rx = gMech.rxn[k];
    double fwd, rev;
    oneway<NS>(rx, s, fwd, rev);
    sh[w][k] = rx.reversible ? fwd - rev : fwd;
  }
  __syncwarp();
  double omega[NS];
#pragma unroll
  for (int n = 0; n < NS; n++) omega[n] = 0.0;
  for (int k = 0; k < nr; k++) {
    const Rxn &rx = kMech.rxn[k];
    const double rp = sh[w][k];
    for (int j = 0; j < rx.nnet; j++) omega[rx.netsp[j]] += rx.netnuMW[j] * rp;
  }
  // every lane has read T above; one writes the new guess
  if (lane == 0) a.T[r] = st.T;
  if (lane >= NE) return;
  const int l = lane;
  const double dt = *a.dt;
  double dq = 0.0;
#pragma unroll
  for (int n = 0; n < NS; n++)
    if (l == 5 + n) dq = omega[n];
  const long long at = l * cap + r;
  double first = 0.0;
  for (int m = 0; m < a.ncomb; m++) {
    const RCombine &cb = a.comb[m];
    auto val = [&](int n) {
      const int src = cb.src[n];
      return src == -1 ? dq : src == -2 ? first : cb.X[n][at];
    };
    auto weight = [&](int n) { return term_weight(cb.w[n], cb.step && n == cb.nterms - 1, dt); };
    double acc = term_first(weight(0), val(0));
    for (int n = 1; n < cb.nterms; n++) acc = term_next(acc, weight(n), val(n));
    if (m == 0) first = acc;
    if (cb.write) cb.out[at] = acc;
  }
}

// a reactor's Q and starting T from its primitives p, u, v, w, T, Y...
// (the reference's fromprims, peregrine/simulator/euler/kernels/state/fromprims.mako)
template <int NS>
__global__ void k_reactor_prims(const double *__restrict__ prims, double *__restrict__ Q, double *__restrict__ T,
                                const int row, const long long cap) {
  constexpr int NE = 4 + NS;
  double q[NE], Qc[NE];
#pragma unroll
  for (int l = 0; l < NE; l++) q[l] = prims[l];
  const State th = fromprims<NS>(q, Qc);
#pragma unroll
  for (int l = 0; l < NE; l++) Q[l * cap + row] = Qc[l];
  T[row] = th.T;
}

}  // namespace pgb
