// The fused passes' faces on uniform blocks: every face's area vector along
// its own axis, the cells evenly spaced (BlockDev.uniform), so the face's
// gradients need no gradient arrays.  One launch forms the faces of all three
// axes of every uniform block, a face a thread.
//
// With the zero metrics left out, alpha damping along axis A
// (peregrine/simulator/navstokes/kernels/flux/alpha-damping.mako:13-58) reads
// of the species and the temperature only their derivative along A, which is
// the central difference of the four cells LL, L, R, RR the reconstruction
// reads anyway, and of the velocity four derivatives across it, formed here
// from the neighbours' velocities.  The general faces (k_rface, react.cuh)
// read 185 doubles a face of nine species, 72 of them gradients and 12
// metrics; these read 98, and the stage needs no gradient pass and no
// gradient halo.  With Lewis diffusion the species' coefficients are one
// value over the Lewis numbers, so one of the NS is read.
//
// The species are walked twice, so few of their values are live at once: the
// first walk takes the diffusion fluxes and the moments of both
// reconstructed sides, the second the upwind side's mass fraction, whose
// flux is the mass flux times it for HLLC and AUSM+-up (both waves of HLLC's
// star form sum to the star mass flux), a blend of both for Rusanov.
#pragma once
#include "layout.cuh"
#include "physics.cuh"
#include "plain.cuh"

namespace pgb {

constexpr int UF_TH = RF_TH;  // threads a CTA
constexpr int UF_UNROLL = 2;  // species a turn of the walks

// one side's mixture as the walk over the species gathers it: R, h298 and
// cp's coefficients in ln T (thermally perfect; a fit's terms past its own
// are stored as zeros) or cp alone in cc[0]
template <bool TPG>
struct SideMix {
  static constexpr int NT = TPG ? MAXT : 1;
  double R, h298, cc[NT];
  __device__ __forceinline__ void zero() {
    R = h298 = 0.0;
#pragma unroll
    for (int t = 0; t < NT; t++) cc[t] = 0.0;
  }
  __device__ __forceinline__ void add(const int n, const double Y) {
    R = fma(Y, kSp.Rsp[n], R);
    h298 = fma(Y, kSp.h298R[n], h298);
#pragma unroll
    for (int t = 0; t < NT; t++) cc[t] = fma(Y, TPG ? kSp.cppolyR[n * MAXT + t] : kSp.cp0[n], cc[t]);
  }
  // frompT (physics.cuh) from the gathered moments
  __device__ __forceinline__ void close(const double p, const double T, RSide &s) const {
    double c, h;
    if (TPG) {
      const double u = log(T) - kSp.lnT0;
      double hcoeff = 0.0;
      c = h = 0.0;
#pragma unroll
      for (int m = NT - 1; m >= 0; m--) {
        c = c * u + cc[m];
        hcoeff = cc[m] - (m + 1) * hcoeff;
        h = h * u + hcoeff;
      }
      h = h * T + h298;
    } else {
      c = cc[0];
      h = c * T + h298;
    }
    const double RT = R * T;
    s.p = p;
    s.rho = p / RT;
    s.e = h - RT;
    s.c = sqrt(c / (c - R) * RT);
  }
};

// HLLC, Rusanov and AUSM+-up (physics.cuh:hllc, rusanov, ausmup) on an area
// vector S along axis A: F[0..4], and the species' flux as a YL + b YR
template <int FN, int A>
__device__ __forceinline__ void riemann_axis(const RSide &L, const RSide &R, const double S, double *F, double &a,
                                             double &b) {
  const double area = fabs(S), sg = S < 0.0 ? -1.0 : 1.0;
  const double unL = sg * (A == 0 ? L.u : A == 1 ? L.v : L.w), unR = sg * (A == 0 ? R.u : A == 1 ? R.v : R.w);
  if (FN == FN_HLLC) {
    const double SL = unL - L.c, SR = unR + R.c;
    const double mL = L.rho * (SL - unL), mR = R.rho * (SR - unR);
    const double Sstar = (R.p - L.p + mL * unL - mR * unR) / (mL - mR);
    const bool left = SL >= 0.0 || Sstar >= 0.0;
    const bool star = left ? SL < 0.0 : SR >= 0.0;
    const double rho = left ? L.rho : R.rho, p = left ? L.p : R.p, e = left ? L.e : R.e;
    const double u = left ? L.u : R.u, v = left ? L.v : R.v, w = left ? L.w : R.w;
    const double U = left ? unL : unR, SX = left ? SL : SR;
    const double et = e + 0.5 * (u * u + v * v + w * w);
    const double mdot = U * rho * area;
    F[0] = mdot;
    F[1] = mdot * u, F[2] = mdot * v, F[3] = mdot * w;
    F[1 + A] += p * S;
    F[4] = mdot * et + U * p * area;
    if (star) {
      const double rhostar = rho * ((SX - U) / (SX - Sstar));
      const double drho = rhostar - rho, dU = rhostar * (Sstar - U);
      const double jump = SX * area;
      F[0] += jump * drho;
      F[1] += jump * (drho * u + (A == 0 ? dU * sg : 0.0));
      F[2] += jump * (drho * v + (A == 1 ? dU * sg : 0.0));
      F[3] += jump * (drho * w + (A == 2 ? dU * sg : 0.0));
      F[4] += jump * (drho * et + dU * (Sstar + p / (rho * (SX - U))));
    }
    a = left ? F[0] : 0.0;
    b = left ? 0.0 : F[0];
  } else if (FN == FN_RUSANOV) {
    const double lam = fmax(fabs(unL) + L.c, fabs(unR) + R.c) * area;
    const double UL = unL * area, UR = unR * area;
    a = 0.5 * L.rho * (UL + lam), b = 0.5 * R.rho * (UR - lam);
    F[0] = a + b;
    F[1] = a * L.u + b * R.u, F[2] = a * L.v + b * R.v, F[3] = a * L.w + b * R.w;
    F[1 + A] += 0.5 * (L.p + R.p) * S;
    const double eL = L.e + 0.5 * (L.u * L.u + L.v * L.v + L.w * L.w);
    const double eR = R.e + 0.5 * (R.u * R.u + R.v * R.v + R.w * R.w);
    F[4] = a * eL + b * eR + 0.5 * (UR * R.p + UL * L.p);
  } else {
    const double zero[1] = {0.0};
    const double Sv[3] = {A == 0 ? S : 0.0, A == 1 ? S : 0.0, A == 2 ? S : 0.0};
    ausmup<1>(L, R, zero, zero, Sv, F);
    const bool left = F[0] > 0.0;
    a = left ? F[0] : 0.0;
    b = left ? 0.0 : F[0];
  }
}

// the face of axis A of a uniform block whose high-side cell is R into
// F[NE]; FN 0 is kepaec on the cells as they are, else a Riemann solver on
// MUSCL's sides under limiter lim.  Q, st, tr, hs the block's own arrays;
// st's fields ST_U.. hold the cells' velocities.  gr, when given, holds the
// cells' velocity gradients (a bounded block's: its halo cells' are set by the
// boundaries); lo, hi: the low or high cell is a boundary's halo cell whose
// gradient is the other's.  M the block's metrics, of which the face reads its
// own area: a block is uniform to 1e-12, and its first face's area for every
// face put that much of p times an area into the momentum, 3.4e-13 of it after
// five RK3 steps of the 192 x 96 x 96 channel where the face's own leaves
// 2.7e-14 (against float64 off each cell's own; 14.5 ms for 14.3).
template <int NS, int A, int FN, bool KOREN, bool VISC, bool TPG>
__device__ __forceinline__ void uface(const BlockDev &B, const double *__restrict__ Q, const double *__restrict__ st,
                                      const double *__restrict__ tr, const double *__restrict__ hs, const double *__restrict__ gr,
                                      const double *__restrict__ M, const bool lo, const bool hi, const int limiter,
                                      const long long R, double *__restrict__ Fo, double *sh) {
  const int lim = KOREN ? LIM_KOREN : limiter;
  constexpr int B1 = (A + 1) % 3, B2 = (A + 2) % 3;
  const int step[3] = {1, B.X, B.X * B.Y};
  const int d = step[A];
  const long long v = B.vol;
  Q += R, st += R;
  const double S = M[(M_S + 4 * A) * v + R];
  double F[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  double rho = 0.0, kor = 0.0;
  const double hJ = 0.5 * B.Jd[A];
  // the derivative along A from LL, L, R, RR: the sides' mean, damped toward
  // the jump the sides' extrapolations leave at the face
  const double damp = VISC ? B.damp[A] : 0.0, xL = B.xL[A], xR = B.xR[A];
  auto along = [&](const double LL, const double L, const double Rr, const double RR) {
    const double dL = hJ * (Rr - LL), dR = hJ * (RR - L), gL = lo ? dR : dL, gR = hi ? dL : dR;
    return 0.5 * (gR + gL) + damp * ((Rr + gR * xR) - (L + gL * xL));
  };
  if (VISC) {
    tr += R, hs += R;
    const double mu = 0.5 * (tr[0] + tr[-d]), kappa = 0.5 * (tr[v] + tr[v - d]);
    rho = 0.5 * (Q[0] + Q[-d]);
    kor = 0.5 * kSp.lewis[0] * (tr[2 * v] + tr[2 * v - d]);
    const double lambda = 0.0 - 2.0 / 3.0 * mu;
    double g[3];  // the velocity's derivatives along A
    double uf[3];
#pragma unroll
    for (int m = 0; m < 3; m++) {
      const double *u = st + (ST_U + m) * v;
      const double uL = u[-d], uR = u[0];
      g[m] = along(u[-2 * d], uL, uR, u[d]);
      uf[m] = 0.5 * (uR + uL);
    }
    // across A: the mean of the two cells' central differences
    auto across = [&](const int m, const int b) {
      if (gr) return 0.5 * (gr[(3 * m + b) * v + R] + gr[(3 * m + b) * v + R - d]);
      const double *u = st + (ST_U + m) * v;
      const int s = step[b];
      const double gL = u[s - d] - u[-s - d], gR = u[s] - u[-s];
      return 0.25 * B.Jd[b] * (gR + gL);
    };
    const double d1 = across(B1, B1), d2 = across(B2, B2), a1 = across(A, B1), a2 = across(A, B2);
    const double div = g[A] + d1 + d2;
    double t[3];
    t[A] = -2.0 * mu * g[A] - lambda * div;
    t[B1] = -mu * (g[B1] + a1);
    t[B2] = -mu * (g[B2] + a2);
#pragma unroll
    for (int m = 0; m < 3; m++) F[1 + m] = t[m] * S;
    const double *T = st + v;
    const double heat = -kappa * (along(T[-2 * d], T[-d], T[0], T[d]) * S);
    F[4] = (uf[0] * t[0] + uf[1] * t[1] + uf[2] * t[2]) * S + heat;
  }
  // the first walk over the species: the diffusion fluxes, the sides' moments
  SideMix<TPG> ml, mr;
  if (FN) ml.zero(), mr.zero();
  double Vc = 0.0, gradYns = 0.0, sumYh = 0.0, Yns = 1.0, YlastL = 1.0, YlastR = 1.0;
  const double riLL = st[2 * v - 2 * d], riL = st[2 * v - d], riR = st[2 * v], riRR = st[2 * v + d];
  if (VISC || FN) {
#pragma unroll UF_UNROLL
    for (int n = 0; n < NS - 1; n++) {
      const double *q = Q + (5 + n) * v;
      const double LL = q[-2 * d] * riLL, L = q[-d] * riL, Rr = q[0] * riR, RR = q[d] * riRR;
      if (FN) {
        const double yl = muscl_left(lim, LL, L, Rr), yr = muscl_right(lim, L, Rr, RR);
        ml.add(n, yl), mr.add(n, yr);
        YlastL -= yl, YlastR -= yr;
      }
      if (VISC) {
        const double D = kor * kSp.lewisinv[n];
        const double gradY = along(LL, L, Rr, RR) * S;
        gradYns -= gradY;
        Vc += D * gradY;
        const double h = 0.5 * (hs[n * v] + hs[n * v - d]), Yk = 0.5 * (Rr + L);
        const double J = -rho * D * gradY;
        sh[n * UF_TH] = J;
        Yns -= Yk;
        sumYh += Yk * h;
        F[4] += J * h;
      }
    }
    if (FN) ml.add(NS - 1, YlastL), mr.add(NS - 1, YlastR);
  }
  double corr = 0.0;
  if (VISC) {
    constexpr int n = NS - 1;
    const double D = kor * kSp.lewisinv[n];
    Vc += D * gradYns;
    corr = rho * Vc;
    const double h = 0.5 * (hs[n * v] + hs[n * v - d]);
    F[4] += corr * sumYh + (-rho * D * gradYns + Yns * corr) * h;
  }
  // the advective flux, F[0..4] added, the species' by a YL + b YR
  double a, b;
  if (FN == 0) {
    auto side = [&](const int o) {
      KSide x;
      x.u = st[ST_U * v + o], x.v = st[(ST_U + 1) * v + o], x.w = st[(ST_U + 2) * v + o];
      x.p = st[o], x.rho = st[3 * v + o], x.e = st[4 * v + o];
      x.th = st[5 * v + o] / st[6 * v + o] * st[v + o];
      return x;
    };
    const KSide l = side(-d), r = side(0);
    double G[5], C;
    kepaec(l, r, A == 0 ? S : 0.0, A == 1 ? S : 0.0, A == 2 ? S : 0.0, G, C);
#pragma unroll
    for (int q = 0; q < 5; q++) F[q] += G[q];
    a = b = 0.5 * C;
  } else {
    RSide l, r;
    auto sides = [&](const double *f, double &fl, double &fr) {
      const double LL = f[-2 * d], L = f[-d], Rr = f[0], RR = f[d];
      fl = muscl_left(lim, LL, L, Rr), fr = muscl_right(lim, L, Rr, RR);
    };
    double pl, pr, Tl, Tr;
    sides(st, pl, pr);
    sides(st + v, Tl, Tr);
    ml.close(pl, Tl, l);
    mr.close(pr, Tr, r);
    sides(st + ST_U * v, l.u, r.u);
    sides(st + (ST_U + 1) * v, l.v, r.v);
    sides(st + (ST_U + 2) * v, l.w, r.w);
    double G[5];
    riemann_axis<FN, A>(l, r, S, G, a, b);
#pragma unroll
    for (int q = 0; q < 5; q++) F[q] += G[q];
  }
  Fo += R;
#pragma unroll
  for (int q = 0; q < 5; q++) Fo[q * v] = F[q];
  // the second walk: the advected mass fraction and the correction velocity's share
#pragma unroll UF_UNROLL
  for (int n = 0; n < NS - 1; n++) {
    const double *q = Q + (5 + n) * v;
    const double L = q[-d] * riL, Rr = q[0] * riR;
    double f;
    if (FN == 0) {
      f = a * (Rr + L);
    } else if (FN == FN_RUSANOV) {
      const double LL = q[-2 * d] * riLL, RR = q[d] * riRR;
      f = a * muscl_left(lim, LL, L, Rr) + b * muscl_right(lim, L, Rr, RR);
    } else {
      // one of a, b is zero: the upwind side alone, its slope from the cell
      // behind it (the right side is the left's mirror image)
      const bool left = b == 0.0;
      const double far = left ? q[-2 * d] * riLL : q[d] * riRR;
      f = (a + b) * muscl_left(lim, far, left ? L : Rr, left ? Rr : L);
    }
    if (VISC) f += sh[n * UF_TH] + 0.5 * (Rr + L) * corr;
    Fo[(5 + n) * v] = f;
  }
}

// the velocity's gradients on the interior of the uniform blocks, rows u, v, w
// of the gradient arrays, from the velocity the cell pass keeps
template <int NS>
__global__ void __launch_bounds__(256) k_vgrads(const BlockDev *__restrict__ blks, int b,
                                                const double *__restrict__ stall, double *__restrict__ gall,
                                                const int2 *__restrict__ ctab = nullptr) {
  PGB_WHERE(B, t);
  if (t >= (long long)B.nx * B.ny * B.nz) return;
  const long long c = inner_cell(B, t), v = B.vol;
  const double *st = stall + SW * B.cv + ST_U * v + c;
  double *g = gall + 3 * (3 + NS) * B.cv + c;
  const int step[3] = {1, B.X, B.X * B.Y};
#pragma unroll
  for (int m = 0; m < 3; m++)
#pragma unroll
    for (int e = 0; e < 3; e++)
      g[(3 * m + e) * v] = 0.5 * (st[m * v + step[e]] - st[m * v - step[e]]) * B.Jd[e];
}

// the faces of every uniform block, all three axes in one launch
template <int NS, int FN, bool KOREN, bool VISC, bool TPG>
__global__ void __launch_bounds__(UF_TH, TPG ? 4 : 5) k_ufaces(const BlockDev *__restrict__ blks, const double *__restrict__ Qall,
                                                     const double *__restrict__ stall, const double *__restrict__ trall,
                                                     const double *__restrict__ hall,
                                                     const double *__restrict__ gall,
                                                     const double *__restrict__ met, double *F0, double *F1,
                                                     double *F2, const int lim, const unsigned n0, const unsigned n1,
                                                     const int2 *__restrict__ ctab) {
  constexpr int NE = 4 + NS;
  unsigned t;
  int row;
  const int axis = face_work(n0, n1, ctab, row, t);
  const BlockDev &B = blks[row];
  if (!B.uniform) return;
  long long R;
  int pos;
  if (!face_cell(B, axis, t, R, pos)) return;
  const bool lo = pos == 0 && (B.bcg >> (2 * axis) & 1);
  const bool hi = pos == (axis == 0 ? B.nx : axis == 1 ? B.ny : B.nz) && (B.bcg >> (2 * axis + 1) & 1);
  const double *gr = VISC && gall ? gall + 3 * (NE - 1) * B.cv : nullptr;
  const double *Q = Qall + NE * B.cv, *st = stall + SW * B.cv, *M = met + M_NCOMP * B.cv;
  const double *tr = VISC ? trall + (2 + NS) * B.cv : nullptr, *hs = VISC ? hall + NS * B.cv : nullptr;
  const long long at = NE * B.cv;
  __shared__ double flux[VISC ? (NS > 1 ? NS - 1 : 1) * UF_TH : 1];
  double *sh = flux + (VISC ? threadIdx.x : 0);
  if (axis == 0) uface<NS, 0, FN, KOREN, VISC, TPG>(B, Q, st, tr, hs, gr, M, lo, hi, lim, R, F0 + at, sh);
  else if (axis == 1) uface<NS, 1, FN, KOREN, VISC, TPG>(B, Q, st, tr, hs, gr, M, lo, hi, lim, R, F1 + at, sh);
  else uface<NS, 2, FN, KOREN, VISC, TPG>(B, Q, st, tr, hs, gr, M, lo, hi, lim, R, F2 + at, sh);
}

// every field the faces read of a halo cell, in one pass over the halo's
// boxes (and the cells no box holds): grid plane 0 copies Q, plane 1 the
// state (p .. c, and with uvel the velocity), plane 2 the transport (all of
// it with full, else mu, kappa and the first species') and the enthalpies;
// the momentum and the velocity turned across a rotational periodic.  A halo
// cell's values are its source's: its Q, and the last T its Newton would
// start from, are.
struct HaloFields {
  double *Q, *state, *tr, *hsp;
  int uvel, full;
  const HaloPatch *boxes;
  const int2 *cta;
  const HaloEntry *rest;
  long long nrest;
  const double *rots;
};
template <int NS, bool ROT>
__global__ void __launch_bounds__(256) k_halo_fields(const HaloFields f) {
  constexpr int NE = 4 + NS;
  const int2 w = f.cta[blockIdx.x];
  const int t = w.y * 256 + (int)threadIdx.x;
  long long dcv, scv;
  int didx, sidx, dvol, svol, rot;
  if (w.x < 0) {
    if (t >= f.nrest) return;
    const HaloEntry h = f.rest[t];
    dcv = h.dcv, scv = h.scv, didx = h.didx, sidx = h.sidx, dvol = h.dvol, svol = h.svol, rot = h.rot;
  } else {
    const HaloPatch &p = f.boxes[w.x];
    if (t >= p.cells) return;
    const int x0 = t % p.n0, r = t / p.n0, x1 = r % p.n1, x2 = r / p.n1;
    didx = p.d0 + x0 * p.dst[0] + x1 * p.dst[1] + x2 * p.dst[2];
    sidx = p.s0 + x0 * p.sst[0] + x1 * p.sst[1] + x2 * p.sst[2];
    dcv = p.dcv, scv = p.scv, dvol = p.dvol, svol = p.svol, rot = p.rot;
  }
  if (blockIdx.z == 0) {
    halo_copy<NE, ROT>(f.Q, NE, 1, f.rots, dcv, didx, dvol, scv, sidx, svol, rot, NE);
  } else if (blockIdx.z == 1) {
    halo_copy<8, false>(f.state, 8, HALO_SCALARS, f.rots, dcv, didx, dvol, scv, sidx, svol, 0, SW);
    if (f.uvel)
      halo_copy<3, ROT>(f.state, 3, 0, f.rots, dcv, didx + (long long)ST_U * dvol, dvol, scv,
                        sidx + (long long)ST_U * svol, svol, rot, SW);
  } else {
    halo_copy<3, false>(f.tr, 3, HALO_SCALARS, f.rots, dcv, didx, dvol, scv, sidx, svol, 0, 2 + NS);
    halo_copy<NS, false>(f.hsp, NS, HALO_SCALARS, f.rots, dcv, didx, dvol, scv, sidx, svol, 0, NS);
    if (NS > 1 && f.full)
      halo_copy<NS - 1, false>(f.tr, NS - 1, HALO_SCALARS, f.rots, dcv, didx + 3LL * dvol, dvol, scv,
                               sidx + 3LL * svol, svol, 0, 2 + NS);
  }
}

}  // namespace pgb
