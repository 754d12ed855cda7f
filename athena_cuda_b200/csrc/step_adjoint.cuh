// step_adjoint.cuh -- the discrete adjoint of one CTU+CT step, the adjoint
// of the ghost-zone fill and of the dt rule, and the generic ghost fill the
// tangent-linear model uses.
//
// Every stage of the step (step_generic.cuh) is reversed by one or two
// per-item functors.  Inputs of the reverse step: the step's input state S^n
// (ghosts filled), its dt, the tape of the recorded forward step (the
// GenPlane planes), and the adjoint of the step's output, lout (the cells the
// step writes: the interior, B1i column ie+1 and B2i row je+1).  Output: lin,
// the adjoint of every plane entry of S^n the step reads (ghosts included),
// and per-item contributions to the adjoint of dt in the plane A_DT.
//
// Adjoints are GATHERED, never scattered: each stage first stores the adjoint
// of its own outputs per cell or face, and the stage before it collects, for
// each of its outputs, the contributions of every consumer in a fixed order.
// No atomics are involved, so the adjoint is deterministic and a kernel never
// has two threads writing one location.
//
// Reference steps reversed (src/__integrate_2d__.c): 13, 11b, 11a, 9 (update
// and CT), 9 (corner EMF, :632-702), 8c, 8b, 7, 6b, 6a, 5b, 5a, 4 (corrector),
// 3-4 (half-step EMF), 2e, 1e (predictor Riemann), 2b-2d, 1b-1d (PLM and
// source terms), 2a, 1a (cons -> prim); set_bvals (src/set_bvals.c:114-145)
// and new_dt (src/new_dt.c:25-100).
#pragma once

#include "mhd_adjoint.cuh"
#include "step_generic.cuh"

namespace athb {

// Adjoint workspace planes.
enum AdjPlane {
  A_DTY = 0,     // dt terms of the corrector's y faces, then of the PLM in y
  A_DTC = 1,     // ... of the corrector's cells
  A_PLMYD = 2,   // the density's share of the PLM source term in y
  A_FX2 = 3,     // corrector x flux (7)
  A_FY2 = 10,    // corrector y flux (7)
  A_ECC1 = 17,   // cell emf3 at t^{n+1/2}
  A_ULX = 18, A_URX = 25,   // corrector L/R states at x faces (7 each)
  A_ULY = 32, A_URY = 39,
  A_B1F = 46,    // half-step b1 at x faces, from the corrector flux
  A_B2F = 47,
  A_HALF = 48,   // half-step d, M1, M2, B1c, B2c of a cell (correct_e)
  A_LB1F = 53,   // half-step b1: every consumer
  A_LB2F = 54,
  A_FX = 56, A_FY = 63,     // predictor fluxes (7 each)
  A_WLNX = 70, A_WRTX = 77, A_WLNY = 84, A_WRTY = 91,  // PLM outputs (7 each)
  A_BNX = 98, A_BNY = 99,   // normal face field at predictor faces
  A_SRCX = 100, A_SRCY = 101,  // the PLM source term of a cell
  A_WXM = 102, A_WX0 = 109, A_WXP = 116,  // PLM inputs: cell c-1, c, c+1 (x)
  A_WYM = 123, A_WY0 = 130, A_WYP = 137,
  A_DT = 144,    // per-item contributions to the adjoint of dt
  A_TMP = 145,   // scratch (objective per cell)
  NADJ = 146
};

struct AdjArgs {
  const double* in;     // S^n, ghosts filled
  const double* tape;   // GenPlane planes of the recorded step
  const double* lout;   // adjoint of S^{n+1} (cells the step writes)
  double* lin;          // adjoint of S^n (adj_update writes it, later stages add)
  double* adj;          // AdjPlane planes
  StepCoef<double> c;   // dt^n and its factors, exactly as the forward formed them
  long long ps;
  int pitch;
  int is, ie, js, je;
  double dx1, dx2;
  Eos eos;
  FastEos fe;           // constants of the fast forms
  ATHB_MEM long long o(int j, int i) const { return (long long)j * pitch + i; }
  ATHB_MEM double s(int p, long long off) const { ATHB_CHECK_OFF(off, ps); return ro(in + p * ps + off); }
  ATHB_MEM double t(int p, long long off) const { ATHB_CHECK_OFF(off, ps); return ro(tape + p * ps + off); }
  ATHB_MEM double lo(int p, long long off) const { ATHB_CHECK_OFF(off, ps); return ro(lout + p * ps + off); }
  ATHB_MEM double& li(int p, long long off) const { ATHB_CHECK_OFF(off, ps); return lin[p * ps + off]; }
  ATHB_MEM double& a(int p, long long off) const { ATHB_CHECK_OFF(off, ps); return adj[p * ps + off]; }
  ATHB_MEM double av(int p, long long off) const { ATHB_CHECK_OFF(off, ps); return ro(adj + p * ps + off); }
  // av (lo) at off where in holds, else 0, without a branch before the load: a
  // gather's loads then all start at once.  safe: a place of the array.
  ATHB_MEM double av_if(bool in, int p, long long off, long long safe) const {
    const double x = av(p, in ? off : safe);
    return in ? x : 0.0;
  }
  ATHB_MEM double lo_if(bool in, int p, long long off, long long safe) const {
    const double x = lo(p, in ? off : safe);
    return in ? x : 0.0;
  }

 private:
  // What a stage reads through s, t, lo and av it never writes (each stage's
  // output planes are others than its input planes), so these are read-only
  // loads, which the compiler may move above the stage's stores: the small
  // stages are otherwise chains of one memory round trip per plane.
  ATHB_MEM static double ro(const double* q) {
#if defined(__CUDA_ARCH__)
    return __ldg(q);
#else
    return *q;
#endif
  }
};

// lin[p[k]] += v[k] at one place, all loads before the first store.
template <int N>
ATHB_HD void lin_add(const AdjArgs& a, long long o, const int (&p)[N], const double (&v)[N]) {
  double x[N];
#pragma unroll
  for (int k = 0; k < N; k++) x[k] = a.li(p[k], o);
#pragma unroll
  for (int k = 0; k < N; k++) a.li(p[k], o) = x[k] + v[k];
}

// x / dx1, x / dx2 with the launch's reciprocals (the same bits)
ATHB_HD double per_dx1(const AdjArgs& a, double x) { return any_quot(x, a.dx1, a.fe.r_dx1); }
ATHB_HD double per_dx2(const AdjArgs& a, double x) { return any_quot(x, a.dx2, a.fe.r_dx2); }

ATHB_HD bool in_range(const GenRange& r, int j, int i) { return j >= r.j0 && j <= r.j1 && i >= r.i0 && i <= r.i1; }

ATHB_HD Cons1 adj_cons(const AdjArgs& a, int base, long long o) {
  Cons1 u;
  u.d = a.av(base + 0, o); u.mx = a.av(base + 1, o); u.my = a.av(base + 2, o); u.mz = a.av(base + 3, o);
  u.e = a.av(base + 4, o); u.by = a.av(base + 5, o); u.bz = a.av(base + 6, o);
  return u;
}
ATHB_HD void adj_put_cons(const AdjArgs& a, int base, long long o, const Cons1& u) {
  a.a(base + 0, o) = u.d; a.a(base + 1, o) = u.mx; a.a(base + 2, o) = u.my; a.a(base + 3, o) = u.mz;
  a.a(base + 4, o) = u.e; a.a(base + 5, o) = u.by; a.a(base + 6, o) = u.bz;
}
ATHB_HD Prim1 adj_prim(const AdjArgs& a, int base, long long o) {
  Prim1 w;
  w.d = a.av(base + 0, o); w.vx = a.av(base + 1, o); w.vy = a.av(base + 2, o); w.vz = a.av(base + 3, o);
  w.p = a.av(base + 4, o); w.by = a.av(base + 5, o); w.bz = a.av(base + 6, o);
  return w;
}
ATHB_HD void adj_put_prim(const AdjArgs& a, int base, long long o, const Prim1& w) {
  a.a(base + 0, o) = w.d; a.a(base + 1, o) = w.vx; a.a(base + 2, o) = w.vy; a.a(base + 3, o) = w.vz;
  a.a(base + 4, o) = w.p; a.a(base + 5, o) = w.by; a.a(base + 6, o) = w.bz;
}
ATHB_HD Cons1 tape_cons(const AdjArgs& a, int base, long long o) {
  Cons1 u;
  u.d = a.t(base + 0, o); u.mx = a.t(base + 1, o); u.my = a.t(base + 2, o); u.mz = a.t(base + 3, o);
  u.e = a.t(base + 4, o); u.by = a.t(base + 5, o); u.bz = a.t(base + 6, o);
  return u;
}
ATHB_HD Prim1 tape_prim(const AdjArgs& a, int base, long long o) {
  Prim1 w;
  w.d = a.t(base + 0, o); w.vx = a.t(base + 1, o); w.vy = a.t(base + 2, o); w.vz = a.t(base + 3, o);
  w.p = a.t(base + 4, o); w.by = a.t(base + 5, o); w.bz = a.t(base + 6, o);
  return w;
}
ATHB_HD Cons1 state_cons(const AdjArgs& a, long long o, int dir) {
  Cons1 u;
  u.d = a.s(P_D, o);
  u.e = a.s(P_E, o);
  if (dir == 0) {
    u.mx = a.s(P_M1, o); u.my = a.s(P_M2, o); u.mz = a.s(P_M3, o); u.by = a.s(P_B2C, o); u.bz = a.s(P_B3C, o);
  } else {
    u.mx = a.s(P_M2, o); u.my = a.s(P_M3, o); u.mz = a.s(P_M1, o); u.by = a.s(P_B3C, o); u.bz = a.s(P_B1C, o);
  }
  return u;
}

// Corner-EMF coefficients of corner (j,i) from the fluxes on the tape
// (full = 0: predictor fluxes G_FX/G_FY; 1: corrector fluxes G_FX2/G_FY2).
ATHB_HD void corner_k(const AdjArgs& a, int full, int j, int i, double k[8]) {
  const int fx = full ? G_FX2 : G_FX, fy = full ? G_FY2 : G_FY;
  const long long o = a.o(j, i);
  corner_emf_coeffs(a.t(fx, o - a.pitch), a.t(fx, o), a.t(fy, o - 1), a.t(fy, o), k);
}

// The corner emf reversed at place (j,i): t[m] is the adjoint of corner input m
// of the one corner where this place is that input (corners (j,i), (j,i+1),
// (j+1,i) and (j+1,i+1)).  lb1 and lb2 give the adjoints of the face fields
// that CT forms from the emf, zero where there is no such face; the emf's own
// adjoint is formed here from six faces of each kind, which are in L1, instead
// of in a launch and a plane of its own.
template <class B1, class B2>
ATHB_HD void corner_terms(const AdjArgs& a, int full, const GenRange& K, double w1, double w2, int j, int i,
                          const B1& lb1, const B2& lb2, double t[8]) {
  double b1[3][2], b2[2][3];
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      b1[r][c] = lb1(j - 1 + r, i + c);
      b2[c][r] = lb2(j + c, i - 1 + r);
    }
#pragma unroll
  for (int m = 0; m < 8; m++) t[m] = 0.0;
#pragma unroll
  for (int r = 0; r < 2; r++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const bool in = in_range(K, j + r, i + c);
      const double e = in ? w1 * (b1[r + 1][c] - b1[r][c]) + w2 * (b2[r][c] - b2[r][c + 1]) : 0.0;
      double k[8];
      corner_k(a, full, in ? j + r : K.j0, in ? i + c : K.i0, k);
      if (r == 0 && c == 0) { t[1] = k[1] * e; t[3] = k[3] * e; t[7] = k[7] * e; }
      else if (r == 0) { t[2] = k[2] * e; t[6] = k[6] * e; }
      else if (c == 0) { t[0] = k[0] * e; t[5] = k[5] * e; }
      else t[4] = k[4] * e;
    }
}

// ===========================================================================
// Reverse of step 9/11/13 (update): the cell planes, the face fields b1, b2,
// the corner emf of the full step, and what they leave to the corrector's
// fluxes and to the half-step cell emf.  One item per place of the whole
// array: it writes every plane of lin and A_DT (zero where the update adds
// nothing), so neither is cleared before.  Fluxes and cell emf are gathered
// over [is-1, ie+1] x [js-1, je+1].
// ===========================================================================
ATHB_HD void adj_update(const AdjArgs& a, int j, int i) {
  const long long o = a.o(j, i), P = a.pitch;
  // b1 at x face (jj,ii), ii in [is, ie+1], jj in [js, je]
  auto lb1 = [&](int jj, int ii) {
    const bool in = jj >= a.js && jj <= a.je && ii >= a.is && ii <= a.ie + 1;
    const long long q = a.o(jj, ii);
    return (a.lo_if(in, P_B1I, q, o) + 0.5 * a.lo_if(in && ii <= a.ie, P_B1C, q, o)) +
           0.5 * a.lo_if(in && ii - 1 >= a.is, P_B1C, q - 1, o);
  };
  // b2 at y face (jj,ii), jj in [js, je+1], ii in [is, ie]
  auto lb2 = [&](int jj, int ii) {
    const bool in = jj >= a.js && jj <= a.je + 1 && ii >= a.is && ii <= a.ie;
    const long long q = a.o(jj, ii);
    return (a.lo_if(in, P_B2I, q, o) + 0.5 * a.lo_if(in && jj <= a.je, P_B2C, q, o)) +
           0.5 * a.lo_if(in && jj - 1 >= a.js, P_B2C, q - P, o);
  };
  double v[NSTATE], dtb = 0.0;
#pragma unroll
  for (int p = 0; p < NSTATE; p++) v[p] = 0.0;
  const GenRange corners = range_emf1(a.is, a.ie, a.js, a.je);
  const GenRange interior = range_interior(a.is, a.ie, a.js, a.je);
  if (in_range(corners, j, i)) {
    if (j <= a.je) {
      v[P_B1I] = lb1(j, i);
      dtb += per_dx2(a, -v[P_B1I] * (a.t(G_EMF1, o + P) - a.t(G_EMF1, o)));
    }
    if (i <= a.ie) {
      v[P_B2I] = lb2(j, i);
      dtb += per_dx1(a, v[P_B2I] * (a.t(G_EMF1, o + 1) - a.t(G_EMF1, o)));
    }
  }
  if (in_range(interior, j, i)) {
    const double ld = a.lo(P_D, o), l1 = a.lo(P_M1, o), l2 = a.lo(P_M2, o), l3 = a.lo(P_M3, o), le = a.lo(P_E, o);
    const double lb3 = a.lo(P_B3C, o) + a.lo(P_B3I, o);
    // d -= dtodx1 (fx(o+1) - fx(o)) ... ; d -= dtodx2 (fy(o+P) - fy(o)) ...
    double g1 = 0.0, g2 = 0.0;
    g1 += ld * (a.t(G_FX2 + 0, o + 1) - a.t(G_FX2 + 0, o));
    g1 += l1 * (a.t(G_FX2 + 1, o + 1) - a.t(G_FX2 + 1, o));
    g1 += l2 * (a.t(G_FX2 + 2, o + 1) - a.t(G_FX2 + 2, o));
    g1 += l3 * (a.t(G_FX2 + 3, o + 1) - a.t(G_FX2 + 3, o));
    g1 += le * (a.t(G_FX2 + 4, o + 1) - a.t(G_FX2 + 4, o));
    g1 += lb3 * (a.t(G_FX2 + 6, o + 1) - a.t(G_FX2 + 6, o));
    g2 += ld * (a.t(G_FY2 + 0, o + P) - a.t(G_FY2 + 0, o));
    g2 += l2 * (a.t(G_FY2 + 1, o + P) - a.t(G_FY2 + 1, o));
    g2 += l3 * (a.t(G_FY2 + 2, o + P) - a.t(G_FY2 + 2, o));
    g2 += l1 * (a.t(G_FY2 + 3, o + P) - a.t(G_FY2 + 3, o));
    g2 += le * (a.t(G_FY2 + 4, o + P) - a.t(G_FY2 + 4, o));
    g2 += lb3 * (a.t(G_FY2 + 5, o + P) - a.t(G_FY2 + 5, o));
    dtb += per_dx1(a, -g1) - per_dx2(a, g2);
    v[P_D] = ld; v[P_M1] = l1; v[P_M2] = l2; v[P_M3] = l3; v[P_E] = le; v[P_B3C] = lb3;
  }
#pragma unroll
  for (int p = 0; p < NSTATE; p++) a.li(p, o) = v[p];
  a.a(A_DT, o) = dtb;

  if (j < a.js - 1 || j > a.je + 1 || i < a.is - 1 || i > a.ie + 1) return;
  double t[8];
  corner_terms(a, 1, corners, a.c.dtodx2, a.c.dtodx1, j, i, lb1, lb2, t);
  auto lcell = [&](int p, int jj, int ii) {
    const bool in = in_range(interior, jj, ii);
    const long long q = a.o(jj, ii);
    return p == P_B3C ? a.lo_if(in, P_B3C, q, o) + a.lo_if(in, P_B3I, q, o) : a.lo_if(in, p, q, o);
  };
  // x face (j,i) in the corrector range
  if (in_range(range_correct_x(a.is, a.ie, a.js, a.je), j, i)) {
    constexpr int map[7] = {P_D, P_M1, P_M2, P_M3, P_E, -1, P_B3C};
#pragma unroll
    for (int c = 0; c < 7; c++)
      if (map[c] >= 0) a.a(A_FX2 + c, o) = a.c.dtodx1 * (lcell(map[c], j, i) - lcell(map[c], j, i - 1));
    a.a(A_FX2 + 5, o) = t[1] + t[0];
  }
  // y face (j,i)
  if (in_range(range_correct_y(a.is, a.ie, a.js, a.je), j, i)) {
    constexpr int map[7] = {P_D, P_M2, P_M3, P_M1, P_E, P_B3C, -1};
#pragma unroll
    for (int c = 0; c < 7; c++)
      if (map[c] >= 0) a.a(A_FY2 + c, o) = a.c.dtodx2 * (lcell(map[c], j, i) - lcell(map[c], j - 1, i));
    a.a(A_FY2 + 6, o) = t[3] + t[2];
  }
  a.a(A_ECC1, o) = t[7] + t[6] + t[5] + t[4];
}

// ===========================================================================
// Reverse of the corrector (steps 4-8).
// ===========================================================================
// Corrector L/R states of x face (j,i), rebuilt exactly as gen_correct_x.
ATHB_HD void correct_x_states(const AdjArgs& a, int j, int i, Cons1& ul, Cons1& ur, double& b1f) {
  const long long o = a.o(j, i), P = a.pitch;
  const StepCoef<double>& c = a.c;
  b1f = a.s(P_B1I, o) - c.hdtodx2 * (a.t(G_EMF0, o + P) - a.t(G_EMF0, o));
  ul = tape_cons(a, G_ULX, o);
  ur = tape_cons(a, G_URX, o);
  {
    const long long on = o + P - 1, oc = o - 1;
    ul.d -= c.hdtodx2 * (a.t(G_FY + 0, on) - a.t(G_FY + 0, oc));
    ul.mx -= c.hdtodx2 * (a.t(G_FY + 3, on) - a.t(G_FY + 3, oc));
    ul.my -= c.hdtodx2 * (a.t(G_FY + 1, on) - a.t(G_FY + 1, oc));
    ul.mz -= c.hdtodx2 * (a.t(G_FY + 2, on) - a.t(G_FY + 2, oc));
    ul.e -= c.hdtodx2 * (a.t(G_FY + 4, on) - a.t(G_FY + 4, oc));
    ul.bz -= c.hdtodx2 * (a.t(G_FY + 5, on) - a.t(G_FY + 5, oc));
  }
  {
    const long long on = o + P, oc = o;
    ur.d -= c.hdtodx2 * (a.t(G_FY + 0, on) - a.t(G_FY + 0, oc));
    ur.mx -= c.hdtodx2 * (a.t(G_FY + 3, on) - a.t(G_FY + 3, oc));
    ur.my -= c.hdtodx2 * (a.t(G_FY + 1, on) - a.t(G_FY + 1, oc));
    ur.mz -= c.hdtodx2 * (a.t(G_FY + 2, on) - a.t(G_FY + 2, oc));
    ur.e -= c.hdtodx2 * (a.t(G_FY + 4, on) - a.t(G_FY + 4, oc));
    ur.bz -= c.hdtodx2 * (a.t(G_FY + 5, on) - a.t(G_FY + 5, oc));
  }
  {
    const long long ow = o - 1;
    const double dbx = a.s(P_B1I, o) - a.s(P_B1I, ow);
    const double B1 = a.s(P_B1C, ow), B2 = a.s(P_B2C, ow), B3 = a.s(P_B3C, ow);
    const double V3 = ratio(a.s(P_M3, ow), a.s(P_D, ow));
    ul.mx += c.hdtodx1 * B1 * dbx;
    ul.my += c.hdtodx1 * B2 * dbx;
    ul.mz += c.hdtodx1 * B3 * dbx;
    ul.bz += c.hdtodx1 * V3 * dbx;
    ul.e += c.hdtodx1 * B3 * V3 * dbx;
  }
  {
    const double dbx = a.s(P_B1I, o + 1) - a.s(P_B1I, o);
    const double B1 = a.s(P_B1C, o), B2 = a.s(P_B2C, o), B3 = a.s(P_B3C, o);
    const double V3 = ratio(a.s(P_M3, o), a.s(P_D, o));
    ur.mx += c.hdtodx1 * B1 * dbx;
    ur.my += c.hdtodx1 * B2 * dbx;
    ur.mz += c.hdtodx1 * B3 * dbx;
    ur.bz += c.hdtodx1 * V3 * dbx;
    ur.e += c.hdtodx1 * B3 * V3 * dbx;
  }
}

ATHB_HD void correct_y_states(const AdjArgs& a, int j, int i, Cons1& ul, Cons1& ur, double& b2f) {
  const long long o = a.o(j, i), P = a.pitch;
  const StepCoef<double>& c = a.c;
  b2f = a.s(P_B2I, o) + c.hdtodx1 * (a.t(G_EMF0, o + 1) - a.t(G_EMF0, o));
  ul = tape_cons(a, G_ULY, o);
  ur = tape_cons(a, G_URY, o);
  {
    const long long oe = o - P + 1, oc = o - P;
    ul.d -= c.hdtodx1 * (a.t(G_FX + 0, oe) - a.t(G_FX + 0, oc));
    ul.mx -= c.hdtodx1 * (a.t(G_FX + 2, oe) - a.t(G_FX + 2, oc));
    ul.my -= c.hdtodx1 * (a.t(G_FX + 3, oe) - a.t(G_FX + 3, oc));
    ul.mz -= c.hdtodx1 * (a.t(G_FX + 1, oe) - a.t(G_FX + 1, oc));
    ul.e -= c.hdtodx1 * (a.t(G_FX + 4, oe) - a.t(G_FX + 4, oc));
    ul.by -= c.hdtodx1 * (a.t(G_FX + 6, oe) - a.t(G_FX + 6, oc));
  }
  {
    const long long oe = o + 1, oc = o;
    ur.d -= c.hdtodx1 * (a.t(G_FX + 0, oe) - a.t(G_FX + 0, oc));
    ur.mx -= c.hdtodx1 * (a.t(G_FX + 2, oe) - a.t(G_FX + 2, oc));
    ur.my -= c.hdtodx1 * (a.t(G_FX + 3, oe) - a.t(G_FX + 3, oc));
    ur.mz -= c.hdtodx1 * (a.t(G_FX + 1, oe) - a.t(G_FX + 1, oc));
    ur.e -= c.hdtodx1 * (a.t(G_FX + 4, oe) - a.t(G_FX + 4, oc));
    ur.by -= c.hdtodx1 * (a.t(G_FX + 6, oe) - a.t(G_FX + 6, oc));
  }
  {
    const long long osn = o - P;
    const double dby = a.s(P_B2I, o) - a.s(P_B2I, osn);
    const double B1 = a.s(P_B1C, osn), B2 = a.s(P_B2C, osn), B3 = a.s(P_B3C, osn);
    const double V3 = ratio(a.s(P_M3, osn), a.s(P_D, osn));
    ul.mz += c.hdtodx2 * B1 * dby;
    ul.mx += c.hdtodx2 * B2 * dby;
    ul.my += c.hdtodx2 * B3 * dby;
    ul.by += c.hdtodx2 * V3 * dby;
    ul.e += c.hdtodx2 * B3 * V3 * dby;
  }
  {
    const double dby = a.s(P_B2I, o + P) - a.s(P_B2I, o);
    const double B1 = a.s(P_B1C, o), B2 = a.s(P_B2C, o), B3 = a.s(P_B3C, o);
    const double V3 = ratio(a.s(P_M3, o), a.s(P_D, o));
    ur.mz += c.hdtodx2 * B1 * dby;
    ur.mx += c.hdtodx2 * B2 * dby;
    ur.my += c.hdtodx2 * B3 * dby;
    ur.by += c.hdtodx2 * V3 * dby;
    ur.e += c.hdtodx2 * B3 * V3 * dby;
  }
}

// dt adjoint of the transverse and source terms of one corrector state
// (x face: transverse terms are x2-flux differences (hdtodx2), sources use
// hdtodx1; y face: the other way round).
ATHB_HD double correct_x_dtb(const AdjArgs& a, int j, int i, const Cons1& lul, const Cons1& lur) {
  const long long o = a.o(j, i), P = a.pitch;
  double g2 = 0.0, g1 = 0.0;
  {
    const long long on = o + P - 1, oc = o - 1;
    g2 -= lul.d * (a.t(G_FY + 0, on) - a.t(G_FY + 0, oc)) + lul.mx * (a.t(G_FY + 3, on) - a.t(G_FY + 3, oc)) +
          lul.my * (a.t(G_FY + 1, on) - a.t(G_FY + 1, oc)) + lul.mz * (a.t(G_FY + 2, on) - a.t(G_FY + 2, oc)) +
          lul.e * (a.t(G_FY + 4, on) - a.t(G_FY + 4, oc)) + lul.bz * (a.t(G_FY + 5, on) - a.t(G_FY + 5, oc));
  }
  {
    const long long on = o + P, oc = o;
    g2 -= lur.d * (a.t(G_FY + 0, on) - a.t(G_FY + 0, oc)) + lur.mx * (a.t(G_FY + 3, on) - a.t(G_FY + 3, oc)) +
          lur.my * (a.t(G_FY + 1, on) - a.t(G_FY + 1, oc)) + lur.mz * (a.t(G_FY + 2, on) - a.t(G_FY + 2, oc)) +
          lur.e * (a.t(G_FY + 4, on) - a.t(G_FY + 4, oc)) + lur.bz * (a.t(G_FY + 5, on) - a.t(G_FY + 5, oc));
  }
  {
    const long long ow = o - 1;
    const double dbx = a.s(P_B1I, o) - a.s(P_B1I, ow);
    const double B1 = a.s(P_B1C, ow), B2 = a.s(P_B2C, ow), B3 = a.s(P_B3C, ow);
    const double V3 = ratio(a.s(P_M3, ow), a.s(P_D, ow));
    g1 += dbx * (B1 * lul.mx + B2 * lul.my + B3 * lul.mz + V3 * lul.bz + B3 * V3 * lul.e);
  }
  {
    const double dbx = a.s(P_B1I, o + 1) - a.s(P_B1I, o);
    const double B1 = a.s(P_B1C, o), B2 = a.s(P_B2C, o), B3 = a.s(P_B3C, o);
    const double V3 = ratio(a.s(P_M3, o), a.s(P_D, o));
    g1 += dbx * (B1 * lur.mx + B2 * lur.my + B3 * lur.mz + V3 * lur.bz + B3 * V3 * lur.e);
  }
  return per_dx1(a, 0.5 * g1) + per_dx2(a, 0.5 * g2);
}
ATHB_HD double correct_y_dtb(const AdjArgs& a, int j, int i, const Cons1& lul, const Cons1& lur) {
  const long long o = a.o(j, i), P = a.pitch;
  double g1 = 0.0, g2 = 0.0;
  {
    const long long oe = o - P + 1, oc = o - P;
    g1 -= lul.d * (a.t(G_FX + 0, oe) - a.t(G_FX + 0, oc)) + lul.mx * (a.t(G_FX + 2, oe) - a.t(G_FX + 2, oc)) +
          lul.my * (a.t(G_FX + 3, oe) - a.t(G_FX + 3, oc)) + lul.mz * (a.t(G_FX + 1, oe) - a.t(G_FX + 1, oc)) +
          lul.e * (a.t(G_FX + 4, oe) - a.t(G_FX + 4, oc)) + lul.by * (a.t(G_FX + 6, oe) - a.t(G_FX + 6, oc));
  }
  {
    const long long oe = o + 1, oc = o;
    g1 -= lur.d * (a.t(G_FX + 0, oe) - a.t(G_FX + 0, oc)) + lur.mx * (a.t(G_FX + 2, oe) - a.t(G_FX + 2, oc)) +
          lur.my * (a.t(G_FX + 3, oe) - a.t(G_FX + 3, oc)) + lur.mz * (a.t(G_FX + 1, oe) - a.t(G_FX + 1, oc)) +
          lur.e * (a.t(G_FX + 4, oe) - a.t(G_FX + 4, oc)) + lur.by * (a.t(G_FX + 6, oe) - a.t(G_FX + 6, oc));
  }
  {
    const long long osn = o - P;
    const double dby = a.s(P_B2I, o) - a.s(P_B2I, osn);
    const double B1 = a.s(P_B1C, osn), B2 = a.s(P_B2C, osn), B3 = a.s(P_B3C, osn);
    const double V3 = ratio(a.s(P_M3, osn), a.s(P_D, osn));
    g2 += dby * (B1 * lul.mz + B2 * lul.mx + B3 * lul.my + V3 * lul.by + B3 * V3 * lul.e);
  }
  {
    const double dby = a.s(P_B2I, o + P) - a.s(P_B2I, o);
    const double B1 = a.s(P_B1C, o), B2 = a.s(P_B2C, o), B3 = a.s(P_B3C, o);
    const double V3 = ratio(a.s(P_M3, o), a.s(P_D, o));
    g2 += dby * (B1 * lur.mz + B2 * lur.mx + B3 * lur.my + V3 * lur.by + B3 * V3 * lur.e);
  }
  return per_dx1(a, 0.5 * g1) + per_dx2(a, 0.5 * g2);
}

// The adjoint of the face flux: the fast form where it applies, else the
// general one, out of line.  The outputs are set.
template <int FLUX>
ATHB_COLD void face_adj_general(const Cons1* ul, const Cons1* ur, const Prim1* wl, const Prim1* wr, double bn,
                                const Eos* eos, const Cons1* fb, Cons1* ulb, Cons1* urb, Prim1* wlb, Prim1* wrb,
                                double* bnb) {
  zero(*ulb); zero(*urb); zero(*wlb); zero(*wrb);
  *bnb = 0.0;
  riemann_adj<FLUX>(*ul, *ur, *wl, *wr, bn, *eos, *fb, *ulb, *urb, *wlb, *wrb, *bnb);
}
template <int FLUX>
ATHB_HD void face_adj(const AdjArgs& a, const Cons1& ul, const Cons1& ur, const Prim1& wl, const Prim1& wr, double bn,
                      const Cons1& fb, Cons1& ulb, Cons1& urb, Prim1& wlb, Prim1& wrb, double& bnb) {
  if (FLUX == kFluxHlle) {
    zero(ulb); zero(urb); zero(wlb); zero(wrb);
    bnb = 0.0;
    flux_hlle_adj(ul, ur, wl, wr, bn, a.eos, fb, ulb, urb, wlb, wrb, bnb);
    return;
  }
  if (flux_roe_adj_fast(ul, ur, wl, wr, bn, a.eos, a.fe.r_gamma_1, fb, ulb, urb, wlb, wrb, bnb) && a.fe.ok) return;
  const Cons1 u = ul, v = ur, f = fb;
  const Prim1 w = wl, x = wr;
  const Eos eos = a.eos;
  Cons1 ub, vb;
  Prim1 wb, xb;
  double bb;
  face_adj_general<FLUX>(&u, &v, &w, &x, bn, &eos, &f, &ub, &vb, &wb, &xb, &bb);
  ulb = ub; urb = vb; wlb = wb; wrb = xb;
  bnb = bb;
}
// prim_to_cons with the launch's 1/(gamma - 1)
ATHB_HD Cons1 face_cons(const AdjArgs& a, const Prim1& w, double bn) {
  return a.fe.ok ? cons_of(w, bn, a.eos, a.fe.r_gamma_1) : prim_to_cons(w, bn, a.eos);
}

template <int FLUX>
ATHB_HD void adj_correct_x(const AdjArgs& a, int j, int i) {
  const long long o = a.o(j, i);
  const double dt0 = a.a(A_DT, o);
  Cons1 ul, ur;
  double b1f;
  correct_x_states(a, j, i, ul, ur, b1f);
  const double dil = any_recip(ul.d), dir = any_recip(ur.d);
  const Prim1 wl = prim_of(ul, b1f, dil, a.eos), wr = prim_of(ur, b1f, dir, a.eos);
  Cons1 ulb, urb;
  Prim1 wlb, wrb;
  double b1fb;
  face_adj<FLUX>(a, ul, ur, wl, wr, b1f, adj_cons(a, A_FX2, o), ulb, urb, wlb, wrb, b1fb);
  cons_to_prim_adj(ul, b1f, a.eos, dil, wlb, ulb, b1fb);
  cons_to_prim_adj(ur, b1f, a.eos, dir, wrb, urb, b1fb);
  a.a(A_DT, o) = dt0 + correct_x_dtb(a, j, i, ulb, urb);
  adj_put_cons(a, A_ULX, o, ulb);
  adj_put_cons(a, A_URX, o, urb);
  a.a(A_B1F, o) = b1fb;
}

template <int FLUX>
ATHB_HD void adj_correct_y(const AdjArgs& a, int j, int i) {
  const long long o = a.o(j, i);
  Cons1 ul, ur;
  double b2f;
  correct_y_states(a, j, i, ul, ur, b2f);
  const double dil = any_recip(ul.d), dir = any_recip(ur.d);
  const Prim1 wl = prim_of(ul, b2f, dil, a.eos), wr = prim_of(ur, b2f, dir, a.eos);
  Cons1 ulb, urb;
  Prim1 wlb, wrb;
  double b2fb;
  face_adj<FLUX>(a, ul, ur, wl, wr, b2f, adj_cons(a, A_FY2, o), ulb, urb, wlb, wrb, b2fb);
  cons_to_prim_adj(ul, b2f, a.eos, dil, wlb, ulb, b2fb);
  cons_to_prim_adj(ur, b2f, a.eos, dir, wrb, urb, b2fb);
  a.a(A_DTY, o) = correct_y_dtb(a, j, i, ulb, urb);
  adj_put_cons(a, A_ULY, o, ulb);
  adj_put_cons(a, A_URY, o, urb);
  a.a(A_B2F, o) = b2fb;
}

// step 7 reversed: cells [is-1, ie+1] x [js-1, je+1]
ATHB_HD void adj_correct_e(const AdjArgs& a, int j, int i) {
  const long long o = a.o(j, i), P = a.pitch;
  const StepCoef<double>& c = a.c;
  const double dfx0 = a.t(G_FX + 0, o + 1) - a.t(G_FX + 0, o), dfy0 = a.t(G_FY + 0, o + P) - a.t(G_FY + 0, o);
  const double dfx1 = a.t(G_FX + 1, o + 1) - a.t(G_FX + 1, o), dfy3 = a.t(G_FY + 3, o + P) - a.t(G_FY + 3, o);
  const double dfx2 = a.t(G_FX + 2, o + 1) - a.t(G_FX + 2, o), dfy1 = a.t(G_FY + 1, o + P) - a.t(G_FY + 1, o);
  const double d = a.s(P_D, o) - c.hdtodx1 * dfx0 - c.hdtodx2 * dfy0;
  const double M1 = a.s(P_M1, o) - c.hdtodx1 * dfx1 - c.hdtodx2 * dfy3;
  const double M2 = a.s(P_M2, o) - c.hdtodx1 * dfx2 - c.hdtodx2 * dfy1;
  const double b1f_c = a.s(P_B1I, o) - c.hdtodx2 * (a.t(G_EMF0, o + P) - a.t(G_EMF0, o));
  const double b1f_e = a.s(P_B1I, o + 1) - c.hdtodx2 * (a.t(G_EMF0, o + P + 1) - a.t(G_EMF0, o + 1));
  const double b2f_c = a.s(P_B2I, o) + c.hdtodx1 * (a.t(G_EMF0, o + 1) - a.t(G_EMF0, o));
  const double b2f_n = a.s(P_B2I, o + P) + c.hdtodx1 * (a.t(G_EMF0, o + P + 1) - a.t(G_EMF0, o + P));
  const double B1c = 0.5 * (b1f_c + b1f_e);
  const double B2c = 0.5 * (b2f_c + b2f_n);
  const double rd = any_recip(d);
  const double e = any_quot(B1c * M2 - B2c * M1, d, rd);
  const double lam = a.av(A_ECC1, o);
  const double ld = any_quot(-lam * e, d, rd), lM1 = any_quot(-lam * B2c, d, rd), lM2 = any_quot(lam * B1c, d, rd);
  const int p[3] = {P_D, P_M1, P_M2};
  const double v[3] = {ld, lM1, lM2};
  lin_add(a, o, p, v);
  a.a(A_HALF + 0, o) = ld;
  a.a(A_HALF + 1, o) = lM1;
  a.a(A_HALF + 2, o) = lM2;
  a.a(A_HALF + 3, o) = any_quot(lam * M2, d, rd);
  a.a(A_HALF + 4, o) = any_quot(-lam * M1, d, rd);
  a.a(A_DTC, o) = per_dx1(a, 0.5 * (-(ld * dfx0 + lM1 * dfx1 + lM2 * dfx2))) +
                  per_dx2(a, 0.5 * (-(ld * dfy0 + lM1 * dfy3 + lM2 * dfy1)));
}

// Every consumer of the half-step face fields: x faces [is-1, ie+2] x
// [js-1, je+1] and y faces [is-1, ie+1] x [js-1, je+2]; items over
// [is-1, ie+2] x [js-1, je+2].  The dt terms of the corrector's y faces and
// cells join A_DT here, in the order x faces, y faces, cells.
ATHB_HD void adj_half_faces(const AdjArgs& a, int j, int i) {
  const long long o = a.o(j, i), P = a.pitch;
  const GenRange E = range_correct_e(a.is, a.ie, a.js, a.je);
  const bool xface = j <= a.je + 1, yface = i <= a.ie + 1;
  const GenRange CX = range_correct_x(a.is, a.ie, a.js, a.je), CY = range_correct_y(a.is, a.ie, a.js, a.je);
  const double dt0 = (a.a(A_DT, o) + a.av_if(in_range(CY, j, i), A_DTY, o, o)) + a.av_if(in_range(E, j, i), A_DTC, o, o);
  const double b10 = xface ? a.li(P_B1I, o) : 0.0, b20 = yface ? a.li(P_B2I, o) : 0.0;
  double dtb = 0.0;
  if (xface) {
    const double lb = (a.av_if(in_range(CX, j, i), A_B1F, o, o) + 0.5 * a.av_if(in_range(E, j, i), A_HALF + 3, o, o)) +
                      0.5 * a.av_if(in_range(E, j, i - 1), A_HALF + 3, o - 1, o);
    a.a(A_LB1F, o) = lb;
    a.li(P_B1I, o) = b10 + lb;
    dtb += per_dx2(a, -lb * (a.t(G_EMF0, o + P) - a.t(G_EMF0, o)) * 0.5);
  }
  if (yface) {
    const double lb = (a.av_if(in_range(CY, j, i), A_B2F, o, o) + 0.5 * a.av_if(in_range(E, j, i), A_HALF + 4, o, o)) +
                      0.5 * a.av_if(in_range(E, j - 1, i), A_HALF + 4, o - P, o);
    a.a(A_LB2F, o) = lb;
    a.li(P_B2I, o) = b20 + lb;
    dtb += per_dx1(a, lb * (a.t(G_EMF0, o + 1) - a.t(G_EMF0, o)) * 0.5);
  }
  a.a(A_DT, o) = dt0 + dtb;
}

// The predictor fluxes and the t^n cell emf, gathered from the corrector
// (transverse terms), correct_e and the half-step corner emf (reversed here
// from the half-step face fields): [is-2, ie+2] x [js-2, je+2].
ATHB_HD void adj_flux1(const AdjArgs& a, int j, int i) {
  const long long o = a.o(j, i);
  const StepCoef<double>& c = a.c;
  const GenRange CX = range_correct_x(a.is, a.ie, a.js, a.je), CY = range_correct_y(a.is, a.ie, a.js, a.je);
  const GenRange E = range_correct_e(a.is, a.ie, a.js, a.je), K = range_emf0(a.is, a.ie, a.js, a.je);
  auto lb1 = [&](int jj, int ii) { return a.av_if(jj >= a.js - 1 && jj <= a.je + 1 && ii >= a.is - 1 && ii <= a.ie + 2, A_LB1F, a.o(jj, ii), o); };
  auto lb2 = [&](int jj, int ii) { return a.av_if(jj >= a.js - 1 && jj <= a.je + 2 && ii >= a.is - 1 && ii <= a.ie + 1, A_LB2F, a.o(jj, ii), o); };
  auto half = [&](int q, int jj, int ii) { return a.av_if(in_range(E, jj, ii), A_HALF + q, a.o(jj, ii), o); };
  double t[8];
  corner_terms(a, 0, K, c.hdtodx2, c.hdtodx1, j, i, lb1, lb2, t);
  // x face (j,i) of the predictor
  if (in_range(range_riemann_x(a.is, a.ie, a.js, a.je), j, i)) {
    double f[7] = {0, 0, 0, 0, 0, 0, 0};
    // correct_y transverse terms: (u.d, u.mx, u.my, u.mz, u.e, u.by) <- fx (0, 2, 3, 1, 4, 6)
    auto addy = [&](int base, int jj, int ii, double w) {
      const bool in = in_range(CY, jj, ii);
      const long long q = a.o(jj, ii);
      f[0] += w * a.av_if(in, base + 0, q, o); f[2] += w * a.av_if(in, base + 1, q, o);
      f[3] += w * a.av_if(in, base + 2, q, o); f[1] += w * a.av_if(in, base + 3, q, o);
      f[4] += w * a.av_if(in, base + 4, q, o); f[6] += w * a.av_if(in, base + 5, q, o);
    };
    addy(A_ULY, j + 1, i - 1, -c.hdtodx1);
    addy(A_ULY, j + 1, i, c.hdtodx1);
    addy(A_URY, j, i - 1, -c.hdtodx1);
    addy(A_URY, j, i, c.hdtodx1);
    // correct_e: d, M1, M2 of cells (j,i) and (j,i-1)
    f[0] += c.hdtodx1 * (half(0, j, i) - half(0, j, i - 1));
    f[1] += c.hdtodx1 * (half(1, j, i) - half(1, j, i - 1));
    f[2] += c.hdtodx1 * (half(2, j, i) - half(2, j, i - 1));
    // half-step corner emf: fx_by of corner (j,i), fx_by_s of corner (j+1,i)
    f[5] = t[1] + t[0];
    for (int q = 0; q < 7; q++) a.a(A_FX + q, o) = f[q];
  }
  // y face (j,i)
  if (in_range(range_riemann_y(a.is, a.ie, a.js, a.je), j, i)) {
    double f[7] = {0, 0, 0, 0, 0, 0, 0};
    // correct_x transverse terms: (u.d, u.mx, u.my, u.mz, u.e, u.bz) <- fy (0, 3, 1, 2, 4, 5)
    auto addx = [&](int base, int jj, int ii, double w) {
      const bool in = in_range(CX, jj, ii);
      const long long q = a.o(jj, ii);
      f[0] += w * a.av_if(in, base + 0, q, o); f[3] += w * a.av_if(in, base + 1, q, o);
      f[1] += w * a.av_if(in, base + 2, q, o); f[2] += w * a.av_if(in, base + 3, q, o);
      f[4] += w * a.av_if(in, base + 4, q, o); f[5] += w * a.av_if(in, base + 6, q, o);
    };
    addx(A_ULX, j - 1, i + 1, -c.hdtodx2);
    addx(A_ULX, j, i + 1, c.hdtodx2);
    addx(A_URX, j - 1, i, -c.hdtodx2);
    addx(A_URX, j, i, c.hdtodx2);
    // correct_e: d <- fy0, M1 <- fy3, M2 <- fy1
    f[0] += c.hdtodx2 * (half(0, j, i) - half(0, j - 1, i));
    f[3] += c.hdtodx2 * (half(1, j, i) - half(1, j - 1, i));
    f[1] += c.hdtodx2 * (half(2, j, i) - half(2, j - 1, i));
    // corner emf: fy_bz of corner (j,i), fy_bz_w of corner (j,i+1)
    f[6] = t[3] + t[2];
    for (int q = 0; q < 7; q++) a.a(A_FY + q, o) = f[q];
  }
  // t^n cell emf of cell (j,i) -> the state
  {
    const double v = t[7] + t[6] + t[5] + t[4];
    if (v != 0.0) {
      const double d = a.s(P_D, o), M1 = a.s(P_M1, o), M2 = a.s(P_M2, o), B1 = a.s(P_B1C, o), B2 = a.s(P_B2C, o);
      const double rd = any_recip(d), e = any_quot(B1 * M2 - B2 * M1, d, rd);
      const int p[5] = {P_B1C, P_M2, P_B2C, P_M1, P_D};
      const double w[5] = {any_quot(v * M2, d, rd), any_quot(v * B1, d, rd), -any_quot(v * M1, d, rd),
                           -any_quot(v * B2, d, rd), -any_quot(v * e, d, rd)};
      lin_add(a, o, p, w);
    }
  }
}

// The corrector's MHD source terms (steps 5b, 6b) back to the state: cells
// [is-1, ie+1] x [js-1, je+1] and the face fields of x faces [is-1, ie+2] x
// [js-1, je+1], y faces [is-1, ie+1] x [js-1, je+2].
ATHB_HD void adj_sources(const AdjArgs& a, int j, int i) {
  const long long o = a.o(j, i), P = a.pitch;
  const double h1 = a.c.hdtodx1, h2 = a.c.hdtodx2;
  const GenRange CX = range_correct_x(a.is, a.ie, a.js, a.je), CY = range_correct_y(a.is, a.ie, a.js, a.je);
  // v3 of the three cells whose source terms reach the faces of (j,i)
  const double rdc = any_recip(a.s(P_D, o)), V3c = any_quot(a.s(P_M3, o), a.s(P_D, o), rdc);
  const double V3w = ratio(a.s(P_M3, o - 1), a.s(P_D, o - 1)), V3s = ratio(a.s(P_M3, o - P), a.s(P_D, o - P));
  // λ of dbx of face (jj,ii)'s left (ul) or right (ur) state, with its cell
  auto dbx = [&](int base, int jj, int ii, long long cell, double V3) {
    const bool in = in_range(CX, jj, ii);
    const long long q = a.o(jj, ii);
    const double B1 = a.s(P_B1C, cell), B2 = a.s(P_B2C, cell), B3 = a.s(P_B3C, cell);
    return h1 * (B1 * a.av_if(in, base + 1, q, o) + B2 * a.av_if(in, base + 2, q, o) + B3 * a.av_if(in, base + 3, q, o) +
                 V3 * a.av_if(in, base + 6, q, o) + B3 * V3 * a.av_if(in, base + 4, q, o));
  };
  auto dby = [&](int base, int jj, int ii, long long cell, double V3) {
    const bool in = in_range(CY, jj, ii);
    const long long q = a.o(jj, ii);
    const double B1 = a.s(P_B1C, cell), B2 = a.s(P_B2C, cell), B3 = a.s(P_B3C, cell);
    return h2 * (B1 * a.av_if(in, base + 3, q, o) + B2 * a.av_if(in, base + 1, q, o) + B3 * a.av_if(in, base + 2, q, o) +
                 V3 * a.av_if(in, base + 5, q, o) + B3 * V3 * a.av_if(in, base + 4, q, o));
  };
  // cell (j,i)
  if (in_range(range_correct_e(a.is, a.ie, a.js, a.je), j, i)) {
    const double B3 = a.s(P_B3C, o);
    const double d = a.s(P_D, o), V3 = V3c;
    double lB1 = 0, lB2 = 0, lB3 = 0, lV3 = 0;
    auto add = [&](bool in, double w, int base, long long q, int m1, int m2, int m3, int mv) {
      const double l4 = a.av_if(in, base + 4, q, o);
      lB1 += w * a.av_if(in, base + m1, q, o);
      lB2 += w * a.av_if(in, base + m2, q, o);
      lB3 += w * (a.av_if(in, base + m3, q, o) + V3 * l4);
      lV3 += w * (a.av_if(in, base + mv, q, o) + B3 * l4);
    };
    const double dx = a.s(P_B1I, o + 1) - a.s(P_B1I, o), dy = a.s(P_B2I, o + P) - a.s(P_B2I, o);
    add(in_range(CX, j, i + 1), h1 * dx, A_ULX, o + 1, 1, 2, 3, 6);   // ul of x face (j,i+1)
    add(in_range(CX, j, i), h1 * dx, A_URX, o, 1, 2, 3, 6);           // ur of x face (j,i)
    add(in_range(CY, j + 1, i), h2 * dy, A_ULY, o + P, 3, 1, 2, 5);   // ul of y face (j+1,i): mz<-B1, mx<-B2, my<-B3, by<-V3
    add(in_range(CY, j, i), h2 * dy, A_URY, o, 3, 1, 2, 5);           // ur of y face (j,i)
    const int p[5] = {P_B1C, P_B2C, P_B3C, P_M3, P_D};
    const double v[5] = {lB1, lB2, lB3, any_quot(lV3, d, rdc), -any_quot(lV3 * V3, d, rdc)};
    lin_add(a, o, p, v);
  }
  // x face (j,i): B1i through dbx of ul/ur of x faces i, i+1, i-1
  if (j <= a.je + 1 && j >= a.js - 1 && i >= a.is - 1 && i <= a.ie + 2)
    a.li(P_B1I, o) += dbx(A_ULX, j, i, o - 1, V3w) - dbx(A_ULX, j, i + 1, o, V3c) - dbx(A_URX, j, i, o, V3c) +
                      dbx(A_URX, j, i - 1, o - 1, V3w);
  // y face (j,i)
  if (i <= a.ie + 1 && i >= a.is - 1 && j >= a.js - 1 && j <= a.je + 2)
    a.li(P_B2I, o) += dby(A_ULY, j, i, o - P, V3s) - dby(A_ULY, j + 1, i, o, V3c) - dby(A_URY, j, i, o, V3c) +
                      dby(A_URY, j - 1, i, o - P, V3s);
}

// Both, items over [is-2, ie+2] x [js-2, je+2]: they read the same corrector
// adjoints, and neither reads what the other writes.
ATHB_HD void adj_flux1_sources(const AdjArgs& a, int j, int i) {
  adj_flux1(a, j, i);
  if (i >= a.is - 1 && j >= a.js - 1) adj_sources(a, j, i);
}

// ===========================================================================
// Reverse of the predictor.
// ===========================================================================
// Predictor face (j,i) of sweep dir: faces of range_riemann_x / _y.
template <int FLUX>
ATHB_HD void adj_riemann(const AdjArgs& a, int dir, int j, int i) {
  const long long o = a.o(j, i);
  const long long step = dir == 0 ? 1 : a.pitch;
  const Prim1 wl = tape_prim(a, dir == 0 ? G_WLNX : G_WLNY, o - step);
  const Prim1 wr = tape_prim(a, dir == 0 ? G_WRTX : G_WRTY, o);
  const double bn = a.s(dir == 0 ? P_B1I : P_B2I, o);
  const Cons1 ul = face_cons(a, wl, bn), ur = face_cons(a, wr, bn);
  Cons1 ulb, urb;
  Prim1 wlb, wrb;
  double bnb;
  face_adj<FLUX>(a, ul, ur, wl, wr, bn, adj_cons(a, dir == 0 ? A_FX : A_FY, o), ulb, urb, wlb, wrb, bnb);
  const GenRange C = dir == 0 ? range_correct_x(a.is, a.ie, a.js, a.je) : range_correct_y(a.is, a.ie, a.js, a.je);
  if (in_range(C, j, i)) {
    addto(ulb, adj_cons(a, dir == 0 ? A_ULX : A_ULY, o));
    addto(urb, adj_cons(a, dir == 0 ? A_URX : A_URY, o));
  }
  prim_to_cons_adj(wl, bn, a.fe.r_gamma_1, ulb, wlb, bnb);
  prim_to_cons_adj(wr, bn, a.fe.r_gamma_1, urb, wrb, bnb);
  adj_put_prim(a, dir == 0 ? A_WLNX : A_WLNY, o - step, wlb);
  adj_put_prim(a, dir == 0 ? A_WRTX : A_WRTY, o, wrb);
  a.a(dir == 0 ? A_BNX : A_BNY, o) = bnb;
}

// plm_cell_adj out of line, from the conserved states: cells outside the ranges
// of the fast form.
ATHB_COLD void plm_adj_general(Cons1 um, Cons1 u0, Cons1 up, double bxm, double bx0, double bxp, double dtodx, Eos eos,
                               Prim1 wlb, Prim1 wrb, Prim1* wmb, Prim1* w0b, Prim1* wpb, double* bxcb,
                               double* dtodxb) {
  Prim1 x, y, z;
  zero(x); zero(y); zero(z);
  double bb = 0.0, tb = 0.0;
  plm_cell_adj(cons_to_prim(um, bxm, eos), cons_to_prim(u0, bx0, eos), cons_to_prim(up, bxp, eos), bx0, dtodx, eos, wlb,
               wrb, x, y, z, bb, tb);
  *wmb = x; *w0b = y; *wpb = z;
  *bxcb = bb;
  *dtodxb = tb;
}

// PLM + source term of cell (j,i) of sweep dir: cells of range_plm.  Both
// sweeps run in one launch: the y sweep's shares of the density and of dt,
// which the x sweep adds to as well, go to planes that adj_prim adds.
ATHB_HD void adj_plm(const AdjArgs& a, int dir, int j, int i) {
  const long long o = a.o(j, i);
  const long long step = dir == 0 ? 1 : a.pitch;
  // faces fed by this cell: wln -> face c+1, wrt -> face c
  const GenRange F = dir == 0 ? range_riemann_x(a.is, a.ie, a.js, a.je) : range_riemann_y(a.is, a.ie, a.js, a.je);
  const int jn = dir == 0 ? j : j + 1, in_ = dir == 0 ? i + 1 : i;
  Prim1 lwl, lwr;
  if (in_range(F, jn, in_)) lwl = adj_prim(a, dir == 0 ? A_WLNX : A_WLNY, o); else zero(lwl);
  if (in_range(F, j, i)) lwr = adj_prim(a, dir == 0 ? A_WRTX : A_WRTY, o); else zero(lwr);
  // source term: wln.(by|bz) += hdt*src, wrt.(by|bz) += hdt*src
  const double lsum = dir == 0 ? (lwl.by + lwr.by) : (lwl.bz + lwr.bz);
  const double mt = a.s(dir == 0 ? P_M2 : P_M1, o);
  const int bnp = dir == 0 ? P_B1I : P_B2I, bxp = dir == 0 ? P_B1C : P_B2C;
  const double rdx = dir == 0 ? a.fe.r_dx1 : a.fe.r_dx2;
  const double db = (a.s(bnp, o + step) - a.s(bnp, o)) * rdx;
  const Cons1 um = state_cons(a, o - step, dir), u0 = state_cons(a, o, dir), up = state_cons(a, o + step, dir);
  const double bxm = a.s(bxp, o - step), bx0 = a.s(bxp, o), bxq = a.s(bxp, o + step);
  const double dt0 = dir == 0 ? a.a(A_DT, o) : 0.0;
  // PLM
  const double hdtodx = dir == 0 ? a.c.hdtodx1 : a.c.hdtodx2;
  double di = recip(u0.d);
  const Prim1 wm = prim_of(um, bxm, recip(um.d), a.eos), w0 = prim_of(u0, bx0, di, a.eos),
              wp = prim_of(up, bxq, recip(up.d), a.eos);
  Prim1 wmb, w0b, wpb;
  double bxcb, dtodxb;
  bool fast = !(outside<-100, 100>(hdtodx) | cell_outside(um, bxm, wm.p) | cell_outside(u0, bx0, w0.p) |
                cell_outside(up, bxq, wp.p));
  if (fast) fast = plm_cell_adj_fast(wm, w0, wp, di, bx0, hdtodx, a.eos, lwl, lwr, wmb, w0b, wpb, bxcb, dtodxb);
  if (!fast) {
    Prim1 x, y, z;
    double bb, tb;
    plm_adj_general(um, u0, up, bxm, bx0, bxq, dir == 0 ? a.c.dtodx1 : a.c.dtodx2, a.eos, lwl, lwr, &x, &y, &z, &bb,
                    &tb);
    wmb = x; w0b = y; wpb = z;
    bxcb = bb;
    dtodxb = tb;
    di = 1.0 / u0.d;
  }
  // source term: src = (mt / d) db, d(B)/dx in db
  const double v0 = mt * di, lsrc = a.c.hdt * lsum;
  double dtb = 0.5 * v0 * db * lsum;
  const double ld = -(lsrc * v0 * di * db);
  if (dir == 0) {
    const int p[3] = {P_M2, P_D, P_B1C};
    const double v[3] = {lsrc * db * di, ld, bxcb};
    lin_add(a, o, p, v);
  } else {
    const int p[2] = {P_M1, P_B2C};
    const double v[2] = {lsrc * db * di, bxcb};
    lin_add(a, o, p, v);
    a.a(A_PLMYD, o) = ld;
  }
  a.a(dir == 0 ? A_SRCX : A_SRCY, o) = lsrc;
  adj_put_prim(a, dir == 0 ? A_WXM : A_WYM, o, wmb);
  adj_put_prim(a, dir == 0 ? A_WX0 : A_WY0, o, w0b);
  adj_put_prim(a, dir == 0 ? A_WXP : A_WYP, o, wpb);
  dtb += dtodxb * rdx;
  if (dir == 0) a.a(A_DT, o) = dt0 + dtb;
  else a.a(A_DTY, o) = dtb;
}

// Primitive-variable adjoints of cell (j,i) of sweep dir gathered from the PLM
// of cells c-1, c, c+1, back through cons -> prim, and the adjoint of the
// normal face field of face (j,i) (Riemann states, source terms), returned.
// Cells of the PLM range widened by one along the sweep.
ATHB_HD double adj_prim_gather(const AdjArgs& a, int dir, int j, int i, double di, Cons1& ub, double& bxb) {
  const long long o = a.o(j, i);
  const long long step = dir == 0 ? 1 : a.pitch;
  const GenRange L = range_plm(a.is, a.ie, a.js, a.je);
  const int jm = dir == 0 ? j : j - 1, im = dir == 0 ? i - 1 : i;   // previous cell along the sweep
  const int jp = dir == 0 ? j : j + 1, ip = dir == 0 ? i + 1 : i;   // next cell
  const bool in0 = in_range(L, j, i), inm = in_range(L, jm, im), inp = in_range(L, jp, ip);
  auto sum = [&](int k) {
    return (a.av_if(in0, (dir == 0 ? A_WX0 : A_WY0) + k, o, o) + a.av_if(inm, (dir == 0 ? A_WXP : A_WYP) + k, o - step, o)) +
           a.av_if(inp, (dir == 0 ? A_WXM : A_WYM) + k, o + step, o);
  };
  const Prim1 lw{sum(0), sum(1), sum(2), sum(3), sum(4), sum(5), sum(6)};
  cons_to_prim_adj(state_cons(a, o, dir), a.s(dir == 0 ? P_B1C : P_B2C, o), a.eos, di, lw, ub, bxb);
  // normal face field at face (j,i)
  const GenRange F = dir == 0 ? range_riemann_x(a.is, a.ie, a.js, a.je) : range_riemann_y(a.is, a.ie, a.js, a.je);
  const int mtp = dir == 0 ? P_M2 : P_M1;
  const int src = dir == 0 ? A_SRCX : A_SRCY;
  const double bn = a.av_if(in_range(F, j, i), dir == 0 ? A_BNX : A_BNY, o, o);
  // src(c) = (Mt/d)(c) (B(c+1) - B(c)) / dx: face (j,i) is B(c) of cell (j,i) and B(c+1) of the previous cell
  const long long om = inm ? o - step : o;
  const double s0 = a.av_if(in0, src, o, o) * any_quot(a.s(mtp, o), a.s(P_D, o), di);
  const double sm = a.av_if(inm, src, om, o) * ratio(a.s(mtp, om), a.s(P_D, om));
  return dir == 0 ? (bn - per_dx1(a, s0)) + per_dx1(a, sm) : (bn - per_dx2(a, s0)) + per_dx2(a, sm);
}

// Both sweeps of cell (j,i) onto lin, one read and one write of each plane;
// items over [is-3, ie+3] x [js-3, je+3].
ATHB_HD void adj_prim(const AdjArgs& a, int j, int i) {
  const long long o = a.o(j, i);
  const bool gx = j >= a.js - 2 && j <= a.je + 2, gy = i >= a.is - 2 && i <= a.ie + 2;
  if (!gx && !gy) return;
  const bool plm = gx && gy;   // range_plm
  const double di = any_recip(a.s(P_D, o));
  const int p[10] = {P_D, P_E, P_M1, P_M2, P_M3, P_B1C, P_B2C, P_B3C, P_B1I, P_B2I};
  double v[10];
#pragma unroll
  for (int k = 0; k < 10; k++) v[k] = a.li(p[k], o);
  if (plm) {
    a.a(A_DT, o) += a.av(A_DTY, o);
    v[0] += a.av(A_PLMYD, o);
  }
  if (gx) {
    Cons1 ub;
    zero(ub);
    double bxb = 0.0;
    v[8] += adj_prim_gather(a, 0, j, i, di, ub, bxb);
    v[0] += ub.d; v[1] += ub.e; v[2] += ub.mx; v[3] += ub.my; v[4] += ub.mz;
    v[6] += ub.by; v[7] += ub.bz; v[5] += bxb;
  }
  if (gy) {
    Cons1 ub;
    zero(ub);
    double bxb = 0.0;
    v[9] += adj_prim_gather(a, 1, j, i, di, ub, bxb);
    v[0] += ub.d; v[1] += ub.e; v[3] += ub.mx; v[4] += ub.my; v[2] += ub.mz;
    v[7] += ub.by; v[5] += ub.bz; v[6] += bxb;
  }
#pragma unroll
  for (int k = 0; k < 10; k++) a.li(p[k], o) = v[k];
}

// ===========================================================================
// Ghost zones (src/set_bvals.c:114-145): the generic fill and its adjoint.
// ===========================================================================
constexpr int kNghostA = 4;   // ghost layers (nghost, src/defs.h:82)

struct GhostGeom {
  int is, ie, js, je, sx, sy;
  int bc[4];
};

// Source index of ghost position k along one direction (lo..hi interior, the
// normal-field kind keeps hi+1 interior), flip for a reflecting wall; the
// reference's index sets (src/set_bvals.c: reflect / outflow / periodic).
ATHB_HD int ghost_map1(int k, int lo, int hi, bool bnorm, int bc_in, int bc_out, bool& flip) {
  flip = false;
  if (k < lo) {
    const int m = lo - k;
    if (bc_in == BC_REFLECT) { flip = true; return lo + (m - 1); }
    if (bc_in == BC_OUTFLOW) return lo;
    return hi - (m - 1);
  }
  if (k > hi + (bnorm ? 1 : 0)) {
    const int m = k - hi;
    if (bc_out == BC_REFLECT) { flip = true; return bnorm ? hi - (m - 2) : hi - (m - 1); }
    if (bc_out == BC_OUTFLOW) return hi;
    return lo + (m - 1);
  }
  return k;
}

// Generic fill of frame cell (j,i) of every plane: x2 map then x1 map.
template <class T>
ATHB_HD void gen_ghost(const Planes<T>& s, long long ps, int pitch, const GhostGeom& g, int j, int i) {
  const bool gxa = i < g.is || i > g.ie, gya = j < g.js || j > g.je;
  for (int kind = 0; kind < 3; kind++) {
    const int ie_int = g.ie + (kind == 1 ? 1 : 0), je_int = g.je + (kind == 2 ? 1 : 0);
    const bool gx = i < g.is || i > ie_int, gy = j < g.js || j > je_int;
    if (!gx && !gy) continue;
    bool f1 = false, f2 = false;
    const int sj = gy ? ghost_map1(j, g.js, g.je, kind == 2, g.bc[2], g.bc[3], f2) : j;
    const int si = gx ? ghost_map1(i, g.is, g.ie, kind == 1, g.bc[0], g.bc[1], f1) : i;
    const long long so = (long long)sj * pitch + si, o = (long long)j * pitch + i;
    if (kind == 0) {
      for (int p = 0; p < 8; p++) {
        T v = s.get(p * ps + so);
        if ((p == P_M1 && f1) || (p == P_M2 && f2)) v = -v;
        s.set(p * ps + o, v);
      }
      s.set(P_B3I * ps + o, s.get(P_B3I * ps + so));
    } else {
      const int p = kind == 1 ? P_B1I : P_B2I;
      s.set(p * ps + o, s.get(p * ps + so));
    }
  }
  (void)gxa; (void)gya;
}

// The kind of a plane at the boundaries: 1 for B1i, 2 for B2i, else 0.
ATHB_HD int plane_kind(int p) { return p == P_B1I ? 1 : p == P_B2I ? 2 : 0; }

// The fill reversed on plane p at place (j,i), one the step writes: the ghost
// rows that copy row j added (x2), in every column, then the ghost columns
// that copy column i, each with its ghost rows added first (x1): the order of
// the fill backwards.  Ghosts are read and never written, so one pass does it.
// One item per plane and place (11 times the threads, none with a chain of 11
// planes).
ATHB_HD void fold_ghost(double* l, long long ps, int pitch, const GhostGeom& g, int p, int j, int i) {
  const int kind = plane_kind(p), ie_int = g.ie + (kind == 1 ? 1 : 0), je_int = g.je + (kind == 2 ? 1 : 0);
  if (j < g.js || j > je_int || i < g.is || i > ie_int) return;
  double* q = l + p * ps;
  int row[2 * kNghostA];   // 0, or the ghost row's sign: rows js-4..js-1, je_int+1..je_int+4
#pragma unroll
  for (int k = 0; k < 2 * kNghostA; k++) {
    const int jj = k < kNghostA ? g.js - kNghostA + k : je_int + 1 + (k - kNghostA);
    bool f = false;
    row[k] = jj < 0 || jj >= g.sy || ghost_map1(jj, g.js, g.je, kind == 2, g.bc[2], g.bc[3], f) != j ? 0
             : p == P_M2 && f                                                                        ? -1
                                                                                                     : 1;
  }
  auto column = [&](int ii) {
    double v = q[(long long)j * pitch + ii];
#pragma unroll
    for (int k = 0; k < 2 * kNghostA; k++) {
      if (row[k] == 0) continue;
      const int jj = k < kNghostA ? g.js - kNghostA + k : je_int + 1 + (k - kNghostA);
      const double x = q[(long long)jj * pitch + ii];
      v += row[k] < 0 ? -x : x;
    }
    return v;
  };
  double v = column(i);
#pragma unroll
  for (int k = 0; k < 2 * kNghostA; k++) {   // the ghost columns: is-4..is-1, ie_int+1..ie_int+4
    const int ii = k < kNghostA ? g.is - kNghostA + k : ie_int + 1 + (k - kNghostA);
    bool f = false;
    if (ii < 0 || ii >= g.sx || ghost_map1(ii, g.is, g.ie, kind == 1, g.bc[0], g.bc[1], f) != i) continue;
    const double x = column(ii);
    v += (p == P_M1 && f) ? -x : x;
  }
  q[(long long)j * pitch + i] = v;
}
// Zero plane p at a place that is not one the step writes (ghosts after the
// fold), so the folded adjoint is exactly the interior one.
ATHB_HD void clear_frame(double* l, long long ps, int pitch, const GhostGeom& g, int p, int j, int i) {
  const int kind = plane_kind(p);
  const bool keep = j >= g.js && j <= g.je + (kind == 2 ? 1 : 0) && i >= g.is && i <= g.ie + (kind == 1 ? 1 : 0);
  if (!keep) l[p * ps + (long long)j * pitch + i] = 0.0;
}

}  // namespace athb
