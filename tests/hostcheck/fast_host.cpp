// Host build of mhd_fast.cuh for tests/test_fast_physics_cpu.py: each entry
// runs the fast and the general form on the same operands and returns their
// outputs.
#include <cmath>

#include "mhd_adjoint.cuh"

using namespace athb;

namespace {
Prim1 prim(const double* w) { return Prim1{w[0], w[1], w[2], w[3], w[4], w[5], w[6]}; }
void put(const Prim1& w, double* o) {
  o[0] = w.d; o[1] = w.vx; o[2] = w.vy; o[3] = w.vz; o[4] = w.p; o[5] = w.by; o[6] = w.bz;
}
void put(const Cons1& u, double* o) {
  o[0] = u.d; o[1] = u.mx; o[2] = u.my; o[3] = u.mz; o[4] = u.e; o[5] = u.by; o[6] = u.bz;
}
}  // namespace

extern "C" {

// op 0: 1/x, 1: sqrt(x), 2: y/x with the reciprocal of x, 3: 1/sqrt(x) from the root's by-product,
// 4: the by-product itself, 1/(2 sqrt(x)) to about an ulp
void fast_ops(int op, int n, const double* x, const double* y, double* fast, double* plain) {
  for (int k = 0; k < n; k++) {
    double h;
    switch (op) {
    case 0: fast[k] = recip(x[k]); plain[k] = 1.0 / x[k]; break;
    case 1: fast[k] = root(x[k]); plain[k] = std::sqrt(x[k]); break;
    case 2: fast[k] = quot(y[k], x[k], recip(x[k])); plain[k] = y[k] / x[k]; break;
    case 4: root(x[k], fast[k]); plain[k] = 0.5 / std::sqrt(x[k]); break;
    default: {
      const double g = root(x[k], h);
      fast[k] = recip_of_root(g, h);
      plain[k] = 1.0 / std::sqrt(x[k]);
    }
    }
  }
}

// n cells: w = 3 primitive states (m, 0, p) of 7 each, bx = their normal
// fields (3 each); out: 14 values of each form.  took[k]: the fast form
// vouches for them.
void fast_plm(int n, const double* w, const double* bx, const double* dtodx, double gamma, int* took, double* fast,
              double* plain) {
  const Eos eos{gamma, gamma - 1.0, gamma - 2.0};
  for (int k = 0; k < n; k++) {
    Prim1 p[3];
    bool bad = false;
    for (int c = 0; c < 3; c++) {
      p[c] = prim(w + 21 * k + 7 * c);
      Cons1 u = prim_to_cons(p[c], bx[3 * k + c], eos);
      bad |= cell_outside(u, bx[3 * k + c], p[c].p);
    }
    Prim1 l, r;
    plm_cell(p[0], p[1], p[2], bx[3 * k + 1], dtodx[k], eos, l, r);
    put(l, plain + 14 * k);
    put(r, plain + 14 * k + 7);
    const bool done = plm_cell_fast(p[0], p[1], p[2], recip(p[1].d), bx[3 * k + 1], 0.5 * dtodx[k], eos, l, r);
    took[k] = !bad && done;
    put(l, fast + 14 * k);
    put(r, fast + 14 * k + 7);
  }
}

// Adjoints of n cells as fast_plm's, lam = adjoints of the left and right
// states; out: 23 values of each form (m, 0, p states, normal field, dtodx).
void fast_plm_adj(int n, const double* w, const double* bx, const double* dtodx, const double* lam, double gamma,
                  int* took, double* fast, double* plain) {
  const Eos eos{gamma, gamma - 1.0, gamma - 2.0};
  for (int k = 0; k < n; k++) {
    Prim1 p[3];
    for (int c = 0; c < 3; c++) p[c] = prim(w + 21 * k + 7 * c);
    const Prim1 ll = prim(lam + 14 * k), lr = prim(lam + 14 * k + 7);
    Prim1 m, z, q;
    double b = 0.0, t = 0.0;
    zero(m); zero(z); zero(q);
    plm_cell_adj(p[0], p[1], p[2], bx[3 * k + 1], dtodx[k], eos, ll, lr, m, z, q, b, t);
    double* o = plain + 23 * k;
    put(m, o); put(z, o + 7); put(q, o + 14);
    o[21] = b; o[22] = t;
    took[k] = plm_cell_adj_fast(p[0], p[1], p[2], recip(p[1].d), bx[3 * k + 1], 0.5 * dtodx[k], eos, ll, lr, m, z, q,
                                b, t);
    o = fast + 23 * k;
    put(m, o); put(z, o + 7); put(q, o + 14);
    o[21] = b; o[22] = t;
  }
}

// n faces: w = left and right primitive states, bx the normal field, lam the
// adjoint of the flux; out: the adjoints of Ul, Ur, Wl, Wr and of the field.
void fast_roe_adj(int n, const double* w, const double* bx, const double* lam, double gamma, int* took, double* fast,
                  double* plain) {
  const Eos eos{gamma, gamma - 1.0, gamma - 2.0};
  for (int k = 0; k < n; k++) {
    const Prim1 wl = prim(w + 14 * k), wr = prim(w + 14 * k + 7), l = prim(lam + 7 * k);
    const Cons1 ul = prim_to_cons(wl, bx[k], eos), ur = prim_to_cons(wr, bx[k], eos);
    const Cons1 fb{l.d, l.vx, l.vy, l.vz, l.p, l.by, l.bz};
    for (int form = 0; form < 2; form++) {
      Cons1 a, b;
      Prim1 c, d;
      double t = 0.0;
      zero(a); zero(b); zero(c); zero(d);
      if (form) flux_roe_adj(ul, ur, wl, wr, bx[k], eos, fb, a, b, c, d, t);
      else took[k] = flux_roe_adj_fast(ul, ur, wl, wr, bx[k], eos, 1.0 / eos.gamma_1, fb, a, b, c, d, t);
      double* o = (form ? plain : fast) + 29 * k;
      put(a, o); put(b, o + 7); put(c, o + 14); put(d, o + 21);
      o[28] = t;
    }
  }
}

// n faces: w = left and right primitive states, bx the normal field.
void fast_flux(int hlle, int n, const double* w, const double* bx, double gamma, int* took, double* fast,
               double* plain) {
  const Eos eos{gamma, gamma - 1.0, gamma - 2.0};
  for (int k = 0; k < n; k++) {
    const Prim1 wl = prim(w + 14 * k), wr = prim(w + 14 * k + 7);
    const Cons1 ul = prim_to_cons(wl, bx[k], eos), ur = prim_to_cons(wr, bx[k], eos);
    Cons1 F{};
    unsigned fails;
    if (hlle) {
      took[k] = flux_hlle_fast(ul, ur, wl, wr, bx[k], eos, F);
      put(flux_hlle(ul, ur, wl, wr, bx[k], eos), plain + 7 * k);
    } else {
      took[k] = flux_roe_fast(ul, ur, wl, wr, bx[k], eos, 1.0 / eos.gamma_1, F, fails);
      put(flux_roe(ul, ur, wl, wr, bx[k], eos), plain + 7 * k);
    }
    put(F, fast + 7 * k);
  }
}

// n faces as fast_flux's through face_flux, and riemann; fallback[k]: the Roe
// solver knows an intermediate state that fails its test.
void fast_face(int hlle, int n, const double* w, const double* bx, double gamma, int* fallback, double* fast,
               double* plain) {
  const Eos eos{gamma, gamma - 1.0, gamma - 2.0};
  const FastEos fe = make_fast_eos(eos, 0.01, 0.01);
  for (int k = 0; k < n; k++) {
    const Prim1 wl = prim(w + 14 * k), wr = prim(w + 14 * k + 7);
    const Cons1 ul = prim_to_cons(wl, bx[k], eos), ur = prim_to_cons(wr, bx[k], eos);
    Cons1 F;
    unsigned fails = 0;
    if (!hlle) (void)flux_roe_fast(ul, ur, wl, wr, bx[k], eos, fe.r_gamma_1, F, fails);
    fallback[k] = fails != 0;
    put(hlle ? face_flux<kFluxHlle>(ul, ur, wl, wr, bx[k], eos, fe) : face_flux<kFluxRoe>(ul, ur, wl, wr, bx[k], eos, fe),
        fast + 7 * k);
    put(hlle ? riemann<kFluxHlle>(ul, ur, wl, wr, bx[k], eos) : riemann<kFluxRoe>(ul, ur, wl, wr, bx[k], eos),
        plain + 7 * k);
  }
}

}  // extern "C"
