// Continuous collision detection: swept boxes, coplanarity-cubic time of
// impact (ccd/ccd.py:166-427, ccd/cubic_roots.py:7-193), all root arithmetic
// in double.  This file is compiled with -fmad=false: every operation rounds
// on its own, in source order, so the TOI is reproducible bit for bit by a
// plain IEEE evaluation.
#include <type_traits>

#include "bodies.cuh"
#include "common.cuh"
#include "geom.cuh"
#include "lbvh.cuh"
#include "records.cuh"
#include "tree.cuh"

namespace ipcb {
int check_launch(const char* where);

namespace {

constexpr int kFindIters = 200;  // bound on the bracketed Newton/bisection loop
constexpr double kXError = 1e-10;  // cubic_roots.py:4

struct Q4 {
  double c[4];
};
struct D3v {
  double v[3];
};

IPCB_D double evaluate(const Q4& p, double x) { return p.c[0] + x * (p.c[1] + x * (p.c[2] + x * p.c[3])); }
IPCB_D double multi_sign(double a, double b) { return b < 0.0 ? -a : a; }
IPCB_D bool diff_sign(double y0, double yr) { return y0 * yr < 0.0; }
IPCB_D double dmin(double a, double b) { return a < b ? a : b; }
IPCB_D double dmax(double a, double b) { return a > b ? a : b; }

IPCB_D D3v deflate(const Q4& p, double root) {
  D3v d;
  d.v[2] = p.c[3];
  d.v[1] = p.c[2] + root * d.v[2];
  d.v[0] = p.c[1] + root * d.v[1];
  return d;
}

IPCB_D double find_closed(const Q4& p, const Q4& dp, double x0, double x1, double y0, double y1, int& status) {
  (void)y1;
  double xr = (x0 + x1) / 2.0;
  double yr = evaluate(p, xr);
  double xb0 = x0, xb1 = x1;
  if (x1 - x0 <= kXError * 2.0) return xr;
  for (int it = 0;; ++it) {
    if (it >= kFindIters) {
      status |= IPCB_STATUS_ROOT_ITERS;
      break;
    }
    if (diff_sign(y0, yr)) xb1 = xr;
    else xb0 = xr;
    double dy = evaluate(dp, xr);
    double dx = yr / dy;
    double xn = xr - dx;
    if (xn > xb0 && xn < xb1) {
      double step = fabs(xr - xn);
      xr = xn;
      if (step > kXError) yr = evaluate(p, xr);
      else break;
    } else {
      xr = (xb0 + xb1) / 2.0;
      yr = evaluate(p, xr);
      if (xb0 == xr || xb1 == xr || xb1 - xb0 <= 2.0 * kXError) break;
    }
  }
  return xr;
}

IPCB_D int quadratic_roots(const D3v& q, double x0, double x1, double* roots) {
  double c = q.v[0], b = q.v[1], a = q.v[2];
  double delta = b * b - 4.0 * a * c;
  int ret = 0;
  roots[0] = roots[1] = 0.0;
  if (delta > 0.0) {
    double d = sqrt(delta);
    double qq = -(b + multi_sign(d, b)) * 0.5;
    double rv0 = qq / a, rv1 = c / qq;
    double xa = dmin(rv0, rv1), xb = dmax(rv0, rv1);
    if (xa >= x0 && xa <= x1) roots[ret++] = xa;
    if (xb >= x0 && xb <= x1) roots[ret++] = xb;
  } else if (delta < 0.0) {
    ret = 0;
  } else {
    double r0 = -0.5 * b / a;
    roots[0] = r0;
    if (r0 >= x0 && r0 <= x1) ret = 1;
  }
  return ret;
}

// cubic_roots.py:96-193: real roots in [x0, x1], ascending.
IPCB_D int cubic_roots(const Q4& p, double x0, double x1, double* roots, int& status) {
  roots[0] = roots[1] = roots[2] = 0.0;
  double y0 = evaluate(p, x0), y1 = evaluate(p, x1);
  double a = p.c[3] * 3.0, b_2 = p.c[2], c = p.c[1];
  Q4 dp{{c, 2.0 * b_2, a, 0.0}};
  double delta_4 = b_2 * b_2 - a * c;
  double q2[2];
  if (delta_4 > 0.0) {
    double d_2 = sqrt(delta_4);
    double q = -(b_2 + multi_sign(d_2, b_2));
    double rv0 = q / a, rv1 = c / q;
    double xa = dmin(rv0, rv1), xb = dmax(rv0, rv1);
    if (diff_sign(y0, y1)) {
      if (xa >= x1 || xb <= x0 || (xa <= x0 && xb >= x1)) {
        roots[0] = find_closed(p, dp, x0, x1, y0, y1, status);
        return 1;
      }
    } else {
      if (xa >= x1 || xb <= x0 || (xa <= x0 && xb >= x1)) return 0;
    }
    if (xa > x0) {
      double ya = evaluate(p, xa);
      if (diff_sign(y0, ya)) {
        roots[0] = find_closed(p, dp, x0, xa, y0, ya, status);
        if (diff_sign(ya, y1) || (xb < x1 && diff_sign(ya, evaluate(p, xb)))) {
          int r = quadratic_roots(deflate(p, roots[0]), xa, x1, q2);
          roots[1] = q2[0];
          roots[2] = q2[1];
          return r + 1;
        }
        return 1;
      }
      if (xb < x1) {
        double yb = evaluate(p, xb);
        if (diff_sign(ya, yb)) {
          roots[0] = find_closed(p, dp, xa, xb, ya, yb, status);
          if (diff_sign(yb, y1)) {
            int r = quadratic_roots(deflate(p, roots[0]), xb, x1, q2);
            roots[1] = q2[0];
            roots[2] = q2[1];
            return r + 1;
          }
          return 1;
        }
        if (diff_sign(yb, y1)) {
          roots[0] = find_closed(p, dp, xb, x1, yb, y1, status);
          return 1;
        }
      } else if (diff_sign(ya, y1)) {
        roots[0] = find_closed(p, dp, xa, x1, ya, y1, status);
        return 1;
      }
    } else {
      double yb = evaluate(p, xb);
      if (diff_sign(y0, yb)) {
        roots[0] = find_closed(p, dp, x0, xb, y0, yb, status);
        if (diff_sign(yb, y1)) {
          int r = quadratic_roots(deflate(p, roots[0]), xb, x1, q2);
          roots[1] = q2[0];
          roots[2] = q2[1];
          return r + 1;
        }
        return 1;
      }
      if (diff_sign(yb, y1)) {
        roots[0] = find_closed(p, dp, xb, x1, yb, y1, status);
        return 1;
      }
    }
    return 0;
  }
  if (diff_sign(y0, y1)) {
    roots[0] = find_closed(p, dp, x0, x1, y0, y1, status);
    return 1;
  }
  return 0;
}

// ccd.py:293-300: coefficients of prod_k (b_k + t a_k), ascending powers
IPCB_D Q4 cubic_binomial(double a0, double a1, double a2, double b0, double b1, double b2) {
  Q4 r;
  r.c[0] = b0 * b1 * b2;
  r.c[1] = a0 * b1 * b2 + b0 * b1 * a2 + b0 * a1 * b2;
  r.c[2] = a0 * a1 * b2 + a0 * b1 * a2 + b0 * a1 * a2;
  r.c[3] = a0 * a1 * a2;
  return r;
}

// det(B + t A) for 3x3 matrices given by columns (ccd.py:252-290)
IPCB_D Q4 det_polynomial(const d3* A, const d3* B) {
  // M[r][c] = col_c[r]
  auto m = [](const d3* C, int r, int c) -> double { return r == 0 ? C[c].x : (r == 1 ? C[c].y : C[c].z); };
  Q4 pos{{0, 0, 0, 0}}, neg{{0, 0, 0, 0}};
  const int P[3][3][2] = {{{0, 0}, {1, 1}, {2, 2}}, {{0, 1}, {1, 2}, {2, 0}}, {{0, 2}, {1, 0}, {2, 1}}};
  const int N[3][3][2] = {{{0, 0}, {1, 2}, {2, 1}}, {{0, 1}, {1, 0}, {2, 2}}, {{0, 2}, {1, 1}, {2, 0}}};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    Q4 t = cubic_binomial(m(A, P[k][0][0], P[k][0][1]), m(A, P[k][1][0], P[k][1][1]), m(A, P[k][2][0], P[k][2][1]),
                          m(B, P[k][0][0], P[k][0][1]), m(B, P[k][1][0], P[k][1][1]), m(B, P[k][2][0], P[k][2][1]));
#pragma unroll
    for (int q = 0; q < 4; ++q) pos.c[q] = pos.c[q] + t.c[q];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    Q4 t = cubic_binomial(m(A, N[k][0][0], N[k][0][1]), m(A, N[k][1][0], N[k][1][1]), m(A, N[k][2][0], N[k][2][1]),
                          m(B, N[k][0][0], N[k][0][1]), m(B, N[k][1][0], N[k][1][1]), m(B, N[k][2][0], N[k][2][1]));
#pragma unroll
    for (int q = 0; q < 4; ++q) neg.c[q] = neg.c[q] + t.c[q];
  }
  Q4 r;
#pragma unroll
  for (int q = 0; q < 4; ++q) r.c[q] = pos.c[q] - neg.c[q];
  return r;
}

// ccd.py:226-249: roots in [0,1] of det[p1-p0 ...] coplanarity polynomial
IPCB_D int coplanar_roots(const d3* p0, const d3* p1, double* roots, int& status) {
  const int cols[4][3] = {{1, 2, 3}, {0, 2, 3}, {0, 1, 3}, {0, 1, 2}};
  Q4 acc{{0, 0, 0, 0}};
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    d3 A[3], B[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      B[c] = p0[cols[m][c]];
      A[c] = p1[cols[m][c]] - p0[cols[m][c]];
    }
    Q4 d = det_polynomial(A, B);
    double sg = (m & 1) ? -1.0 : 1.0;
    if (m == 0) acc = d;
    else
#pragma unroll
      for (int q = 0; q < 4; ++q) acc.c[q] = sg > 0 ? acc.c[q] + d.c[q] : acc.c[q] - d.c[q];
  }
  return cubic_roots(acc, 0.0, 1.0, roots, status);
}

IPCB_D d3 lerp(d3 a, d3 b, double t) { return a * (1.0 - t) + b * t; }

// Least-squares coordinates of the coplanar configuration (ipctkwp
// beta_gamma_pt/ee, restated): PT solves x0 - x1 = beta e1 + gamma e2,
// EE solves x2 - x0 = beta ea + gamma eb.
IPCB_D void solve2(double a11, double a12, double a22, double b1, double b2, double& be, double& ga) {
  double det = a11 * a22 - a12 * a12;
  be = (b1 * a22 - a12 * b2) / det;
  ga = (a11 * b2 - a12 * b1) / det;
}

IPCB_D bool verify_pt(const d3* x) {
  d3 e1 = x[2] - x[1], e2 = x[3] - x[1], w = x[0] - x[1];
  double be, ga;
  solve2(dot(e1, e1), dot(e1, e2), dot(e2, e2), dot(e1, w), dot(e2, w), be, ga);
  const double tol = 1e-8;
  return be >= -tol && ga >= -tol && be + ga <= 1.0 + tol;
}

IPCB_D bool verify_ee(const d3* x) {
  d3 ea = x[1] - x[0], eb = x[3] - x[2], w = x[2] - x[0];
  double be, ga;
  solve2(dot(ea, ea), dot(ea, eb), dot(eb, eb), dot(ea, w), dot(eb, w), be, ga);
  const double tol = 1e-8;
  return be >= -tol && be <= 1.0 + tol && -ga >= -tol && -ga <= 1.0 + tol;
}

// ccd.py:304-357
template <int KIND>
IPCB_D double collision_time(const d3* p0, const d3* p1, int& status) {
  double roots[3];
  int nr = coplanar_roots(p0, p1, roots, status);
  double root = 1.0;
  bool ok = false;
  for (int i = 0; i < nr; ++i) {
    root = roots[i];
    d3 xt[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) xt[k] = lerp(p0[k], p1[k], root);
    ok = KIND == 0 ? verify_ee(xt) : verify_pt(xt);
    if (ok) break;
  }
  return ok ? root : 1.0;
}

template <class S>
IPCB_D d3 ld(const S* __restrict__ x, int i) {
  return mk3((double)__ldg(x + 3 * i), (double)__ldg(x + 3 * i + 1), (double)__ldg(x + 3 * i + 2));
}

IPCB_D void store_toi(float* toi, double t) { atomic_min_nonneg(toi, __double2float_rz(t)); }
IPCB_D void store_toi(double* toi, double t) { atomic_min_nonneg(toi, t); }

// Optional output of new_intersections (contact.py:587-670): every pair whose
// time of impact is < 1 is appended as a record (append_ccd, contact.py:186-197:
// a1a2b1b2, e0e1 = (query primitive, hit primitive), l0 = 2 thickness,
// alpha = toi, lam = 0); records beyond the capacity are only counted.
struct Sink {
  ipcb_contacts L;
  double l0;
  int on;
};

template <class S>
IPCB_D void sink_append(const Sink& k, int4 ids, int e0, int e1, double t) {
  if (!k.on) return;
  const int idx = atomicAdd(k.L.cnt, 1);
  if (idx >= k.L.capacity) return;
  reinterpret_cast<int4*>(k.L.a1a2b1b2)[idx] = ids;
  reinterpret_cast<int2*>(k.L.e0e1)[idx] = make_int2(e0, e1);
  static_cast<S*>(k.L.l0)[idx] = S(k.l0);
  static_cast<S*>(k.L.alpha)[idx] = sizeof(S) == 4 ? S(__double2float_rz(t)) : S(t);
  static_cast<S*>(k.L.lam)[idx] = S(0);
}

template <class S>
__global__ void k_add_dx(const S* __restrict__ x, const S* __restrict__ dx, S* __restrict__ x1, int n3) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n3) x1[i] = x[i] - dx[i];
}

template <class S, int NV>
__global__ void k_swept(const S* __restrict__ x0, const S* __restrict__ x1, const int* __restrict__ prims, int n,
                        double pad, float* __restrict__ lo, float* __restrict__ hi) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    int k = __ldg(prims + NV * i + v);
    d3 a = ld(x0, k), b = ld(x1, k);
    mn[0] = dmin(mn[0], dmin(a.x, b.x)); mx[0] = dmax(mx[0], dmax(a.x, b.x));
    mn[1] = dmin(mn[1], dmin(a.y, b.y)); mx[1] = dmax(mx[1], dmax(a.y, b.y));
    mn[2] = dmin(mn[2], dmin(a.z, b.z)); mx[2] = dmax(mx[2], dmax(a.z, b.z));
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lo[3 * i + k] = __double2float_rd(mn[k] - pad);
    hi[3 * i + k] = __double2float_ru(mx[k] + pad);
  }
}

// Candidate pairs are staged in a list so the cubic solves run one pair per
// thread (balanced) instead of inside divergent traversal loops (layout of the
// workspace: cand_list, cand_order).  When a pair finds the list full the
// overflow flag is raised and an inline pass solves every pair of the query
// during traversal, so the result never depends on the capacity.
struct CandList {
  int* count;
  int* overflow;  // set by a collect pass that dropped pairs (the inline pass then redoes the query)
  int2* pairs;
  int capacity;
};


// ---- exact skip of pairs that cannot reach contact within the step ----
// The primitives move linearly, so their distance obeys
//   d(t) >= d(0) - t * (max_a |dx_a - m| + max_b |dx_b - m|)
// for any common translation m (the vertex-mean here).  A verified root needs
// the primitives to touch up to the barycentric tolerance of the root check
// (1e-8 in parameter units), so a pair with d(0) - motion above a margin of
// 1e-6 (1 + extent) returns 1 from the cubic path; skipping it does not change
// the TOI.
IPCB_D double seg_seg_dist(d3 p1, d3 q1, d3 p2, d3 q2) {
  d3 d1 = q1 - p1, d2 = q2 - p2, r = p1 - p2;
  double a = dot(d1, d1), e = dot(d2, d2), f = dot(d2, r);
  double s = 0, t = 0;
  if (a <= 1e-30 && e <= 1e-30) {
  } else if (a <= 1e-30) {
    t = fmin(fmax(f / e, 0.0), 1.0);
  } else {
    double c = dot(d1, r);
    if (e <= 1e-30) {
      s = fmin(fmax(-c / a, 0.0), 1.0);
    } else {
      double b = dot(d1, d2), den = a * e - b * b;
      s = den > 0 ? fmin(fmax((b * f - c * e) / den, 0.0), 1.0) : 0.0;
      t = (b * s + f) / e;
      if (t < 0) {
        t = 0;
        s = fmin(fmax(-c / a, 0.0), 1.0);
      } else if (t > 1) {
        t = 1;
        s = fmin(fmax((b - c) / a, 0.0), 1.0);
      }
    }
  }
  d3 w = (p1 + d1 * s) - (p2 + d2 * t);
  return sqrt(dot(w, w));
}

IPCB_D double pt_dist(d3 p, d3 a, d3 b, d3 c) {
  d3 ab = b - a, ac = c - a, ap = p - a;
  double d1 = dot(ab, ap), d2 = dot(ac, ap);
  if (d1 <= 0 && d2 <= 0) return sqrt(dot(ap, ap));
  d3 bp = p - b;
  double d3v = dot(ab, bp), d4 = dot(ac, bp);
  if (d3v >= 0 && d4 <= d3v) return sqrt(dot(bp, bp));
  double vc = d1 * d4 - d3v * d2;
  if (vc <= 0 && d1 >= 0 && d3v <= 0) {
    d3 w = p - (a + ab * (d1 / (d1 - d3v)));
    return sqrt(dot(w, w));
  }
  d3 cp = p - c;
  double d5 = dot(ab, cp), d6 = dot(ac, cp);
  if (d6 >= 0 && d5 <= d6) return sqrt(dot(cp, cp));
  double vb = d5 * d2 - d1 * d6;
  if (vb <= 0 && d2 >= 0 && d6 <= 0) {
    d3 w = p - (a + ac * (d2 / (d2 - d6)));
    return sqrt(dot(w, w));
  }
  double va = d3v * d6 - d5 * d4;
  if (va <= 0 && (d4 - d3v) >= 0 && (d5 - d6) >= 0) {
    d3 w = p - (b + (c - b) * ((d4 - d3v) / ((d4 - d3v) + (d5 - d6))));
    return sqrt(dot(w, w));
  }
  double den = va + vb + vc;
  if (!(fabs(den) > 0)) {  // degenerate triangle: distance to its edges
    return fmin(seg_seg_dist(p, p, a, b), fmin(seg_seg_dist(p, p, a, c), seg_seg_dist(p, p, b, c)));
  }
  d3 w = p - (a + ab * (vb / den) + ac * (vc / den));
  return sqrt(dot(w, w));
}

// KIND 0: (a0, a1 | b0, b1); KIND 1: (p | t0, t1, t2).  Lower bound on the
// time at which the pair can touch: (d(0) - margin) / (relative motion bound),
// 0 when it already touches, infinity when it does not move.  A verified root
// at t needs d(t) within the margin, so no root lies below the bound.
template <int KIND>
IPCB_D double touch_time_bound(const d3* p0, const d3* p1) {
  d3 dx[4];
  d3 m = mk3(0.0, 0.0, 0.0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    dx[k] = p1[k] - p0[k];
    m = m + dx[k];
  }
  m = m * 0.25;
  double ma = 0, mb = 0, ext = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    d3 u = dx[k] - m;
    double l = sqrt(dot(u, u));
    if ((KIND == 0 && k < 2) || (KIND == 1 && k < 1)) ma = fmax(ma, l);
    else mb = fmax(mb, l);
    ext = fmax(ext, fmax(fabs(p0[k].x), fmax(fabs(p0[k].y), fabs(p0[k].z))));
    ext = fmax(ext, fmax(fabs(p1[k].x), fmax(fabs(p1[k].y), fabs(p1[k].z))));
  }
  const double d0 = KIND == 0 ? seg_seg_dist(p0[0], p0[1], p0[2], p0[3]) : pt_dist(p0[0], p0[1], p0[2], p0[3]);
  const double gap = d0 - 1e-6 * (1.0 + ext);
  if (!(gap > 0.0)) return 0.0;
  const double v = ma + mb;
  return v > 0.0 ? gap / v : INFINITY;
}

template <int KIND>
IPCB_D bool cannot_touch(const d3* p0, const d3* p1) {
  d3 dx[4];
  d3 m = mk3(0.0, 0.0, 0.0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    dx[k] = p1[k] - p0[k];
    m = m + dx[k];
  }
  m = m * 0.25;
  double ma = 0, mb = 0, ext = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    d3 u = dx[k] - m;
    double l = sqrt(dot(u, u));
    if ((KIND == 0 && k < 2) || (KIND == 1 && k < 1)) ma = fmax(ma, l);
    else mb = fmax(mb, l);
    ext = fmax(ext, fmax(fabs(p0[k].x), fmax(fabs(p0[k].y), fabs(p0[k].z))));
    ext = fmax(ext, fmax(fabs(p1[k].x), fmax(fabs(p1[k].y), fabs(p1[k].z))));
  }
  double d0 = KIND == 0 ? seg_seg_dist(p0[0], p0[1], p0[2], p0[3]) : pt_dist(p0[0], p0[1], p0[2], p0[3]);
  return d0 - (ma + mb) > 1e-6 * (1.0 + ext);
}

template <class S>
IPCB_D double ee_pair_time(const S* __restrict__ x0, const S* __restrict__ x1, int2 ea, int2 eb, int& st) {
  d3 p0[4] = {ld(x0, ea.x), ld(x0, ea.y), ld(x0, eb.x), ld(x0, eb.y)};
  d3 p1[4] = {ld(x1, ea.x), ld(x1, ea.y), ld(x1, eb.x), ld(x1, eb.y)};
  if (cannot_touch<0>(p0, p1)) return 1.0;
  return collision_time<0>(p0, p1, st);
}

template <class S>
IPCB_D double pt_pair_time(const S* __restrict__ x0, const S* __restrict__ x1, int v, int3 t, int& st) {
  d3 p0[4] = {ld(x0, v), ld(x0, t.x), ld(x0, t.y), ld(x0, t.z)};
  d3 p1[4] = {ld(x1, v), ld(x1, t.x), ld(x1, t.y), ld(x1, t.z)};
  if (cannot_touch<1>(p0, p1)) return 1.0;
  return collision_time<1>(p0, p1, st);
}

constexpr int kQueue = 32;  // per-thread queue of filtered leaf hits (fixed bodies)

IPCB_D int warp_max(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// converged push: one ballot and one atomicAdd per warp; returns false for a
// lane whose pair did not fit (the caller solves it in place)
IPCB_D bool push_converged(const CandList& L, bool has, int a, int b) {
  const unsigned lane = threadIdx.x & 31;
  unsigned m = __ballot_sync(0xffffffffu, has);
  int base = 0;
  if (lane == 0 && m) base = atomicAdd(L.count, __popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  int slot = base + __popc(m & ((1u << lane) - 1u));
  if (has && slot < L.capacity) {
    L.pairs[slot] = make_int2(a, b);
    return true;
  }
  return !has;
}

// Swept boxes over [0, t_end] of the step (tree.cuh functor): over the whole
// step (t_end null or 1) exactly k_swept's.  Only the minimum TOI matters to a
// query without a sink, and a pair whose root is below the TOI stored so far
// is within the touch margin (see touch_time_bound) by that time, so boxes
// over [0, stored TOI] grown by that margin still meet for every pair that can
// lower it: the result is the same minimum, from far fewer pairs when the
// step is much longer than the first contact.
template <class S, int NV>
IPCB_D void swept_box(const S* __restrict__ x0, const S* __restrict__ x1, const int* ids, double pad, double t, f3& lo,
                      f3& hi) {
  double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const d3 a = ld(x0, ids[v]);
    d3 b = ld(x1, ids[v]);
    if (t < 1.0) b = a + (b - a) * t;
    mn[0] = dmin(mn[0], dmin(a.x, b.x)); mx[0] = dmax(mx[0], dmax(a.x, b.x));
    mn[1] = dmin(mn[1], dmin(a.y, b.y)); mx[1] = dmax(mx[1], dmax(a.y, b.y));
    mn[2] = dmin(mn[2], dmin(a.z, b.z)); mx[2] = dmax(mx[2], dmax(a.z, b.z));
  }
  if (t < 1.0) {
    double ext = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) ext = dmax(ext, dmax(fabs(mn[k]), fabs(mx[k])));
    pad += 1e-6 * (1.0 + ext);
  }
  lo = mk3(__double2float_rd(mn[0] - pad), __double2float_rd(mn[1] - pad), __double2float_rd(mn[2] - pad));
  hi = mk3(__double2float_ru(mx[0] + pad), __double2float_ru(mx[1] + pad), __double2float_ru(mx[2] + pad));
}

IPCB_D double current_toi(const float* toi) { return (double)__ldcg(toi); }
IPCB_D double current_toi(const double* toi) { return __ldcg(toi); }

template <class S, int NV>
struct SweptBox {
  const S* x0;
  const S* x1;
  const int* prims;
  double pad;
  const S* t_end;
  IPCB_D void operator()(int p, f3& lo, f3& hi) const {
    int ids[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) ids[k] = __ldg(prims + NV * p + k);
    swept_box<S, NV>(x0, x1, ids, pad, t_end ? current_toi(t_end) : 1.0, lo, hi);
  }
};

// The swept box of the whole step joined with the discrete query's box (x in
// float, padded by reach): one tree for both queries.
template <class S, int NV>
struct BothBox {
  const S* x0;
  const S* x1;
  const int* prims;
  double pad;
  float reach;
  IPCB_D void operator()(int p, f3& lo, f3& hi) const {
    int ids[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) ids[k] = __ldg(prims + NV * p + k);
    swept_box<S, NV>(x0, x1, ids, pad, 1.0, lo, hi);
    f3 a = to_f(load3(x0, ids[0])), b = a;
#pragma unroll
    for (int k = 1; k < NV; ++k) {
      const f3 q = to_f(load3(x0, ids[k]));
      a = mk3(fminf(a.x, q.x), fminf(a.y, q.y), fminf(a.z, q.z));
      b = mk3(fmaxf(b.x, q.x), fmaxf(b.y, q.y), fmaxf(b.z, q.z));
    }
    lo = mk3(fminf(lo.x, a.x - reach), fminf(lo.y, a.y - reach), fminf(lo.z, a.z - reach));
    hi = mk3(fmaxf(hi.x, b.x + reach), fmaxf(hi.y, b.y + reach), fmaxf(hi.z, b.z + reach));
  }
};

// ---- ordered candidate solve (no record sink): the collect pass computes
// each pair's touch-time bound, drops the pairs that cannot touch within the
// step or before the TOI stored so far, and counts the rest in 32 buckets over
// [0, 1]; the solve then takes the pairs in bucket order, so the pairs that
// can touch earliest set the TOI first, and a pair whose bound is at or above
// the TOI stored so far is skipped (it cannot lower the minimum: the result is
// the same minimum, bit for bit); a warp that meets a bucket starting at or
// above the stored TOI stops.  Divergence between pruned and solved pairs and
// the cubic solver's registers stay out of the collect pass.
constexpr int kBuckets = 32;
struct CandOrder {
  int* bcount;   // pairs per bucket
  int* bcursor;  // fill cursors
  int* work;     // next position of the ordered solve
  float* tlb;    // per staged pair: touch-time bound rounded down
  int* order;    // staged pair indices in bucket order
};

IPCB_D int bucket_of(float tl) { return min(kBuckets - 1, (int)(tl * (float)kBuckets)); }

template <int KIND>
IPCB_D int4 pair_ids(const int* __restrict__ prims, int2 pr) {
  if (KIND == 0) {
    const int2 ea = __ldg(reinterpret_cast<const int2*>(prims) + pr.x);
    const int2 eb = __ldg(reinterpret_cast<const int2*>(prims) + pr.y);
    return make_int4(ea.x, ea.y, eb.x, eb.y);
  }
  return make_int4(pr.x, __ldg(prims + 3 * pr.y), __ldg(prims + 3 * pr.y + 1), __ldg(prims + 3 * pr.y + 2));
}

// Lower bound on the time at which a pair can touch, in float: the distance
// along the axis n of the closest points at t = 0 (r = closest point of a -
// closest point of b, d = |r|).  n . (a_i - b_j) is linear in t for every
// vertex pair, and as long as all of them exceed the margin n separates the
// primitives by it: the earliest time one falls to the margin is the bound (a
// verified root needs the primitives within 1e-6 (1 + extent), see
// touch_time_bound).  Only the closing speed along n counts, where the
// distance-over-speed bound charges sliding motion too: a loaded thread flank
// sliding 8e-3 at a gap of 2e-5 keeps a bound near its true touch time.  The
// margin covers the float rounding of the (locally formed) dots, and for
// double positions their rounding to float.
template <class S, int KIND>
IPCB_D float touch_bound(const f3* p, const f3* v, f3 r, float d) {
  if (!(d > 0.f)) return 0.f;
  const float q = 1.0f / d;
  const f3 n = mk3(r.x * q, r.y * q, r.z * q);
  constexpr int NA = KIND == 0 ? 2 : 1;
  float s[4], w[4], size = 0.f, ext = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const f3 l = mk3(p[k].x - p[0].x, p[k].y - p[0].y, p[k].z - p[0].z);
    s[k] = fmaf(n.x, l.x, fmaf(n.y, l.y, n.z * l.z));
    w[k] = fmaf(n.x, v[k].x, fmaf(n.y, v[k].y, n.z * v[k].z));
    const float av = fabsf(v[k].x) + fabsf(v[k].y) + fabsf(v[k].z);
    size += fabsf(l.x) + fabsf(l.y) + fabsf(l.z) + av;
    ext = fmaxf(ext, fmaxf(fabsf(p[k].x), fmaxf(fabsf(p[k].y), fabsf(p[k].z))) + av);
  }
  const float margin = 1.05e-6f * (1.0f + ext) + 1e-6f * size + (sizeof(S) == 8 ? 5e-7f * ext : 0.f);
  float t = 4.0f;
#pragma unroll
  for (int i = 0; i < NA; ++i)
#pragma unroll
    for (int j = NA; j < 4; ++j) {
      const float c = s[i] - s[j] - margin, u = w[j] - w[i];
      if (!(c > 0.f)) t = 0.f;
      else if (u > 0.f) t = fminf(t, c / u);
    }
  return t * 0.9999f;
}

// Closest points at t = 0 (the discrete predicate's float operations): their
// distance, and the difference r.
template <int KIND>
IPCB_D float closest_difference(const f3* p, f3& r) {
  if (KIND == 0) {
    const CPEE c = closest_point_edge_edge(p[0], p[1], p[2], p[3], 1.0e-6f);
    r = (p[0] - p[2]) + (p[1] - p[0]) * c.s - (p[3] - p[2]) * c.t;
    return c.d;
  }
  const CPT c = closest_point_triangle(p[0], p[1], p[2], p[3]);
  r = (p[0] - p[1]) - (p[2] - p[1]) * c.v - (p[3] - p[1]) * (1.0f - c.u - c.v);
  return c.d;
}

// Whether the boxes of the whole step (k_swept's) meet: the query's own test,
// applied to the few pairs that are solved (the tree's boxes may be larger).
template <class S, int KIND>
IPCB_D bool swept_boxes_meet(const S* __restrict__ x0, const S* __restrict__ x1, int4 ids, double pad) {
  const int v[4] = {ids.x, ids.y, ids.z, ids.w};
  constexpr int NA = KIND == 0 ? 2 : 1;
  f3 alo, ahi, blo, bhi;
  swept_box<S, NA>(x0, x1, v, pad, 1.0, alo, ahi);
  swept_box<S, 4 - NA>(x0, x1, v + NA, pad, 1.0, blo, bhi);
  return alo.x <= bhi.x && blo.x <= ahi.x && alo.y <= bhi.y && blo.y <= ahi.y && alo.z <= bhi.z && blo.z <= ahi.z;
}

template <class S>
IPCB_D void load_motion(const S* __restrict__ x0, const S* __restrict__ x1, int i, f3& p, f3& v) {
  const d3 a = ld(x0, i), b = ld(x1, i);
  p = mk3((float)a.x, (float)a.y, (float)a.z);
  v = mk3((float)(b.x - a.x), (float)(b.y - a.y), (float)(b.z - a.z));
}
IPCB_D void load_motion(const float* __restrict__ x0, const float* __restrict__ x1, int i, f3& p, f3& v) {
  p = load3(x0, i);
  const f3 b = load3(x1, i);
  v = mk3(b.x - p.x, b.y - p.y, b.z - p.z);
}

// What a query does with its pairs.
enum Mode {
  kStage,   // CCD: stage the pairs that can lower the TOI
  kInline,  // CCD: solve them in place (the staging list overflowed)
  kBoth     // the discrete test and record, and CCD staging
};

// One queued pair a lane (has), converged over the warp: the closest points
// (the discrete predicate's exact float operations, so kBoth appends what the
// discrete query appends), the touch bound along their axis, and the pair is
// staged or solved.
template <class S, int KIND, int MODE>
IPCB_D void take_pairs(const S* __restrict__ x0, const S* __restrict__ x1, const int* __restrict__ prims, bool has,
                       int2 pr, double pair_pad, float l0f, S l0, const ipcb_contacts& out, const CandList& cand,
                       const CandOrder& o, int* hist, S* toi, const Sink& sink, int& st) {
  const unsigned lane = threadIdx.x & 31;
  bool want = false, accept = false;
  float tl = 4.0f;
  int4 ids = make_int4(0, 0, 0, 0);
  if (has) {
    ids = pair_ids<KIND>(prims, pr);
    f3 p[4], v[4], r;
    load_motion(x0, x1, ids.x, p[0], v[0]);
    load_motion(x0, x1, ids.y, p[1], v[1]);
    load_motion(x0, x1, ids.z, p[2], v[2]);
    load_motion(x0, x1, ids.w, p[3], v[3]);
    const float d = closest_difference<KIND>(p, r);
    if (MODE == kBoth) accept = d < l0f;
    tl = touch_bound<S, KIND>(p, v, r, sqrtf(dot(r, r)));
    // cannot touch within the step, or (only the minimum wanted) cannot lower it
    want = tl <= 1.0f && (sink.on || (double)tl < current_toi(toi));
  }
  if (MODE == kBoth) {
    const int slot = warp_reserve(out.cnt, accept);
    if (accept) {
      if (KIND == 0) write_record<S>(out, slot, ids.x, ids.y, ids.z, ids.w, pr.x, pr.y, l0);
      else write_record<S>(out, slot, ids.x, ids.z, ids.y, ids.w, pr.x, pr.y, l0);  // (p, tri[1], tri[0], tri[2])
    }
  }
  if (MODE == kInline) {
    if (want && (pair_pad < 0.0 || swept_boxes_meet<S, KIND>(x0, x1, ids, pair_pad))) {
      const d3 p0[4] = {ld(x0, ids.x), ld(x0, ids.y), ld(x0, ids.z), ld(x0, ids.w)};
      const d3 p1[4] = {ld(x1, ids.x), ld(x1, ids.y), ld(x1, ids.z), ld(x1, ids.w)};
      const double tt = collision_time<KIND>(p0, p1, st);
      if (tt < 1.0) {
        store_toi(toi, tt);
        sink_append<S>(sink, ids, pr.x, pr.y, tt);
      }
    }
    return;
  }
  const unsigned m = __ballot_sync(0xffffffffu, want);
  if (!m) return;
  int base = 0;
  if (lane == 0) base = atomicAdd(cand.count, __popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (want) {
    const int slot = base + __popc(m & ((1u << lane) - 1u));
    if (slot < cand.capacity) {
      cand.pairs[slot] = pr;
      o.tlb[slot] = tl;
      atomicAdd(hist + bucket_of(tl), 1);
    } else {
      *cand.overflow = 1;  // the inline pass redoes the query
    }
  }
}

// The CCD edge-edge query over the packed tree of swept boxes: a warp per
// block of 32 edges in Morton order (tree.cuh); pairs that survive the box and
// topology tests are bounded on full warps and staged.  kInline (run only when
// *gate is set: the staging list overflowed) solves every pair in place.
// lo / hi: the queries' boxes, or null for the tree's own leaf boxes.
// 64 registers (8 blocks a SM; 96 unbounded): the walk issues about 7,900
// instructions a block in short dependent runs, and the spills (around the
// flush) cost less than the missing warps (screw and nut iteration 1.59 ->
// 1.45 ms, from 3.37 with a traversal per thread).
template <class S, int MODE>
__global__ void __launch_bounds__(32 * tree::kWarps, MODE == kInline ? 1 : 8) k_ee_collect(
    const S* __restrict__ x0, const S* __restrict__ x1, const int* __restrict__ edges, const int* __restrict__ body,
    const __grid_constant__ tree::View v, const int* __restrict__ order, int first, int count, int nsub, int items,
    const float* __restrict__ lo, const float* __restrict__ hi, double pair_pad, int exclude, float thickness,
    ipcb_contacts out, CandList cand, CandOrder o, S* toi, int* status, Sink sink, const int* gate) {
  __shared__ tree::Block blocks[tree::kWarps];
  __shared__ int hist[kBuckets];
  if (MODE == kInline && *gate == 0) return;
  if (threadIdx.x < kBuckets) hist[threadIdx.x] = 0;
  __syncthreads();
  tree::Block& B = blocks[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const float l0f = xmul(thickness, 2.0f);
  const S l0 = S(thickness) * S(2.0);
  int st = 0;
  for (int item = blockIdx.x * tree::kWarps + (threadIdx.x >> 5); item < items; item += gridDim.x * tree::kWarps) {
    const int qb = (first >> 5) + item / nsub, sub = item % nsub;
    const int t = qb * 32 + lane;
    // queries: the edges of Morton rank first .. first + count - 1
    const bool active = t >= first && t < first + count;
    const int i = active ? __ldg(order + t) : 0;
    const int2 ea = __ldg(reinterpret_cast<const int2*>(edges) + i);
    f3 qlo = mk3(tree::kBig, tree::kBig, tree::kBig), qhi = mk3(-tree::kBig, -tree::kBig, -tree::kBig);
    if (active) {
      if (lo) {
        qlo = mk3(__ldg(lo + 3 * i), __ldg(lo + 3 * i + 1), __ldg(lo + 3 * i + 2));
        qhi = mk3(__ldg(hi + 3 * i), __ldg(hi + 3 * i + 1), __ldg(hi + 3 * i + 2));
      } else {
        const float4 l = __ldg(v.lv[0] + 2 * (size_t)t), h = __ldg(v.lv[0] + 2 * (size_t)t + 1);
        qlo = mk3(l.x, l.y, l.z);
        qhi = mk3(h.x, h.y, h.z);
      }
    }
    const int bi = exclude ? __ldg(body + ea.x) : 0;
    __syncwarp();
    B.qlo[lane] = make_float4(qlo.x, qlo.y, qlo.z, __int_as_float(i));
    B.qhi[lane] = make_float4(qhi.x, qhi.y, qhi.z, __int_as_float(bi));
    B.ev[lane] = ea;
    __syncwarp();
    int nq = 0;
    auto flush = [&](int n) {
      const bool has = lane < n;
      const int2 pr = has ? B.queue[nq - n + lane] : make_int2(0, 0);
      const int a = __float_as_int(B.qlo[pr.x].w);
      // the reference's (lower id, higher id) pair
      take_pairs<S, 0, MODE>(x0, x1, edges, has, make_int2(min(a, pr.y), max(a, pr.y)), pair_pad, l0f, l0, out, cand, o,
                             hist, toi, sink, st);
    };
    tree::for_segments(active, qlo, qhi, [&](bool in, f3 glo, f3 ghi) {
    tree::for_block_pairs<true>(v, glo, ghi, qb, sub, nsub, B.stack, [&](int tb) {
      tree::block_pair<true>(
          v, B, qb, tb, in, qlo, qhi, glo, ghi, nq,
          [&](int j) {
            int3 e = make_int3(-1, -1, 0);
            if (j >= 0) {
              const int2 w = __ldg(reinterpret_cast<const int2*>(edges) + j);
              e = make_int3(w.x, w.y, exclude ? __ldg(body + w.x) : 0);
            }
            return e;
          },
          [&](int q, int3 e) {
            const int2 w = B.ev[q];
            if (w.x == e.x || w.x == e.y || w.y == e.x || w.y == e.y) return false;
            return !(exclude && __float_as_int(B.qhi[q].w) == e.z);
          },
          flush);
    });
    });
    __syncwarp();
    if (nq) flush(nq);
  }
  if (st) atomicOr(status, st);
  if (MODE == kInline) return;
  __syncthreads();
  if (threadIdx.x < kBuckets && hist[threadIdx.x]) atomicAdd(o.bcount + threadIdx.x, hist[threadIdx.x]);
}

// The CCD point-triangle query: blocks of 32 vertices of the visiting order.
template <class S, int MODE>
__global__ void __launch_bounds__(32 * tree::kWarps, MODE == kInline ? 1 : 8) k_pt_collect(
    const S* __restrict__ x0, const S* __restrict__ x1, const int* __restrict__ tris, const int* __restrict__ body,
    const __grid_constant__ tree::View v, const int* __restrict__ order, int first, int count, int nsub, int items,
    double pad, double pair_pad, float qpad, int exclude, float thickness, ipcb_contacts out, CandList cand,
    CandOrder o, S* toi, int* status, Sink sink, const int* gate) {
  __shared__ tree::Block blocks[tree::kWarps];
  __shared__ int hist[kBuckets];
  if (MODE == kInline && *gate == 0) return;
  if (threadIdx.x < kBuckets) hist[threadIdx.x] = 0;
  __syncthreads();
  tree::Block& B = blocks[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const float l0f = xmul(thickness, 2.0f);
  const S l0 = S(thickness) * S(2.0);
  int st = 0;
  // boxes up to the TOI stored so far (see swept_box), against the caller's
  // boxes those of the whole step
  const double t_end = sink.on || pair_pad < 0.0 ? 1.0 : dmin(1.0, current_toi(toi));
  for (int item = blockIdx.x * tree::kWarps + (threadIdx.x >> 5); item < items; item += gridDim.x * tree::kWarps) {
    const int sub = item % nsub;
    // queries: the vertices first .. first + count - 1 of the visiting order
    const int t = (item / nsub) * 32 + lane;
    const bool active = t < count;
    const int i = active ? (order ? __ldg(order + first + t) : first + t) : 0;
    f3 qlo = mk3(tree::kBig, tree::kBig, tree::kBig), qhi = mk3(-tree::kBig, -tree::kBig, -tree::kBig);
    if (active) {
      swept_box<S, 1>(x0, x1, &i, pad, t_end, qlo, qhi);
      if (MODE == kBoth) {  // and the discrete query's box
        const f3 p = to_f(load3(x0, i));
        qlo = mk3(fminf(qlo.x, p.x - qpad), fminf(qlo.y, p.y - qpad), fminf(qlo.z, p.z - qpad));
        qhi = mk3(fmaxf(qhi.x, p.x + qpad), fmaxf(qhi.y, p.y + qpad), fmaxf(qhi.z, p.z + qpad));
      }
    }
    const int bi = exclude ? __ldg(body + i) : 0;
    __syncwarp();
    B.qlo[lane] = make_float4(qlo.x, qlo.y, qlo.z, __int_as_float(i));
    B.qhi[lane] = make_float4(qhi.x, qhi.y, qhi.z, __int_as_float(bi));
    __syncwarp();
    int nq = 0;
    auto flush = [&](int n) {
      const bool has = lane < n;
      const int2 pr = has ? B.queue[nq - n + lane] : make_int2(0, 0);
      const int a = __float_as_int(B.qlo[pr.x].w);
      take_pairs<S, 1, MODE>(x0, x1, tris, has, make_int2(a, pr.y), pair_pad, l0f, l0, out, cand, o, hist, toi, sink, st);
    };
    tree::for_segments(active, qlo, qhi, [&](bool in, f3 glo, f3 ghi) {
    tree::for_block_pairs<false>(v, glo, ghi, 0, sub, nsub, B.stack, [&](int tb) {
      tree::block_pair<false>(
          v, B, 0, tb, in, qlo, qhi, glo, ghi, nq,
          [&](int j) {
            int4 e = make_int4(-1, -1, -1, 0);
            if (j >= 0) {
              e = make_int4(__ldg(tris + 3 * j), __ldg(tris + 3 * j + 1), __ldg(tris + 3 * j + 2), 0);
              if (exclude) e.w = __ldg(body + e.x);
            }
            return e;
          },
          [&](int q, int4 e) {
            const int a = __float_as_int(B.qlo[q].w);
            if (a == e.x || a == e.y || a == e.z) return false;
            return !(exclude && __float_as_int(B.qhi[q].w) == e.w);
          },
          flush);
    });
    });
    __syncwarp();
    if (nq) flush(nq);
  }
  if (st) atomicOr(status, st);
  if (MODE == kInline) return;
  __syncthreads();
  if (threadIdx.x < kBuckets && hist[threadIdx.x]) atomicAdd(o.bcount + threadIdx.x, hist[threadIdx.x]);
}

// An early upper bound on the TOI: pairs of a contact list (the discrete
// query's) that the CCD query would meet too -- the same filters, and boxes
// over the whole step that overlap -- are solved before the boxes are formed.
// Each lane takes up to kSeedPairs spread over the list and solves the one
// with the smallest touch-time bound.  Every solved pair is one of the
// query's, so the minimum is unchanged; the list may be of any age.
constexpr int kSeedPairs = 4, kSeedLanes = 8192;

template <class S, int KIND>
__global__ void __launch_bounds__(64) k_seed(const S* __restrict__ x0, const S* __restrict__ x1,
                                             const int* __restrict__ prims, const int* __restrict__ body, int n_a,
                                             int n_b, int exclude, double pad, ipcb_contacts list, S* toi,
                                             int* status) {
  const int n = min(*list.cnt, list.capacity);
  const int m = min(n, kSeedPairs * kSeedLanes);
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  float best = 2.0f;
  int4 ids = make_int4(0, 0, 0, 0);
  for (int q = 0; q < kSeedPairs; ++q) {
    const int k = q * kSeedLanes + g;
    if (k >= m) break;
    int2 pr = reinterpret_cast<const int2*>(list.e0e1)[(long long)k * n / m];
    if (KIND == 0) pr = make_int2(min(pr.x, pr.y), max(pr.x, pr.y));
    if (pr.x < 0 || pr.y < 0 || pr.x >= n_a || pr.y >= n_b) continue;
    const int4 w = pair_ids<KIND>(prims, pr);
    if (w.x == w.z || w.x == w.w || (KIND == 0 ? (w.y == w.z || w.y == w.w) : w.x == w.y)) continue;
    if (exclude && __ldg(body + w.x) == __ldg(body + (KIND == 0 ? w.z : w.y))) continue;
    f3 p[4], v[4], r;
    load_motion(x0, x1, w.x, p[0], v[0]);
    load_motion(x0, x1, w.y, p[1], v[1]);
    load_motion(x0, x1, w.z, p[2], v[2]);
    load_motion(x0, x1, w.w, p[3], v[3]);
    closest_difference<KIND>(p, r);
    const float tl = touch_bound<S, KIND>(p, v, r, sqrtf(dot(r, r)));
    if (tl < best) {
      best = tl;
      ids = w;
    }
  }
  if (!(best <= 1.0f) || (double)best >= current_toi(toi) || !swept_boxes_meet<S, KIND>(x0, x1, ids, pad)) return;
  const d3 p0[4] = {ld(x0, ids.x), ld(x0, ids.y), ld(x0, ids.z), ld(x0, ids.w)};
  const d3 p1[4] = {ld(x1, ids.x), ld(x1, ids.y), ld(x1, ids.z), ld(x1, ids.w)};
  int st = 0;
  const double tt = collision_time<KIND>(p0, p1, st);
  if (tt < 1.0) store_toi(toi, tt);
  if (st) atomicOr(status, st);
}

// one thread per staged candidate; kind 0 EE (edge, edge), 1 PT (vertex, triangle)
// One thread per staged pair, grid-stride.  Without a sink only the minimum
// matters: a pair whose touch-time bound is at or above the TOI stored so far
// (re-read from L2 for every pair; it only decreases) cannot lower it, so its
// cubic is not solved -- the result is the same minimum, bit for bit.  With
// a sink every pair that can touch within the step is solved.
template <class S, int KIND>
__global__ void __launch_bounds__(128) k_cand_toi(const S* __restrict__ x0, const S* __restrict__ x1,
                                                  const int* __restrict__ prims, CandList cand, S* toi,
                                                  int* status, Sink sink, const int* skip_if) {
  if (skip_if && *skip_if) return;  // the inline pass redoes every pair
  const int n = min(*cand.count, cand.capacity);
  int st = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int2 pr = cand.pairs[k];
    const int4 ids = pair_ids<KIND>(prims, pr);
    d3 p0[4] = {ld(x0, ids.x), ld(x0, ids.y), ld(x0, ids.z), ld(x0, ids.w)};
    d3 p1[4] = {ld(x1, ids.x), ld(x1, ids.y), ld(x1, ids.z), ld(x1, ids.w)};
    const double lb = touch_time_bound<KIND>(p0, p1);
    if (lb > 1.0) continue;  // cannot touch within the step
    if (!sink.on && lb >= current_toi(toi)) continue;  // cannot lower the minimum
    const double tt = collision_time<KIND>(p0, p1, st);
    if (tt < 1.0) {
      store_toi(toi, tt);
      sink_append<S>(sink, ids, pr.x, pr.y, tt);
    }
  }
  if (st) atomicOr(status, st);
}

// The staged pairs' indices in bucket order.
__global__ void __launch_bounds__(256) k_cand_bucket(CandList cand, CandOrder o, const int* skip_if) {
  __shared__ int sb[kBuckets], sbase[kBuckets];
  if (*skip_if) return;
  const int n = min(*cand.count, cand.capacity);
  for (int first = blockIdx.x * blockDim.x; first < n; first += gridDim.x * blockDim.x) {
    if (threadIdx.x < kBuckets) sb[threadIdx.x] = 0;
    __syncthreads();
    const int k = first + threadIdx.x;
    int b = -1, local = 0;
    if (k < n) {
      b = bucket_of(o.tlb[k]);
      local = atomicAdd(&sb[b], 1);
    }
    __syncthreads();
    if (threadIdx.x < kBuckets) {
      const int q = threadIdx.x;
      int start = 0;
      for (int c = 0; c < q; ++c) start += o.bcount[c];
      sbase[q] = sb[q] ? start + atomicAdd(o.bcursor + q, sb[q]) : 0;
    }
    __syncthreads();
    // (a second solve of the same list finds the cursors at its end)
    if (b >= 0 && sbase[b] + local < cand.capacity) o.order[sbase[b] + local] = k;
    __syncthreads();
  }
}

template <class S, int KIND>
__global__ void __launch_bounds__(128) k_cand_solve(const S* __restrict__ x0, const S* __restrict__ x1,
                                                    const int* __restrict__ prims, double pair_pad, CandList cand,
                                                    CandOrder o, S* toi, int* status, const int* skip_if) {
  if (skip_if && *skip_if) return;
  int total = 0;
#pragma unroll 1
  for (int q = 0; q < kBuckets; ++q) total += o.bcount[q];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int st = 0;
  for (;;) {
    int base = 0;
    if (lane == 0) base = atomicAdd(o.work, 32);
    base = __shfl_sync(full, base, 0);
    if (base >= total) break;
    const int item = base + lane;
    const int k = item < total ? __ldg(o.order + item) : -1;
    const float tl = k >= 0 ? __ldg(o.tlb + k) : 2.0f;
    const double cur = current_toi(toi);
    // the chunk's first pair starts its bucket range: every later pair lies
    // in this bucket or a later one, so none can lower a TOI at or below it
    const float first = __shfl_sync(full, tl, 0);
    if ((double)bucket_of(first) / kBuckets >= cur) break;
    if (k < 0 || (double)tl >= cur) continue;
    const int2 pr = cand.pairs[k];
    const int4 ids = pair_ids<KIND>(prims, pr);
    if (pair_pad >= 0.0 && !swept_boxes_meet<S, KIND>(x0, x1, ids, pair_pad)) continue;
    d3 p0[4] = {ld(x0, ids.x), ld(x0, ids.y), ld(x0, ids.z), ld(x0, ids.w)};
    d3 p1[4] = {ld(x1, ids.x), ld(x1, ids.y), ld(x1, ids.z), ld(x1, ids.w)};
    const double tt = collision_time<KIND>(p0, p1, st);
    if (tt < 1.0) store_toi(toi, tt);
  }
  if (st) atomicOr(status, st);
}

// ---------------------------------------------------------------- fixed bodies
// frames at q, swept world boxes of the bodies over the step q -> q - dq, the
// singular test at both ends, and the target-frame motion extent
// (_target_motion_extent, fixed_bvh_contacts.py:121-141):
//   d = A0^-1 (A1 - A0), c = A0^-1 (p1 - p0), m = |d mid + c| + |d| ext
template <class S>
__global__ void k_body_frames_swept(int nb, const S* __restrict__ q, const S* __restrict__ dq,
                                    const float* __restrict__ llo, const float* __restrict__ lhi,
                                    double* __restrict__ frames, double* __restrict__ motion,
                                    int* __restrict__ status) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  double p0[3], A0[9], p1[3], A1[9], I[9], w0l[3], w0h[3], w1l[3], w1h[3];
  bodies::load_affine(q, b, p0, A0);
  for (int k = 0; k < 3; ++k) p1[k] = p0[k] - (double)dq[12 * b + k];
  for (int c = 0; c < 3; ++c)
    for (int r = 0; r < 3; ++r) A1[3 * r + c] = A0[3 * r + c] - (double)dq[12 * b + 3 + 3 * c + r];
  const double d0 = bodies::det3(A0), d1 = bodies::det3(A1);
  if (!(fmin(fabs(d0), fabs(d1)) >= 1e-8)) {
    atomicOr(status, IPCB_STATUS_SINGULAR);
    for (int k = 0; k < 9; ++k) I[k] = (k % 4) == 0 ? 1.0 : 0.0;
  } else {
    bodies::inverse3(A0, d0, I);
  }
  double fro = 0.0;
  for (int k = 0; k < 9; ++k) {
    frames[13 * b + k] = I[k];
    fro += I[k] * I[k];
  }
  for (int k = 0; k < 3; ++k) frames[13 * b + 9 + k] = p0[k];
  frames[13 * b + 12] = sqrt(fro);
  const float* lo = llo + 3 * b;
  const float* hi = lhi + 3 * b;
  bodies::world_box(p0, A0, lo, hi, w0l, w0h);
  bodies::world_box(p1, A1, lo, hi, w1l, w1h);
  double* wbox = frames + 13 * (size_t)nb + 6 * b;
  for (int k = 0; k < 3; ++k) {
    wbox[k] = fmin(w0l[k], w1l[k]);
    wbox[3 + k] = fmax(w0h[k], w1h[k]);
  }
  double D[9], cvec[3];
  for (int r = 0; r < 3; ++r) {
    for (int c = 0; c < 3; ++c) {
      double acc = 0.0;
      for (int k = 0; k < 3; ++k) acc += I[3 * r + k] * (A1[3 * k + c] - A0[3 * k + c]);
      D[3 * r + c] = acc;
    }
    cvec[r] = I[3 * r] * (p1[0] - p0[0]) + I[3 * r + 1] * (p1[1] - p0[1]) + I[3 * r + 2] * (p1[2] - p0[2]);
  }
  for (int r = 0; r < 3; ++r) {
    double dc = cvec[r], e = 0.0;
    for (int k = 0; k < 3; ++k) {
      const double mid = 0.5 * ((double)lo[k] + (double)hi[k]), ext = 0.5 * ((double)hi[k] - (double)lo[k]);
      dc += D[3 * r + k] * mid;
      e += fabs(D[3 * r + k]) * ext;
    }
    motion[3 * b + r] = fabs(dc) + e;
  }
}

__global__ void k_swept_pair_cull(int nb, const double* __restrict__ wbox, double pad, int2* __restrict__ pairs,
                                  int capacity, int* __restrict__ count) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int a = (int)(t / nb), b = (int)(t % nb);
  bool hit = false;
  if (a < nb && a < b) {
    hit = true;
    for (int k = 0; k < 3; ++k)
      hit = hit && wbox[6 * a + k] - pad <= wbox[6 * b + 3 + k] && wbox[6 * b + k] - pad <= wbox[6 * a + 3 + k];
  }
  const unsigned lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xffffffffu, hit);
  int base = 0;
  if (lane == 0 && m) base = atomicAdd(count, __popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  const int slot = base + __popc(m & ((1u << lane) - 1u));
  if (hit && slot < capacity) pairs[slot] = make_int2(a, b);
}

// swept local box of world points (x0 and x1 of each) in the target frame,
// inflated by the frame's motion extent and |A^-1|_F pad
template <class S, int NP>
IPCB_D void swept_local_box(const bodies::Frame& f, const double* __restrict__ motion, int tb, const S* __restrict__ x0,
                            const S* __restrict__ x1, const int (&v)[NP], double pad, f3& qlo, f3& qhi) {
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300}, pd[3], a[3];
  for (int k = 0; k < NP; ++k) {
    const d3 p = ld(x0, v[k]), r = ld(x1, v[k]);
    bodies::to_local(f, p.x, p.y, p.z, a);
    for (int c = 0; c < 3; ++c) {
      lo[c] = fmin(lo[c], a[c]);
      hi[c] = fmax(hi[c], a[c]);
    }
    bodies::to_local(f, r.x, r.y, r.z, a);
    for (int c = 0; c < 3; ++c) {
      lo[c] = fmin(lo[c], a[c]);
      hi[c] = fmax(hi[c], a[c]);
    }
  }
  for (int c = 0; c < 3; ++c)
    pd[c] = motion[3 * tb + c] + f.fro * pad + 1e-6 * (1.0 + fmax(fabs(lo[c]), fabs(hi[c])));
  bodies::float_box(lo, hi, pd, qlo, qhi);
}

template <class S>
__global__ void __launch_bounds__(128) k_fixed_ee_collect(const S* __restrict__ x0, const S* __restrict__ x1,
                                                          const int* __restrict__ edges, ipcb_bodies B,
                                                          const int* __restrict__ fixed, const int2* __restrict__ pairs,
                                                          double pad, CandList cand, S* toi, int* status) {
  const int chunks = (B.max_edges + 127) / 128;
  const int pair = blockIdx.x / chunks;
  const int k = (blockIdx.x % chunks) * blockDim.x + threadIdx.x;
  int2 pr = pairs[pair];
  if (fixed && fixed[pr.x] != 0 && fixed[pr.y] == 0) pr = make_int2(pr.y, pr.x);  // query from the moving body
  const int sb = pr.x, tb = pr.y;
  const int s0 = __ldg(B.edge_off + sb), sn = __ldg(B.edge_off + sb + 1) - s0;
  const bool active = k < sn;
  const int i = active ? __ldg(B.edge_ids + s0 + k) : 0;
  const int2 ea = __ldg(reinterpret_cast<const int2*>(edges) + i);
  const int t0 = __ldg(B.edge_off + tb), tn = __ldg(B.edge_off + tb + 1) - t0;
  int st = 0;
  int q[kQueue];
  int nq = 0;
  if (active && tn > 0) {
    const bodies::Frame f = bodies::load_frame(B.frames, tb);
    const int v[2] = {ea.x, ea.y};
    f3 qlo, qhi;
    swept_local_box<S, 2>(f, B.motion, tb, x0, x1, v, pad, qlo, qhi);
    const float4* wide = reinterpret_cast<const float4*>(B.edge_wide[tb]);
    bool ok = traverse4(wide, tn, qlo, qhi, [&](int j) {
      const int e2 = __ldg(B.edge_ids + t0 + j);
      if (nq < kQueue) {
        q[nq++] = e2;
      } else {
        const int2 eb = __ldg(reinterpret_cast<const int2*>(edges) + e2);
        double tt = ee_pair_time(x0, x1, ea, eb, st);
        if (tt < 1.0) store_toi(toi, tt);
      }
    });
    if (!ok) st |= IPCB_STATUS_STACK;
  }
  const int rounds = warp_max(nq);
  for (int r = 0; r < rounds; ++r) {
    const bool has = r < nq;
    const int e2 = has ? q[r] : 0;
    if (!push_converged(cand, has, i, e2)) {
      const int2 eb = __ldg(reinterpret_cast<const int2*>(edges) + e2);
      double tt = ee_pair_time(x0, x1, ea, eb, st);
      if (tt < 1.0) store_toi(toi, tt);
    }
  }
  if (st) atomicOr(status, st);
}

template <class S>
__global__ void __launch_bounds__(128) k_fixed_pt_collect(const S* __restrict__ x0, const S* __restrict__ x1,
                                                          const int* __restrict__ tris, ipcb_bodies B,
                                                          const int2* __restrict__ pairs, double pad, CandList cand,
                                                          S* toi, int* status) {
  const int chunks = (B.max_verts + 127) / 128;
  const int pair = blockIdx.x / chunks, dir = blockIdx.y;
  const int k = (blockIdx.x % chunks) * blockDim.x + threadIdx.x;
  const int2 pr = pairs[pair];
  const int sb = dir ? pr.y : pr.x, tb = dir ? pr.x : pr.y;
  const int s0 = __ldg(B.vert_off + sb), sn = __ldg(B.vert_off + sb + 1) - s0;
  const bool active = k < sn;
  const int i = active ? __ldg(B.vert_ids + s0 + k) : 0;
  const int t0 = __ldg(B.tri_off + tb), tn = __ldg(B.tri_off + tb + 1) - t0;
  int st = 0;
  int q[kQueue];
  int nq = 0;
  if (active && tn > 0) {
    const bodies::Frame f = bodies::load_frame(B.frames, tb);
    const int v[1] = {i};
    f3 qlo, qhi;
    swept_local_box<S, 1>(f, B.motion, tb, x0, x1, v, pad, qlo, qhi);
    const float4* wide = reinterpret_cast<const float4*>(B.tri_wide[tb]);
    bool ok = traverse4(wide, tn, qlo, qhi, [&](int j) {
      const int tr = __ldg(B.tri_ids + t0 + j);
      if (nq < kQueue) {
        q[nq++] = tr;
      } else {
        const int3 tj = make_int3(__ldg(tris + 3 * tr), __ldg(tris + 3 * tr + 1), __ldg(tris + 3 * tr + 2));
        double tt = pt_pair_time(x0, x1, i, tj, st);
        if (tt < 1.0) store_toi(toi, tt);
      }
    });
    if (!ok) st |= IPCB_STATUS_STACK;
  }
  const int rounds = warp_max(nq);
  for (int r = 0; r < rounds; ++r) {
    const bool has = r < nq;
    const int tr = has ? q[r] : 0;
    if (!push_converged(cand, has, i, tr)) {
      const int3 tj = make_int3(__ldg(tris + 3 * tr), __ldg(tris + 3 * tr + 1), __ldg(tris + 3 * tr + 2));
      double tt = pt_pair_time(x0, x1, i, tj, st);
      if (tt < 1.0) store_toi(toi, tt);
    }
  }
  if (st) atomicOr(status, st);
}

// Candidate workspace: a 512-byte header (count, overflow flag, bucket counts
// and cursors, work counter), then per staged pair its int2, its touch-time
// bound (float) and the bucket order (int): 16 bytes a pair.
constexpr size_t kCandHeader = 512;
constexpr size_t kCandPerPair = sizeof(int2) + sizeof(float) + sizeof(int);

inline CandList cand_list(void* ws, size_t ws_bytes) {
  CandList c;
  c.count = (int*)ws;
  c.overflow = (int*)ws + 1;
  c.pairs = (int2*)((char*)ws + kCandHeader);
  size_t cap = ws_bytes > kCandHeader ? (ws_bytes - kCandHeader) / kCandPerPair : 0;
  c.capacity = cap > 0x7fffffff ? 0x7fffffff : (int)cap;
  return c;
}

inline CandOrder cand_order(void* ws, const CandList& c) {
  CandOrder o;
  int* h = (int*)ws;
  o.bcount = h + 2;
  o.bcursor = h + 2 + kBuckets;
  o.work = h + 2 + 2 * kBuckets;
  o.tlb = (float*)(c.pairs + c.capacity);
  o.order = (int*)(o.tlb + c.capacity);
  return o;
}

__global__ void k_pair_time(int kind, int n, const double* __restrict__ a, const double* __restrict__ b,
                            double* __restrict__ t, int* status) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  d3 p0[4], p1[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    p0[k] = mk3(a[12 * i + 3 * k], a[12 * i + 3 * k + 1], a[12 * i + 3 * k + 2]);
    p1[k] = mk3(b[12 * i + 3 * k], b[12 * i + 3 * k + 1], b[12 * i + 3 * k + 2]);
  }
  int st = 0;
  t[i] = kind == 0 ? collision_time<0>(p0, p1, st) : collision_time<1>(p0, p1, st);
  if (st) atomicOr(status, st);
}

__global__ void k_cubic(int n, const double* __restrict__ coef, double x0, double x1, double* __restrict__ roots,
                        int* __restrict__ nr, int* status) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Q4 p{{coef[4 * i], coef[4 * i + 1], coef[4 * i + 2], coef[4 * i + 3]}};
  int st = 0;
  double r[3];
  nr[i] = cubic_roots(p, x0, x1, r, st);
  roots[3 * i] = r[0];
  roots[3 * i + 1] = r[1];
  roots[3 * i + 2] = r[2];
  if (st) atomicOr(status, st);
}

// One CCD query of one kind (KIND 0: edges first .. first + count - 1 in
// Morton rank; 1: the vertices of those places of the visiting order).
template <class S>
struct Query {
  const ipcb_soup* soup;
  const S* x1;
  const ipcb_lbvh* bvh;
  const float *lower, *upper;  // EE: query boxes (null: the tree's leaf boxes)
  double pad;                  // of the swept boxes formed here
  double pair_pad;             // of the pairs' own box test; < 0: the caller's boxes decide
  float reach, thickness;      // kBoth: the discrete query's
  const int* order;            // PT: visiting order or null
  int exclude, first, count;
  ipcb_contacts out;           // kBoth: records
  void* ws;
  CandList cand;
  S* toi;
  int* status;
  Sink sink;
  cudaStream_t st;
};

constexpr int kInlineBlocks = 148 * 2;

template <class S, int KIND, int MODE>
void collect(const Query<S>& q) {
  const S* x0 = (const S*)q.soup->x;
  const tree::View v = tree::view(q.bvh);
  const CandOrder o = cand_order(q.ws, q.cand);
  const int blocks = KIND == 0 ? ((q.first + q.count - 1) >> 5) - (q.first >> 5) + 1 : div_up(q.count, 32);
  const int nsub = tree::share(blocks), items = blocks * nsub;
  int grid = div_up(items, tree::kWarps);
  if (MODE == kInline) grid = min(grid, kInlineBlocks);
  const int* gate = MODE == kInline ? q.cand.overflow : nullptr;
  if (KIND == 0)
    k_ee_collect<S, MODE><<<grid, 32 * tree::kWarps, 0, q.st>>>(
        x0, q.x1, q.soup->edges, q.soup->body, v, q.bvh->sorted, q.first, q.count, nsub, items, q.lower, q.upper,
        q.pair_pad, q.exclude, q.thickness, q.out, q.cand, o, q.toi, q.status, q.sink, gate);
  else
    k_pt_collect<S, MODE><<<grid, 32 * tree::kWarps, 0, q.st>>>(
        x0, q.x1, q.soup->triangles, q.soup->body, v, q.order, q.first, q.count, nsub, items, q.pad, q.pair_pad,
        q.reach, q.exclude, q.thickness, q.out, q.cand, o, q.toi, q.status, q.sink, gate);
}

constexpr int kHeaderWords = 2 + 2 * kBuckets + 1;  // zero when a query starts staging

// The staged pairs (in bucket order without a sink), then -- a small grid that
// returns at once unless the staging list overflowed -- every pair in place.
template <class S, int KIND>
void solve(const Query<S>& q) {
  const S* x0 = (const S*)q.soup->x;
  const int* prims = KIND == 0 ? q.soup->edges : q.soup->triangles;
  const CandList& c = q.cand;
  if (c.capacity && q.sink.on) {  // every pair that collides is a record: solve them all
    k_cand_toi<S, KIND><<<min(div_up(c.capacity, 128), 2048), 128, 0, q.st>>>(x0, q.x1, prims, c, q.toi, q.status,
                                                                              q.sink, c.overflow);
  } else if (c.capacity) {
    const CandOrder o = cand_order(q.ws, c);
    k_cand_bucket<<<min(div_up(c.capacity, 256), 148 * 4), 256, 0, q.st>>>(c, o, c.overflow);
    k_cand_solve<S, KIND><<<148 * 3, 128, 0, q.st>>>(x0, q.x1, prims, q.pair_pad, c, o, q.toi, q.status, c.overflow);
  }
  collect<S, KIND, kInline>(q);
}

// Boxes given (EE: also the query boxes), and with them what a pair is: stage
// and solve.
template <class S, int KIND>
void run_boxes(Query<S> q) {
  q.pair_pad = -1.0;
  cudaMemsetAsync(q.ws, 0, kHeaderWords * sizeof(int), q.st);
  collect<S, KIND, kStage>(q);
  solve<S, KIND>(q);
}

// Boxes formed here, over the step up to the TOI the seeds give.
template <class S, int KIND>
void run_step(const Query<S>& q, const ipcb_contacts* seeds) {
  const S* x0 = (const S*)q.soup->x;
  const int* prims = KIND == 0 ? q.soup->edges : q.soup->triangles;
  if (seeds)
    k_seed<S, KIND><<<kSeedLanes / 64, 64, 0, q.st>>>(x0, q.x1, prims, q.soup->body,
                                                      KIND == 0 ? q.soup->n_edges : q.soup->n_verts,
                                                      KIND == 0 ? q.soup->n_edges : q.soup->n_tris, q.exclude, q.pad,
                                                      *seeds, q.toi, q.status);
  tree::refit(q.bvh, SweptBox<S, KIND == 0 ? 2 : 3>{x0, q.x1, prims, q.pad, q.toi}, q.st, (int*)q.ws,
              kHeaderWords);
  collect<S, KIND, kStage>(q);
  solve<S, KIND>(q);
}

// Boxes of both queries; the discrete records and the staged CCD pairs (solve
// takes those).
template <class S, int KIND>
void run_both(const Query<S>& q, float box_reach) {
  const int* prims = KIND == 0 ? q.soup->edges : q.soup->triangles;
  tree::refit(q.bvh, BothBox<S, KIND == 0 ? 2 : 3>{(const S*)q.soup->x, q.x1, prims, q.pad, box_reach}, q.st,
              (int*)q.ws, kHeaderWords);
  collect<S, KIND, kBoth>(q);
}

template <class S>
Query<S> make_query(const ipcb_soup* soup, const void* x1, const ipcb_lbvh* bvh, double pad, int exclude, int first,
                    int count, void* toi, int* status, void* ws, size_t ws_bytes, ipcb_stream s) {
  Query<S> q{};
  q.soup = soup;
  q.x1 = (const S*)x1;
  q.bvh = bvh;
  q.pad = q.pair_pad = pad;
  q.exclude = exclude;
  q.first = first;
  q.count = count;
  q.ws = ws;
  q.cand = cand_list(ws, ws_bytes);
  q.toi = (S*)toi;
  q.status = status;
  q.st = (cudaStream_t)s;
  return q;
}

inline bool query_ok(const ipcb_soup* soup, const void* x1, const ipcb_lbvh* bvh, const void* toi, const int* status,
                     const void* ws, size_t ws_bytes, int prims) {
  return x1 && bvh && toi && status && ws && ws_bytes >= kCandHeader && bvh->n == prims;
}

inline bool range_ok(int first, int count, int n) {
  return first >= 0 && count >= 0 && first <= n && count <= n - first;
}

// f(Query<S>) in the soup's scalar
template <class F>
void in_scalar(const ipcb_soup* soup, F&& f) {
  if (soup->fp64) f((double*)nullptr);
  else f((float*)nullptr);
}

}  // namespace
}  // namespace ipcb

using namespace ipcb;


extern "C" {

int ipcb_add_dx(const ipcb_soup* soup, const void* dx, void* x1, ipcb_stream s) {
  if (!soup || !dx || !x1) return IPCB_E_ARG;
  int n3 = 3 * soup->n_verts;
  if (n3 == 0) return IPCB_OK;
  if (soup->fp64)
    k_add_dx<double><<<div_up(n3, 256), 256, 0, (cudaStream_t)s>>>((const double*)soup->x, (const double*)dx,
                                                                   (double*)x1, n3);
  else
    k_add_dx<float><<<div_up(n3, 256), 256, 0, (cudaStream_t)s>>>((const float*)soup->x, (const float*)dx,
                                                                  (float*)x1, n3);
  return check_launch("ipcb_add_dx");
}

int ipcb_swept_edge_aabbs(const ipcb_soup* soup, const void* x1, double pad, float* lower, float* upper,
                          ipcb_stream s) {
  if (!soup || !x1 || !lower || !upper) return IPCB_E_ARG;
  int n = soup->n_edges;
  if (n == 0) return IPCB_OK;
  if (soup->fp64)
    k_swept<double, 2><<<div_up(n, 256), 256, 0, (cudaStream_t)s>>>((const double*)soup->x, (const double*)x1,
                                                                    soup->edges, n, pad, lower, upper);
  else
    k_swept<float, 2><<<div_up(n, 256), 256, 0, (cudaStream_t)s>>>((const float*)soup->x, (const float*)x1,
                                                                   soup->edges, n, pad, lower, upper);
  return check_launch("ipcb_swept_edge_aabbs");
}

int ipcb_swept_triangle_aabbs(const ipcb_soup* soup, const void* x1, double pad, float* lower, float* upper,
                              ipcb_stream s) {
  if (!soup || !x1 || !lower || !upper) return IPCB_E_ARG;
  int n = soup->n_tris;
  if (n == 0) return IPCB_OK;
  if (soup->fp64)
    k_swept<double, 3><<<div_up(n, 256), 256, 0, (cudaStream_t)s>>>((const double*)soup->x, (const double*)x1,
                                                                    soup->triangles, n, pad, lower, upper);
  else
    k_swept<float, 3><<<div_up(n, 256), 256, 0, (cudaStream_t)s>>>((const float*)soup->x, (const float*)x1,
                                                                   soup->triangles, n, pad, lower, upper);
  return check_launch("ipcb_swept_triangle_aabbs");
}

size_t ipcb_toi_workspace(int capacity) { return kCandHeader + (size_t)(capacity > 0 ? capacity : 0) * kCandPerPair; }

int ipcb_edge_edge_toi_range(const ipcb_soup* soup, const void* x1, const ipcb_lbvh* bvh, const float* lower,
                             const float* upper, int exclude_same_body, int first, int count, void* toi, int* status,
                             void* ws, size_t ws_bytes, ipcb_stream s) {
  if (!soup || !lower || !upper || !query_ok(soup, x1, bvh, toi, status, ws, ws_bytes, soup->n_edges) ||
      !range_ok(first, count, soup->n_edges))
    return IPCB_E_ARG;
  if (count == 0) return IPCB_OK;
  in_scalar(soup, [&](auto* scalar) {
    using S = std::remove_pointer_t<decltype(scalar)>;
    Query<S> q = make_query<S>(soup, x1, bvh, 0.0, exclude_same_body, first, count, toi, status, ws, ws_bytes, s);
    q.lower = lower;
    q.upper = upper;
    run_boxes<S, 0>(q);
  });
  return check_launch("ipcb_edge_edge_toi");
}

int ipcb_edge_edge_toi(const ipcb_soup* soup, const void* x1, const ipcb_lbvh* bvh, const float* lower,
                       const float* upper, int exclude_same_body, void* toi, int* status, void* ws, size_t ws_bytes,
                       ipcb_stream s) {
  if (!soup) return IPCB_E_ARG;
  return ipcb_edge_edge_toi_range(soup, x1, bvh, lower, upper, exclude_same_body, 0, soup->n_edges, toi, status, ws,
                                  ws_bytes, s);
}

int ipcb_point_triangle_toi_range(const ipcb_soup* soup, const void* x1, const ipcb_lbvh* bvh, double pad,
                                  int exclude_same_body, int first, int count, void* toi, int* status, void* ws,
                                  size_t ws_bytes, ipcb_stream s) {
  if (!soup || !query_ok(soup, x1, bvh, toi, status, ws, ws_bytes, soup->n_tris) ||
      !range_ok(first, count, soup->n_verts))
    return IPCB_E_ARG;
  if (count == 0 || soup->n_tris == 0) return IPCB_OK;
  in_scalar(soup, [&](auto* scalar) {
    using S = std::remove_pointer_t<decltype(scalar)>;
    run_boxes<S, 1>(make_query<S>(soup, x1, bvh, pad, exclude_same_body, first, count, toi, status, ws, ws_bytes, s));
  });
  return check_launch("ipcb_point_triangle_toi");
}

int ipcb_point_triangle_toi(const ipcb_soup* soup, const void* x1, const ipcb_lbvh* bvh, double pad,
                            int exclude_same_body, void* toi, int* status, void* ws, size_t ws_bytes,
                            ipcb_stream s) {
  if (!soup) return IPCB_E_ARG;
  return ipcb_point_triangle_toi_range(soup, x1, bvh, pad, exclude_same_body, 0, soup->n_verts, toi, status, ws,
                                       ws_bytes, s);
}

static bool list_ok(const ipcb_contacts* l) {
  return l && l->cnt && (l->capacity <= 0 || (l->a1a2b1b2 && l->e0e1 && l->l0 && l->alpha && l->lam));
}
static bool seeds_ok(const ipcb_contacts* seeds) {
  return !seeds || (seeds->cnt && (seeds->capacity <= 0 || seeds->e0e1));
}

int ipcb_edge_edge_step(const ipcb_soup* soup, const void* x1, double pad, const ipcb_lbvh* bvh,
                        const ipcb_contacts* seeds, int exclude_same_body, int first, int count, void* toi, int* status,
                        void* ws, size_t ws_bytes, ipcb_stream s) {
  if (!soup || !(pad >= 0.0) || !seeds_ok(seeds) ||
      !query_ok(soup, x1, bvh, toi, status, ws, ws_bytes, soup->n_edges) || !range_ok(first, count, soup->n_edges))
    return IPCB_E_ARG;
  if (count == 0) return IPCB_OK;
  in_scalar(soup, [&](auto* scalar) {
    using S = std::remove_pointer_t<decltype(scalar)>;
    run_step<S, 0>(make_query<S>(soup, x1, bvh, pad, exclude_same_body, first, count, toi, status, ws, ws_bytes, s),
                   seeds);
  });
  return check_launch("ipcb_edge_edge_step");
}

int ipcb_point_triangle_step(const ipcb_soup* soup, const void* x1, double pad, const ipcb_lbvh* bvh,
                             const int* query_order, const ipcb_contacts* seeds, int exclude_same_body, int first,
                             int count, void* toi, int* status, void* ws, size_t ws_bytes, ipcb_stream s) {
  if (!soup || !(pad >= 0.0) || !seeds_ok(seeds) ||
      !query_ok(soup, x1, bvh, toi, status, ws, ws_bytes, soup->n_tris) || !range_ok(first, count, soup->n_verts))
    return IPCB_E_ARG;
  if (count == 0 || soup->n_tris == 0) return IPCB_OK;
  in_scalar(soup, [&](auto* scalar) {
    using S = std::remove_pointer_t<decltype(scalar)>;
    Query<S> q = make_query<S>(soup, x1, bvh, pad, exclude_same_body, first, count, toi, status, ws, ws_bytes, s);
    q.order = query_order;
    run_step<S, 1>(q, seeds);
  });
  return check_launch("ipcb_point_triangle_step");
}

int ipcb_edge_edge_both(const ipcb_soup* soup, const void* x1, double pad, const ipcb_lbvh* bvh, float thickness,
                        float box_pad, int exclude_same_body, ipcb_contacts* out, void* toi, int* status, void* ws,
                        size_t ws_bytes, ipcb_stream s) {
  if (!soup || !(pad >= 0.0) || !list_ok(out) || !query_ok(soup, x1, bvh, toi, status, ws, ws_bytes, soup->n_edges))
    return IPCB_E_ARG;
  if (soup->n_edges == 0) return IPCB_OK;
  in_scalar(soup, [&](auto* scalar) {
    using S = std::remove_pointer_t<decltype(scalar)>;
    Query<S> q = make_query<S>(soup, x1, bvh, pad, exclude_same_body, 0, soup->n_edges, toi, status, ws, ws_bytes, s);
    q.thickness = thickness;
    q.out = *out;
    run_both<S, 0>(q, box_pad);
  });
  return check_launch("ipcb_edge_edge_both");
}

int ipcb_point_triangle_both(const ipcb_soup* soup, const void* x1, double pad, const ipcb_lbvh* bvh, float thickness,
                             float query_pad, const int* query_order, int exclude_same_body, ipcb_contacts* out,
                             void* toi, int* status, void* ws, size_t ws_bytes, ipcb_stream s) {
  if (!soup || !(pad >= 0.0) || !list_ok(out) || !query_ok(soup, x1, bvh, toi, status, ws, ws_bytes, soup->n_tris))
    return IPCB_E_ARG;
  if (soup->n_verts == 0 || soup->n_tris == 0) return IPCB_OK;
  in_scalar(soup, [&](auto* scalar) {
    using S = std::remove_pointer_t<decltype(scalar)>;
    Query<S> q = make_query<S>(soup, x1, bvh, pad, exclude_same_body, 0, soup->n_verts, toi, status, ws, ws_bytes, s);
    q.order = query_order;
    q.thickness = thickness;
    q.reach = query_pad;
    q.out = *out;
    run_both<S, 1>(q, 0.f);
  });
  return check_launch("ipcb_point_triangle_both");
}

int ipcb_edge_edge_solve(const ipcb_soup* soup, const void* x1, double pad, const ipcb_lbvh* bvh,
                         int exclude_same_body, void* toi, int* status, void* ws, size_t ws_bytes, ipcb_stream s) {
  if (!soup || !(pad >= 0.0) || !query_ok(soup, x1, bvh, toi, status, ws, ws_bytes, soup->n_edges)) return IPCB_E_ARG;
  if (soup->n_edges == 0) return IPCB_OK;
  in_scalar(soup, [&](auto* scalar) {
    using S = std::remove_pointer_t<decltype(scalar)>;
    solve<S, 0>(
        make_query<S>(soup, x1, bvh, pad, exclude_same_body, 0, soup->n_edges, toi, status, ws, ws_bytes, s));
  });
  return check_launch("ipcb_edge_edge_solve");
}

int ipcb_point_triangle_solve(const ipcb_soup* soup, const void* x1, double pad, const ipcb_lbvh* bvh,
                              const int* query_order, int exclude_same_body, void* toi, int* status, void* ws,
                              size_t ws_bytes, ipcb_stream s) {
  if (!soup || !(pad >= 0.0) || !query_ok(soup, x1, bvh, toi, status, ws, ws_bytes, soup->n_tris)) return IPCB_E_ARG;
  if (soup->n_verts == 0 || soup->n_tris == 0) return IPCB_OK;
  in_scalar(soup, [&](auto* scalar) {
    using S = std::remove_pointer_t<decltype(scalar)>;
    Query<S> q = make_query<S>(soup, x1, bvh, pad, exclude_same_body, 0, soup->n_verts, toi, status, ws, ws_bytes, s);
    q.order = query_order;
    solve<S, 1>(q);
  });
  return check_launch("ipcb_point_triangle_solve");
}

int ipcb_edge_edge_intersections(const ipcb_soup* soup, const void* x1, const ipcb_lbvh* bvh, const float* lower,
                                 const float* upper, int exclude_same_body, double thickness, void* toi,
                                 const ipcb_contacts* out, int* status, void* ws, size_t ws_bytes, ipcb_stream s) {
  if (!soup || !lower || !upper || !list_ok(out) ||
      !query_ok(soup, x1, bvh, toi, status, ws, ws_bytes, soup->n_edges))
    return IPCB_E_ARG;
  if (soup->n_edges == 0) return IPCB_OK;
  in_scalar(soup, [&](auto* scalar) {
    using S = std::remove_pointer_t<decltype(scalar)>;
    Query<S> q = make_query<S>(soup, x1, bvh, 0.0, exclude_same_body, 0, soup->n_edges, toi, status, ws, ws_bytes, s);
    q.lower = lower;
    q.upper = upper;
    q.sink = Sink{*out, thickness * 2.0, 1};
    run_boxes<S, 0>(q);
  });
  return check_launch("ipcb_edge_edge_intersections");
}

int ipcb_point_triangle_intersections(const ipcb_soup* soup, const void* x1, const ipcb_lbvh* bvh, double pad,
                                      int exclude_same_body, double thickness, void* toi, const ipcb_contacts* out,
                                      int* status, void* ws, size_t ws_bytes, ipcb_stream s) {
  if (!soup || !list_ok(out) || !query_ok(soup, x1, bvh, toi, status, ws, ws_bytes, soup->n_tris)) return IPCB_E_ARG;
  if (soup->n_verts == 0 || soup->n_tris == 0) return IPCB_OK;
  in_scalar(soup, [&](auto* scalar) {
    using S = std::remove_pointer_t<decltype(scalar)>;
    Query<S> q = make_query<S>(soup, x1, bvh, pad, exclude_same_body, 0, soup->n_verts, toi, status, ws, ws_bytes, s);
    q.sink = Sink{*out, thickness * 2.0, 1};
    run_boxes<S, 1>(q);
  });
  return check_launch("ipcb_point_triangle_intersections");
}

int ipcb_collision_time(int kind, int n, const double* p_t0, const double* p_t1, double* t, int* status,
                        ipcb_stream s) {
  if (n < 0 || (kind != 0 && kind != 1)) return IPCB_E_ARG;
  if (n == 0) return IPCB_OK;
  if (!p_t0 || !p_t1 || !t || !status) return IPCB_E_ARG;
  k_pair_time<<<div_up(n, 128), 128, 0, (cudaStream_t)s>>>(kind, n, p_t0, p_t1, t, status);
  return check_launch("ipcb_collision_time");
}

int ipcb_cubic_roots(int n, const double* coef, double x0, double x1, double* roots, int* n_roots, int* status,
                     ipcb_stream s) {
  if (n < 0) return IPCB_E_ARG;
  if (n == 0) return IPCB_OK;
  if (!coef || !roots || !n_roots || !status) return IPCB_E_ARG;
  k_cubic<<<div_up(n, 128), 128, 0, (cudaStream_t)s>>>(n, coef, x0, x1, roots, n_roots, status);
  return check_launch("ipcb_cubic_roots");
}


static bool bodies_ok(const ipcb_bodies* B) {
  return B && B->n_bodies > 0 && B->local_lower && B->local_upper && B->edge_off && B->edge_ids && B->tri_off &&
         B->tri_ids && B->vert_off && B->vert_ids && B->edge_wide && B->tri_wide && B->frames && B->motion;
}

int ipcb_body_pairs_swept(const ipcb_bodies* B, int fp64, const void* q, const void* dq, double padding, int* pairs,
                          int capacity, int* count, int* status, ipcb_stream s) {
  if (!bodies_ok(B) || !q || !dq || !pairs || capacity < 0 || !count || !status) return IPCB_E_ARG;
  cudaStream_t st = (cudaStream_t)s;
  const int nb = B->n_bodies;
  if (fp64)
    k_body_frames_swept<double><<<div_up(nb, 128), 128, 0, st>>>(nb, (const double*)q, (const double*)dq,
                                                                  B->local_lower, B->local_upper, B->frames,
                                                                  B->motion, status);
  else
    k_body_frames_swept<float><<<div_up(nb, 128), 128, 0, st>>>(nb, (const float*)q, (const float*)dq,
                                                                 B->local_lower, B->local_upper, B->frames,
                                                                 B->motion, status);
  k_swept_pair_cull<<<div_up((long long)nb * nb, 256), 256, 0, st>>>(nb, B->frames + 13 * (size_t)nb, padding,
                                                                     (int2*)pairs, capacity, count);
  return check_launch("ipcb_body_pairs_swept");
}

int ipcb_fixed_edge_edge_toi(const ipcb_soup* soup, const void* x1, const ipcb_bodies* B, const int* fixed,
                             const int* pairs, int n_pairs, double pad, void* toi, int* status, void* ws,
                             size_t ws_bytes, ipcb_stream s) {
  if (!soup || !x1 || !bodies_ok(B) || !pairs || n_pairs < 0 || !toi || !status || !ws || ws_bytes < kCandHeader)
    return IPCB_E_ARG;
  if (n_pairs == 0 || B->max_edges == 0) return IPCB_OK;
  cudaStream_t st = (cudaStream_t)s;
  CandList c = cand_list(ws, ws_bytes);
  cudaMemsetAsync(c.count, 0, sizeof(int), st);
  dim3 grid(div_up(B->max_edges, 128) * n_pairs);
  const int gc = min(div_up(c.capacity > 0 ? c.capacity : 1, 128), 2048);
  if (soup->fp64) {
    k_fixed_ee_collect<double><<<grid, 128, 0, st>>>((const double*)soup->x, (const double*)x1, soup->edges, *B,
                                                     fixed, (const int2*)pairs, pad, c, (double*)toi, status);
    if (c.capacity)
      k_cand_toi<double, 0><<<gc, 128, 0, st>>>((const double*)soup->x, (const double*)x1, soup->edges, c,
                                              (double*)toi, status, Sink{}, nullptr);
  } else {
    k_fixed_ee_collect<float><<<grid, 128, 0, st>>>((const float*)soup->x, (const float*)x1, soup->edges, *B, fixed,
                                                    (const int2*)pairs, pad, c, (float*)toi, status);
    if (c.capacity)
      k_cand_toi<float, 0><<<gc, 128, 0, st>>>((const float*)soup->x, (const float*)x1, soup->edges, c, (float*)toi,
                                             status, Sink{}, nullptr);
  }
  return check_launch("ipcb_fixed_edge_edge_toi");
}

int ipcb_fixed_point_triangle_toi(const ipcb_soup* soup, const void* x1, const ipcb_bodies* B, const int* pairs,
                                  int n_pairs, double pad, void* toi, int* status, void* ws, size_t ws_bytes,
                                  ipcb_stream s) {
  if (!soup || !x1 || !bodies_ok(B) || !pairs || n_pairs < 0 || !toi || !status || !ws || ws_bytes < kCandHeader)
    return IPCB_E_ARG;
  if (n_pairs == 0 || B->max_verts == 0) return IPCB_OK;
  cudaStream_t st = (cudaStream_t)s;
  CandList c = cand_list(ws, ws_bytes);
  cudaMemsetAsync(c.count, 0, sizeof(int), st);
  dim3 grid(div_up(B->max_verts, 128) * n_pairs, 2);
  const int gc = min(div_up(c.capacity > 0 ? c.capacity : 1, 128), 2048);
  if (soup->fp64) {
    k_fixed_pt_collect<double><<<grid, 128, 0, st>>>((const double*)soup->x, (const double*)x1, soup->triangles, *B,
                                                     (const int2*)pairs, pad, c, (double*)toi, status);
    if (c.capacity)
      k_cand_toi<double, 1><<<gc, 128, 0, st>>>((const double*)soup->x, (const double*)x1, soup->triangles, c,
                                              (double*)toi, status, Sink{}, nullptr);
  } else {
    k_fixed_pt_collect<float><<<grid, 128, 0, st>>>((const float*)soup->x, (const float*)x1, soup->triangles, *B,
                                                    (const int2*)pairs, pad, c, (float*)toi, status);
    if (c.capacity)
      k_cand_toi<float, 1><<<gc, 128, 0, st>>>((const float*)soup->x, (const float*)x1, soup->triangles, c,
                                             (float*)toi, status, Sink{}, nullptr);
  }
  return check_launch("ipcb_fixed_point_triangle_toi");
}

}  // extern "C"
