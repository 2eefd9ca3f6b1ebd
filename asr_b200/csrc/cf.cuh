// Device continued fractions and terminators: cf_species (src/asr_chain.f90:67-167), sqrt_tail / cf_green
// (src/reference/asr_greens.f90:12-22, :80-90) and the real Beer-Pettifor asymptote (src/reference/asr_terminator.f90:39-67).
//
// LAPACK zgeev (the reference's eigenvalues of the m x m chain matrix) is replaced by the implicit-shift QL iteration for a
// complex symmetric tridiagonal matrix (eigenvalues only): the EISPACK tql1 / Numerical Recipes tqli scheme carried over
// to complex symmetric matrices with complex plane rotations (Cullum & Willoughby, Lanczos Algorithms for Large Symmetric
// Eigenvalue Computations, Vol. 1, ch. 6, CMTQL1).  dsterf (real tridiagonal eigenvalues) is replaced by Sturm-sequence
// bisection for the extreme eigenvalue.
#pragma once
#include <cfloat>
#include <cmath>

#include "common.cuh"

namespace asrb {

constexpr int CF_NMAX = 128;   // longest chain the device fractions take

__host__ __device__ inline double inv_sqrt(double x) {
#ifdef __CUDA_ARCH__
  return rsqrt(x);
#else
  return 1.0 / std::sqrt(x);
#endif
}
// |re| + |im|: within a factor sqrt(2) of the modulus, for the tests that compare with DBL_EPSILON
__host__ __device__ __forceinline__ double cabs1(double2 a) { return fabs(a.x) + fabs(a.y); }

// r = sqrt(w) (principal, as csqrt_p) and ir = 1 / r from two reciprocal square roots: with 1/|w| = |w|^2 ^ -1/2,
// sqrt(w) = (t, |w.y| / 2t) or its mirror for t = ((|w| + |w.x|) / 2)^1/2, and 1 / sqrt(w) = conj(sqrt(w)) / |w|.  The four
// divisions, two square roots and a hypot of csqrt_p and two cdiv of a plane rotation are its whole latency, and one
// rotation waits for the last.  Moduli whose square leaves the double range take csqrt_p and cdiv.
__host__ __device__ __forceinline__ void csqrt_inv(double2 w, double2& r, double2& ir) {
  const double q = w.x * w.x + w.y * w.y;
  if (q > 1e-290 && q < 1e290) {
    const double rq = inv_sqrt(q), t2 = 0.5 * (q * rq + fabs(w.x)), rt = inv_sqrt(t2);
    const double t = t2 * rt, o = 0.5 * fabs(w.y) * rt;
    r = w.x >= 0.0 ? make_double2(t, copysign(o, w.y)) : make_double2(o, copysign(t, w.y));
    ir = make_double2(r.x * rq, -r.y * rq);
  } else {
    r = csqrt_p(w);
    ir = cmag(r) == 0.0 ? make_double2(0.0, 0.0) : cdiv(make_double2(1.0, 0.0), r);
  }
}

// eigenvalues of the complex symmetric tridiagonal (d[0..n-1], e[0..n-2]) in place in d; e is destroyed.  0 = converged.
__host__ __device__ inline int cs_tridiag_eig(int n, double2* d, double2* e) {
  if (n <= 0) return 0;
  e[n - 1] = make_double2(0.0, 0.0);
  for (int l = 0; l < n; ++l) {
    int iter = 0;
    for (;;) {
      int m;
      for (m = l; m < n - 1; ++m)
        if (cabs1(e[m]) <= DBL_EPSILON * (cabs1(d[m]) + cabs1(d[m + 1]))) break;
      if (m == l) break;
      if (++iter > 60) return 1;
      double2 g = cdiv(csub(d[l + 1], d[l]), cscale(e[l], 2.0));
      double2 r, ir;
      r = csqrt_p(cadd(cmul(g, g), make_double2(1.0, 0.0)));
      double2 gp = cadd(g, r), gm = csub(g, r);
      double2 den = cabs1(gp) >= cabs1(gm) ? gp : gm;
      g = cadd(csub(d[m], d[l]), cdiv(e[l], den));
      double2 s = make_double2(1.0, 0.0), c = make_double2(1.0, 0.0), p = make_double2(0.0, 0.0);
      double2 dn = d[m];   // d[i + 1] of the next rotation
      bool early = false;
      for (int i = m - 1; i >= l; --i) {
        const double2 ei = e[i], di = d[i];
        double2 f = cmul(s, ei), b = cmul(c, ei);
        csqrt_inv(cadd(cmul(f, f), cmul(g, g)), r, ir);
        e[i + 1] = r;
        if (r.x == 0.0 && r.y == 0.0) {
          d[i + 1] = csub(dn, p);
          e[m] = make_double2(0.0, 0.0);
          early = true;
          break;
        }
        s = cmul(f, ir);
        c = cmul(g, ir);
        g = csub(dn, p);
        r = cadd(cmul(csub(di, g), s), cscale(cmul(c, b), 2.0));
        p = cmul(s, r);
        d[i + 1] = cadd(g, p);
        g = csub(cmul(c, r), b);
        dn = di;
      }
      if (early) continue;
      d[l] = csub(d[l], p);
      e[l] = g;
      e[m] = make_double2(0.0, 0.0);
    }
  }
  return 0;
}

// extreme (by real part) eigenvalues of the chain matrix with a[m-1] replaced by am; returns 0 on success
__host__ __device__ inline int chain_extremes(const double2* a, const double2* b, int m, double2 am, double2* wd, double2* we,
                                              double2& lo, double2& hi) {
  for (int j = 0; j < m; ++j) wd[j] = a[j];
  wd[m - 1] = am;
  for (int j = 0; j < m - 1; ++j) we[j] = b[j];
  if (cs_tridiag_eig(m, wd, we)) return 1;
  int ilo = 0, ihi = 0;
  for (int j = 1; j < m; ++j) {
    if (wd[j].x < wd[ilo].x) ilo = j;
    if (wd[j].x > wd[ihi].x) ihi = j;
  }
  lo = wd[ilo];
  hi = wd[ihi];
  return 0;
}

// tail parameters (aa, bb) of cf_species (src/asr_chain.f90:80-101): hull extremes, Beer-Pettifor fixed point, avg2 or
// none.  wd, we: work (m).
__host__ __device__ inline void cf_tail_dev(const double2* a, const double2* b, int m, int tail, double2* wd, double2* we,
                                            int* nfall, double2& aa, double2& bb) {
  bool ok = false;
  double2 lo, hi;
  if (m >= 2 && tail != 0) ok = chain_extremes(a, b, m, a[m - 1], wd, we, lo, hi) == 0;
  if (ok) {
    aa = cscale(cadd(lo, hi), 0.5);
    bb = cscale(csub(hi, lo), 0.25);
    if (tail == 2) {   // bp_fixed_point, src/asr_chain.f90:126-156
      bool done = false;
      for (int it = 0; it < 200 && !done; ++it) {
        double2 l1, h1, l2, h2;
        if (chain_extremes(a, b, m, cadd(a[m - 1], bb), wd, we, l1, h1)) { if (nfall) ++*nfall; done = true; break; }
        if (chain_extremes(a, b, m, csub(a[m - 1], bb), wd, we, l2, h2)) { if (nfall) ++*nfall; done = true; break; }
        double2 an = cscale(cadd(h1, l2), 0.5), bn = cscale(csub(h1, l2), 0.25);
        if (cmag(csub(an, aa)) + cmag(csub(bn, bb)) < 1.0e-12 * (1.0 + cmag(bn))) { aa = an; bb = bn; done = true; break; }
        aa = an;
        bb = bn;
      }
      if (!done) {
        if (nfall) ++*nfall;
        chain_extremes(a, b, m, a[m - 1], wd, we, lo, hi);
        aa = cscale(cadd(lo, hi), 0.5);
        bb = cscale(csub(hi, lo), 0.25);
      }
    }
  } else {
    aa = a[m - 1];
    bb = m > 1 ? b[m - 2] : make_double2(0.0, 0.0);
  }
  if (tail == 3 && m >= 3) {
    aa = cscale(cadd(a[m - 1], a[m - 2]), 0.5);
    bb = csqrt_p(cscale(cadd(cmul(b[m - 2], b[m - 2]), cmul(b[m - 3], b[m - 3])), 0.5));
  }
  if (tail == 0) { aa = make_double2(0.0, 0.0); bb = make_double2(0.0, 0.0); }
}

#ifdef __CUDACC__
// The roots of one chain's two Beer-Pettifor problems, T with +bb and with -bb in the last diagonal entry, for one warp.
struct BpRoots {
  double2 a[CF_NMAX], b2[CF_NMAX];        // diagonal and squared off-diagonal, scaled to entries of order one
  double2 lam[2][2][CF_NMAX];             // [buffer][+bb, -bb][root]
};
// one Ehrlich-Aberth sweep over the m roots of both problems, from buffer `cur` into the other one (all roots at once; a thread
// takes the roots t, t + 32, ..): with N = p / p' of the characteristic polynomial (its three-term recurrence) a root moves by
// N / (1 - N sum_j 1 / (x - x_j)).  al: the last diagonal entries.  True when every root moved less than 1e-11: the sweep's
// convergence is cubic, so what is left is below the rounding of the entries.
__device__ inline bool bp_sweep(BpRoots& R, int m, int cur, const double2 (&al)[2]) {
  bool settled = true;
  for (int i = threadIdx.x & 31; i < m; i += 32) {
    double2 x[2], p0[2], pm[2], q0[2], qm[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      x[u] = R.lam[cur][u][i];
      p0[u] = make_double2(1.0, 0.0);
      pm[u] = q0[u] = qm[u] = make_double2(0.0, 0.0);
    }
    for (int k = 0; k < m; ++k) {
      const double2 ak = R.a[k], c = k > 0 ? R.b2[k - 1] : make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const double2 t = csub(x[u], k == m - 1 ? al[u] : ak);
        const double2 q1 = cadd(csub(cmul(t, q0[u]), cmul(c, qm[u])), p0[u]), p1 = csub(cmul(t, p0[u]), cmul(c, pm[u]));
        pm[u] = p0[u];
        p0[u] = p1;
        qm[u] = q0[u];
        q0[u] = q1;
      }
    }
    // sum_j 1 / (x - x_j) as a fraction num / den: one division a root, none in the loop
    double2 num[2], den[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      num[u] = make_double2(0.0, 0.0);
      den[u] = make_double2(1.0, 0.0);
    }
    for (int j = 0; j < m; ++j) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const double2 d = csub(x[u], R.lam[cur][u][j]);
        const bool other = d.x != 0.0 || d.y != 0.0;   // not itself
        const double2 n1 = cadd(cmul(num[u], d), den[u]), d1 = cmul(den[u], d);
        num[u] = other ? n1 : num[u];
        den[u] = other ? d1 : den[u];
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {   // p / p' / (1 - p / p' num / den)
      double2 step = make_double2(0.0, 0.0);
      if (p0[u].x != 0.0 || p0[u].y != 0.0)
        step = cdiv(cmul(p0[u], den[u]), csub(cmul(q0[u], den[u]), cmul(p0[u], num[u])));
      if (!(cabs1(step) <= 1.0e-11)) settled = false;
      R.lam[cur ^ 1][u][i] = csub(x[u], step);
    }
  }
  __syncwarp();
  return __all_sync(0xffffffffu, settled);
}
// the warp's sums of N values a thread
template <int N>
__device__ __forceinline__ void warp_sums(double (&v)[N]) {
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], off);
}
// the roots of both problems from those in buffer `cur`: settled within 24 sweeps, and complete (sum and sum of squares of the
// roots against the traces of T and T^2, tr and tr2 without the last entry)
__device__ inline bool bp_roots(BpRoots& R, int m, int& cur, const double2 (&al)[2], double2 tr, double2 tr2) {
  int left = 24;
  for (bool ok = false; !ok; cur ^= 1) {
    if (left-- == 0) return false;
    ok = bp_sweep(R, m, cur, al);
  }
  double v[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int i = threadIdx.x & 31; i < m; i += 32)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const double2 x = R.lam[cur][u][i], q = cmul(x, x);
      v[4 * u] += x.x;
      v[4 * u + 1] += x.y;
      v[4 * u + 2] += q.x;
      v[4 * u + 3] += q.y;
    }
  warp_sums(v);
  bool good = true;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const double2 e1 = csub(make_double2(v[4 * u], v[4 * u + 1]), cadd(tr, al[u]));
    const double2 e2 = csub(make_double2(v[4 * u + 2], v[4 * u + 3]), cadd(tr2, cmul(al[u], al[u])));
    good = good && cabs1(e1) <= 1.0e-11 * m && cabs1(e2) <= 1.0e-10 * m;
  }
  return good;
}
// the root of problem u with the largest (sgn = 1) or smallest (-1) real part
__device__ inline double2 bp_edge(const BpRoots& R, int m, int cur, int u, double sgn) {
  double best = -1.0 / 0.0;
  int at = 0;
  for (int i = threadIdx.x & 31; i < m; i += 32)
    if (sgn * R.lam[cur][u][i].x > best) { best = sgn * R.lam[cur][u][i].x; at = i; }
  for (int off = 16; off > 0; off >>= 1) {
    const double v = __shfl_xor_sync(0xffffffffu, best, off);
    const int w = __shfl_xor_sync(0xffffffffu, at, off);
    if (v > best || (v == best && w < at)) { best = v; at = w; }
  }
  return R.lam[cur][u][at];
}

// cf_tail_dev by one warp (live: there is a chain, the same for the whole warp); every thread gets the tail.  nf: tail fallbacks.
// Only the Beer-Pettifor tail uses more than one thread: its map bb -> (edge of T + bb, edge of T - bb) is iterated as
// written there, up to 200 times, but after the hull's eigenvalue problem (plane rotations, one thread) the spectra are
// followed from one iteration to the next by bp_roots, all roots at once, some three sweeps an iteration (17 us with its checks at 20 levels;
// the rotations, a serial chain, took 265 us).  Roots that do not settle or are not complete, near-defective chains, are
// left to the rotations, for good after the third time.
__device__ inline void cf_tail_warp(bool live, const double2* a, const double2* b, int m, int tail, BpRoots& R, double2* wd, double2* we,
                                    int& nf, double2& aa, double2& bb) {
  const int t = threadIdx.x & 31;
  nf = 0;
  aa = bb = make_double2(0.0, 0.0);
  if (!live) return;
  double2 lo, hi;
  int eig = 0;
  if (t == 0) {
    if (tail != 2) cf_tail_dev(a, b, m, tail, wd, we, nullptr, aa, bb);
    else if (m >= 2 && chain_extremes(a, b, m, a[m - 1], wd, we, lo, hi) == 0) {
      eig = 1;
      aa = cscale(cadd(lo, hi), 0.5);
      bb = cscale(csub(hi, lo), 0.25);
    } else {   // the last coefficients
      aa = a[m - 1];
      bb = m > 1 ? b[m - 2] : make_double2(0.0, 0.0);
    }
  }
  __syncwarp();
  auto bcast = [](double2 v) { return make_double2(__shfl_sync(0xffffffffu, v.x, 0), __shfl_sync(0xffffffffu, v.y, 0)); };
  aa = bcast(aa);
  bb = bcast(bb);
  if (!__shfl_sync(0xffffffffu, eig, 0)) return;
  const double2 a0 = aa, b0 = bb;
  // a power of two that brings the largest entry to order one
  double big = 0.0;
  for (int k = t; k < m; k += 32) big = fmax(big, fmax(cabs1(a[k]), k < m - 1 ? cabs1(b[k]) : 0.0));
  for (int off = 16; off > 0; off >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, off));
  const int ex = big > 0.0 && big < 1e300 ? ilogb(big) : 0;
  const double sc = scalbn(1.0, -ex), us = scalbn(1.0, ex);
  double2 tr = make_double2(0.0, 0.0), tr2 = tr;
  for (int k = t; k < m; k += 32) {
    const double2 ak = cscale(a[k], sc), bk = k < m - 1 ? cscale(b[k], sc) : make_double2(0.0, 0.0), c = cmul(bk, bk);
    R.a[k] = ak;
    R.b2[k] = c;
    if (k < m - 1) { tr = cadd(tr, ak); tr2 = cadd(tr2, cadd(cmul(ak, ak), cscale(c, 2.0))); }
  }
  double trs[4] = {tr.x, tr.y, tr2.x, tr2.y};
  warp_sums(trs);
  tr = make_double2(trs[0], trs[1]);
  tr2 = make_double2(trs[2], trs[3]);
  if (t == 0)
    for (int k = 0; k < m; ++k) R.lam[0][0][k] = R.lam[0][1][k] = cscale(wd[k], sc);
  __syncwarp();
  int cur = 0, lost = 0;
  for (int it = 0; it < 200; ++it) {
    const double2 ap = cadd(a[m - 1], bb), am = csub(a[m - 1], bb);
    const double2 al[2] = {cscale(ap, sc), cscale(am, sc)};
    double2 h1, l2;
    if (lost < 3 && bp_roots(R, m, cur, al, tr, tr2)) {
      h1 = cscale(bp_edge(R, m, cur, 0, 1.0), us);
      l2 = cscale(bp_edge(R, m, cur, 1, -1.0), us);
    } else {
      ++lost;
      int bad = 0;
      double2 edge = make_double2(0.0, 0.0);
      if (t < 2) {
        bad = chain_extremes(a, b, m, t ? am : ap, wd, we, lo, hi);
        edge = t ? lo : hi;
        if (!bad)
          for (int k = 0; k < m; ++k) R.lam[cur][t][k] = cscale(wd[k], sc);
      }
      __syncwarp();
      if (__any_sync(0xffffffffu, bad)) { ++nf; return; }   // an eigenvalue failure keeps the last iterate
      h1 = bcast(edge);
      l2 = make_double2(__shfl_sync(0xffffffffu, edge.x, 1), __shfl_sync(0xffffffffu, edge.y, 1));
    }
    const double2 an = cscale(cadd(h1, l2), 0.5), bn = cscale(csub(h1, l2), 0.25);
    const bool done = cmag(csub(an, aa)) + cmag(csub(bn, bb)) < 1.0e-12 * (1.0 + cmag(bn));
    aa = an;
    bb = bn;
    if (__shfl_sync(0xffffffffu, (int)done, 0)) return;
  }
  ++nf;   // no fixed point within 200 iterations: the hull
  aa = a0;
  bb = b0;
}
#endif

// the square-root terminator of the tail (aa, bb) at z, on the branch with |bb g| minimal (src/asr_chain.f90:103-110)
__host__ __device__ inline double2 cf_tail_term(double2 z, double2 aa, double2 bb) {
  double2 d = csub(z, aa), tl = make_double2(0.0, 0.0);
  if (cmag(bb) >= 1.0e-14) {   // |bb| < 1e-14: no tail
    double2 bb2 = cmul(bb, bb);
    double2 s = csqrt_p(csub(cmul(d, d), cscale(bb2, 4.0)));
    double2 g1 = cdiv(csub(d, s), cscale(bb2, 2.0)), g2 = cdiv(cadd(d, s), cscale(bb2, 2.0));
    tl = cmag(cmul(bb, g1)) <= cmag(cmul(bb, g2)) ? cmul(bb2, g1) : cmul(bb2, g2);
  }
  return tl;
}

// g11 of the chain (a, b) of depth m at z with the square-root tail (aa, bb)
__host__ __device__ inline double2 cf_green_dev(const double2* a, const double2* b, int m, double2 z, double2 aa, double2 bb) {
  double2 tl = cf_tail_term(z, aa, bb);
  double2 one = make_double2(1.0, 0.0);
  double2 gt = cdiv(one, csub(csub(z, a[m - 1]), tl));
  for (int j = m - 2; j >= 0; --j) gt = cdiv(one, csub(csub(z, a[j]), cmul(cmul(b[j], b[j]), gt)));
  return gt;
}

// cf_species: g11 of the chain (a, b) of depth m at z with the tail (0 none, 1 hull, 2 bp, 3 avg2).  wd, we: work (m).
__host__ __device__ inline double2 cf_species_dev(const double2* a, const double2* b, int m, double2 z, int tail, double2* wd,
                                                  double2* we, int* nfall, double2* edges) {
  double2 aa, bb;
  cf_tail_dev(a, b, m, tail, wd, we, nfall, aa, bb);
  if (edges) { edges[0] = aa; edges[1] = bb; }
  return cf_green_dev(a, b, m, z, aa, bb);
}

// cf_species with the projection f = sum_k c_k prod_{j<k} (b_j gt_{j+1}) gt_1 (src/asr_chain.f90:111-122); closed: the exact
// fraction without tail (cf_closed, src/asr_ed3.f90:221-236).  gt: work (m); wd, we: work (m).
__host__ __device__ inline double2 cf_species_f_dev(const double2* a, const double2* b, const double2* c, int m, double2 z, int tail,
                                                    bool closed, double2* gt, double2* wd, double2* we, int* nfall, double2& f) {
  double2 tl = make_double2(0.0, 0.0);
  if (!closed) {
    double2 aa, bb;
    cf_tail_dev(a, b, m, tail, wd, we, nfall, aa, bb);
    tl = cf_tail_term(z, aa, bb);
  }
  double2 one = make_double2(1.0, 0.0);
  gt[m - 1] = cdiv(one, csub(csub(z, a[m - 1]), tl));
  for (int j = m - 2; j >= 0; --j) gt[j] = cdiv(one, csub(csub(z, a[j]), cmul(cmul(b[j], b[j]), gt[j + 1])));
  f = make_double2(0.0, 0.0);
  double2 prod = gt[0];
  for (int k = 0; k < m; ++k) {
    f = cadd(f, cmul(c[k], prod));
    if (k < m - 1) prod = cmul(prod, cmul(b[k], gt[k + 1]));
  }
  return gt[0];
}

// cf_species with the factors pv_k = [g]_{k1} = gt_1 prod_{j<k} (b_j gt_{j+1}) of the projections f = sum_k c_k pv_k
// (src/asr_chain.f90:111-122, the pv output used by edc_green_proj); pv (m) receives them, the return value is g11.
__host__ __device__ inline double2 cf_species_pv_dev(const double2* a, const double2* b, int m, double2 z, double2 aa, double2 bb,
                                                     double2* pv) {
  double2 tl = cf_tail_term(z, aa, bb);
  double2 one = make_double2(1.0, 0.0);
  pv[m - 1] = cdiv(one, csub(csub(z, a[m - 1]), tl));   // gt in place, then turned into the products
  for (int j = m - 2; j >= 0; --j) pv[j] = cdiv(one, csub(csub(z, a[j]), cmul(cmul(b[j], b[j]), pv[j + 1])));
  double2 g11 = pv[0], prod = pv[0];
  for (int k = 0; k < m; ++k) {
    double2 gnext = k < m - 1 ? pv[k + 1] : make_double2(0.0, 0.0);
    pv[k] = prod;
    if (k < m - 1) prod = cmul(prod, cmul(b[k], gnext));
  }
  return g11;
}

// ---- real chains (plain mode)
#ifdef __CUDACC__
// Number of eigenvalues below x of the real tridiagonal (d, e2 = e^2; last diagonal entry dl) from the signs of the leading
// minors p_j = (d_j - x) p_{j-1} - e2_{j-1} p_{j-2}, rescaled before they leave the double range; a zero minor takes the
// sign of its predecessor.  No division: the quotients of successive minors are a chain of dependent divisions.
__device__ inline int sturm_minors(int n, const double* d, const double* e2, double dl, double x) {
  int cnt = 0;
  double p0 = 1.0, p1 = (n > 1 ? d[0] : dl) - x;
  bool neg = p1 < 0.0;
  cnt += neg;
  for (int i = 1; i < n; ++i) {
    const double p2 = ((i < n - 1 ? d[i] : dl) - x) * p1 - e2[i - 1] * p0;
    p0 = p1;
    p1 = p2;
    if (p1 != 0.0 && (p1 < 0.0) != neg) { ++cnt; neg = !neg; }
    const double m = fabs(p1);
    if (m > 1e150) { p0 *= 1e-150; p1 *= 1e-150; }
    else if (m < 1e-150 && fabs(p0) < 1e-150) { p0 *= 1e150; p1 *= 1e150; }
  }
  return cnt;
}
// The extreme eigenvalue of the real tridiagonal with last diagonal entry dl, by the 16 threads of a half warp (thread h of
// 16; mask: its half): every step cuts the bracket into 17 and keeps the section where the count passes the target, to the
// resolution of a double.  (lo, hi): Gershgorin bounds.
__device__ inline double tridiag_extreme_half(int n, const double* d, const double* e2, double dl, double lo, double hi, bool upper,
                                              int h, unsigned mask) {
  const int target = upper ? n : 1;
  for (int it = 0; it < 64; ++it) {
    const double w = hi - lo, x = lo + w * ((h + 1) * (1.0 / 17.0));
    const double mid = 0.5 * (lo + hi);
    if (mid <= lo || mid >= hi) break;
    const unsigned ge = __ballot_sync(mask, sturm_minors(n, d, e2, dl, x) >= target) & mask;   // the sections at and above the edge
    const unsigned g = ge >> (mask == 0xffff0000u ? 16 : 0);
    const int k = g ? __ffs(g) - 1 : 16;   // the first such point
    const double nlo = k == 0 ? lo : lo + w * (k * (1.0 / 17.0)), nhi = k == 16 ? hi : lo + w * ((k + 1) * (1.0 / 17.0));
    if (nlo <= lo && nhi >= hi) break;
    lo = nlo;
    hi = nhi;
  }
  return 0.5 * (lo + hi);
}
// bp_asymptote (src/reference/asr_terminator.f90:39-67) by one warp: the upper edge of T + B on the lower half of the warp,
// the lower edge of T - B on the upper half; d, e2: work (n) shared by the warp
__device__ inline void bp_asymptote_warp(const double* a, const double* b, int n, double* d, double* e2, double& ainf, double& binf) {
  const int t = threadIdx.x & 31, h = t & 15;
  const bool upper = t < 16;
  const unsigned mask = upper ? 0x0000ffffu : 0xffff0000u;
  for (int i = t; i < n; i += 32) {
    d[i] = a[i];
    e2[i] = b[i] * b[i];
  }
  __syncwarp();
  double A = 0.5 * (a[n - 1] + a[n - 2]);
  double B = sqrt(0.5 * (b[n - 1] * b[n - 1] + b[n - 2] * b[n - 2]));
  for (int it = 0; it < 500; ++it) {
    const double dl = upper ? a[n - 1] + B : a[n - 1] - B;
    double lo = dl, hi = dl;   // Gershgorin bounds, a little widened
    for (int i = 0; i < n; ++i) {
      const double r = (i > 0 ? fabs(b[i - 1]) : 0.0) + (i < n - 1 ? fabs(b[i]) : 0.0), x = i < n - 1 ? d[i] : dl;
      lo = fmin(lo, x - r);
      hi = fmax(hi, x + r);
    }
    const double span = hi - lo;
    lo -= 1e-12 * (span + 1.0);
    hi += 1e-12 * (span + 1.0);
    const double e = tridiag_extreme_half(n, d, e2, dl, lo, hi, upper, h, mask);
    __syncwarp();
    const double ep = __shfl_sync(0xffffffffu, e, 0), em = __shfl_sync(0xffffffffu, e, 16);
    const double an = 0.5 * (ep + em), bn = 0.25 * (ep - em);
    const bool conv = fabs(an - A) + fabs(bn - B) < 1.0e-13;
    A = an;
    B = bn;
    if (conv) break;
  }
  ainf = A;
  binf = B;
}
#endif
// sqrt_tail + cf_green (src/reference/asr_greens.f90:12-22, :80-90)
__host__ __device__ inline double2 terminated_green_dev(const double* a, const double* b, int n, double2 z, double ainf, double binf,
                                                        bool has_tail) {
  double2 tl = make_double2(0.0, 0.0);
  if (has_tail) {
    double2 w = make_double2(z.x - ainf, z.y);
    double2 s = csqrt_p(csub(cmul(w, w), make_double2(4.0 * binf * binf, 0.0)));
    double d2 = 2.0 * binf * binf;
    double2 g1 = cscale(csub(w, s), 1.0 / d2), g2 = cscale(cadd(w, s), 1.0 / d2);
    double2 g = cmag(g1) <= cmag(g2) ? g1 : g2;
    tl = cscale(g, binf * binf);
  }
  double2 one = make_double2(1.0, 0.0);
  double2 g = cdiv(one, csub(make_double2(z.x - a[n - 1], z.y), tl));
  for (int i = n - 2; i >= 0; --i) g = cdiv(one, csub(make_double2(z.x - a[i], z.y), cscale(g, b[i] * b[i])));
  return g;
}


// ---- reverse mode of cf_species (tails none, hull, avg2): abar_k += w dG/da_k, bbar_k += w dG/db_k.  G is holomorphic in
// (a, b) away from the branch choices, so the complex derivatives compose.  The hull edges are extreme eigenvalues of
// the chain matrix T; for a simple eigenvalue of a complex symmetric matrix d(lambda) = v^T dT v / (v^T v), with v from
// inverse iteration on T - lambda.  wd, we, wx: work (m).  Returns 0 on success.
__host__ __device__ inline int tridiag_solve_shift(int m, const double2* a, const double2* b, double2 lam, const double2* rhs,
                                                   double2* x, double2* wd, double2* we) {
  // (T - lam) x = rhs, Thomas algorithm on the complex symmetric tridiagonal (no pivoting; lam is perturbed off the
  // eigenvalue by the caller)
  double2 dd = csub(a[0], lam);
  if (cmag(dd) == 0.0) dd = make_double2(1e-300, 0.0);
  wd[0] = dd;
  x[0] = rhs[0];
  for (int j = 1; j < m; ++j) {
    double2 l = cdiv(b[j - 1], wd[j - 1]);
    we[j - 1] = l;
    double2 d = csub(csub(a[j], lam), cmul(l, b[j - 1]));
    if (cmag(d) == 0.0) d = make_double2(1e-300, 0.0);
    wd[j] = d;
    x[j] = csub(rhs[j], cmul(l, x[j - 1]));
  }
  x[m - 1] = cdiv(x[m - 1], wd[m - 1]);
  for (int j = m - 2; j >= 0; --j) x[j] = cdiv(csub(x[j], cmul(b[j], x[j + 1])), wd[j]);
  return 0;
}

// eigenvector t (scaled to max modulus 1) of the complex symmetric tridiagonal (a, b) at the simple eigenvalue lam: two
// steps of inverse iteration at a shift next to lam; returns t.t (the bilinear, not the Hermitian, square)
__host__ __device__ inline double2 eig_vec(int m, const double2* a, const double2* b, double2 lam, double2* v, double2* t,
                                           double2* wd, double2* we) {
  double sc = 0.0;
  for (int j = 0; j < m; ++j) sc = fmax(sc, cmag(a[j]) + (j < m - 1 ? cmag(b[j]) : 0.0));
  double2 mu = cadd(lam, make_double2(1e-10 * (sc + 1.0), 1e-10 * (sc + 1.0)));
  for (int j = 0; j < m; ++j) t[j] = make_double2(1.0 / sqrt((double)m), 0.0);
  for (int it = 0; it < 3; ++it) {
    tridiag_solve_shift(m, a, b, mu, t, v, wd, we);
    double nr = 0.0;
    for (int j = 0; j < m; ++j) nr = fmax(nr, cmag(v[j]));
    for (int j = 0; j < m; ++j) t[j] = cscale(v[j], 1.0 / nr);
  }
  double2 vv = make_double2(0.0, 0.0);
  for (int j = 0; j < m; ++j) vv = cadd(vv, cmul(t[j], t[j]));
  return vv;
}

// abar_j += w dlam/da_j, bbar_j += w dlam/db_j with dlam = v^T dT v / (v^T v)
__host__ __device__ inline void eig_grad(int m, const double2* a, const double2* b, double2 lam, double2 w, double2* abar,
                                         double2* bbar, double2* v, double2* t, double2* wd, double2* we) {
  double2 vv = eig_vec(m, a, b, lam, v, t, wd, we);
  double2 f = cdiv(w, vv);
  for (int j = 0; j < m; ++j) abar[j] = cadd(abar[j], cmul(f, cmul(t[j], t[j])));
  for (int j = 0; j < m - 1; ++j) bbar[j] = cadd(bbar[j], cmul(f, cscale(cmul(t[j], t[j + 1]), 2.0)));
}

// dlam / da_{m-1} = v_{m-1}^2 / (v^T v): the sensitivity of the eigenvalue to the last diagonal entry
__host__ __device__ inline double2 eig_last_sens(int m, const double2* a, const double2* b, double2 lam, double2* v, double2* t,
                                                 double2* wd, double2* we) {
  double2 vv = eig_vec(m, a, b, lam, v, t, wd, we);
  return cdiv(cmul(t[m - 1], t[m - 1]), vv);
}

// w: seed; work arrays of length >= m each: gt, v, t, wd, we.  Returns G.
__host__ __device__ inline double2 cf_species_adjoint(const double2* a, const double2* b, int m, double2 z, int tail, double2 w,
                                                       double2* abar, double2* bbar, double2* gt, double2* v, double2* t, double2* wd,
                                                       double2* we) {
  // forward: tail parameters
  double2 aa = make_double2(0, 0), bb = make_double2(0, 0), lo, hi, ep = make_double2(0, 0), em = make_double2(0, 0);
  int kind = 0;   // 0 none / finite, 1 hull, 2 last coefficients, 3 avg2, 4 Beer-Pettifor fixed point, 5 tail held fixed
  if (tail == 2 && m >= 2 && chain_extremes(a, b, m, a[m - 1], wd, we, lo, hi) == 0) {
    // the fixed point as cf_tail_dev iterates it (src/asr_chain.f90:126-156): converged -> differentiated implicitly;
    // not converged -> the hull values (differentiated as the hull); an eigenvalue failure keeps the last iterate, whose
    // dependence on (a, b) is not followed (kind 5)
    aa = cscale(cadd(lo, hi), 0.5);
    bb = cscale(csub(hi, lo), 0.25);
    kind = 1;
    for (int it = 0; it < 200; ++it) {
      double2 l1, h1, l2, h2;
      if (chain_extremes(a, b, m, cadd(a[m - 1], bb), wd, we, l1, h1) ||
          chain_extremes(a, b, m, csub(a[m - 1], bb), wd, we, l2, h2)) { kind = 5; break; }
      double2 an = cscale(cadd(h1, l2), 0.5), bn = cscale(csub(h1, l2), 0.25);
      if (cmag(csub(an, aa)) + cmag(csub(bn, bb)) < 1.0e-12 * (1.0 + cmag(bn))) {
        aa = an; bb = bn; ep = h1; em = l2; kind = 4;
        break;
      }
      aa = an;
      bb = bn;
    }
    if (kind == 1) {   // not converged within 200 iterations: the hull
      aa = cscale(cadd(lo, hi), 0.5);
      bb = cscale(csub(hi, lo), 0.25);
    }
  } else if (tail == 3 && m >= 3) {
    aa = cscale(cadd(a[m - 1], a[m - 2]), 0.5);
    bb = csqrt_p(cscale(cadd(cmul(b[m - 2], b[m - 2]), cmul(b[m - 3], b[m - 3])), 0.5));
    kind = 3;
  } else if (tail == 1 && m >= 2 && chain_extremes(a, b, m, a[m - 1], wd, we, lo, hi) == 0) {
    aa = cscale(cadd(lo, hi), 0.5);
    bb = cscale(csub(hi, lo), 0.25);
    kind = 1;
  } else if (tail != 0 && m >= 1) {   // eigenvalue failure or m = 1: the last coefficients (src/asr_chain.f90:95)
    aa = a[m - 1];
    bb = m > 1 ? b[m - 2] : make_double2(0.0, 0.0);
    kind = 2;
  }
  double2 d = csub(z, aa), tl = make_double2(0, 0), sroot = make_double2(0, 0);
  double sig = 0.0;
  bool has_tail = cmag(bb) >= 1.0e-14;
  if (has_tail) {
    double2 bb2 = cmul(bb, bb);
    sroot = csqrt_p(csub(cmul(d, d), cscale(bb2, 4.0)));
    double2 g1 = cdiv(csub(d, sroot), cscale(bb2, 2.0)), g2 = cdiv(cadd(d, sroot), cscale(bb2, 2.0));
    if (cmag(cmul(bb, g1)) <= cmag(cmul(bb, g2))) { tl = cmul(bb2, g1); sig = 1.0; }
    else { tl = cmul(bb2, g2); sig = -1.0; }
  }
  double2 one = make_double2(1.0, 0.0);
  gt[m - 1] = cdiv(one, csub(csub(z, a[m - 1]), tl));
  for (int j = m - 2; j >= 0; --j) gt[j] = cdiv(one, csub(csub(z, a[j]), cmul(cmul(b[j], b[j]), gt[j + 1])));
  const double2 G = gt[0];
  // reverse: gbar_j is the adjoint of gt_j
  double2 gbar = w;
  double2 tbar = make_double2(0, 0);
  for (int j = 0; j < m; ++j) {
    double2 Dbar = cmul(cscale(cmul(gt[j], gt[j]), -1.0), gbar);   // d gt / dD = -gt^2
    abar[j] = csub(abar[j], Dbar);
    if (j < m - 1) {
      bbar[j] = csub(bbar[j], cscale(cmul(cmul(b[j], gt[j + 1]), Dbar), 2.0));
      gbar = csub(make_double2(0, 0), cmul(cmul(b[j], b[j]), Dbar));
    } else {
      tbar = csub(make_double2(0, 0), Dbar);
    }
  }
  if (has_tail && kind != 0) {
    // T = (d - sig s) / 2, s^2 = d^2 - 4 bb^2, d = z - aa
    double2 aabar = cscale(cmul(tbar, csub(cscale(cdiv(d, sroot), sig), one)), 0.5);
    double2 bbbar = cmul(tbar, cscale(cdiv(bb, sroot), 2.0 * sig));
    if (kind == 3) {
      abar[m - 1] = cadd(abar[m - 1], cscale(aabar, 0.5));
      abar[m - 2] = cadd(abar[m - 2], cscale(aabar, 0.5));
      double2 f = cdiv(bbbar, cscale(bb, 2.0));   // d bb / d b_j = b_j / (2 bb)
      bbar[m - 2] = cadd(bbar[m - 2], cmul(f, b[m - 2]));
      bbar[m - 3] = cadd(bbar[m - 3], cmul(f, b[m - 3]));
    } else if (kind == 2) {
      abar[m - 1] = cadd(abar[m - 1], aabar);
      if (m > 1) bbar[m - 2] = cadd(bbar[m - 2], bbbar);
    } else if (kind == 4) {
      // bb = phi(bb) = (ep(a_m + bb) - em(a_m - bb)) / 4 and aa = (ep + em) / 2 at the fixed point.  With the
      // sensitivities pv = d ep / d a_m, pu = d em / d a_m (eigenvectors of the two shifted chain matrices):
      // d phi / d bb = (pv + pu) / 4, partial d aa / d bb = (pv - pu) / 2, and the adjoint of the fixed point
      // lam = (bbbar + aabar (pv - pu) / 2) / (1 - (pv + pu) / 4); the eigenvalue seeds are aabar / 2 +- lam / 4.
      double2* am = gt;   // gt is no longer needed: the shifted diagonal
      for (int j = 0; j < m; ++j) am[j] = a[j];
      am[m - 1] = cadd(a[m - 1], bb);
      double2 pv = eig_last_sens(m, am, b, ep, v, t, wd, we);
      am[m - 1] = csub(a[m - 1], bb);
      double2 pu = eig_last_sens(m, am, b, em, v, t, wd, we);
      double2 den = csub(one, cscale(cadd(pv, pu), 0.25));
      double2 lam = cdiv(cadd(bbbar, cmul(aabar, cscale(csub(pv, pu), 0.5))), den);
      double2 wp = cadd(cscale(aabar, 0.5), cscale(lam, 0.25)), wm = csub(cscale(aabar, 0.5), cscale(lam, 0.25));
      am[m - 1] = cadd(a[m - 1], bb);
      eig_grad(m, am, b, ep, wp, abar, bbar, v, t, wd, we);
      am[m - 1] = csub(a[m - 1], bb);
      eig_grad(m, am, b, em, wm, abar, bbar, v, t, wd, we);
    } else if (kind == 5) {
      // tail held fixed
    } else {
      // aa = (lo + hi)/2, bb = (hi - lo)/4
      double2 wlo = csub(cscale(aabar, 0.5), cscale(bbbar, 0.25)), whi = cadd(cscale(aabar, 0.5), cscale(bbbar, 0.25));
      eig_grad(m, a, b, lo, wlo, abar, bbar, v, t, wd, we);
      eig_grad(m, a, b, hi, whi, abar, bbar, v, t, wd, we);
    }
  }
  return G;
}

// kernels of cf.cu
void cf_eval(cudaStream_t s, const double2* a, const double2* b, const int* m, int ld, int nchain, const double2* z, int nz, int tail,
             double2* g, double2* edges, int* nfall);
__global__ void k_real_tail(const double* a, const double* b, const int* n, int ld, int method, double* ainf, double* binf);
__global__ void k_real_green(const double* a, const double* b, const int* n, int ld, int nchain, const double* ainf,
                             const double* binf, int method, const double2* z, int nz, double2* g);

}  // namespace asrb
