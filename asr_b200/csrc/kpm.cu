// Kernel polynomial method on an explicit supercell: kpm_moments / kpm_dos (src/reference/asr_kpm.f90:39-87) on the
// realisation operator lmto_real_op (src/reference/asr_lmto_realization.f90:120-191), generalised to n species.
//
// Layout: the nvec random vectors are the innermost index, x[(site * 9 + l) * V + v] with V = 64, so that each orbital
// load of a site is coalesced; the FP64 step of the scaled recurrence (k_cheb_d) keeps pairs of vectors in the order of the
// tensor-core fragments instead (dmma.cuh, cheb_at()).  The bond blocks sit in shared memory; d and c per species are tiny
// tables there too.  One Chebyshev step is one kernel:
//     t_{n+1} = 2 (H t_n - cen t_n) / sc - t_{n-1}   (n = 0: t_1 = (H t_0 - cen t_0) / sc),  H = e + c + d S d  (o = 0)
// with the FP64 partial dots r . t_{n+1}, t_{n+1} . t_{n+1} and t_{n+1} . t_n per vector.  The Rademacher vectors r are
// regenerated from a counter-based hash (splitmix64) instead of being read.  Two moment sets come out of one matvec
// with the Chebyshev doubling identities mu_2n = 2 <t_n|t_n> - mu_0, mu_2n+1 = 2 <t_n+1|t_n> - mu_1 (H symmetric), or
// one moment per matvec as the reference does (mu_n = <r|t_n>).
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "dmma.cuh"
#include "ffma2.cuh"
#include "op.h"

struct asr_supercell {
  asr_ctx* ctx = nullptr;
  int n = 0, ns = 0, nsp = 0;
  bool o_zero = true, e_zero = true;
  int* d_nbr = nullptr;          // (ns, n) 0-based
  uint8_t* d_spc = nullptr;      // (n) 0-based species
  double* d_par = nullptr;       // c, d, o, e: 4 x (9, nsp)
  std::vector<double> par_h;     // host copy of the same
  double* d_blocks = nullptr;    // [1 + ns][l][l']
  float* d_blocks_f = nullptr;
};

namespace asrb {
namespace {

constexpr int KV = 64;           // vectors per site row
constexpr int KSITES = 4;        // sites per 256-thread block row

__host__ __device__ inline uint64_t splitmix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ULL;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
  return x ^ (x >> 31);
}
// Rademacher entry q of vector v: +1 if bit 63 of splitmix64(seed * phi + (v << 40) + q) is clear
__device__ __forceinline__ double rademacher(uint64_t seed, uint64_t v, uint64_t q) {
  return (splitmix64(seed * 0x9E3779B97F4A7C15ULL + (v << 40) + q) >> 63) ? -1.0 : 1.0;
}

template <typename ST> __device__ __forceinline__ ST fma_t(ST a, ST b, ST c);
template <> __device__ __forceinline__ double fma_t<double>(double a, double b, double c) { return fma(a, b, c); }
template <> __device__ __forceinline__ float fma_t<float>(float a, float b, float c) { return fmaf(a, b, c); }

struct ScView {
  int n, ns, nsp;
  const int* nbr;
  const uint8_t* spc;
  const double* par;   // c | d | o | e, each (9, nsp)
};

// y = h x = c x + d S (d x) for one (site, vector): acc over the on-site and ns bond blocks
template <typename ST>
__device__ __forceinline__ void h_site(const ScView& S, const ST* Bs, const double* ps, const ST* x, int i, int v, double* y) {
  ST acc[9];
  for (int l = 0; l < 9; ++l) acc[l] = (ST)0;
  int si = S.spc[i];
  {
    ST u[9];
    for (int l = 0; l < 9; ++l) u[l] = (ST)ps[9 * S.nsp + l + 9 * si] * x[((size_t)i * 9 + l) * KV + v];
    for (int l = 0; l < 9; ++l)
      for (int lp = 0; lp < 9; ++lp) acc[l] = fma_t<ST>(Bs[l * 9 + lp], u[lp], acc[l]);
  }
  for (int k = 0; k < S.ns; ++k) {
    int j = S.nbr[k + (size_t)S.ns * i];
    int sj = S.spc[j];
    const ST* Bk = Bs + (size_t)(k + 1) * 81;
    ST u[9];
    for (int l = 0; l < 9; ++l) u[l] = (ST)ps[9 * S.nsp + l + 9 * sj] * x[((size_t)j * 9 + l) * KV + v];
    for (int l = 0; l < 9; ++l)
      for (int lp = 0; lp < 9; ++lp) acc[l] = fma_t<ST>(Bk[l * 9 + lp], u[lp], acc[l]);
  }
  for (int l = 0; l < 9; ++l)
    y[l] = ps[l + 9 * si] * (double)x[((size_t)i * 9 + l) * KV + v] + ps[9 * S.nsp + l + 9 * si] * (double)acc[l];
}

// smem: blocks [(1 + ns) * 81] (ST), then parameters 4 * 9 * nsp (double)
template <typename ST>
__device__ __forceinline__ void load_smem(const ScView& S, const ST* blocks, ST*& Bs, double*& ps) {
  extern __shared__ unsigned char sm_raw[];
  ps = (double*)sm_raw;
  Bs = (ST*)(ps + 4 * 9 * S.nsp);
  for (int q = threadIdx.x; q < 4 * 9 * S.nsp; q += blockDim.x) ps[q] = S.par[q];
  for (int q = threadIdx.x; q < (S.ns + 1) * 81; q += blockDim.x) Bs[q] = blocks[q];
  __syncthreads();
}

// one Chebyshev step, o = 0: t_new = 2 (H t - cen t)/sc - t_old (first: (H t - cen t)/sc); partial dots per vector:
// part[blk][v] = (r . t_new, t_new . t_new, t_new . t)
template <typename ST>
__global__ void __launch_bounds__(KSITES * KV) k_cheb(ScView S, const ST* __restrict__ blocks, const ST* __restrict__ t,
                                                      const ST* __restrict__ told, ST* __restrict__ tnew, double cen, double isc,
                                                      bool first, bool has_e, uint64_t seed, int v0, double* part) {
  ST* Bs;
  double* ps;
  load_smem<ST>(S, blocks, Bs, ps);
  const int v = threadIdx.x % KV, row = threadIdx.x / KV;
  double rt = 0.0, tt = 0.0, tp = 0.0;
  for (int i = blockIdx.x * KSITES + row; i < S.n; i += gridDim.x * KSITES) {
    double y[9];
    h_site<ST>(S, Bs, ps, t, i, v, y);
    int si = S.spc[i];
    for (int l = 0; l < 9; ++l) {
      size_t q = ((size_t)i * 9 + l) * KV + v;
      double tl = (double)t[q];
      double hy = y[l] + (has_e ? ps[27 * S.nsp + l + 9 * si] * tl : 0.0);
      double tn = first ? (hy - cen * tl) * isc : 2.0 * (hy - cen * tl) * isc - (double)told[q];
      ST ts = (ST)tn;
      tnew[q] = ts;
      double tr = (double)ts;
      rt += rademacher(seed, (uint64_t)(v0 + v), (uint64_t)i * 9 + l) * tr;
      tt += tr * tr;
      tp += tr * tl;
    }
  }
  __shared__ double red[KSITES][KV][3];
  red[row][v][0] = rt; red[row][v][1] = tt; red[row][v][2] = tp;
  __syncthreads();
  if (row == 0) {
    for (int r = 1; r < KSITES; ++r) { rt += red[r][v][0]; tt += red[r][v][1]; tp += red[r][v][2]; }
    double* out = part + ((size_t)blockIdx.x * KV + v) * 3;
    out[0] = rt; out[1] = tt; out[2] = tp;
  }
}

// Chebyshev step for o = 0 on d-scaled vectors u = d o t (per site and orbital, d of the site's species): with
// h t = c t + d S (d t), the recurrence t' = 2 (H t - cen t) / sc - t_old becomes
//   u' = 2 ((c + e - cen) o u + d^2 o S u) / sc - u_old,
// so the gathered neighbour rows need neither their species nor a scaling.  Partial dots of t (weights 1/d^2, 1/d):
// part[blk][v] = (r . t', t' . t', t' . t).  Both kernels take two vectors as one 2-component value, one site per warp:
// FP32 (k_cheb_f) the orbital-major rows and paired FMAs of ffma2.cuh, FP64 (k_cheb_d) the layout and tensor-core products
// of dmma.cuh.
struct UCoef {   // tables per (orbital, species), 9 nsp each: c + e - cen | d^2 | 1 / d^2 | 1 / d
  const double* p;
  int np;
};
constexpr int KW = 8;            // warps (sites) per block
constexpr int KP = KV / 2;       // vector pairs of a site

// u' of one (orbital, pair) from the S application's acc, and its shares of the dots
template <bool WANT_R>
struct ChebOut {
  double2 rt, tt, tp;
  __device__ __forceinline__ void zero() { rt = tt = tp = make_double2(0.0, 0.0); }
  template <typename T2, typename A2>
  __device__ __forceinline__ T2 step(const double* cs, int np, int q, T2 uo, A2 acc, double2 uold, double isc, bool first, uint64_t seed,
                                     uint64_t v, uint64_t row) {
    const double yx = cs[q] * (double)uo.x + cs[np + q] * (double)acc.x, yy = cs[q] * (double)uo.y + cs[np + q] * (double)acc.y;
    T2 us;
    us.x = first ? yx * isc : 2.0 * yx * isc - uold.x;
    us.y = first ? yy * isc : 2.0 * yy * isc - uold.y;
    const double ux = (double)us.x, uy = (double)us.y, w2 = cs[2 * np + q];
    tt.x += w2 * ux * ux;
    tt.y += w2 * uy * uy;
    tp.x += w2 * ux * (double)uo.x;
    tp.y += w2 * uy * (double)uo.y;
    if (WANT_R) {
      rt.x += rademacher(seed, v, row) * ux * cs[3 * np + q];
      rt.y += rademacher(seed, v + 1, row) * uy * cs[3 * np + q];
    }
    return us;
  }
};
// the block's sums of the pairs' dots (pair < 0: none) into part, in a fixed order
__device__ __forceinline__ void cheb_reduce(double2 rt, double2 tt, double2 tp, int pair, double* part) {
  __shared__ double2 red[KW][KP][3];
  const int w = threadIdx.x / 32, t = threadIdx.x % 32;
  for (int k = 0; k < 3; ++k) red[w][t][k] = make_double2(0.0, 0.0);
  __syncwarp();
  if (pair >= 0) { red[w][pair][0] = rt; red[w][pair][1] = tt; red[w][pair][2] = tp; }
  __syncthreads();
  if (threadIdx.x < 3 * KP) {
    const int v = threadIdx.x / 3, k = threadIdx.x % 3;
    double2 s = red[0][v][k];
    for (int q = 1; q < KW; ++q) s = cadd(s, red[q][v][k]);
    double* out = part + ((size_t)blockIdx.x * KV + 2 * v) * 3 + k;
    out[0] = s.x;
    out[3] = s.y;
  }
}

// FP32: thread = pair.  The neighbour indices of a site are read once, one per thread.  Per output the FMAs run over the
// on-site block, then the slots, nine source orbitals each; the rows of the next slot are in flight while a slot is
// multiplied.  Bound by the shared-memory block reads (25 broadcasts per slot and site; L1 data pipe 73 %, FMA pipe 46 %,
// issue 0.51 a cycle) and the gathers' latency.  256,000 sites x 64 vectors: 1.73 ms per step (29 TFLOP/s) at two blocks per SM; 2.11 ms without the prefetch, 1.90 / 2.24 ms at three
// blocks (80 registers) without / with it; one vector per thread and scalar FMAs 2.49 ms.
template <bool WANT_R>
__global__ void __launch_bounds__(KW * 32, 2) k_cheb_f(ScView S, const float* __restrict__ blocks, const double* __restrict__ coef,
                                                    const float2* __restrict__ u, const float2* __restrict__ uold,
                                                    float2* __restrict__ unew, double isc, bool first, uint64_t seed, int v0,
                                                    double* part) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const int np = 9 * S.nsp;
  double* cs = (double*)sm_raw;
  float* Bs = (float*)(cs + 4 * np);   // (9 nsp doubles four times: a multiple of 16 bytes)
  for (int q = threadIdx.x; q < 4 * np; q += blockDim.x) cs[q] = coef[q];
  for (int q = threadIdx.x; q < (S.ns + 1) * 81; q += blockDim.x)
    BlockAcc<float>::put(Bs + (q / 81) * BlockAcc<float>::BLK, (q / 9) % 9, q % 9, (double)blocks[q]);
  __syncthreads();
  const int t = threadIdx.x % 32, w = threadIdx.x / 32;
  ChebOut<WANT_R> D;
  D.zero();
  for (int i = blockIdx.x * KW + w; i < S.n; i += gridDim.x * KW) {
    BlockAcc<float> A;
    A.zero();
    const float2* ui = u + (size_t)i * MNODE + t;
    const int nb = t < S.ns ? S.nbr[t + (size_t)S.ns * i] : 0;
    float2 x[9];
#pragma unroll
    for (int l = 0; l < 9; ++l) x[l] = ui[l * KP];
    A.mac(Bs, x);
    float2 y[9];
    auto fetch = [&](int k, float2 (&v)[9]) {
      const int j = k < 32 ? __shfl_sync(0xffffffffu, nb, k) : S.nbr[k + (size_t)S.ns * i];
      const float2* src = u + (size_t)j * MNODE + t;
#pragma unroll
      for (int l = 0; l < 9; ++l) v[l] = src[l * KP];
    };
    if (S.ns) fetch(0, x);
#pragma unroll 1
    for (int k = 0; k < S.ns; k += 2) {
      if (k + 1 < S.ns) fetch(k + 1, y);
      A.mac(Bs + (k + 1) * BlockAcc<float>::BLK, x);
      if (k + 1 < S.ns) {
        if (k + 2 < S.ns) fetch(k + 2, x);
        A.mac(Bs + (k + 2) * BlockAcc<float>::BLK, y);
      }
    }
    float2 acc[9];
    A.out(acc);
    const int si = S.spc[i];
#pragma unroll
    for (int l = 0; l < 9; ++l) {
      const float2 uo = ui[l * KP];
      float2 ol = make_float2(0.f, 0.f);
      if (!first) ol = uold[(size_t)i * MNODE + l * KP + t];
      unew[(size_t)i * MNODE + l * KP + t] = D.step(cs, np, l + 9 * si, uo, acc[l], make_double2(ol.x, ol.y), isc, first, seed,
                                                    (uint64_t)(v0 + 2 * t), (uint64_t)i * 9 + l);
    }
  }
  cheb_reduce(D.rt, D.tt, D.tp, t, part);
}

// FP64: NJ octets of pairs (16 vectors each).  Bound by the FP64 tensor pipe (60 % of its cycles, and the largest stall) and the
// gathers' latency, as the chain step.  48,668 sites x 64 vectors: 0.41 ms per step (23.4 TFLOP/s); plain FP64 FMAs, one vector per thread, 1.31 ms.
template <bool WANT_R, int NJ>
__global__ void __launch_bounds__(KW * 32, 2) k_cheb_d(ScView S, const double* __restrict__ blocks, const double* __restrict__ coef,
                                                       const double2* __restrict__ u, const double2* __restrict__ uold,
                                                       double2* __restrict__ unew, double isc, bool first, uint64_t seed, int v0,
                                                       double* part) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const int np = 9 * S.nsp, ns1 = S.ns + 1, ldl = (ns1 + 3) & ~3;
  double* cs = (double*)sm_raw;
  double* Bs = cs + 4 * np;                                   // [1 + ns][l'][MB_ROW], then zeros
  uint32_t* opw = (uint32_t*)(Bs + (ns1 + 1) * MB);           // the identity
  int2* links = (int2*)(opw + 12) + (threadIdx.x / 32) * ldl;
  for (int q = threadIdx.x; q < 4 * np; q += blockDim.x) cs[q] = coef[q];
  for (int q = threadIdx.x; q < ns1 * 81; q += blockDim.x) Bs[(q / 81) * MB + (q % 9) * MB_ROW + (q / 9) % 9] = blocks[q];
  for (int q = threadIdx.x; q < MB; q += blockDim.x) Bs[ns1 * MB + q] = 0.0;
  if (threadIdx.x < 9) opw[threadIdx.x] = op_word(threadIdx.x, 0u);
  __syncthreads();
  const int t = threadIdx.x % 32, w = threadIdx.x / 32, c = t & 3, n = t >> 2;
  auto off = [](int j) { return j; };
  ChebOut<WANT_R> D;   // of the pair this thread owns: row n of octet c (c < NJ)
  D.zero();
  for (int i = blockIdx.x * KW + w; i < S.n; i += gridDim.x * KW) {
    __syncwarp();
    for (int k = t; k < ns1; k += 32) links[k] = make_int2(k ? S.nbr[k - 1 + (size_t)S.ns * i] : i, k);
    __syncwarp();
    const int si = S.spc[i];
    NodeAcc<NJ> A;
    A.zero();
    A.run(links, ns1, u, off, (const char*)Bs, opw, ns1, t);
    const double2 a8 = quad_own<NJ>(A.c8, c);
    const size_t q = (size_t)i * MNODE;
    double2 rt[NJ], tt[NJ], tp[NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int pair = n + 8 * j;
      const size_t at = q + mnode_at(2 * c, pair);
      double2 uo[2], ol[2], un[2];
      ldg2(u + at, uo[0], uo[1]);
      ol[0] = ol[1] = make_double2(0.0, 0.0);
      if (!first) ldg2_cs(uold + at, ol[0], ol[1]);
      ChebOut<WANT_R> P;
      P.zero();
#pragma unroll
      for (int e = 0; e < 2; ++e)
        un[e] = P.step(cs, np, 2 * c + e + 9 * si, uo[e], A.out(j, e), ol[e], isc, first, seed, (uint64_t)(v0 + 2 * pair),
                       (uint64_t)i * 9 + 2 * c + e);
      stg2(unew + at, un[0], un[1]);
      rt[j] = P.rt; tt[j] = P.tt; tp[j] = P.tp;
    }
    const double2 otp = quad_own<NJ>(tp, c), ott = quad_own<NJ>(tt, c);
    D.tp = cadd(D.tp, otp);
    D.tt = cadd(D.tt, ott);
    if (WANT_R) D.rt = cadd(D.rt, quad_own<NJ>(rt, c));
    if (c < NJ) {
      const size_t at = q + 256 + n + 8 * c;
      double2 ol = make_double2(0.0, 0.0);
      if (!first) ol = __ldcs(uold + at);
      unew[at] = D.step(cs, np, 8 + 9 * si, u[at], a8, ol, isc, first, seed, (uint64_t)(v0 + 2 * (n + 8 * c)), (uint64_t)i * 9 + 8);
    }
  }
  cheb_reduce(D.rt, D.tt, D.tp, c < NJ ? n + 8 * c : -1, part);
}

// shared memory of the two kernels
size_t cheb_f_smem(int nsp, int ns) { return (size_t)36 * nsp * sizeof(double) + (size_t)(ns + 1) * BlockAcc<float>::BLK * sizeof(float); }
size_t cheb_d_smem(int nsp, int ns) {
  return (size_t)36 * nsp * sizeof(double) + (size_t)(ns + 2) * MB * sizeof(double) + 12 * sizeof(uint32_t) +
         (size_t)KW * ((ns + 4) & ~3) * sizeof(int2);
}

// element (site, orbital, vector) of the d-scaled vectors, as the kernels above keep them
template <typename ST>
__device__ __forceinline__ size_t cheb_at(size_t site, int l, int v) {
  return std::is_same<ST, double>::value ? 2 * (site * MNODE + mnode_at(l, v >> 1)) + (v & 1) : (site * 9 + l) * KV + v;
}

// u_0 = d o r (d of each site's species)
template <typename ST>
__global__ void k_rademacher_init_scaled(ScView S, uint64_t seed, int v0, ST* t) {
  size_t tot = (size_t)S.n * 9 * KV;
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += (size_t)gridDim.x * blockDim.x) {
    int v = (int)(q % KV);
    size_t e = q / KV;   // site * 9 + l
    int site = (int)(e / 9), l = (int)(e % 9);
    double d = S.par[9 * S.nsp + l + 9 * S.spc[site]];
    t[cheb_at<ST>(site, l, v)] = (ST)(d * rademacher(seed, (uint64_t)(v0 + v), (uint64_t)e));
  }
}

// general operator (o != 0): w = h x (stored, FP64 math, ST storage)
template <typename ST>
__global__ void __launch_bounds__(KSITES * KV) k_h(ScView S, const ST* __restrict__ blocks, const ST* __restrict__ x,
                                                   bool oscale, ST* __restrict__ w) {
  ST* Bs;
  double* ps;
  load_smem<ST>(S, blocks, Bs, ps);
  const int v = threadIdx.x % KV, row = threadIdx.x / KV;
  for (int i = blockIdx.x * KSITES + row; i < S.n; i += gridDim.x * KSITES) {
    double y[9];
    h_site<ST>(S, Bs, ps, x, i, v, y);
    int si = S.spc[i];
    for (int l = 0; l < 9; ++l) {
      double f = oscale ? ps[18 * S.nsp + l + 9 * si] : 1.0;   // o h x when requested
      w[((size_t)i * 9 + l) * KV + v] = (ST)(f * y[l]);
    }
  }
}

// general Chebyshev combination: y = e t + w1 - w3 (w1 = h t, w3 = h o h t)
template <typename ST>
__global__ void __launch_bounds__(KSITES * KV) k_cheb_comb(ScView S, const ST* __restrict__ t, const ST* __restrict__ w1,
                                                           const ST* __restrict__ w3, const ST* __restrict__ told,
                                                           ST* __restrict__ tnew, double cen, double isc, bool first,
                                                           uint64_t seed, int v0, double* part) {
  const int v = threadIdx.x % KV, row = threadIdx.x / KV;
  double rt = 0.0, tt = 0.0, tp = 0.0;
  for (int i = blockIdx.x * KSITES + row; i < S.n; i += gridDim.x * KSITES) {
    int si = S.spc[i];
    for (int l = 0; l < 9; ++l) {
      size_t q = ((size_t)i * 9 + l) * KV + v;
      double tl = (double)t[q];
      double hy = S.par[27 * S.nsp + l + 9 * si] * tl + (double)w1[q] - (double)w3[q];
      double tn = first ? (hy - cen * tl) * isc : 2.0 * (hy - cen * tl) * isc - (double)told[q];
      ST ts = (ST)tn;
      tnew[q] = ts;
      double tr = (double)ts;
      rt += rademacher(seed, (uint64_t)(v0 + v), (uint64_t)i * 9 + l) * tr;
      tt += tr * tr;
      tp += tr * tl;
    }
  }
  __shared__ double red[KSITES][KV][3];
  red[row][v][0] = rt; red[row][v][1] = tt; red[row][v][2] = tp;
  __syncthreads();
  if (row == 0) {
    for (int r = 1; r < KSITES; ++r) { rt += red[r][v][0]; tt += red[r][v][1]; tp += red[r][v][2]; }
    double* out = part + ((size_t)blockIdx.x * KV + v) * 3;
    out[0] = rt; out[1] = tt; out[2] = tp;
  }
}

template <typename ST>
__global__ void k_rademacher_init(int n, uint64_t seed, int v0, ST* t) {
  size_t tot = (size_t)n * 9 * KV;
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += (size_t)gridDim.x * blockDim.x) {
    int v = (int)(q % KV);
    size_t e = q / KV;   // site * 9 + l
    t[q] = (ST)rademacher(seed, (uint64_t)(v0 + v), (uint64_t)e);
  }
}

// sum of the block partials per vector in a fixed order: out[v][3].  32 of the 3 KV columns per block, the rows over its
// warps with eight loads in flight (one thread per vector over all rows in turn took 0.11 ms a step, 4-9 % of a run).
__global__ void k_kpm_reduce(const double* part, int nblk, double* out) {
  __shared__ double sm[8][32];
  const int t = threadIdx.x % 32, w = threadIdx.x / 32, col = blockIdx.x * 32 + t;
  const double* p = part + col;
  double s = 0.0;
  int q = w;
  for (; q + 56 < nblk; q += 64) {
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = p[(size_t)(q + 8 * j) * KV * 3];
#pragma unroll
    for (int j = 0; j < 8; ++j) s += v[j];
  }
  for (; q < nblk; q += 8) s += p[(size_t)q * KV * 3];
  sm[w][t] = s;
  __syncthreads();
  if (w == 0) {
    for (int j = 1; j < 8; ++j) s += sm[j][t];
    out[col] = s;
  }
}

template <typename T>
struct DevBuf {
  T* p = nullptr;
  DevMem mem;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { mem.put(); }
  int alloc(size_t n) {
    if (!mem.get(std::max<size_t>(n, 1) * sizeof(T))) {
      set_error("kpm: device allocation of %zu bytes failed", n * sizeof(T));
      return ASR_ENOMEM;
    }
    p = (T*)mem.p;
    return ASR_OK;
  }
};

// blocks of the scaled steps: as many as run at once (each prepares its tables once and takes every grid-th group of sites)
int cheb_grid(const asr_ctx* ctx) { return ctx->num_sms * 2; }

// one scaled step on nv <= KV vectors
void cheb_scaled(asr_ctx* ctx, const ScView& S, const float* blocks, const double* coef, const float* u, const float* uold, float* unew,
                 double isc, bool first, bool want_r, int, uint64_t seed, int v0, double* part, int grid) {
  auto k = want_r ? k_cheb_f<true> : k_cheb_f<false>;
  k<<<grid, KW * 32, cheb_f_smem(S.nsp, S.ns), ctx->stream>>>(S, blocks, coef, (const float2*)u, (const float2*)uold, (float2*)unew, isc,
                                                             first, seed, v0, part);
}
void cheb_scaled(asr_ctx* ctx, const ScView& S, const double* blocks, const double* coef, const double* u, const double* uold,
                 double* unew, double isc, bool first, bool want_r, int nv, uint64_t seed, int v0, double* part, int grid) {
  // octets of vector pairs in use: 16 vectors each; three run as four
  auto k = nv <= 16 ? (want_r ? k_cheb_d<true, 1> : k_cheb_d<false, 1>)
         : nv <= 32 ? (want_r ? k_cheb_d<true, 2> : k_cheb_d<false, 2>) : (want_r ? k_cheb_d<true, 4> : k_cheb_d<false, 4>);
  k<<<grid, KW * 32, cheb_d_smem(S.nsp, S.ns), ctx->stream>>>(S, blocks, coef, (const double2*)u, (const double2*)uold, (double2*)unew, isc,
                                                             first, seed, v0, part);
}

template <typename ST>
int kpm_run(asr_ctx* ctx, asr_supercell* sc, double cen, double scl, int nmom, int v0, int nvec, uint64_t seed, bool doubling,
            double* mu) {
  cudaStream_t s = ctx->stream;
  const int n = sc->n;
  ScView S{n, sc->ns, sc->nsp, sc->d_nbr, sc->d_spc, sc->d_par};
  const ST* blocks = std::is_same<ST, double>::value ? (const ST*)sc->d_blocks : (const ST*)sc->d_blocks_f;
  const size_t nel = (size_t)n * 9 * KV;
  const size_t smem = 4 * 9 * sc->nsp * sizeof(double) + (size_t)(sc->ns + 1) * 81 * sizeof(ST);
  const bool general = !sc->o_zero;
  const int grid = ctx->num_sms * 4;
  const size_t one = nel * sizeof(ST);
  ctx->mem->room((general ? 6 : 3) * one, general ? ctx->plan_bytes({one, one, one, one, one, one}) : ctx->plan_bytes({one, one, one}));
  DevBuf<ST> T0, T1, T2, W1, W2, W3;
  ASR_TRY(T0.alloc(nel)); ASR_TRY(T1.alloc(nel)); ASR_TRY(T2.alloc(nel));
  if (general) { ASR_TRY(W1.alloc(nel)); ASR_TRY(W2.alloc(nel)); ASR_TRY(W3.alloc(nel)); }
  DevBuf<double> part, red;
  ASR_TRY(part.alloc((size_t)grid * KV * 3));
  // all reduced dots of the run: (nsteps, KV, 3)
  const int nsteps = doubling ? std::max(1, (nmom + 1) / 2) : std::max(1, nmom - 1);
  ASR_TRY(red.alloc((size_t)nsteps * KV * 3));
  for (int m = 0; m < nmom; ++m) mu[m] = 0.0;
  const double isc = 1.0 / scl;
  const double dim = 9.0 * n;
  std::vector<double> hred((size_t)nsteps * KV * 3);
  // coefficients of the d-scaled recurrence (o = 0): c + e - cen, d^2, 1/d^2, 1/d per (orbital, species)
  DevBuf<double> ucoef;
  bool dpos = true;
  if (!general) {
    const int np = 9 * sc->nsp;
    std::vector<double> hc(4 * (size_t)np);
    for (int q = 0; q < np; ++q) {
      double c = sc->par_h[q], d = sc->par_h[np + q], e = sc->par_h[3 * np + q];
      if (d == 0.0) dpos = false;
      hc[q] = c + e - cen;
      hc[np + q] = d * d;
      hc[2 * np + q] = d != 0.0 ? 1.0 / (d * d) : 0.0;
      hc[3 * np + q] = d != 0.0 ? 1.0 / d : 0.0;
    }
    if (dpos) {
      ASR_TRY(ucoef.alloc(hc.size()));
      ASR_CUDA(cudaMemcpyAsync(ucoef.p, hc.data(), hc.size() * sizeof(double), cudaMemcpyHostToDevice, s));
    }
  }
  const bool scaled = !general && dpos;
  if (scaled) {   // the scaled steps' static sums come on top of up to 48 KB of tables
    if (std::is_same<ST, float>::value)
      for (auto k : {k_cheb_f<true>, k_cheb_f<false>}) ASR_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 48 * 1024));
    else
      for (auto k : {k_cheb_d<true, 1>, k_cheb_d<false, 1>, k_cheb_d<true, 2>, k_cheb_d<false, 2>, k_cheb_d<true, 4>, k_cheb_d<false, 4>})
        ASR_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 48 * 1024));
  }
  const int sgrid = std::min(cheb_grid(ctx), (n + KW - 1) / KW);
  for (int vb = 0; vb < nvec; vb += KV) {
    const int nv = std::min(KV, nvec - vb);
    if (scaled) k_rademacher_init_scaled<ST><<<ctx->num_sms * 8, 256, 0, s>>>(S, seed, v0 + vb, T0.p);
    else k_rademacher_init<ST><<<ctx->num_sms * 8, 256, 0, s>>>(n, seed, v0 + vb, T0.p);
    ST *ta = T0.p, *tb = T1.p, *tc = T2.p;   // t_{k-1}, t_k, t_{k+1}
    // step 0: t_1 = (H t_0 - cen t_0) / sc
    for (int k = 0; k < nsteps; ++k) {
      const ST* tin = (k == 0) ? ta : tb;
      const ST* told = (k == 0) ? nullptr : ta;
      ST* tout = (k == 0) ? tb : tc;
      const int ps = ctx->prof_start(s);
      if (scaled) {
        // <r|t> is needed for every step without doubling, and for mu_1 (step 0) with it
        cheb_scaled(ctx, S, blocks, ucoef.p, tin, told, tout, isc, k == 0, !doubling || k == 0, nv, seed, v0 + vb, part.p, sgrid);
      } else if (!general) {
        k_cheb<ST><<<grid, KSITES * KV, smem, s>>>(S, blocks, tin, told, tout, cen, isc, k == 0, !sc->e_zero, seed, v0 + vb, part.p);
      } else {
        k_h<ST><<<grid, KSITES * KV, smem, s>>>(S, blocks, tin, false, W1.p);
        k_h<ST><<<grid, KSITES * KV, smem, s>>>(S, blocks, tin, true, W2.p);    // o h t
        k_h<ST><<<grid, KSITES * KV, smem, s>>>(S, blocks, W2.p, false, W3.p);
        k_cheb_comb<ST><<<grid, KSITES * KV, 0, s>>>(S, tin, W1.p, W3.p, told, tout, cen, isc, k == 0, seed, v0 + vb, part.p);
      }
      {   // algorithmic work of one Chebyshev step: read t_k and t_{k-1}, write t_{k+1}, one species byte per site; flops
          // 2 x 81 x (1 + slots) per site and vector per S application (one for o = 0, three for the general operator)
        const double sapp = general ? 3.0 : 1.0;
        const double streams = general ? 9.0 : 3.0;
        ctx->prof_stop(s, ps, ASR_KERNEL_KPM, (double)n * (KV * streams * 9 * sizeof(ST) + 1.0),
                       sapp * (double)n * KV * 2.0 * 81.0 * (1 + sc->ns));
      }
      k_kpm_reduce<<<KV * 3 / 32, 256, 0, s>>>(part.p, scaled ? sgrid : grid, red.p + (size_t)k * KV * 3);
      if (k > 0) { ST* t_ = ta; ta = tb; tb = tc; tc = t_; }
    }
    ASR_CUDA(cudaGetLastError());
    ASR_CUDA(cudaMemcpyAsync(hred.data(), red.p, hred.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
    ASR_CUDA(cudaStreamSynchronize(s));
    // moments of the vectors of this block: step k produced t_{k+1}; dots (r.t_{k+1}, t_{k+1}.t_{k+1}, t_{k+1}.t_k)
    for (int v = 0; v < nv; ++v) {
      auto R = [&](int k, int c) { return hred[((size_t)k * KV + v) * 3 + c]; };
      double m0 = 1.0;   // <r|r> / dim for a Rademacher vector
      double m1 = R(0, 0) / dim;
      if (!doubling) {
        mu[0] += m0;
        if (nmom > 1) mu[1] += m1;
        for (int m = 2; m < nmom; ++m) mu[m] += R(m - 1, 0) / dim;
      } else {
        // t_0 . t_0 = dim, t_1 . t_0 = r . t_1
        mu[0] += m0;
        if (nmom > 1) mu[1] += m1;
        for (int m = 2; m < nmom; ++m) {
          int nh = m / 2;   // mu_2n = 2 t_n.t_n/dim - mu_0 ; mu_2n+1 = 2 t_n+1.t_n/dim - mu_1
          double val;
          if (m % 2 == 0) val = 2.0 * R(nh - 1, 1) / dim - m0;   // t_nh . t_nh is from step nh - 1
          else val = 2.0 * R(nh, 2) / dim - m1;                  // t_{nh+1} . t_nh from step nh
          mu[m] += val;
        }
      }
    }
  }
  for (int m = 0; m < nmom; ++m) mu[m] /= (double)nvec;
  return ASR_OK;
}

}  // namespace
}  // namespace asrb

using namespace asrb;

extern "C" {

int asr_supercell_build(asr_ctx* ctx, int nsite, int nslot, const int* nbr, const int* spc, int nsp, const double* c,
                        const double* d, const double* o, const double* e, const double* block, const double* block0,
                        asr_supercell** out) {
  if (!ctx || !out || !nbr || !spc || !c || !d || !block || nsite < 1 || nslot < 0 || nsp < 1 || nsp > 255) {
    set_error("asr_supercell_build: bad argument");
    return ASR_EINVAL;
  }
  *out = nullptr;
  for (size_t q = 0; q < (size_t)nslot * nsite; ++q)
    if (nbr[q] < 1 || nbr[q] > nsite) { set_error("asr_supercell_build: neighbour index out of range"); return ASR_EINVAL; }
  std::vector<uint8_t> sp(nsite);
  for (int i = 0; i < nsite; ++i) {
    if (spc[i] < 1 || spc[i] > nsp) { set_error("asr_supercell_build: species index out of range"); return ASR_EINVAL; }
    sp[i] = (uint8_t)(spc[i] - 1);
  }
  ASR_ON_DEVICE(ctx->device);
  asr_supercell* sc = new asr_supercell();
  sc->ctx = ctx; sc->n = nsite; sc->ns = nslot; sc->nsp = nsp;
  std::vector<int> nb((size_t)nslot * nsite);
  for (size_t q = 0; q < nb.size(); ++q) nb[q] = nbr[q] - 1;
  std::vector<double> par(4 * 9 * (size_t)nsp, 0.0);
  for (int q = 0; q < 9 * nsp; ++q) {
    par[q] = c[q];
    par[9 * nsp + q] = d[q];
    par[18 * nsp + q] = o ? o[q] : 0.0;
    par[27 * nsp + q] = e ? e[q] : 0.0;
    if (par[18 * nsp + q] != 0.0) sc->o_zero = false;
    if (par[27 * nsp + q] != 0.0) sc->e_zero = false;
  }
  std::vector<double> B((size_t)(nslot + 1) * 81, 0.0);
  for (int l = 0; l < 9; ++l)
    for (int lp = 0; lp < 9; ++lp) {
      if (block0) B[l * 9 + lp] = block0[l + 9 * lp];
      for (int k = 0; k < nslot; ++k) B[(size_t)(k + 1) * 81 + l * 9 + lp] = block[l + 9 * (lp + 9 * (size_t)k)];
    }
  std::vector<float> Bf(B.begin(), B.end());
  cudaStream_t s = ctx->stream;
  DevStore* st = ctx->mem;
  bool ok = dev_alloc(st, s, &sc->d_nbr, std::max<size_t>(nb.size(), 1) * sizeof(int)) && dev_alloc(st, s, &sc->d_spc, nsite) &&
            dev_alloc(st, s, &sc->d_par, par.size() * sizeof(double)) && dev_alloc(st, s, &sc->d_blocks, B.size() * sizeof(double)) &&
            dev_alloc(st, s, &sc->d_blocks_f, Bf.size() * sizeof(float));
  if (!ok) {
    asr_supercell_free(sc);
    set_error("asr_supercell_build: device allocation failed");
    return ASR_ENOMEM;
  }
  cudaMemcpyAsync(sc->d_nbr, nb.data(), nb.size() * sizeof(int), cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(sc->d_spc, sp.data(), nsite, cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(sc->d_par, par.data(), par.size() * sizeof(double), cudaMemcpyHostToDevice, s);
  sc->par_h = par;
  cudaMemcpyAsync(sc->d_blocks, B.data(), B.size() * sizeof(double), cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(sc->d_blocks_f, Bf.data(), Bf.size() * sizeof(float), cudaMemcpyHostToDevice, s);
  ASR_CUDA(cudaStreamSynchronize(s));
  *out = sc;
  return ASR_OK;
}

int asr_supercell_free(asr_supercell* sc) {
  if (!sc) return ASR_OK;
  DeviceGuard dg;
  dg.set(sc->ctx->device);
  cudaFree(sc->d_nbr); cudaFree(sc->d_spc); cudaFree(sc->d_par); cudaFree(sc->d_blocks); cudaFree(sc->d_blocks_f);
  delete sc;
  return ASR_OK;
}

int asr_supercell_apply(asr_supercell* sc, const double* x, double* y, int nvec) {
  if (!sc || !x || !y || nvec < 1) { set_error("asr_supercell_apply: bad argument"); return ASR_EINVAL; }
  asr_ctx* ctx = sc->ctx;
  ASR_ENTER(ctx);
  cudaStream_t s = ctx->stream;
  const int n = sc->n;
  const size_t nel = (size_t)n * 9 * KV;
  ScView S{n, sc->ns, sc->nsp, sc->d_nbr, sc->d_spc, sc->d_par};
  const size_t smem = 4 * 9 * sc->nsp * sizeof(double) + (size_t)(sc->ns + 1) * 81 * sizeof(double);
  const int grid = ctx->num_sms * 4;
  for (int vb = 0; vb < nvec; vb += KV) {
    int nv = std::min(KV, nvec - vb);
    std::vector<double> hx(nel, 0.0), hy(nel);
    for (int v = 0; v < nv; ++v)
      for (size_t q = 0; q < (size_t)n * 9; ++q) hx[q * KV + v] = x[(size_t)(vb + v) * n * 9 + q];
    DevBuf<double> X, W1, W2, W3;
    ASR_TRY(X.alloc(nel)); ASR_TRY(W1.alloc(nel)); ASR_TRY(W2.alloc(nel)); ASR_TRY(W3.alloc(nel));
    ASR_CUDA(cudaMemcpyAsync(X.p, hx.data(), nel * sizeof(double), cudaMemcpyHostToDevice, s));
    k_h<double><<<grid, KSITES * KV, smem, s>>>(S, sc->d_blocks, X.p, false, W1.p);
    k_h<double><<<grid, KSITES * KV, smem, s>>>(S, sc->d_blocks, X.p, true, W2.p);   // o h x
    k_h<double><<<grid, KSITES * KV, smem, s>>>(S, sc->d_blocks, W2.p, false, W3.p);
    ASR_CUDA(cudaGetLastError());
    std::vector<double> w1(nel), w3(nel);
    ASR_CUDA(cudaMemcpyAsync(w1.data(), W1.p, nel * sizeof(double), cudaMemcpyDeviceToHost, s));
    ASR_CUDA(cudaMemcpyAsync(w3.data(), W3.p, nel * sizeof(double), cudaMemcpyDeviceToHost, s));
    ASR_CUDA(cudaStreamSynchronize(s));
    // y = e x + h x - h o h x (real_apply, src/reference/asr_lmto_realization.f90:149-191)
    std::vector<double> par(4 * 9 * (size_t)sc->nsp);
    ASR_CUDA(cudaMemcpy(par.data(), sc->d_par, par.size() * sizeof(double), cudaMemcpyDeviceToHost));
    std::vector<uint8_t> sp(n);
    ASR_CUDA(cudaMemcpy(sp.data(), sc->d_spc, n, cudaMemcpyDeviceToHost));
    for (int v = 0; v < nv; ++v)
      for (int i = 0; i < n; ++i)
        for (int l = 0; l < 9; ++l) {
          size_t q = (size_t)i * 9 + l;
          double ev = par[27 * sc->nsp + l + 9 * sp[i]];
          y[(size_t)(vb + v) * n * 9 + q] = ev * x[(size_t)(vb + v) * n * 9 + q] + w1[q * KV + v] - w3[q * KV + v];
        }
  }
  return ASR_OK;
}

int asr_kpm_moments(asr_ctx* ctx, asr_supercell* sc, double cen, double scl, int nmom, int v0, int nvec, uint64_t seed,
                    int precision, int doubling, double* mu) {
  if (!ctx || !sc || !mu || nmom < 1 || nvec < 1 || !(scl > 0.0)) { set_error("kpm_moments: bad argument"); return ASR_EINVAL; }
  ASR_ENTER(ctx);
  if (precision == ASR_FP32) return kpm_run<float>(ctx, sc, cen, scl, nmom, v0, nvec, seed, doubling != 0, mu);
  return kpm_run<double>(ctx, sc, cen, scl, nmom, v0, nvec, seed, doubling != 0, mu);
}

// kpm_dos (src/reference/asr_kpm.f90:68-87): Jackson kernel, host
int asr_kpm_dos(const double* mu, int nmom, double cen, double scl, const double* e, int ne, double* rho) {
  if (!mu || !e || !rho || nmom < 1 || ne < 0 || !(scl > 0.0)) { set_error("kpm_dos: bad argument"); return ASR_EINVAL; }
  const double pi = 3.14159265358979323846;
  std::vector<double> g(nmom);
  for (int n = 0; n < nmom; ++n)
    g[n] = ((nmom - n + 1) * std::cos(pi * n / (nmom + 1)) + std::sin(pi * n / (nmom + 1)) / std::tan(pi / (nmom + 1))) / (nmom + 1);
  for (int i = 0; i < ne; ++i) {
    double x = (e[i] - cen) / scl;
    if (std::fabs(x) >= 1.0) { rho[i] = 0.0; continue; }
    double th = std::acos(x), s = g[0] * mu[0];
    for (int n = 1; n < nmom; ++n) s += 2.0 * g[n] * mu[n] * std::cos(n * th);
    rho[i] = s / (pi * std::sqrt(1.0 - x * x) * scl);
  }
  return ASR_OK;
}

}  // extern "C"
