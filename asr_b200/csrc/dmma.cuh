// FP64 tensor-core products of the 9 x 9 bond blocks (mma.sync m16n8k4, f64), shared by the chain step and the
// KPM step, and the vector layout that feeds them.
//
// A warp multiplies one node by the blocks of its neighbours for 8 NJ "rows": lanes of a chain tile, or pairs of random
// vectors.  Thread t holds row n = t / 4 of each octet j < NJ and column c = t % 4 of the contraction:
//   A (16 x 4): the two components (re, im) of a row are the matrix rows n and n + 8, so one 16-byte load of the vector is
//               the thread's whole fragment;
//   B (4 x 8):  entry (k = c, column n) of the transposed block, read from shared memory;
//   C (16 x 8): the rows' outputs l = 2 c and 2 c + 1.
// The four columns of a step are the source orbitals 0-3, then 4-7 of one neighbour; orbital 8 of four neighbours is one
// more step, so nothing is padded but the last group of four.  The group operation of a link (orbital permutation
// and signs) sits in the B fragment: the source orbitals are read in storage order and the block row pi^-1(p) with the sign
// of p is taken instead.  The ninth output (l = 8) does not fit the 8-wide tile: it is one FP64 FMA per component and
// source orbital, summed over the four columns at the end (1/9 of the work; padding N to 16 would double it).
// Measured rate of the instruction on a B200 (register operands): 37.1 TFLOP/s, the FP64 peak, against 28 TFLOP/s of a
// stream of plain FP64 FMAs; 34.4 TFLOP/s for the 8 + 1 mix.
//
// Layout.  A node's 9 x 32 values are stored as two quads of orbitals, [quad][lane][4 orbitals], then orbital 8, [lane].
// The fragment load of a quad then reads 128 contiguous bytes per eight threads (4 L1 wavefronts per 512-byte load);
// orbital-major rows would put the four columns of every eight threads on four lines (16 wavefronts: the L1 data pipe 91 %
// busy, 3.9 ms per launch of the fcc ternary workload; the first form in this layout took 2.6).
#pragma once
#include "common.cuh"

namespace asrb {

constexpr int MB_ROW = 12;           // doubles per block row in shared memory: 8 + 1 outputs, 3 pads (rows 4 k banks apart)
constexpr int MB = 9 * MB_ROW;       // doubles per block
constexpr int MNODE = 9 * 32;        // elements of a node (32 lanes, or 32 pairs of vectors)

// element of (orbital l, lane) within a node
__host__ __device__ __forceinline__ int mnode_at(int l, int lane) { return l < 8 ? (l >> 2) * 128 + lane * 4 + (l & 3) : 256 + lane; }

__device__ __forceinline__ void dmma_16x8x4(double (&c)[4], double a0, double a1, double b) {
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b));
}
// Complex arithmetic with every rounding written out (explicit FMAs and uncontractible products): a lane gets the same bits
// from every instantiation that computes it, whatever the compiler would contract there.
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -__dmul_rn(a.y, b.y)), fma(a.x, b.y, __dmul_rn(a.y, b.x)));
}
__device__ __forceinline__ double2 zfma(double2 a, double2 b, double2 c) {   // a b + c
  return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)); }
__device__ __forceinline__ double2 zscale(double2 a, double s) { return make_double2(__dmul_rn(a.x, s), __dmul_rn(a.y, s)); }
__device__ __forceinline__ double2 zneg(double2 a) { return make_double2(-a.x, -a.y); }

// the sign bit of x flipped where bit 31 of m is set
__device__ __forceinline__ double xor_sign(double x, unsigned m) {
  return __hiloint2double(__double2hiint(x) ^ (int)(m & 0x80000000u), __double2loint(x));
}

__device__ __forceinline__ double2 shfl_xor2(double2 v, int m) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}

// Sum of v[j] over the four threads of a quad, left with the thread whose column c = t % 4 equals j (NJ = 2: threads j and
// j + 2; NJ = 1: all four).  The same order for every NJ.
template <int NJ>
__device__ __forceinline__ double2 quad_own(const double2 (&v)[NJ], int c) {
  if constexpr (NJ == 4) {
    double2 r[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double2 mine = (c & 1) ? v[2 * h + 1] : v[2 * h], other = (c & 1) ? v[2 * h] : v[2 * h + 1];
      r[h] = zadd(mine, shfl_xor2(other, 1));
    }
    const double2 mine = (c & 2) ? r[1] : r[0], other = (c & 2) ? r[0] : r[1];
    return zadd(mine, shfl_xor2(other, 2));
  } else if constexpr (NJ == 2) {
    const double2 mine = (c & 1) ? v[1] : v[0], other = (c & 1) ? v[0] : v[1];
    const double2 r = zadd(mine, shfl_xor2(other, 1));
    return zadd(r, shfl_xor2(r, 2));
  } else {
    const double2 r = zadd(v[0], shfl_xor2(v[0], 1));
    return zadd(r, shfl_xor2(r, 2));
  }
}

// two adjacent elements (32 bytes)
__device__ __forceinline__ void ldg2(const double2* p, double2& a, double2& b) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y) : "l"(p));
}
__device__ __forceinline__ void ldg2_cs(const double2* p, double2& a, double2& b) {   // read once
  asm volatile("ld.global.cs.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y) : "l"(p));
}
__device__ __forceinline__ void stg2(double2* p, double2 a, double2 b) {
  asm volatile("st.global.v4.f64 [%4], {%0, %1, %2, %3};" ::"d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y), "l"(p) : "memory");
}
__device__ __forceinline__ void stg2_cs(double2* p, double2 a, double2 b) {
  asm volatile("st.global.cs.v4.f64 [%4], {%0, %1, %2, %3};" ::"d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y), "l"(p) : "memory");
}

// word of source orbital p under an operation: its block row l (pi(l) = p) as a byte offset, the sign in bit 31
__host__ __device__ __forceinline__ uint32_t op_word(int l, uint32_t sign) { return (uint32_t)(l * MB_ROW * 8) | sign << 31; }

// Accumulators of one node: c[j] the outputs l = 2 c, 2 c + 1 of row n of octet j as {re, re, im, im}; c8[j] the thread's
// column of the output l = 8.
template <int NJ>
struct NodeAcc {
  double c[NJ][4];
  double2 c8[NJ];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.0;
      c8[j] = make_double2(0.0, 0.0);
    }
  }
  __device__ __forceinline__ double2 out(int j, int e) const { return make_double2(c[j][e], c[j][2 + e]); }
  // one step of depth 4: x the thread's elements (row n of octet j, column c), B the block (byte address), wd the operation
  // word of the column's source orbital
  __device__ __forceinline__ void step(const double2 (&x)[NJ], const char* B, int n, uint32_t wd) {
    const double* Br = (const double*)(B + (wd & 0x7fffffffu));
    const double b = xor_sign(Br[n], wd), q = xor_sign(Br[8], wd);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      dmma_16x8x4(c[j], x[j].x, x[j].y, b);
      c8[j].x = fma(q, x[j].x, c8[j].x);
      c8[j].y = fma(q, x[j].y, c8[j].y);
    }
  }
  // The products of a node over its list of cnt neighbours {node, block | operation << 16}.  in: element 0 of node 0, off(j)
  // the octet j, Bs the blocks, opw the operation words, zero the block of zeros.  The loads run one step ahead of the
  // products.
  template <typename Off>
  __device__ __forceinline__ void run(const int2* list, int cnt, const double2* __restrict__ in, Off off, const char* Bs,
                                      const uint32_t* opw, int zero, int t) {
    const int cc = t & 3, n = t >> 2;
    auto load = [&](double2 (&v)[NJ], const double2* p, int step) {
#pragma unroll
      for (int j = 0; j < NJ; ++j) v[j] = p[step * off(j)];
    };
    double2 x[NJ], y[NJ];
    int2 e = list[0];
    const double2* src = in + (size_t)e.x * MNODE + 4 * n + cc;
    load(x, src, 32);
    for (int k = 0; k < cnt; ++k) {   // source orbitals 0-3 (x) and 4-7 (y) of every neighbour
      load(y, src + 128, 32);
      const char* B = Bs + (e.y & 0xffff) * (MB * 8);
      const uint32_t* wd = opw + (e.y >> 16) * 9 + cc;
      const uint32_t w0 = wd[0], w1 = wd[4];
      e = list[min(k + 1, cnt - 1)];
      src = in + (size_t)e.x * MNODE + 4 * n + cc;
      step(x, B, n, w0);
      if (k + 1 < cnt) load(x, src, 32);
      step(y, B, n, w1);
    }
    // source orbital 8, four neighbours a step; a pad column multiplies the first entry's row by the block of zeros
    auto entry = [&](int g) { return list[g + cc < cnt ? g + cc : 0]; };
    e = entry(0);
    load(x, in + (size_t)e.x * MNODE + 256 + n, 8);
    for (int g = 0; g < cnt; g += 4) {
      const int blk = g + cc < cnt ? e.y & 0xffff : zero, o = e.y >> 16;
      if (g + 4 < cnt) {
        e = entry(g + 4);
        load(y, in + (size_t)e.x * MNODE + 256 + n, 8);
      }
      step(x, Bs + blk * (MB * 8), n, opw[o * 9 + 8]);
#pragma unroll
      for (int j = 0; j < NJ; ++j) x[j] = y[j];
    }
  }
};

}  // namespace asrb
