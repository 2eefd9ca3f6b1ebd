#pragma once
#include "common.cuh"

namespace asrb {

constexpr int RW = 12;   // padded row of a shared-memory block (16-byte aligned pairs for FP64 and FP32)

// FP32 block products of the chain step and of the KPM step, for one 2-component value (a complex lane, or two random vectors)
// per thread: acc_l += sum_lp B[l][lp] x[lp] over the nine rows of one shared-memory block, the
// nine products of a row added in the order lp = 0 .. 8 (the FP64 kernel's products: dmma.cuh).  Rows 2p and 2p + 1 (p < 4)
// interleaved as {B[2p][lp], B[2p+1][lp]} pairs (18 floats, padded to 20), then row 8 alone (padded to 12); one paired
// FMA (__ffma2_rn, each half rounded as a scalar FMA) updates one component of two rows, so the bits are those of the
// scalar products with half their FMA instructions and no more shared-memory bytes.
template <typename ST> struct BlockAcc;
template <> struct BlockAcc<float> {
  static constexpr int BLK = 4 * 20 + 12;
  __device__ static void put(float* blk, int l, int lp, double v) {
    if (l < 8) blk[(l >> 1) * 20 + 2 * lp + (l & 1)] = (float)v;
    else blk[80 + lp] = (float)v;
  }
  float2 ax[4], ay[4], a8;   // {row 2p, row 2p + 1} of the real and of the imaginary parts; row 8
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int p = 0; p < 4; ++p) { ax[p] = make_float2(0.f, 0.f); ay[p] = ax[p]; }
    a8 = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void mac(const float* __restrict__ blk, const float2* x) {
#pragma unroll
    for (int lp = 0; lp < 8; lp += 2) {
      const float2 x0 = make_float2(x[lp].x, x[lp].x), y0 = make_float2(x[lp].y, x[lp].y);
      const float2 x1 = make_float2(x[lp + 1].x, x[lp + 1].x), y1 = make_float2(x[lp + 1].y, x[lp + 1].y);
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float4 bb = *(const float4*)(blk + p * 20 + 2 * lp);
        ax[p] = __ffma2_rn(make_float2(bb.x, bb.y), x0, ax[p]);
        ay[p] = __ffma2_rn(make_float2(bb.x, bb.y), y0, ay[p]);
        ax[p] = __ffma2_rn(make_float2(bb.z, bb.w), x1, ax[p]);
        ay[p] = __ffma2_rn(make_float2(bb.z, bb.w), y1, ay[p]);
      }
    }
    {
      const float2 x8 = make_float2(x[8].x, x[8].x), y8 = make_float2(x[8].y, x[8].y);
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float2 bb = *(const float2*)(blk + p * 20 + 16);
        ax[p] = __ffma2_rn(bb, x8, ax[p]);
        ay[p] = __ffma2_rn(bb, y8, ay[p]);
      }
    }
    const float* r8 = blk + 80;
#pragma unroll
    for (int lp = 0; lp < 8; lp += 2) {
      const float2 bb = *(const float2*)(r8 + lp);
      a8.x = fmaf(bb.x, x[lp].x, a8.x);
      a8.y = fmaf(bb.x, x[lp].y, a8.y);
      a8.x = fmaf(bb.y, x[lp + 1].x, a8.x);
      a8.y = fmaf(bb.y, x[lp + 1].y, a8.y);
    }
    a8.x = fmaf(r8[8], x[8].x, a8.x);
    a8.y = fmaf(r8[8], x[8].y, a8.y);
  }
  __device__ __forceinline__ void out(float2* acc) const {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      acc[2 * p] = make_float2(ax[p].x, ay[p].x);
      acc[2 * p + 1] = make_float2(ax[p].y, ay[p].y);
    }
    acc[8] = a8;
  }
};


}  // namespace asrb
