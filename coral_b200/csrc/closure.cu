// Learned subgrid closure: a small stencil network that predicts, on a coarse
// grid, the subgrid part of every quadratic variable,
//   tau_q = P(q_fine) - q(P(fields_fine))        (P: truncation to the coarse modes),
// from the resolved full variables.  Inside the time step its outputs are added
// to the pointwise products before their forward transform, so they reach the
// explicit nonlinear term K_hat through the recipe's own NL operator (the
// divergence and quasi-inverse integration of the subgrid fluxes).  The
// reference has no learned closure; its nonlinear terms are the products of
// src/plane_layer/PL_IMEX_timestepping_marching.f90:279-352.
//
// Network (every grid point independently):
//   x  = 5 channels (u, v, w, T scaled by in_scale, and the wall-normal
//        coordinate z' in [-1, 1]) at the 27 points of the 3 x 3 x 3 stencil
//        (periodic in x and y, zero beyond the walls): 135 inputs
//   h1 = tanh(W0 x + b0)      64
//   h2 = tanh(W1 h1 + b1)     64
//   h3 = tanh(W2 h2 + b2)     64
//   y  = W3 h3 + b3           9 outputs, tau_q = out_scale[q] y_q
// Weights are used in BF16 (FP32 master copies for the optimiser), biases,
// activations and every accumulation in FP32.  Inference, training (forward,
// backward; loss = mean over points of sum_q (y_q - target_q / out_scale[q])^2)
// and Adam are the kernels below.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/coral_b200.h"
#include "device.hpp"
#include "host.hpp"

namespace coral {
namespace {

constexpr int kCin = 5, kTaps = 27, kIn = kCin * kTaps, kHid = 64, kOut = 9;
// flat parameter layout: W0 [kHid][kIn], b0, W1 [kHid][kHid], b1, W2 [kHid][kHid], b2, W3 [kOut][kHid], b3
constexpr int oW0 = 0, oB0 = oW0 + kHid * kIn, oW1 = oB0 + kHid, oB1 = oW1 + kHid * kHid, oW2 = oB1 + kHid,
              oB2 = oW2 + kHid * kHid, oW3 = oB2 + kHid, oB3 = oW3 + kOut * kHid, kNParam = oB3 + kOut;
constexpr int kGradBuckets = 4;  // copies of the gradient that the training CTAs add into

struct NetDev {
  const __nv_bfloat16* w16;  // kNParam (biases too, unused in BF16)
  const float* w32;          // master copies (the biases are read from here)
  float in_scale[4], out_scale[kOut];
};

// ------------------------------------------------------------------------------
// The network's products on the tensor cores, in FP32 precision: weights are
// BF16 as they are; an FP32 activation (or gradient) is the exact sum of three
// BF16 numbers, h = bf16(h) + bf16(rest) + bf16(rest), so h W is three BF16
// products with FP32 accumulation.  (Relative error of tau against FP64, rms, for
// inputs of 1 | 0.1 | 0.01 | 1e-5: 1.5e-7 | 1.8e-7 | 2.0e-7 | 1.9e-7; of scalar FP32
// sums in one chain 2.8e-7 | 3.3e-7 | 3.1e-7 | 3.1e-7.)
//
// A warp takes 16 points through all layers with its activations in registers: the
// accumulator layout of mma.m16n8k16 (rows = points, columns = features) is the
// A-operand layout of the next layer's k step.  Lane = 4 g + q holds rows g and g + 8
// and columns 2 q, 2 q + 1 of every 8-column tile.
// Legacy MMAs, not tcgen05: their accumulators stay in registers from layer to
// layer, and the tensor pipe is a third busy; the issue slots (48%: splitting,
// tanh, the stencil's addresses) and the instruction cache bound the kernel.  One
// thread per point with its activations in shared memory (4 warps per SM): 2606 us
// for 96 x 96 x 72 points; this kernel: 392 us at 3 CTAs per SM (4: 404, 5: 408).
//
// The order of layer 0's 135 inputs is free: k step ks < 7 gives lane column q
// channel q and taps 4 ks .. 4 ks + 3, the last two steps hold channel 4 (z').
// ------------------------------------------------------------------------------
constexpr int kK0 = 9;  // k steps of layer 0 (144 inputs, 9 of them zero)
__device__ __forceinline__ int input_of(int ks, int q, int slot) {  // column c * kTaps + tap, -1: none
  if (ks < 7) {
    const int tap = 4 * ks + slot;
    return tap < kTaps ? q * kTaps + tap : -1;
  }
  const int tap = 16 * (ks - 7) + 4 * q + slot;
  return tap < kTaps ? 4 * kTaps + tap : -1;
}

__device__ __forceinline__ void mma16816(float (&d)[4], const unsigned (&a)[4], uint2 b, const float (&c)[4]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
// two floats as one operand of the packed FP32 instructions
__device__ __forceinline__ unsigned long long pair2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpair2(unsigned long long p, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// c += a b, a in three planes: the step's products are summed from zero, smallest
// plane first, and added to c in one rounding (the tensor core's own additions
// truncate: with c as their accumulator the error against FP64 doubled)
__device__ __forceinline__ void mma_planes(float (&c)[4], const unsigned (&a)[3][4], uint2 b) {
  const float zero[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  float t2[4], t1[4], t0[4];
  mma16816(t2, a[2], b, zero);
  mma16816(t1, a[1], b, t2);
  mma16816(t0, a[0], b, t1);
#pragma unroll
  for (int e = 0; e < 4; e += 2) unpair2(add2(pair2(c[e], c[e + 1]), pair2(t0[e], t0[e + 1])), c[e], c[e + 1]);
}
__device__ __forceinline__ unsigned pack2(float lo, float hi) {
  unsigned r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// (a, b) as three packed BF16 pairs whose sum they are
__device__ __forceinline__ void split3(float a, float b, unsigned& p0, unsigned& p1, unsigned& p2) {
  p0 = pack2(a, b);
  a -= __uint_as_float(p0 << 16);
  b -= __uint_as_float(p0 & 0xffff0000u);
  p1 = pack2(a, b);
  a -= __uint_as_float(p1 << 16);
  b -= __uint_as_float(p1 & 0xffff0000u);
  p2 = pack2(a, b);
}
// the same for any value: the first plane is cut off, not rounded, so that finite
// values up to the largest FP32 stay finite (rounding takes those above 3.396e38 to
// infinity, and two of opposite sign to NaN); infinities have zero rests
__device__ __forceinline__ void split3_any(float a, float b, unsigned& p0, unsigned& p1, unsigned& p2) {
  p0 = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
  a -= __uint_as_float(p0 << 16);
  b -= __uint_as_float(p0 & 0xffff0000u);
  p1 = pack2(a, b);
  a -= __uint_as_float(p1 << 16);
  b -= __uint_as_float(p1 & 0xffff0000u);
  p2 = pack2(a, b);
  const unsigned keep = ((p0 & 0x7f80u) == 0x7f80u ? 0u : 0xffffu) | ((p0 & 0x7f800000u) == 0x7f800000u ? 0u : 0xffff0000u);
  p1 &= keep;
  p2 &= keep;
}
// B operands of the layers in shared memory, one 32-lane row of 8 bytes per (k step,
// 8-column tile)
constexpr int fW0 = 0, fW1 = fW0 + kK0 * 8, fW2 = fW1 + 32, fW3 = fW2 + 32, kFwdTiles = fW3 + 8;
__device__ __forceinline__ void pack_weights(uint2* B, const __nv_bfloat16* w) {
  const unsigned short* u = reinterpret_cast<const unsigned short*>(w);
#pragma unroll 4
  for (int e = threadIdx.x; e < kFwdTiles * 32; e += blockDim.x) {
    const int tile = e >> 5, lane = e & 31, g = lane >> 2, q = lane & 3;
    unsigned v[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int k = 2 * q + (s & 1) + 8 * (s >> 1);  // row of the k step
      int at = -1;
      if (tile < fW1) {
        const int i = input_of(tile / 8, q, s);
        at = i < 0 ? -1 : oW0 + ((tile % 8) * 8 + g) * kIn + i;
      } else if (tile < fW3) {
        const int t = (tile - fW1) % 32;
        at = (tile < fW2 ? oW1 : oW2) + ((t % 8) * 8 + g) * kHid + (t / 8) * 16 + k;
      } else {
        const int t = tile - fW3, o = (t % 2) * 8 + g;
        at = o < kOut ? oW3 + o * kHid + (t / 2) * 16 + k : -1;
      }
      v[s] = at < 0 ? 0u : u[at];
    }
    B[e] = make_uint2(v[0] | v[1] << 16, v[2] | v[3] << 16);
  }
}

// a point: offsets of the 3 x 3 neighbouring columns at its z
struct PointRow {
  unsigned col[9];
  int z;
  bool lo, hi;  // z - 1, z + 1 inside
};
__device__ __forceinline__ void point_row(PointRow& r, long long lin, int NYA, int NXA, int NZA) {
  const unsigned u = (unsigned)lin, t = u / NZA;  // (13 doubles a point: fewer than 2^32 points fit on the device)
  const int y = (int)(t / NXA), x = (int)(t - (unsigned)y * NXA);
  r.z = (int)(u - t * NZA);
  r.lo = r.z > 0;
  r.hi = r.z + 1 < NZA;
  const int yn[3] = {y > 0 ? y - 1 : NYA - 1, y, y + 1 < NYA ? y + 1 : 0};
  const int xn[3] = {x > 0 ? x - 1 : NXA - 1, x, x + 1 < NXA ? x + 1 : 0};
#pragma unroll
  for (int k = 0; k < 9; ++k) r.col[k] = ((unsigned)yn[k / 3] * NXA + xn[k % 3]) * NZA + r.z;
}
// z' at z + dz, dz = (q + i) mod 3 - 1
struct PointZeta {
  float v[3];
};
__device__ __forceinline__ PointZeta point_zeta(const PointRow& r, const double* zeta, int q) {
  PointZeta zt;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int dz = (q + i) % 3 - 1;
    zt.v[i] = (dz < 0 ? r.lo : dz > 0 ? r.hi : true) ? (float)zeta[r.z + dz] : 0.0f;
  }
  return zt;
}
// input of slot s of k step ks (channel field f of this lane column, scaled by sc)
template <int KS, int S, typename F>
__device__ __forceinline__ float point_input(const PointRow& r, const PointZeta& zt, const F* f, float sc, int q) {
  if constexpr (KS < 7) {
    constexpr int tap = 4 * KS + S;
    if constexpr (tap >= kTaps) {
      return 0.0f;
    } else {
      constexpr int dz = tap % 3 - 1;
      const bool in = dz < 0 ? r.lo : dz > 0 ? r.hi : true;
      return in ? (float)f[(long long)r.col[tap / 3] + dz] * sc : 0.0f;
    }
  } else {
    return 16 * (KS - 7) + 4 * q + S < kTaps ? zt.v[(S + KS - 7) % 3] : 0.0f;
  }
}
// the A operand of k step KS in three BF16 planes
template <int KS, typename F>
__device__ __forceinline__ void input_planes(unsigned (&a)[3][4], const PointRow (&r)[2], const PointZeta (&z)[2],
                                             const F* f, float sc, int q) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    split3_any(point_input<KS, 0>(r[i], z[i], f, sc, q), point_input<KS, 1>(r[i], z[i], f, sc, q), a[0][i], a[1][i],
               a[2][i]);
    split3_any(point_input<KS, 2>(r[i], z[i], f, sc, q), point_input<KS, 3>(r[i], z[i], f, sc, q), a[0][2 + i],
               a[1][2 + i], a[2][2 + i]);
  }
}
// the A operand of k step j from the accumulators of tiles 2 j, 2 j + 1
__device__ __forceinline__ void act_planes(unsigned (&a)[3][4], const float (&t0)[4], const float (&t1)[4]) {
  split3(t0[0], t0[1], a[0][0], a[1][0], a[2][0]);
  split3(t0[2], t0[3], a[0][1], a[1][1], a[2][1]);
  split3(t1[0], t1[1], a[0][2], a[1][2], a[2][2]);
  split3(t1[2], t1[3], a[0][3], a[1][3], a[2][3]);
}

template <int KS, typename F>
__device__ __forceinline__ void layer0_step(float (&c)[8][4], const uint2* B, const PointRow (&r)[2],
                                            const PointZeta (&z)[2], const F* f, float sc, int q, int lane) {
  unsigned a[3][4];
  input_planes<KS>(a, r, z, f, sc, q);
#pragma unroll
  for (int n = 0; n < 8; ++n) mma_planes(c[n], a, B[(fW0 + KS * 8 + n) * 32 + lane]);
  if constexpr (KS + 1 < kK0) layer0_step<KS + 1>(c, B, r, z, f, sc, q, lane);
}
// c = b (one float per column; 0 past ncol) in every row
template <int NT>
__device__ __forceinline__ void bias_tiles(float (&c)[NT][4], const float* b, int ncol, int q) {
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const int o = n * 8 + 2 * q;
    c[n][0] = c[n][2] = o < ncol ? b[o] : 0.0f;
    c[n][1] = c[n][3] = o + 1 < ncol ? b[o + 1] : 0.0f;
  }
}
// c += h W, h of 64 columns
template <int NT>
__device__ __forceinline__ void hidden_product(float (&c)[NT][4], const float (&h)[8][4], const uint2* B, int lane) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    unsigned a[3][4];
    act_planes(a, h[2 * j], h[2 * j + 1]);
#pragma unroll
    for (int n = 0; n < NT; ++n) mma_planes(c[n], a, B[(j * NT + n) * 32 + lane]);
  }
}

// tanh of two values at once: an odd polynomial below 0.5 (least-maximum fit of the
// relative error to tanh, 1.5e-8, by iteratively reweighted least squares), above it
// 1 - 2 / (e^{2|x|} + 1), where the subtraction loses nothing, so relative accuracy
// holds down to the smallest x.  Cut at 15, where the quotient is below half a last
// bit; NaN stays.  Packed in pairs, as the issue slots bound the kernel (96 x 96 x 72
// points: tanhf 443 us, this 390 with the sums of mma_planes in pairs too, 410 without).
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float ex2_approx(float a) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float rcp_approx(float a) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ void tanh_pair(float& x0, float& x1) {
  const float a0 = fabsf(x0), a1 = fabsf(x1);
  const unsigned long long x = pair2(x0, x1), y = mul2(x, x);
  unsigned long long p = fma2(pair2(0.017241491f, 0.017241491f), y, pair2(-0.053045493f, -0.053045493f));
  p = fma2(p, y, pair2(0.13325879f, 0.13325879f));
  p = fma2(p, y, pair2(-0.33333144f, -0.33333144f));
  float s0, s1, t0, t1, q0, q1;
  unpair2(fma2(x, mul2(p, y), x), s0, s1);
  constexpr float k = 2.8853900817779268f;  // 2 / ln 2
  unpair2(mul2(pair2(min_nan(a0, 15.0f), min_nan(a1, 15.0f)), pair2(k, k)), t0, t1);
  unpair2(add2(pair2(ex2_approx(t0), ex2_approx(t1)), pair2(1.0f, 1.0f)), t0, t1);
  unpair2(fma2(pair2(rcp_approx(t0), rcp_approx(t1)), pair2(-2.0f, -2.0f), pair2(1.0f, 1.0f)), q0, q1);
  x0 = a0 < 0.5f ? s0 : copysignf(q0, x0);
  x1 = a1 < 0.5f ? s1 : copysignf(q1, x1);
}

// Inference on a grid: point p is grid point p (linear [y][x][z]) of fields
// (double, [4][y][x][z]); tau_q = out_scale[q] y_q (double).  Warps walk the
// tiles of 16 points with a stride of the grid size.
constexpr int kInferThreads = 128, kInferCtas = 3;  // CTAs per SM
constexpr size_t kInferSmem = (size_t)kFwdTiles * 32 * sizeof(uint2);
__global__ void __launch_bounds__(kInferThreads, kInferCtas) k_closure_infer(NetDev net, const double* fields, int NYA,
                                                                            int NXA, int NZA, const double* zeta,
                                                                            long long npts, double* tau) {
  extern __shared__ __align__(16) uint2 Bs[];
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  pack_weights(Bs, net.w16);
  __syncthreads();
  const double* f = fields + (long long)q * npts;
  float sc = net.in_scale[0];
#pragma unroll
  for (int i = 1; i < 4; ++i) sc = q == i ? net.in_scale[i] : sc;
  const long long ntile = (npts + 15) / 16, stride = (long long)gridDim.x * (kInferThreads / 32);
  for (long long tile = (long long)blockIdx.x * (kInferThreads / 32) + (threadIdx.x >> 5); tile < ntile; tile += stride) {
    float h[8][4];
    {
      PointRow r[2];
      PointZeta z[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const long long p = tile * 16 + 8 * i + g;
        point_row(r[i], p < npts ? p : npts - 1, NYA, NXA, NZA);
        z[i] = point_zeta(r[i], zeta, q);
      }
      bias_tiles<8>(h, net.w32 + oB0, kHid, q);
      layer0_step<0>(h, Bs, r, z, f, sc, q, lane);
    }
    // (one copy of the code for both hidden layers: it is the instruction cache that
    // the unrolled layers press on)
#pragma unroll 1
    for (int layer = 0; layer < 2; ++layer) {
      float c[8][4];
      bias_tiles<8>(c, net.w32 + (layer ? oB2 : oB1), kHid, q);
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; e += 2) tanh_pair(h[n][e], h[n][e + 1]);
      hidden_product<8>(c, h, Bs + (layer ? fW2 : fW1) * 32, lane);
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) h[n][e] = c[n][e];
    }
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; e += 2) tanh_pair(h[n][e], h[n][e + 1]);
    float y[2][4];
    bias_tiles<2>(y, net.w32 + oB3, kOut, q);
    hidden_product<2>(y, h, Bs + fW3 * 32, lane);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const long long p = tile * 16 + 8 * (e >> 1) + g;
      if (p < npts) {
        const int o = 2 * q + (e & 1);
        tau[(long long)o * npts + p] = (double)(y[0][e] * net.out_scale[o]);
        if (o == 0) tau[8 * npts + p] = (double)(y[1][e] * net.out_scale[8]);
      }
    }
  }
}

// ---- training ------------------------------------------------------------------
// FP32 on the FP32 units: a batch of some thousand points is too small to fill the
// chip with tensor-core tiles, and the products of two FP32 operands would take six
// BF16 products each.  A CTA takes kTP points at a time with their inputs,
// activations and gradients in shared memory ([feature][point]) and the weights in
// FP32 (k-major for the forward, row-major for the backward products); every
// product is a register tile (forward and backward 4 features x 4 points a thread,
// weight gradients 4 x 4 or 4 x 9 features), so that a shared-memory access feeds
// eight or more multiply-adds.  (One thread per point, one multiply-add per two
// accesses, 64 CTAs: 240 us for 8192 points; now 53 us.)
// The CTAs' gradients are added (atomically) into kGradBuckets copies, which the
// next reader sums: shorter chains of FP32 additions, fewer collisions.
constexpr int kTrainThreads = 256, kTP = 64, kTR = kTP + 4;  // row stride: 8 rows' 16-byte reads hit distinct banks
constexpr int kWR = kHid + 4;  // row stride of the k-major weights
constexpr int sF0 = 0, sF1 = sF0 + kIn * kWR, sF2 = sF1 + kHid * kWR, sR1 = sF2 + kHid * kWR, sR2 = sR1 + kHid * kHid, sW3 = sR2 + kHid * kHid, sX = sW3 + kOut * kHid, sH1 = sX + kIn * kTR,
              sH2 = sH1 + kHid * kTR, sH3 = sH2 + kHid * kTR, sY = sH3 + kHid * kTR, kTrainFloats = sY + kOut * kTR;
constexpr size_t kTrainSmem = (size_t)kTrainFloats * sizeof(float);
static_assert(sX % 4 == 0 && sH1 % 4 == 0 && sF1 % 4 == 0 && kTP == kHid && kTrainThreads == 4 * kTP, "layout");

// acc[o][p] += sum_k W[k][4 ob + o] in[k][4 pb + p] (row stride LD of W).  The k are
// summed in runs of CH, the runs then: a smaller rounding error than one chain.
template <int NK, int CH, int LD>
__device__ __forceinline__ void tile_product(float (&acc)[4][4], const float* W, const float* in, int ob, int pb) {
  static_assert(NK % CH == 0, "whole runs");
#pragma unroll 1
  for (int k0 = 0; k0 < NK; k0 += CH) {
    float run[4][4];
#pragma unroll
    for (int o = 0; o < 4; ++o)
#pragma unroll
      for (int p = 0; p < 4; ++p) run[o][p] = 0.0f;
#pragma unroll
    for (int k = k0; k < k0 + CH; ++k) {
      const float4 w = *reinterpret_cast<const float4*>(W + k * LD + 4 * ob);
      const float4 x = *reinterpret_cast<const float4*>(in + k * kTR + 4 * pb);
      const float wv[4] = {w.x, w.y, w.z, w.w}, xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int o = 0; o < 4; ++o)
#pragma unroll
        for (int p = 0; p < 4; ++p) run[o][p] = fmaf(wv[o], xv[p], run[o][p]);
    }
#pragma unroll
    for (int o = 0; o < 4; ++o)
#pragma unroll
      for (int p = 0; p < 4; ++p) acc[o][p] += run[o][p];
  }
}
template <int NI>
__device__ __forceinline__ void train_forward(const float* W, const float* b, const float* in, float* out, int ob, int pb) {
  float acc[4][4];
#pragma unroll
  for (int o = 0; o < 4; ++o)
#pragma unroll
    for (int p = 0; p < 4; ++p) acc[o][p] = b[4 * ob + o];
  tile_product<NI, NI == kIn ? 27 : 16, kWR>(acc, W, in, ob, pb);
#pragma unroll
  for (int o = 0; o < 4; ++o)
    *reinterpret_cast<float4*>(out + (4 * ob + o) * kTR + 4 * pb) =
        make_float4(tanhf(acc[o][0]), tanhf(acc[o][1]), tanhf(acc[o][2]), tanhf(acc[o][3]));
}
// h <- (sum_k W[k][i] d[k]) (1 - h^2): the gradient at a tanh layer's inputs, in place
template <int NK>
__device__ __forceinline__ void train_back(const float* W, const float* d, float* h, int ib, int pb) {
  float acc[4][4];
#pragma unroll
  for (int o = 0; o < 4; ++o)
#pragma unroll
    for (int p = 0; p < 4; ++p) acc[o][p] = 0.0f;
  tile_product<NK, NK == kOut ? 9 : 16, kHid>(acc, W, d, ib, pb);
#pragma unroll
  for (int o = 0; o < 4; ++o) {
    float4* row = reinterpret_cast<float4*>(h + (4 * ib + o) * kTR + 4 * pb);
    const float4 v = *row;
    *row = make_float4(acc[o][0] * (1.0f - v.x * v.x), acc[o][1] * (1.0f - v.y * v.y), acc[o][2] * (1.0f - v.z * v.z),
                       acc[o][3] * (1.0f - v.w * v.w));
  }
}
// grad[o][i] += sum_p d[o][p] h[i][p] for the thread's 4 o and its M i = il + 16 m;
// runs of 16 points
template <int NI>
__device__ __forceinline__ void train_wgrad(float* grad, const float* d, const float* h, int t) {
  constexpr int M = (NI + 15) / 16;
  const int o0 = 4 * (t >> 4), il = t & 15;
  float acc[M][4];
#pragma unroll
  for (int m = 0; m < M; ++m)
#pragma unroll
    for (int o = 0; o < 4; ++o) acc[m][o] = 0.0f;
#pragma unroll 1
  for (int p0 = 0; p0 < kTP; p0 += 16) {
    float run[M][4];
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int o = 0; o < 4; ++o) run[m][o] = 0.0f;
#pragma unroll
    for (int p = p0; p < p0 + 16; p += 4) {
      float4 dv[4];
#pragma unroll
      for (int o = 0; o < 4; ++o) dv[o] = *reinterpret_cast<const float4*>(d + (o0 + o) * kTR + p);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int i = il + 16 * m;
        const float4 hv = *reinterpret_cast<const float4*>(h + (i < NI ? i : il) * kTR + p);
#pragma unroll
        for (int o = 0; o < 4; ++o)
          run[m][o] = fmaf(dv[o].w, hv.w, fmaf(dv[o].z, hv.z, fmaf(dv[o].y, hv.y, fmaf(dv[o].x, hv.x, run[m][o]))));
      }
    }
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int o = 0; o < 4; ++o) acc[m][o] += run[m][o];
  }
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int i = il + 16 * m;
    if (i < NI)
#pragma unroll
      for (int o = 0; o < 4; ++o) atomicAdd(grad + (o0 + o) * NI + i, acc[m][o]);
  }
}
__device__ __forceinline__ float row_sum(const float* d) {
  float s = 0.0f;
  for (int p = 0; p < kTP; p += 4) {
    const float4 v = *reinterpret_cast<const float4*>(d + p);
    s += (v.x + v.y) + (v.z + v.w);
  }
  return s;
}

// Loss (mean over the points of sum_q (y_q - target_q / out_scale[q])^2) and its
// gradient, added to loss and grad: point points[p] = snapshot * npoint + linear
// index of the float data set.
__global__ void __launch_bounds__(kTrainThreads, 1) k_closure_train(NetDev net, const float* fields, int NYA, int NXA,
                                                                   int NZA, const double* zeta, const long long* points,
                                                                   long long npts, const float* targets, float* grad,
                                                                   double* loss) {
  extern __shared__ __align__(16) float sm[];
  const int t = threadIdx.x, pt = t & (kTP - 1), part = t / kTP;  // part 0 .. 3
  const int ob = t >> 4, pb = t & 15;
  const long long npoint = (long long)NYA * NXA * NZA;
  {  // the weights, 8 at a time (every matrix starts on a 16-byte boundary)
    const uint4* w16 = reinterpret_cast<const uint4*>(net.w16);
    auto expand = [&](int off, int n, auto&& put) {
#pragma unroll 4
      for (int v = t; v < n / 8; v += kTrainThreads) {
        const uint4 u = w16[off / 8 + v];
        const unsigned uv[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int k = 0; k < 8; ++k)
          put(8 * v + k, __uint_as_float(k & 1 ? uv[k / 2] & 0xffff0000u : uv[k / 2] << 16));
      }
    };
    static_assert(oW1 % 8 == 0 && oW2 % 8 == 0 && oW3 % 8 == 0 && kHid * kIn % 8 == 0 && kOut * kHid % 8 == 0, "vectors");
    expand(oW0, kHid * kIn, [&](int e, float w) { sm[sF0 + e % kIn * kWR + e / kIn] = w; });
    expand(oW1, kHid * kHid, [&](int e, float w) { sm[sF1 + e % kHid * kWR + e / kHid] = sm[sR1 + e] = w; });
    expand(oW2, kHid * kHid, [&](int e, float w) { sm[sF2 + e % kHid * kWR + e / kHid] = sm[sR2 + e] = w; });
    expand(oW3, kOut * kHid, [&](int e, float w) { sm[sW3 + e] = w; });
  }
  grad += (size_t)(blockIdx.x % kGradBuckets) * kNParam;
  const float inv = 1.0f / (float)npts;
  double l = 0.0;  // (FP32 within a point only: a chain over a CTA's tiles would grow with the batch)
  for (long long p0 = (long long)blockIdx.x * kTP; p0 < npts; p0 += (long long)gridDim.x * kTP) {
    __syncthreads();  // the weights are in; the previous points are done with
    const bool ok = p0 + pt < npts;
    const long long at = points[ok ? p0 + pt : npts - 1], snap = at / npoint, lin = at - snap * npoint;
    {
      PointRow r;
      point_row(r, lin, NYA, NXA, NZA);
      const float* f = fields + snap * 4 * npoint;
      float* X = sm + sX + pt;
      const float sc = net.in_scale[part];
      f += part * npoint;
#pragma unroll
      for (int k = 0; k < 9; ++k)  // the stencil's columns of this part's channel
#pragma unroll
        for (int dz = -1; dz <= 1; ++dz) {
          const bool in = dz < 0 ? r.lo : dz > 0 ? r.hi : true;
          X[(part * kTaps + 3 * k + dz + 1) * kTR] = in ? f[(long long)r.col[k] + dz] * sc : 0.0f;
        }
      if (part < 3) {  // z' at dz = part - 1, the same in every column
        const bool in = part == 0 ? r.lo : part == 2 ? r.hi : true;
        const float v = in ? (float)zeta[r.z + part - 1] : 0.0f;
#pragma unroll
        for (int k = 0; k < 9; ++k) X[(4 * kTaps + 3 * k + part) * kTR] = v;
      }
    }
    __syncthreads();
    train_forward<kIn>(sm + sF0, net.w32 + oB0, sm + sX, sm + sH1, ob, pb);
    __syncthreads();
    train_forward<kHid>(sm + sF1, net.w32 + oB1, sm + sH1, sm + sH2, ob, pb);
    __syncthreads();
    train_forward<kHid>(sm + sF2, net.w32 + oB2, sm + sH2, sm + sH3, ob, pb);
    __syncthreads();
    {  // y, dL/dy of this point: outputs part, part + 4, part + 8
      float y[3];
#pragma unroll
      for (int m = 0; m < 3; ++m) y[m] = part + 4 * m < kOut ? net.w32[oB3 + part + 4 * m] : 0.0f;
#pragma unroll 8
      for (int k = 0; k < kHid; ++k) {
        const float x = sm[sH3 + k * kTR + pt];
#pragma unroll
        for (int m = 0; m < 3; ++m)
          if (part + 4 * m < kOut) y[m] = fmaf(sm[sW3 + (part + 4 * m) * kHid + k], x, y[m]);
      }
      const float* tg = targets + snap * kOut * npoint + lin;
      float lp = 0.0f;
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const int o = part + 4 * m;
        if (o < kOut) {
          const float d = ok ? y[m] - tg[(long long)o * npoint] / net.out_scale[o] : 0.0f;
          lp += d * d;
          sm[sY + o * kTR + pt] = 2.0f * d * inv;
        }
      }
      l += (double)lp;
    }
    __syncthreads();
    {  // dW3, db3
      float acc[3] = {};
#pragma unroll 4
      for (int p = 0; p < kTP; p += 4) {
        const float4 h = *reinterpret_cast<const float4*>(sm + sH3 + pt * kTR + p);
#pragma unroll
        for (int m = 0; m < 3; ++m)
          if (part + 4 * m < kOut) {
            const float4 d = *reinterpret_cast<const float4*>(sm + sY + (part + 4 * m) * kTR + p);
            acc[m] = fmaf(d.w, h.w, fmaf(d.z, h.z, fmaf(d.y, h.y, fmaf(d.x, h.x, acc[m]))));
          }
      }
#pragma unroll
      for (int m = 0; m < 3; ++m)
        if (part + 4 * m < kOut) atomicAdd(grad + oW3 + (part + 4 * m) * kHid + pt, acc[m]);
      if (t < kOut) atomicAdd(grad + oB3 + t, row_sum(sm + sY + t * kTR));
    }
    __syncthreads();
    train_back<kOut>(sm + sW3, sm + sY, sm + sH3, ob, pb);
    __syncthreads();
    train_wgrad<kHid>(grad + oW2, sm + sH3, sm + sH2, t);
    if (part == 0) atomicAdd(grad + oB2 + pt, row_sum(sm + sH3 + pt * kTR));
    __syncthreads();
    train_back<kHid>(sm + sR2, sm + sH3, sm + sH2, ob, pb);
    __syncthreads();
    train_wgrad<kHid>(grad + oW1, sm + sH2, sm + sH1, t);
    if (part == 0) atomicAdd(grad + oB1 + pt, row_sum(sm + sH2 + pt * kTR));
    __syncthreads();
    train_back<kHid>(sm + sR1, sm + sH2, sm + sH1, ob, pb);
    __syncthreads();
    train_wgrad<kIn>(grad + oW0, sm + sH1, sm + sX, t);
    if (part == 0) atomicAdd(grad + oB0 + pt, row_sum(sm + sH1 + pt * kTR));
  }
  for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  if ((t & 31) == 0 && l != 0.0) atomicAdd(loss, l * inv);
}

__device__ __forceinline__ float grad_sum(const float* g, int i) {
  float s = g[i];
#pragma unroll
  for (int b = 1; b < kGradBuckets; ++b) s += g[(size_t)b * kNParam + i];
  return s;
}
// the buckets' sum into the first one, the others cleared
__global__ void k_grad_sum(float* g) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kNParam; i += gridDim.x * blockDim.x) {
    g[i] = grad_sum(g, i);
#pragma unroll
    for (int b = 1; b < kGradBuckets; ++b) g[(size_t)b * kNParam + i] = 0.0f;
  }
}

// Adam (Kingma & Ba, 2015) on the FP32 master parameters; the BF16 copies are
// refreshed and the gradient cleared
__global__ void k_adam(float* w32, __nv_bfloat16* w16, float* g, float* m, float* v, int n, float lr, float b1,
                       float b2, float eps, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = grad_sum(g, i);
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w32[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w32[i] = wi;
    w16[i] = __float2bfloat16(wi);
#pragma unroll
    for (int b = 0; b < kGradBuckets; ++b) g[(size_t)b * kNParam + i] = 0.0f;
  }
}

__global__ void k_to_bf16(const float* w32, __nv_bfloat16* w16, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    w16[i] = __float2bfloat16(w32[i]);
}

}  // namespace

// ---- the network object ----------------------------------------------------------------
struct ClosureImpl {
  int device = 0;
  float *w32 = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
  __nv_bfloat16* w16 = nullptr;
  double* loss = nullptr;
  double* zeta = nullptr;
  int zeta_n = 0;
  float in_scale[4] = {1, 1, 1, 1}, out_scale[kOut] = {1, 1, 1, 1, 1, 1, 1, 1, 1};
  long long adam_t = 0;
  std::string err;
};

size_t closure_param_count() { return kNParam; }

NetDev net_dev(const ClosureImpl* c) {
  NetDev n{};
  n.w16 = c->w16;
  n.w32 = c->w32;
  for (int i = 0; i < 4; ++i) n.in_scale[i] = c->in_scale[i];
  for (int i = 0; i < kOut; ++i) n.out_scale[i] = c->out_scale[i];
  return n;
}

int device_sms() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 1;
}

void closure_set_smem() {
  static bool done = false;
  if (done) return;
  cudaFuncSetAttribute(k_closure_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInferSmem);
  cudaFuncSetAttribute(k_closure_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem);
  done = true;
}

// z' = (z - center) / (gap / 2) of the Gauss-Chebyshev grid, uploaded once per size
void closure_zeta(ClosureImpl* c, int NZA) {
  if (c->zeta && c->zeta_n == NZA) return;
  if (c->zeta) cudaFree(c->zeta);
  std::vector<double> z(NZA);
  const long double pi = 3.141592653589793238462643383279502884L;
  for (int i = 0; i < NZA; ++i) z[i] = (double)cosl(pi * (2.0L * (i + 1) - 1.0L) / (2.0L * NZA));
  if (cudaMalloc(&c->zeta, NZA * sizeof(double)) != cudaSuccess) throw CoralError(CORAL_ENOMEM, "closure: zeta");
  cudaMemcpy(c->zeta, z.data(), NZA * sizeof(double), cudaMemcpyHostToDevice);
  c->zeta_n = NZA;
}

// inference on a whole grid: 4 full-variable fields [f][y][x][z] (double) -> tau [9][y][x][z]
void closure_infer(ClosureImpl* c, const double* fields, int NYA, int NXA, int NZA, double* tau, cudaStream_t s) {
  closure_set_smem();
  closure_zeta(c, NZA);
  const long long np = (long long)NYA * NXA * NZA;
  // one wave of persistent warps, fewer when there are fewer tiles
  const long long need = (np + kInferThreads / 2 - 1) / (kInferThreads / 2);
  k_closure_infer<<<(unsigned)std::min<long long>(need, kInferCtas * device_sms()), kInferThreads, kInferSmem, s>>>(
      net_dev(c), fields, NYA, NXA, NZA, c->zeta, np, tau);
}

}  // namespace coral

using namespace coral;

struct coral_closure : ClosureImpl {};

namespace {

thread_local std::string g_closure_error;

template <typename F>
int cguard(coral_closure* c, F&& f) {
  if (!c) return CORAL_EBADARG;
  try {
    if (cudaSetDevice(c->device) != cudaSuccess) throw CoralError(CORAL_ECUDA, "cudaSetDevice");
    f();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw CoralError(CORAL_ECUDA, std::string("closure kernel: ") + cudaGetErrorString(e));
    return CORAL_OK;
  } catch (const CoralError& x) {
    c->err = x.what();
    return x.code;
  }
}

}  // namespace

namespace coral {
ClosureImpl* closure_impl(coral_closure* c) { return c; }
}  // namespace coral

extern "C" {

int coral_closure_create(int device, unsigned long long seed, coral_closure** out) {
  if (!out) return CORAL_EBADARG;
  *out = nullptr;
  auto* c = new coral_closure();
  c->device = device;
  if (cudaSetDevice(device) != cudaSuccess) {
    g_closure_error = "closure: no such device";
    delete c;
    return CORAL_ENODEV;
  }
  const size_t n = kNParam;
  bool okm = cudaMalloc(&c->w32, n * 4) == cudaSuccess && cudaMalloc(&c->g, kGradBuckets * n * 4) == cudaSuccess &&
             cudaMalloc(&c->m, n * 4) == cudaSuccess && cudaMalloc(&c->v, n * 4) == cudaSuccess &&
             cudaMalloc(&c->w16, n * 2) == cudaSuccess && cudaMalloc(&c->loss, 8) == cudaSuccess;
  if (!okm) {
    g_closure_error = "closure: device allocation failed";
    coral_closure_destroy(c);
    return CORAL_ENOMEM;
  }
  // Glorot-uniform weights from a 64-bit LCG (Knuth's MMIX constants), zero biases
  std::vector<float> w(n, 0.0f);
  unsigned long long st = seed * 6364136223846793005ull + 1442695040888963407ull;
  auto uni = [&]() {
    st = st * 6364136223846793005ull + 1442695040888963407ull;
    return (double)(st >> 11) * (1.0 / 9007199254740992.0);
  };
  auto fill = [&](int off, int no, int ni) {
    const double a = std::sqrt(6.0 / (double)(no + ni));
    for (int i = 0; i < no * ni; ++i) w[off + i] = (float)((2.0 * uni() - 1.0) * a);
  };
  fill(oW0, kHid, kIn);
  fill(oW1, kHid, kHid);
  fill(oW2, kHid, kHid);
  fill(oW3, kOut, kHid);
  cudaMemcpy(c->w32, w.data(), n * 4, cudaMemcpyHostToDevice);
  cudaMemset(c->g, 0, kGradBuckets * n * 4);
  cudaMemset(c->m, 0, n * 4);
  cudaMemset(c->v, 0, n * 4);
  k_to_bf16<<<64, 256>>>(c->w32, c->w16, (int)n);
  if (cudaDeviceSynchronize() != cudaSuccess) {
    g_closure_error = "closure: initialisation failed";
    coral_closure_destroy(c);
    return CORAL_ECUDA;
  }
  *out = c;
  return CORAL_OK;
}

void coral_closure_destroy(coral_closure* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  cudaFree(c->w32);
  cudaFree(c->g);
  cudaFree(c->m);
  cudaFree(c->v);
  cudaFree(c->w16);
  cudaFree(c->loss);
  if (c->zeta) cudaFree(c->zeta);
  delete c;
}

const char* coral_closure_last_error(const coral_closure* c) { return c ? c->err.c_str() : g_closure_error.c_str(); }

int coral_closure_param_count(void) { return kNParam; }

int coral_closure_set_scales(coral_closure* c, const float* in_scale4, const float* out_scale9) {
  return cguard(c, [&] {
    if (!in_scale4 || !out_scale9) throw CoralError(CORAL_EBADARG, "null scales");
    for (int i = 0; i < 4; ++i) c->in_scale[i] = in_scale4[i];
    for (int i = 0; i < kOut; ++i) {
      if (!(out_scale9[i] > 0.0f)) throw CoralError(CORAL_EBADARG, "output scales must be > 0");
      c->out_scale[i] = out_scale9[i];
    }
  });
}

int coral_closure_get_params(coral_closure* c, float* params, int n) {
  return cguard(c, [&] {
    if (!params || n < kNParam) throw CoralError(CORAL_EBADARG, "buffer smaller than the parameter count");
    if (cudaMemcpy(params, c->w32, kNParam * 4, cudaMemcpyDeviceToHost) != cudaSuccess)
      throw CoralError(CORAL_ECUDA, "copy");
  });
}

int coral_closure_set_params(coral_closure* c, const float* params, int n) {
  return cguard(c, [&] {
    if (!params || n < kNParam) throw CoralError(CORAL_EBADARG, "buffer smaller than the parameter count");
    if (cudaMemcpy(c->w32, params, kNParam * 4, cudaMemcpyHostToDevice) != cudaSuccess)
      throw CoralError(CORAL_ECUDA, "copy");
    k_to_bf16<<<64, 256>>>(c->w32, c->w16, kNParam);
    cudaDeviceSynchronize();
  });
}

int coral_closure_get_gradient(coral_closure* c, float* grad, int n) {
  return cguard(c, [&] {
    if (!grad || n < kNParam) throw CoralError(CORAL_EBADARG, "buffer smaller than the parameter count");
    k_grad_sum<<<(kNParam + 255) / 256, 256>>>(c->g);
    if (cudaMemcpy(grad, c->g, kNParam * 4, cudaMemcpyDeviceToHost) != cudaSuccess)
      throw CoralError(CORAL_ECUDA, "copy");
  });
}

int coral_closure_train(coral_closure* c, const float* inputs, const float* targets, int nsnap, int NXA, int NYA,
                        int NZA, const long long* points, long long npts, float lr, int apply, double* loss) {
  return cguard(c, [&] {
    if (!inputs || !targets || !points || npts <= 0 || nsnap <= 0 || NXA <= 0 || NYA <= 0 || NZA <= 0)
      throw CoralError(CORAL_EBADARG, "closure_train: bad arguments");
    closure_set_smem();
    closure_zeta(c, NZA);
    cudaMemset(c->loss, 0, 8);
    const long long tiles = (npts + kTP - 1) / kTP;
    k_closure_train<<<(unsigned)std::min<long long>(tiles, device_sms()), kTrainThreads, kTrainSmem>>>(
        net_dev(c), inputs, NYA, NXA, NZA, c->zeta, points, npts, targets, c->g, c->loss);
    if (apply) {
      ++c->adam_t;
      const float b1 = 0.9f, b2 = 0.999f;
      k_adam<<<64, 256>>>(c->w32, c->w16, c->g, c->m, c->v, kNParam, lr, b1, b2, 1e-8f,
                          1.0f - std::pow(b1, (float)c->adam_t), 1.0f - std::pow(b2, (float)c->adam_t));
    }
    double l = 0.0;
    if (cudaMemcpy(&l, c->loss, 8, cudaMemcpyDeviceToHost) != cudaSuccess) throw CoralError(CORAL_ECUDA, "loss");
    if (loss) *loss = l;
  });
}

int coral_closure_zero_gradient(coral_closure* c) {
  return cguard(c, [&] { cudaMemset(c->g, 0, (size_t)kGradBuckets * kNParam * 4); });
}

int coral_closure_infer(coral_closure* c, const double* fields, int NXA, int NYA, int NZA, double* tau, void* stream) {
  return cguard(c, [&] {
    if (!fields || !tau) throw CoralError(CORAL_EBADARG, "null buffer");
    closure_infer(c, fields, NYA, NXA, NZA, tau, static_cast<cudaStream_t>(stream));
  });
}

}  // extern "C"
