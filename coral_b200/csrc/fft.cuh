// Shared-memory FFTs for the transform kernels (sm_100a, FP64).
//
// A CTA transforms a batch of lines held contiguously in shared memory
// (line-major, line stride N) with a self-sorting Stockham scheme of radix 4, 3
// and 2 stages (all grid sizes of the plane-layer problems are 2^a 3^b).  The
// twiddles exp(-2 pi i k / N) come from a table computed on the host in long
// double.  Real transforms pack two real lines into one complex line.
#pragma once
#include <cuda_runtime.h>

namespace coral {

struct FftPlan {
  int N;
  int nst;
  int radix[16];
  const double2* tw;      // tw[k] = exp(-2 pi i k / N), k < N (plans chosen at run time)
  const double2* tws[2];  // the compiled plans' twiddles pass by pass (pass_tw_index), per plan variant
};

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
// multiply by -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ double2 mul_mi(double2 a) {
  return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// sin(pi/3), from the mathematics
#define CORAL_SIN60 0.86602540378443864676372317075293618

// Ping-pong batched FFT of nl lines of length p.N stored in A (line stride LS)
// with a plan chosen at run time (lengths without a compile-time plan).  B is
// scratch of the same size.  Returns the buffer that holds the result.
// INV = false: exp(-i), INV = true: exp(+i); no normalisation.
// Must be called by all threads of the CTA (contains __syncthreads).
template <bool INV>
__device__ double2* fft_lines(double2* A, double2* B, int nl, int LS, const FftPlan& p) {
  double2* src = A;
  double2* dst = B;
  const int N = p.N;
  int Ns = 1;
  for (int s = 0; s < p.nst; ++s) {
    const int R = p.radix[s];
    const int nb = N / R;
    const int tstride = N / (Ns * R);
    const int total = nl * nb;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
      const int line = idx / nb;
      const int j = idx - line * nb;
      const int k = j % Ns;
      const double2* sl = src + line * LS;
      double2* dl = dst + line * LS;
      const int od = (j / Ns) * Ns * R + k;
      if (R == 4) {
        double2 a0 = sl[j], a1 = sl[j + nb], a2 = sl[j + 2 * nb], a3 = sl[j + 3 * nb];
        if (Ns > 1) {
          double2 w1 = p.tw[k * tstride], w2 = p.tw[2 * k * tstride], w3 = p.tw[3 * k * tstride];
          if (INV) { w1 = cconj(w1); w2 = cconj(w2); w3 = cconj(w3); }
          a1 = cmul(a1, w1); a2 = cmul(a2, w2); a3 = cmul(a3, w3);
        }
        double2 t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = mul_mi<INV>(csub(a1, a3));
        dl[od] = cadd(t0, t2);
        dl[od + Ns] = cadd(t1, t3);
        dl[od + 2 * Ns] = csub(t0, t2);
        dl[od + 3 * Ns] = csub(t1, t3);
      } else if (R == 3) {
        double2 a0 = sl[j], a1 = sl[j + nb], a2 = sl[j + 2 * nb];
        if (Ns > 1) {
          double2 w1 = p.tw[k * tstride], w2 = p.tw[2 * k * tstride];
          if (INV) { w1 = cconj(w1); w2 = cconj(w2); }
          a1 = cmul(a1, w1); a2 = cmul(a2, w2);
        }
        double2 t = cadd(a1, a2), d = csub(a1, a2);
        double2 m = make_double2(a0.x - 0.5 * t.x, a0.y - 0.5 * t.y);
        // forward: y1 = m - i s d, y2 = m + i s d ; inverse: s -> -s
        const double sd = INV ? -CORAL_SIN60 : CORAL_SIN60;
        double2 isd = make_double2(-sd * d.y, sd * d.x);  // i*s*d
        dl[od] = cadd(a0, t);
        dl[od + Ns] = csub(m, isd);
        dl[od + 2 * Ns] = cadd(m, isd);
      } else {  // R == 2
        double2 a0 = sl[j], a1 = sl[j + nb];
        if (Ns > 1) {
          double2 w1 = p.tw[k * tstride];
          if (INV) w1 = cconj(w1);
          a1 = cmul(a1, w1);
        }
        dl[od] = cadd(a0, a1);
        dl[od + Ns] = csub(a0, a1);
      }
    }
    __syncthreads();
    double2* t = src;
    src = dst;
    dst = t;
    Ns *= R;
  }
  return src;
}

// ---- compile-time plans: register passes ----------------------------------------
// With the length N known at compile time the transform runs as a few passes of
// radix 24, 18, 16, 9, 8, 4, 3 or 2 (in the three-pass plans odd radices come
// first: their strided stores in the first pass hit distinct shared-memory banks;
// the two-pass plans trade that for one pass fewer).  Each thread computes whole
// radix-R butterflies in registers: it loads its R inputs, applies the twiddles,
// waits for every thread to have loaded (so the pass can write in place), and
// stores its R outputs at their Stockham (self-sorting) positions.  Only one
// line buffer is needed.
// A plan is a list of passes; an entry r < 100 is one radix, a 100 + b (or
// (a 100 + b) 100 + c) a pass that takes the radices a, b (, c) one after the other
// in registers, with the arithmetic of separate passes bit for bit (the solves
// turn another rounding of the transforms into 1e-9 of the pressure, so a length
// keeps its radices when its passes are merged).
struct PlanR {
  int nst;
  int r[12];
};
__host__ __device__ constexpr int radix_a(int code) { return code < 100 ? code : code < 10000 ? code / 100 : code / 10000; }
__host__ __device__ constexpr int radix_b(int code) { return code < 100 ? 1 : code < 10000 ? code % 100 : code / 100 % 100; }
__host__ __device__ constexpr int radix_c(int code) { return code < 10000 ? 1 : code % 100; }
__host__ __device__ constexpr int radix_of(int code) { return radix_a(code) * radix_b(code) * radix_c(code); }
__host__ __device__ constexpr PlanR make_planr(int N) {
  switch (N) {
    case 54: return PlanR{2, {303, 302}};
    case 108: return PlanR{2, {403, 303}};
    case 162: return PlanR{2, {303, 30302}};
    case 216: return PlanR{2, {403, 30302}};
    case 324: return PlanR{2, {403, 30303}};
    case 432: return PlanR{2, {404, 30303}};
    case 486: return PlanR{3, {303, 303, 302}};
    default: break;
  }
  PlanR p{0, {}};
  int n = N, a = 0, b = 0;
  while (n % 3 == 0) { n /= 3; ++b; }
  while (n % 2 == 0) { n /= 2; ++a; }
  if (n != 1) return PlanR{0, {}};
  for (; b >= 2; b -= 2) p.r[p.nst++] = 9;
  if (b == 1) p.r[p.nst++] = 3;
  while (a > 0) {
    if (a == 6) { p.r[p.nst++] = 8; p.r[p.nst++] = 8; a = 0; }
    else if (a == 5) { p.r[p.nst++] = 8; p.r[p.nst++] = 4; a = 0; }
    else if (a >= 4) { p.r[p.nst++] = 16; a -= 4; }
    else if (a == 3) { p.r[p.nst++] = 8; a = 0; }
    else if (a == 2) { p.r[p.nst++] = 4; a = 0; }
    else { p.r[p.nst++] = 2; a = 0; }
  }
  return p;
}

// Two-pass plans (more registers per thread, one barrier pair fewer):
// 288 = 18 x 16, 576 = 24 x 24; other lengths keep make_planr.
__host__ __device__ constexpr PlanR make_planr2(int N) {
  if (N == 288) return PlanR{2, {18, 16}};
  if (N == 576) return PlanR{2, {24, 24}};
  return make_planr(N);
}
// make_planr's radices in passes of at most 12 elements: the forward z pass keeps 64
// registers a thread, with which 27-element butterflies spill 1 to 2.4 KB (one | nine
// variables of a 144 x 144 grid, us, run-time plan, 27-element passes, these: 162
// points 50 | 193, 41 | 181, 38 | 160; 216: 53 | 238, 48 | 242, 48 | 215; 324: 63 |
// 378, 100 | 481, 64 | 318; 432: 73 | 600, 115 | 704, 92 | 516)
__host__ __device__ constexpr PlanR make_planr3(int N) {
  switch (N) {
    case 162: return PlanR{3, {303, 303, 2}};
    case 216: return PlanR{3, {403, 3, 302}};
    case 324: return PlanR{3, {4, 303, 303}};
    case 432: return PlanR{3, {4, 403, 303}};
    default: return make_planr(N);
  }
}
// plan variant PV: 0 = make_planr, 1 = make_planr2, 2 = make_planr3 (its radices are
// make_planr's in the same order, so the twiddle tables of variant 0 serve it)
__host__ __device__ constexpr PlanR plan_of(int N, int PV) {
  return PV == 0 ? make_planr(N) : PV == 1 ? make_planr2(N) : make_planr3(N);
}

// cos / sin of 2 pi m / 16 and 2 pi m / 9, from the mathematics (40-digit values)
#define CORAL_C16_1 0.923879532511286756128183189396788287   // cos(pi/8)
#define CORAL_S16_1 0.382683432365089771728459984030398867   // sin(pi/8)
#define CORAL_SQRT1_2 0.707106781186547524400844362104849039 // cos(pi/4)
#define CORAL_C9_1 0.766044443118978035202392650555416674    // cos(2 pi/9)
#define CORAL_S9_1 0.642787609686539326322643409907263433    // sin(2 pi/9)
#define CORAL_C9_2 0.173648177666930348851716626769314796    // cos(4 pi/9)
#define CORAL_S9_2 0.984807753012208059366743024589523014    // sin(4 pi/9)
#define CORAL_C9_4 (-0.93969262078590838405410927732473147)  // cos(8 pi/9)
#define CORAL_S9_4 0.342020143325668733044099614682259581    // sin(8 pi/9)

// cos / sin of 2 pi m / 18 and 2 pi m / 24 (m = 0, 1, ...), from the mathematics
__device__ constexpr double kC18[9] = {1.0, 0.93969262078590838405410927732473147, 0.766044443118978035202392650555416674,
                                       0.5, 0.173648177666930348851716626769314796, -0.173648177666930348851716626769314796,
                                       -0.5, -0.766044443118978035202392650555416674, -0.93969262078590838405410927732473147};
__device__ constexpr double kS18[9] = {0.0, 0.342020143325668733044099614682259581, 0.642787609686539326322643409907263433,
                                       0.866025403784438646763723170752936183, 0.984807753012208059366743024589523014,
                                       0.984807753012208059366743024589523014, 0.866025403784438646763723170752936183,
                                       0.642787609686539326322643409907263433, 0.342020143325668733044099614682259581};
__device__ constexpr double kC24[15] = {1.0, 0.965925826289068286749743199728897368, 0.866025403784438646763723170752936183,
                                        0.707106781186547524400844362104849039, 0.5, 0.258819045102520762348898837624048328,
                                        0.0, -0.258819045102520762348898837624048328, -0.5,
                                        -0.707106781186547524400844362104849039, -0.866025403784438646763723170752936183,
                                        -0.965925826289068286749743199728897368, -1.0,
                                        -0.965925826289068286749743199728897368, -0.866025403784438646763723170752936183};
__device__ constexpr double kS24[15] = {0.0, 0.258819045102520762348898837624048328, 0.5,
                                        0.707106781186547524400844362104849039, 0.866025403784438646763723170752936183,
                                        0.965925826289068286749743199728897368, 1.0, 0.965925826289068286749743199728897368,
                                        0.866025403784438646763723170752936183, 0.707106781186547524400844362104849039, 0.5,
                                        0.258819045102520762348898837624048328, 0.0, -0.258819045102520762348898837624048328,
                                        -0.5};

// a * exp(-i t) (forward) or a * exp(+i t) (inverse), given c = cos t, s = sin t
template <bool INV>
__device__ __forceinline__ double2 rot(double2 a, double c, double s) {
  return INV ? make_double2(a.x * c - a.y * s, a.x * s + a.y * c) : make_double2(a.x * c + a.y * s, a.y * c - a.x * s);
}

template <bool INV>
__device__ __forceinline__ void dft3(double2& a0, double2& a1, double2& a2) {
  const double2 t = cadd(a1, a2), d = csub(a1, a2);
  const double2 m = make_double2(a0.x - 0.5 * t.x, a0.y - 0.5 * t.y);
  const double sd = INV ? -CORAL_SIN60 : CORAL_SIN60;
  const double2 isd = make_double2(-sd * d.y, sd * d.x);  // i s d
  a0 = cadd(a0, t);
  a1 = csub(m, isd);
  a2 = cadd(m, isd);
}
template <bool INV>
__device__ __forceinline__ void dft4(double2& a0, double2& a1, double2& a2, double2& a3) {
  const double2 t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = mul_mi<INV>(csub(a1, a3));
  a0 = cadd(t0, t2);
  a1 = cadd(t1, t3);
  a2 = csub(t0, t2);
  a3 = csub(t1, t3);
}

// in-register DFT of length R, natural order in and out
template <int R, bool INV>
__device__ __forceinline__ void dft(double2 (&x)[R]) {
  if constexpr (R == 2) {
    const double2 t = x[0];
    x[0] = cadd(t, x[1]);
    x[1] = csub(t, x[1]);
  } else if constexpr (R == 3) {
    dft3<INV>(x[0], x[1], x[2]);
  } else if constexpr (R == 4) {
    dft4<INV>(x[0], x[1], x[2], x[3]);
  } else if constexpr (R == 8) {
    // n = 2 n1 + n2, k = k1 + 4 k2
    dft4<INV>(x[0], x[2], x[4], x[6]);
    dft4<INV>(x[1], x[3], x[5], x[7]);
    x[3] = rot<INV>(x[3], CORAL_SQRT1_2, CORAL_SQRT1_2);
    x[5] = mul_mi<INV>(x[5]);
    x[7] = rot<INV>(x[7], -CORAL_SQRT1_2, CORAL_SQRT1_2);
    double2 y[8];
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      y[k1] = cadd(x[2 * k1], x[2 * k1 + 1]);
      y[k1 + 4] = csub(x[2 * k1], x[2 * k1 + 1]);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = y[k];
  } else if constexpr (R == 9) {
    // n = 3 n1 + n2, k = k1 + 3 k2
    dft3<INV>(x[0], x[3], x[6]);
    dft3<INV>(x[1], x[4], x[7]);
    dft3<INV>(x[2], x[5], x[8]);
    // A_{n2}[k1] sits in x[n2 + 3 k1]; twiddle by w9^(n2 k1)
    x[4] = rot<INV>(x[4], CORAL_C9_1, CORAL_S9_1);
    x[7] = rot<INV>(x[7], CORAL_C9_2, CORAL_S9_2);
    x[5] = rot<INV>(x[5], CORAL_C9_2, CORAL_S9_2);
    x[8] = rot<INV>(x[8], CORAL_C9_4, CORAL_S9_4);
    dft3<INV>(x[0], x[1], x[2]);  // k1 = 0 -> X[0], X[3], X[6]
    dft3<INV>(x[3], x[4], x[5]);  // k1 = 1 -> X[1], X[4], X[7]
    dft3<INV>(x[6], x[7], x[8]);  // k1 = 2 -> X[2], X[5], X[8]
    double2 y[9];
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1)
#pragma unroll
      for (int k2 = 0; k2 < 3; ++k2) y[k1 + 3 * k2] = x[3 * k1 + k2];
#pragma unroll
    for (int k = 0; k < 9; ++k) x[k] = y[k];
  } else if constexpr (R == 18) {
    // n = 2 n1 + n2, k = k1 + 9 k2: two 9-point DFTs, twiddles w18^k1, butterflies
    double2 e[9], o[9];
#pragma unroll
    for (int n1 = 0; n1 < 9; ++n1) {
      e[n1] = x[2 * n1];
      o[n1] = x[2 * n1 + 1];
    }
    dft<9, INV>(e);
    dft<9, INV>(o);
#pragma unroll
    for (int k1 = 1; k1 < 9; ++k1) o[k1] = rot<INV>(o[k1], kC18[k1], kS18[k1]);
#pragma unroll
    for (int k1 = 0; k1 < 9; ++k1) {
      x[k1] = cadd(e[k1], o[k1]);
      x[k1 + 9] = csub(e[k1], o[k1]);
    }
  } else if constexpr (R == 24) {
    // n = 3 n1 + n2, k = k1 + 8 k2: three 8-point DFTs, twiddles w24^(n2 k1), 3-point DFTs
    double2 a0[8], a1[8], a2[8];
#pragma unroll
    for (int n1 = 0; n1 < 8; ++n1) {
      a0[n1] = x[3 * n1];
      a1[n1] = x[3 * n1 + 1];
      a2[n1] = x[3 * n1 + 2];
    }
    dft<8, INV>(a0);
    dft<8, INV>(a1);
    dft<8, INV>(a2);
#pragma unroll
    for (int k1 = 1; k1 < 8; ++k1) {
      a1[k1] = rot<INV>(a1[k1], kC24[k1], kS24[k1]);
      a2[k1] = rot<INV>(a2[k1], kC24[2 * k1], kS24[2 * k1]);
    }
#pragma unroll
    for (int k1 = 0; k1 < 8; ++k1) {
      dft3<INV>(a0[k1], a1[k1], a2[k1]);
      x[k1] = a0[k1];
      x[k1 + 8] = a1[k1];
      x[k1 + 16] = a2[k1];
    }
  } else if constexpr (R == 16) {
    // n = 4 n1 + n2, k = k1 + 4 k2
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) dft4<INV>(x[n2], x[n2 + 4], x[n2 + 8], x[n2 + 12]);
    // A_{n2}[k1] sits in x[n2 + 4 k1]; twiddle by w16^(n2 k1)
    x[5] = rot<INV>(x[5], CORAL_C16_1, CORAL_S16_1);      // 1
    x[9] = rot<INV>(x[9], CORAL_SQRT1_2, CORAL_SQRT1_2);  // 2
    x[13] = rot<INV>(x[13], CORAL_S16_1, CORAL_C16_1);    // 3
    x[6] = rot<INV>(x[6], CORAL_SQRT1_2, CORAL_SQRT1_2);  // 2
    x[10] = mul_mi<INV>(x[10]);                            // 4
    x[14] = rot<INV>(x[14], -CORAL_SQRT1_2, CORAL_SQRT1_2);  // 6
    x[7] = rot<INV>(x[7], CORAL_S16_1, CORAL_C16_1);      // 3
    x[11] = rot<INV>(x[11], -CORAL_SQRT1_2, CORAL_SQRT1_2);  // 6
    x[15] = rot<INV>(x[15], -CORAL_C16_1, -CORAL_S16_1);  // 9
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) dft4<INV>(x[4 * k1], x[4 * k1 + 1], x[4 * k1 + 2], x[4 * k1 + 3]);
    double2 y[16];
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) y[k1 + 4 * k2] = x[4 * k1 + k2];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = y[k];
  }
}

// Twiddles of a compiled plan's radices in their order (those of merged passes one by
// one) after the first, one table [r - 1][k] after the other: entry (r, k),
// 1 <= r < R, k < Ns (the product of the earlier radices), is exp(-2 pi i r k / (Ns R)).
// Consecutive lanes take consecutive k, so a load touches consecutive 16-byte words
// (the N-entry table read at stride r touched up to a line per lane).  With the
// padding below, per step at 384^2 x 192: inverse y 2.91 -> 2.48 ms, inverse x 2.38
// -> 2.20, forward x 3.48 -> 3.16, forward y 3.59 -> 3.38, z 9.3 -> 9.07; z at 96
// points 0.54 -> 0.46 ms.
__host__ __device__ constexpr int pass_ns(int N, int PV, int S) {
  int ns = 1;
  for (int q = 0; q < S; ++q) ns *= radix_of(plan_of(N, PV).r[q]);
  return ns;
}
// entries of the tables before radix q (0, 1, 2) of pass S
__host__ __device__ constexpr int pass_tw_offset(int N, int PV, int S, int q = 0) {
  const PlanR p = plan_of(N, PV);
  int o = 0, ns = 1;
  for (int t = 0; t <= S && t < p.nst; ++t) {
    const int r[3] = {radix_a(p.r[t]), radix_b(p.r[t]), radix_c(p.r[t])};
    for (int u = 0; u < 3; ++u) {
      if (t == S && u == q) return o;
      if (ns > 1) o += ns * (r[u] - 1);
      ns *= r[u];
    }
  }
  return o;
}
__host__ __device__ constexpr int pass_tw_len(int N, int PV) { return pass_tw_offset(N, PV, plan_of(N, PV).nst); }
// index into the N-entry table of entry i of the pass tables
__host__ __device__ inline int pass_tw_index(int N, int PV, int i) {
  const PlanR p = plan_of(N, PV);
  int ns = 1;
  for (int t = 0; t < p.nst; ++t) {
    const int r[3] = {radix_a(p.r[t]), radix_b(p.r[t]), radix_c(p.r[t])};
    for (int u = 0; u < 3; ++u) {
      const int n = ns > 1 ? ns * (r[u] - 1) : 0;
      if (i < n) return (i / ns + 1) * (i % ns) * (N / (ns * r[u]));
      i -= n;
      ns *= r[u];
    }
  }
  return 0;
}

// Padding of a line between the first and the second pass of a two-pass plan whose
// first radix is even: its butterflies store R0 consecutive elements each, so 8
// lanes' 16-byte stores at stride R0 would share banks; one element is left out
// after every pad_every butterflies (LINE_FAST: 4 interleaved lines x 2
// butterflies).  Odd radices need none, and later passes store in natural order.
__host__ __device__ constexpr int pad_every(int N, int PV, bool line_fast) {
  const PlanR p = plan_of(N, PV);
  const int r0 = radix_of(p.r[0]);
  if (p.nst != 2 || r0 % 2) return 0;
  if (line_fast) return 1;
  return r0 % 8 == 0 ? 1 : r0 % 4 == 0 ? 2 : 4;
}
__host__ __device__ constexpr int line_len(int N, int PV, bool line_fast) {
  const int e = N ? pad_every(N, PV, line_fast) : 0;
  return e ? N + (N / radix_of(plan_of(N, PV).r[0]) - 1) / e : N;
}
// line stride of the passes that walk 4 interleaved lines: 2 mod 8, so that the
// same position of the lines hits 4 distinct even 16-byte bank groups
__host__ __device__ constexpr int line_stride(int N, int PV) {
  const int n = line_len(N, PV, true);
  return n == N ? N + 2 : (n + 5) / 8 * 8 + 2;
}

// The radices of a merged pass S in registers: x[r] is the element at position j + r N / R of
// the line, k = j mod Ns.  Radix a combines x[r' + r1 (R / a)] over r1 for every r',
// radix b then the results over the next digit, and so on; the twiddle of digit r_b
// has k + r_a Ns in place of k, and the outputs come in order.  tw: the plan's
// tables (null only when no twiddle is needed).
template <int N, int PV, int S, bool INV, int R>
__device__ __forceinline__ void pass_butterfly(double2 (&x)[R], int k, const double2* __restrict__ tw) {
  constexpr int code = plan_of(N, PV).r[S], Ra = radix_a(code), Rb = radix_b(code), Rc = radix_c(code);
  constexpr int Ns = pass_ns(N, PV, S);
  static_assert(R == Ra * Rb * Rc, "radix");
  auto twiddle = [&](double2 v, int at) {
    double2 w = tw[at];
    if (INV) w = cconj(w);
    return cmul(v, w);
  };
  constexpr int M = Rb * Rc;
  double2 y[R];  // y[ra M + r']
#pragma unroll
  for (int q = 0; q < M; ++q) {
    double2 v[Ra];
#pragma unroll
    for (int r = 0; r < Ra; ++r) {
      v[r] = x[q + r * M];
      if (Ns > 1 && r > 0) v[r] = twiddle(v[r], pass_tw_offset(N, PV, S) + (r - 1) * Ns + k);
    }
    dft<Ra, INV>(v);
#pragma unroll
    for (int r = 0; r < Ra; ++r) y[r * M + q] = v[r];
  }
  // digit rb of r' = rb Rc + rc
#pragma unroll
  for (int ra = 0; ra < Ra; ++ra)
#pragma unroll
    for (int rc = 0; rc < Rc; ++rc) {
      double2 v[Rb];
#pragma unroll
      for (int r = 0; r < Rb; ++r) {
        v[r] = y[ra * M + r * Rc + rc];
        if (r > 0 && Ns * Ra > 1)
          v[r] = twiddle(v[r], pass_tw_offset(N, PV, S, 1) + (r - 1) * Ns * Ra + k + ra * Ns);
      }
      dft<Rb, INV>(v);
#pragma unroll
      for (int r = 0; r < Rb; ++r) y[ra * M + r * Rc + rc] = v[r];
    }
  if constexpr (Rc > 1) {
#pragma unroll
    for (int ra = 0; ra < Ra; ++ra)
#pragma unroll
      for (int rb = 0; rb < Rb; ++rb) {
        double2 v[Rc];
#pragma unroll
        for (int r = 0; r < Rc; ++r) {
          v[r] = y[ra * M + rb * Rc + r];
          if (r > 0) v[r] = twiddle(v[r], pass_tw_offset(N, PV, S, 2) + (r - 1) * Ns * Ra * Rb + k + (ra + rb * Ra) * Ns);
        }
        dft<Rc, INV>(v);
#pragma unroll
        for (int r = 0; r < Rc; ++r) y[ra * M + rb * Rc + r] = v[r];
      }
  }
#pragma unroll
  for (int ra = 0; ra < Ra; ++ra)
#pragma unroll
    for (int rb = 0; rb < Rb; ++rb)
#pragma unroll
      for (int rc = 0; rc < Rc; ++rc) x[ra + Ra * (rb + Rb * rc)] = y[ra * M + rb * Rc + rc];
}

// Pass S in place over nl lines (line stride LS) by NT threads; NLMAX bounds nl
// (registers hold ceil(NLMAX N / (R NT)) butterflies per thread); tw: the plan's
// tables; PADE: pad_every of the line as the first pass left it.
template <int N, int PV, int S, bool INV, int NT, int NLMAX, int PADE = 0>
__device__ __forceinline__ void fft_pass(double2* A, int nl, int LS, const double2* __restrict__ tw) {
  constexpr int R = radix_of(plan_of(N, PV).r[S]), Ns = pass_ns(N, PV, S);
  constexpr int NB = N / R;               // butterflies per line
  static_assert(PADE == 0 || NB == Ns, "padding: second of two passes");
  constexpr int BPT = (NLMAX * NB + NT - 1) / NT;
  const int total = nl * NB;
  double2 v[BPT][R];
#pragma unroll
  for (int i = 0; i < BPT; ++i) {
    const int b = threadIdx.x + i * NT;
    if (b < total) {
      const int line = b / NB, j = b - line * NB;
      const double2* sl = A + line * LS + j;
#pragma unroll
      for (int r = 0; r < R; ++r) v[i][r] = sl[r * NB + (PADE ? r / PADE : 0)];
      if constexpr (plan_of(N, PV).r[S] >= 100) {
        pass_butterfly<N, PV, S, INV>(v[i], j % Ns, tw);
      } else {
        if constexpr (Ns > 1) {
          const int k = j % Ns;
          const double2* tp = tw + pass_tw_offset(N, PV, S);
#pragma unroll
          for (int r = 1; r < R; ++r) {
            double2 w = tp[(r - 1) * Ns + k];
            if (INV) w = cconj(w);
            v[i][r] = cmul(v[i][r], w);
          }
        }
        dft<R, INV>(v[i]);
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < BPT; ++i) {
    const int b = threadIdx.x + i * NT;
    if (b < total) {
      const int line = b / NB, j = b - line * NB;
      double2* dl = A + line * LS + (j / Ns) * Ns * R + (j % Ns);
#pragma unroll
      for (int r = 0; r < R; ++r) dl[r * Ns] = v[i][r];
    }
  }
  __syncthreads();
}

// The first pass with its inputs produced by ld(line, k) (k = position in the line)
// instead of read from shared memory; it writes its outputs in place into A, which
// nothing reads during the pass, so it needs no barrier between loads and stores.
// LINE_FAST: consecutive threads take consecutive lines at the same position
// (so that interleaved lines of a global array load together); otherwise
// consecutive positions of one line.
template <int N, bool INV, int NT, int NLMAX, bool LINE_FAST, int PV, class Load>
__device__ __forceinline__ void fft_pass_first(double2* A, int nl, int LS, const double2* __restrict__ tw, Load&& ld) {
  constexpr int R = radix_of(plan_of(N, PV).r[0]);
  constexpr int NB = N / R, PADE = pad_every(N, PV, LINE_FAST);
  constexpr int BPT = (NLMAX * NB + NT - 1) / NT;
  const int total = nl * NB;
#pragma unroll
  for (int i = 0; i < BPT; ++i) {
    const int b = threadIdx.x + i * NT;
    if (b < total) {
      const int line = LINE_FAST ? b % nl : b / NB;
      const int j = LINE_FAST ? b / nl : b - line * NB;
      double2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = ld(line, j + r * NB);
      if constexpr (plan_of(N, PV).r[0] >= 100) pass_butterfly<N, PV, 0, INV>(v, 0, tw);
      else dft<R, INV>(v);
      double2* dl = A + line * LS + j * R + (PADE ? j / PADE : 0);
#pragma unroll
      for (int r = 0; r < R; ++r) dl[r] = v[r];
    }
  }
  __syncthreads();
}

// passes S, S + 1, ... of plan variant PV; tw: the plan's tables; PADE as
// fft_pass's (of pass 1)
template <int N, int S, bool INV, int NT, int NLMAX, int PV = 0, int PADE = 0>
__device__ __forceinline__ void fft_passes(double2* A, int nl, int LS, const double2* tw) {
  if constexpr (S < plan_of(N, PV).nst) {
    fft_pass<N, PV, S, INV, NT, NLMAX, S == 1 ? PADE : 0>(A, nl, LS, tw);
    fft_passes<N, S + 1, INV, NT, NLMAX, PV, PADE>(A, nl, LS, tw);
  }
}

// Batched FFT of nl <= NLMAX lines (line stride LS >= line_len) by NT threads:
// compile-time length NC in place in A (B unused), or the runtime plan (NC == 0)
// ping-ponging through B.  Returns the buffer holding the result.  The inputs are
// produced by ld(line, k) (see fft_pass_first; runtime plans stage them in A
// first), so the caller need not synchronise before; it may read the result
// directly after.
template <int NC, bool INV, int NT, int NLMAX, bool LINE_FAST = false, int PV = 0, class Load>
__device__ __forceinline__ double2* fft_lines_ld(double2* A, double2* B, int nl, int LS, const FftPlan& p,
                                                 Load&& ld) {
  if constexpr (NC == 0) {
    for (int idx = threadIdx.x; idx < nl * p.N; idx += blockDim.x) {
      const int line = idx / p.N, k = idx - line * p.N;
      A[line * LS + k] = ld(line, k);
    }
    __syncthreads();
    return fft_lines<INV>(A, B, nl, LS, p);
  } else {
    static_assert(plan_of(NC, PV).nst > 0, "transform length must be 2^a 3^b");
    fft_pass_first<NC, INV, NT, NLMAX, LINE_FAST, PV>(A, nl, LS, p.tws[PV], ld);
    fft_passes<NC, 1, INV, NT, NLMAX, PV, pad_every(NC, PV, LINE_FAST)>(A, nl, LS, p.tws[PV]);
    return A;
  }
}

// The same of lines already in A (unpadded; the caller has synchronised)
template <int NC, bool INV, int NT, int NLMAX, int PV = 0>
__device__ __forceinline__ double2* fft_lines_n(double2* A, double2* B, int nl, int LS, const FftPlan& p) {
  if constexpr (NC == 0) {
    return fft_lines<INV>(A, B, nl, LS, p);
  } else {
    static_assert(plan_of(NC, PV).nst > 0, "transform length must be 2^a 3^b");
    fft_passes<NC, 0, INV, NT, NLMAX, PV>(A, nl, LS, p.tws[PV % 2]);
    return A;
  }
}

}  // namespace coral
