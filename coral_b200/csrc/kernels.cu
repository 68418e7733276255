// CUDA kernels (sm_100a, FP64) of the plane-layer IMEX timestep.
//
// Layouts (first index slowest, C order), identical in memory to the
// reference's Fortran arrays:
//   state       field[kx][ky][t]          (Fortran field(T, NYAA, NX/2))
//   spectral    spec [kx][ky][n]          (Fortran spec(NZ, NYAA, NX/2))
//   physical    phys [y][x][z]            (Fortran phys(NZAA, NXAA, NYAA))
// Transform intermediates (this build's own choice):
//   Y1 / Q1     [var][y][kx][n]  complex  (after the y transform / before it)
//   Y2 / Q2     [var][y][x][n]   real     (after the x transform / before it)
// The x<->y exchange of the reference's slab decomposition
// (src/slabs.fftw3mpi/domain_decomposition.f90:152-183) is the change of
// layout between the y pass and the x pass, done in shared memory.
#include <algorithm>
#include <cstdio>

#include <string>

#include "../../include/coral_b200.h"
#include "device.hpp"
#include "host.hpp"

namespace coral {

namespace {

constexpr int kNB1 = 4;  // n lines per CTA, inverse / forward y pass
constexpr int kNB2 = 8;  // n lines per CTA, x passes (packed in pairs)
constexpr int kXB3 = 16; // x columns per CTA, inverse z pass (packed in pairs)
constexpr int kQC = 5;   // quadratic variables per FFT batch, forward z pass (one radix-9 / radix-8
                         // butterfly per thread at NZAA = 288)
constexpr int kPadRt = 2;  // line stride N + 2 of the x / y passes with run-time plans
constexpr int kThreads = 256;
// x / y passes: threads per CTA for nl lines of a compiled length N, the most
// that any pass keeps busy, rounded up to whole warps: one butterfly per thread,
// of radix 2, 3 and 4 as many as make 8 or 9 elements (one radix-3 butterfly each
// left the radix-8 passes of 192 = 3 x 8 x 8 with 96 of 256 threads); 256 for the
// run-time plans
__host__ __device__ constexpr int xy_threads(int N, int nl, int pv) {
  if (N == 0) return 256;
  const PlanR p = plan_of(N, pv);
  int m = 32;
  for (int i = 0; i < p.nst; ++i) {
    const int r = radix_of(p.r[i]), per = r <= 4 ? 9 / r : 1, t = (nl * N / r + per - 1) / per;
    m = t > m ? t : m;
  }
  return (m + 31) / 32 * 32;
}
#define kThreadsX xy_threads(NF, kNB2 / 2, PV)
#define kThreadsY xy_threads(NF, 4, kPlanY)
// the pipelined forward y pass reads its first-pass inputs from shared memory:
// plan and threads of its own
constexpr int kPlanYF = 1;
#define kThreadsYF xy_threads(NF, 4, kPlanYF)
#define kMinBlocksYF (kPlanYF ? hot_min_blocks(kThreadsYF) : kMinBlocksY)
// CTAs per SM the kernels with two-pass plans are compiled for: registers
// capped at no fewer than 128 per thread
__host__ __device__ constexpr int hot_min_blocks(int nt) { return 65536 / (nt * 128) > 1 ? 65536 / (nt * 128) : 1; }
// CTAs per SM of the y passes: 3, measured best at 384^2 x 192; fewer where that
// would leave a thread under 64 registers
__host__ __device__ constexpr int y_min_blocks(int nt) { return 65536 / (nt * 64) < 3 ? 65536 / (nt * 64) : 3; }
#define kMinBlocksY y_min_blocks(kThreadsY)
// CTAs per SM of the separate forward z pass
constexpr int kMinBlocksZ = 4;
constexpr int kWPB = 8;  // warps (systems) per CTA in the per-system kernels

__device__ __forceinline__ double2 zero2() { return make_double2(0.0, 0.0); }

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// 16 bytes, or zeros when !valid (then gmem is not read)
__device__ __forceinline__ void cp_async16z(void* smem, const void* gmem, bool valid) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(n) : "memory");
}


// 32-byte global store of two adjacent complex values (256-bit vector access;
// the address must be 32-byte aligned).  (The matching 32-byte load, tried for
// the inverse x pass's packed rows, was slower than two 16-byte loads.)
__device__ __forceinline__ void st32(double2* p, double2 a, double2 b) {
  asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y) : "memory");
}
__device__ __forceinline__ bool aligned32(const void* p) { return ((size_t)p & 31) == 0; }

__device__ __forceinline__ double2 ipow(double k, int e) {
  // (i k)^e by repeated multiplication, as Fortran's complex**integer
  double2 r = make_double2(1.0, 0.0);
  double2 z = make_double2(0.0, k);
  for (int q = 0; q < e; ++q) r = cmul(r, z);
  return r;
}

// ------------------------------------------------------------------------------
// inverse transform, pass 1: spectral build of the full variables + y c2c (e^{+i})
// (compute_full_variables_in_physical_space, marching.f90:436-503, then
//  c2r_transform steps 1-2 and the 0.5 of the x padding, transforms.f90:172-198)
// ------------------------------------------------------------------------------
template <int NF>
__global__ void __launch_bounds__(kThreadsY, kMinBlocksY) k_inv_y(Dims d, const FullVarDev* fv, StateSet st,
                                                     const double2* plain_spec, const double* kxv,
                                                     const double* kyv, double2* Y1, FftPlan py) {
  extern __shared__ double2 sm[];
  const int f = blockIdx.x, n0 = blockIdx.y * kNB1, kx = blockIdx.z;
  const int NYA = NF ? NF : d.NYA, LS = NF ? line_stride(NF, kPlanY) : NYA + kPadRt;
  double2* A = sm;
  double2* B = sm + kNB1 * LS;  // runtime plan only
  // the CTA's build tables in shared memory: per term and line the stencil's
  // state indices and values, the term's state base at this kx and (i kx)^dx,
  // so that the state loads of the first pass depend on no global load
  __shared__ int s_tt[kMaxFullTerms][kNB1][kTabW];
  __shared__ double s_tv[kMaxFullTerms][kNB1][kTabW];
  __shared__ const double2* s_base[kMaxFullTerms];
  __shared__ double2 s_kxf[kMaxFullTerms];
  __shared__ int s_kt[kMaxFullTerms], s_zero[kMaxFullTerms], s_dx[kMaxFullTerms], s_dy[kMaxFullTerms];
  __shared__ double s_dsca[kMaxFullTerms];
  const int nterms = plain_spec ? 0 : fv[f].nterms;
  for (int e = threadIdx.x; e < nterms * kNB1 * kTabW; e += blockDim.x) {
    const int t = e / (kNB1 * kTabW), r = e - t * kNB1 * kTabW, ln = r / kTabW, k = r - ln * kTabW;
    const FullTermDev& ft = fv[f].term[t];
    const int n = n0 + ln;
    s_tt[t][ln][k] = n < d.NZ ? ft.tab_t[n * kTabW + k] : -1;
    s_tv[t][ln][k] = n < d.NZ ? ft.tab_v[n * kTabW + k] : 0.0;
  }
  if (threadIdx.x < nterms) {
    const int t = threadIdx.x;
    const FullTermDev& ft = fv[f].term[t];
    s_zero[t] = ft.zero_kind;
    s_dx[t] = ft.dx;
    s_dy[t] = ft.dy;
    s_dsca[t] = ft.dsca;
    s_kt[t] = ft.zero_kind ? 0 : st.kT[ft.set];
    s_base[t] = ft.zero_kind ? nullptr : st.k[ft.set] + (size_t)kx * NYA * st.kT[ft.set];
    s_kxf[t] = ipow(kxv[kx], ft.dx);
  }
  __syncthreads();
  // the spectral build of (line ln = Chebyshev n0 + ln, ky index iy), produced
  // inside the first FFT pass
  auto ld = [&](int ln, int iy) -> double2 {
    const int n = n0 + ln;
    double2 c = zero2();
    if (n < d.NZ) {
      if (plain_spec) {
        c = plain_spec[((size_t)kx * NYA + iy) * d.NZ + n];
      } else {
        for (int t = 0; t < nterms; ++t) {
          if (s_zero[t]) {
            if (kx == 0 && iy == 0) {
              const FullTermDev& ft = fv[f].term[t];
              const double* zs = st.z[ft.set];
              double s = 0.0;
              for (int k = 0; k < kTabW; ++k) {
                int tt = ft.tab_t[n * kTabW + k];
                if (tt >= 0) s += ft.tab_v[n * kTabW + k] * zs[tt];
              }
              c.x += s * ft.dsca;
            }
          } else {
            const double2* sv = s_base[t] + (size_t)iy * s_kt[t];
            double2 s = zero2();
#pragma unroll
            for (int k = 0; k < kTabW; ++k) {
              const int tt = s_tt[t][ln][k];
              if (tt >= 0) {
                const double w = s_tv[t][ln][k];
                const double2 x = sv[tt];
                s.x += w * x.x;
                s.y += w * x.y;
              }
            }
            s = cscale(s, s_dsca[t]);
            if (s_dx[t] || s_dy[t]) s = cmul(cmul(s, s_kxf[t]), ipow(kyv[iy], s_dy[t]));
            c = cadd(c, s);
          }
        }
      }
    }
    return c;
  };
  const double2* R = fft_lines_ld<NF, true, kThreadsY, kNB1, true, kPlanY>(A, B, kNB1, LS, py, ld);
  for (int idx = threadIdx.x; idx < kNB1 * NYA; idx += blockDim.x) {
    const int ln = idx % kNB1, y = idx / kNB1, n = n0 + ln;
    if (n < d.NZ) {
      const double s = (n == 0) ? 1.0 : 0.5;  // (x2 on Chebyshev index 0) * (0.5 of the x padding)
      Y1[(((size_t)f * NYA + y) * d.NXH + kx) * d.NZ + n] = cscale(R[ln * LS + y], s);
    }
  }
}

// The same pass for full variables whose terms are mean variables followed by
// exactly one kxky variable (the u, v, w, T of the plane-layer recipes): the
// mean terms reach only the (0,0) mode and are summed in the prologue, in term
// order, so that a position's build is one unrolled stencil whose state loads
// do not wait on a loop over terms, and all of a thread's loads in the first
// pass can be in flight at once.  The same arithmetic in the same order as
// k_inv_y (bit for bit).
template <int NF>
__global__ void __launch_bounds__(kThreadsY, kMinBlocksY) k_inv_y1(Dims d, const FullVarDev* fv, StateSet st,
                                                      const double* kxv, const double* kyv, double2* Y1, FftPlan py) {
  extern __shared__ double2 sm[];
  const int f = blockIdx.x, n0 = blockIdx.y * kNB1, kx = blockIdx.z;
  const int NYA = NF ? NF : d.NYA, LS = NF ? line_stride(NF, kPlanY) : NYA + kPadRt;
  double2* A = sm;
  double2* B = sm + kNB1 * LS;  // runtime plan only
  __shared__ int s_tt[kNB1][kTabW];
  __shared__ double s_tv[kNB1][kTabW];
  __shared__ double2 s_zc[kNB1];  // per line, the mean terms' sum at (kx, ky) = (0, 0)
  const int tk = fv[f].nterms - 1;  // the kxky term is the last
  const FullTermDev& ft = fv[f].term[tk];
  for (int e = threadIdx.x; e < kNB1 * kTabW; e += blockDim.x) {
    const int ln = e / kTabW, k = e - ln * kTabW, n = n0 + ln;
    s_tt[ln][k] = n < d.NZ ? ft.tab_t[n * kTabW + k] : -1;
    s_tv[ln][k] = n < d.NZ ? ft.tab_v[n * kTabW + k] : 0.0;
  }
  if (threadIdx.x < kNB1) {
    const int ln = threadIdx.x, n = n0 + ln;
    double2 c = zero2();
    if (kx == 0 && n < d.NZ) {
      for (int t = 0; t < tk; ++t) {  // the mean terms, as k_inv_y's build at iy = 0
        const FullTermDev& fz = fv[f].term[t];
        const double* zs = st.z[fz.set];
        double s = 0.0;
        for (int k = 0; k < kTabW; ++k) {
          const int tt = fz.tab_t[n * kTabW + k];
          if (tt >= 0) s += fz.tab_v[n * kTabW + k] * zs[tt];
        }
        c.x += s * fz.dsca;
      }
    }
    s_zc[ln] = c;
  }
  const int kt = st.kT[ft.set], dx = ft.dx, dy = ft.dy;
  const double2* base = st.k[ft.set] + (size_t)kx * NYA * kt;
  const double dsca = ft.dsca;
  const double2 kxf = ipow(kxv[kx], dx);
  __syncthreads();
  auto ld = [&](int ln, int iy) -> double2 {
    const int n = n0 + ln;
    double2 c = zero2();
    if (n < d.NZ) {
      if (kx == 0 && iy == 0) c = s_zc[ln];
      const double2* sv = base + (size_t)iy * kt;
      double2 s = zero2();
#pragma unroll
      for (int k = 0; k < kTabW; ++k) {
        const int tt = s_tt[ln][k];
        if (tt >= 0) {
          const double w = s_tv[ln][k];
          const double2 x = sv[tt];
          s.x += w * x.x;
          s.y += w * x.y;
        }
      }
      s = cscale(s, dsca);
      if (dx || dy) s = cmul(cmul(s, kxf), ipow(kyv[iy], dy));
      c = cadd(c, s);
    }
    return c;
  };
  const double2* R = fft_lines_ld<NF, true, kThreadsY, kNB1, true, kPlanY>(A, B, kNB1, LS, py, ld);
  // two adjacent Chebyshev rows per thread: one 32-byte store
  for (int idx = threadIdx.x; idx < (kNB1 / 2) * NYA; idx += blockDim.x) {
    const int l0 = 2 * (idx % (kNB1 / 2)), y = idx / (kNB1 / 2), n = n0 + l0;
    // (x2 on Chebyshev index 0) * (0.5 of the x padding)
    const double2 v0 = cscale(R[l0 * LS + y], (n == 0) ? 1.0 : 0.5);
    const double2 v1 = cscale(R[(l0 + 1) * LS + y], 0.5);
    double2* dst = Y1 + (((size_t)f * NYA + y) * d.NXH + kx) * d.NZ + n;
    if (n + 1 < d.NZ && aligned32(dst)) {
      st32(dst, v0, v1);
    } else {
      if (n < d.NZ) dst[0] = v0;
      if (n + 1 < d.NZ) dst[1] = v1;
    }
  }
}

// ------------------------------------------------------------------------------
// inverse transform, pass 2: x c2r with zero padding NX/2 -> NXAA (transforms.f90:197-210)
// two real output lines per complex FFT
// ------------------------------------------------------------------------------
template <int NF, int PV>
__global__ void __launch_bounds__(kThreadsX, hot_min_blocks(kThreadsX)) k_inv_x(Dims d, const double2* Y1, double* Y2, FftPlan px,
                                                                               int y0) {
  extern __shared__ double2 sm[];
  const int f = blockIdx.x, n0 = blockIdx.y * kNB2, y = y0 + blockIdx.z;
  const int NXA = NF ? NF : d.NXA, NP = kNB2 / 2, LS = NF ? line_stride(NF, PV) : NXA + kPadRt;
  double2* A = sm;
  double2* B = sm + NP * LS;  // runtime plan only
  // position p of line m (Chebyshev pair na, na+1): the Hermitian extension of
  // both coefficient rows packed as a + i b, zero padding in between; produced
  // inside the first FFT pass
  const double2* src0 = Y1 + ((size_t)f * d.NYA + y) * d.NXH * d.NZ;
  auto ld = [&](int m, int p) -> double2 {
    const int na = n0 + 2 * m;
    const bool lo = p < d.NXH, hi = p > NXA - d.NXH;  // kx = p, or kx = NXA - p (conjugate)
    if (!lo && !hi) return zero2();
    const int kx = lo ? p : NXA - p;
    const double2* src = src0 + (size_t)kx * d.NZ;
    const double2 a = (na < d.NZ) ? src[na] : zero2();
    const double2 b = (na + 1 < d.NZ) ? src[na + 1] : zero2();
    if (p == 0) return make_double2(a.x, b.x);  // c2r reads only the real part of the DC term
    return lo ? make_double2(a.x - b.y, a.y + b.x)    // a + i b
              : make_double2(a.x + b.y, b.x - a.y);   // conj(a) + i conj(b)
  };
  const double2* R = fft_lines_ld<NF, true, kThreadsX, kNB2 / 2, true, PV>(A, B, NP, LS, px, ld);
  for (int idx = threadIdx.x; idx < NP * NXA; idx += blockDim.x) {
    const int m = idx % NP, x = idx / NP, na = n0 + 2 * m;
    double2 z = R[m * LS + x];
    double* dst = Y2 + (((size_t)f * d.NYA + y) * NXA + x) * d.NZ;
    if (na + 1 < d.NZ && (d.NZ & 1) == 0) {
      *reinterpret_cast<double2*>(dst + na) = z;  // na and NZ even: one 16-byte store
    } else {
      if (na < d.NZ) dst[na] = z.x;
      if (na + 1 < d.NZ) dst[na + 1] = z.y;
    }
  }
}

// The same pass for compiled lengths with the two-pass plan, as a persistent
// kernel: each CTA walks the tiles (full variable, block of kNB2 Chebyshev rows,
// y) with a stride of the grid size; the next tile's input rows (kx < NX/2,
// kNB2 coefficients each) are copied into a staging buffer with cp.async while
// the current tile's second FFT pass and stores run (the first pass reads the
// staging buffer and frees it).  Staging rows are kNB2 + 1 16-byte words apart,
// so that the first pass's reads (4 lines x 2 positions a quarter warp) fall in
// distinct bank groups; the twiddles are in shared memory.  That (line buffer, staging,
// table) admits 3 CTAs per SM at NXAA = 576: registers are sized for 3.
constexpr int kStgX = kNB2 + 1;
#define kThreadsXP xy_threads(NF, kNB2 / 2, 1)
template <int NF>
__global__ void __launch_bounds__(kThreadsXP, 3) k_inv_x_pipe(Dims d, int nf, const double2* Y1,
                                                                                      double* Y2, FftPlan px) {
  constexpr int NT = kThreadsXP, NXA = NF, NP = kNB2 / 2;
  constexpr PlanR P = plan_of(NF, 1);
  constexpr int kTw2 = pass_tw_len(NF, 1);
  static_assert(P.nst == 2, "two-pass plan");
  extern __shared__ double2 sm[];
  __shared__ double2 s_tw[kTw2];
  constexpr int LS = line_stride(NF, 1);
  double2* A = sm;               // NP lines, stride LS
  double2* stg = A + NP * LS;    // staged input [kx][kStgX]
  const int NXH = d.NXH, NZ = d.NZ;
  const int nnb = (NZ + kNB2 - 1) / kNB2;
  const int ntiles = nf * nnb * d.NYA;
  for (int i = threadIdx.x; i < kTw2; i += NT) s_tw[i] = px.tws[1][i];  // read after the loop's first barrier
  auto issue = [&](int tile) {
    if (tile < ntiles) {
      const int f = tile % nf, r = tile / nf, nb = r % nnb, y = r / nnb, n0 = nb * kNB2;
      const double2* src = Y1 + ((size_t)f * d.NYA + y) * NXH * NZ + n0;
      for (int e = threadIdx.x; e < NXH * kNB2; e += NT) {
        const int kx = e / kNB2, ln = e - kx * kNB2;
        const bool ok = n0 + ln < NZ;
        cp_async16z(stg + kx * kStgX + ln, ok ? src + (size_t)kx * NZ + ln : Y1, ok);
      }
    }
    cp_async_commit();
  };
  issue(blockIdx.x);
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int f = tile % nf, r = tile / nf, nb = r % nnb, y = r / nnb, n0 = nb * kNB2;
    cp_async_wait<0>();
    __syncthreads();
    // position p of line m (Chebyshev pair 2m, 2m+1 of the block): as in k_inv_x
    auto ld = [&](int m, int p) -> double2 {
      const bool lo = p < NXH, hi = p > NXA - NXH;
      if (!lo && !hi) return zero2();
      const int kx = lo ? p : NXA - p;
      const double2 a = stg[kx * kStgX + 2 * m], b = stg[kx * kStgX + 2 * m + 1];
      if (p == 0) return make_double2(a.x, b.x);
      return lo ? make_double2(a.x - b.y, a.y + b.x) : make_double2(a.x + b.y, b.x - a.y);
    };
    fft_pass_first<NF, true, NT, NP, true, 1>(A, NP, LS, s_tw, ld);  // ends with a barrier
    issue(tile + gridDim.x);
    fft_passes<NF, 1, true, NT, NP, 1, pad_every(NF, 1, true)>(A, NP, LS, s_tw);
    double* dst0 = Y2 + ((size_t)f * d.NYA + y) * NXA * NZ;
    for (int idx = threadIdx.x; idx < NP * NXA; idx += NT) {
      const int m = idx % NP, x = idx / NP, na = n0 + 2 * m;
      const double2 z = A[m * LS + x];
      double* dst = dst0 + (size_t)x * NZ + na;
      if (na + 1 < NZ && (NZ & 1) == 0) {
        *reinterpret_cast<double2*>(dst) = z;  // na and NZ even: 16-byte aligned
      } else {
        if (na < NZ) dst[0] = z.x;
        if (na + 1 < NZ) dst[1] = z.y;
      }
    }
    __syncthreads();  // A is rewritten by the next tile's first pass
  }
  cp_async_wait<0>();
}

__device__ __forceinline__ void atomic_max_nonneg(unsigned long long* addr, double v) {
  atomicMax(addr, (unsigned long long)__double_as_longlong(v));
}

// Threads of the z kernels for nl lines of a compiled length N: enough for
// one butterfly per thread in the radix >= 8 passes and two in the radix-2/4
// passes (N = 288, 8 lines, plan 18 x 16: 160 threads).
__host__ __device__ constexpr int z_threads(int N, int nl, int pv = kPlanHot) {
  if (N == 0) return 256;
  const PlanR p = plan_of(N, pv);
  int m = 32;
  for (int i = 0; i < p.nst; ++i) {
    const int b = nl * N / radix_of(p.r[i]), per = (radix_of(p.r[i]) <= 4) ? (b + 1) / 2 : b;
    m = per > m ? per : m;
  }
  return (m + 31) / 32 * 32;
}

// ------------------------------------------------------------------------------
// inverse transform, pass 3: z REDFT01 with zero padding NZ -> NZAA (transforms.f90:216-223)
// via an NZAA-point complex FFT (two columns per FFT); also the CFL maxima of
// compute_cfl_based_timestep (marching.f90:219-238) for the first three full variables
// ------------------------------------------------------------------------------
#define kThreadsIZ z_threads(NF, kXB3 / 2, kPlanInvZ)
template <int NF>
__global__ void __launch_bounds__(kThreadsIZ, hot_min_blocks(kThreadsIZ)) k_inv_z(Dims d, const double* Y2, double* phys,
                                                                                 FftPlan pz, const double2* dct_tw,
                                                                                 const double* wz,
                                                                                 unsigned long long* cfl_bits) {
  constexpr int NT = kThreadsIZ;
  extern __shared__ double2 sm[];
  __shared__ double red[NT / 32];
  const int f = blockIdx.x, x0 = blockIdx.y * kXB3, y = blockIdx.z;
  const int N = NF ? NF : d.NZA, NP = kXB3 / 2, LZ = NF ? line_len(NF, kPlanInvZ, false) : N;
  double2* A = sm;
  double2* B = sm + NP * LZ;  // runtime plan only
  const double* src0 = Y2 + (((size_t)f * d.NYA + y) * d.NXA + x0) * d.NZ;
  // X_n and X_{N-n} of the pair's columns, twiddled, packed as va + i vb, produced
  // inside the first FFT pass (as in the fused kernel)
  auto ld = [&](int m, int n) -> double2 {
    const double* sa = src0 + (size_t)(2 * m) * d.NZ;
    const double* sb = sa + d.NZ;
    const bool ha = x0 + 2 * m < d.NXA, hb = x0 + 2 * m + 1 < d.NXA, lo = n < d.NZ, hi = n > 0 && N - n < d.NZ;
    const double a0 = (lo && ha) ? sa[n] : 0.0, a1 = (hi && ha) ? sa[N - n] : 0.0;
    const double b0 = (lo && hb) ? sb[n] : 0.0, b1 = (hi && hb) ? sb[N - n] : 0.0;
    const double2 w = cconj(dct_tw[n]);  // exp(+i pi n / 2N)
    const double2 va = cmul(w, make_double2(a0, -a1));
    const double2 vb = cmul(w, make_double2(b0, -b1));
    return make_double2(va.x - vb.y, va.y + vb.x);
  };
  const double2* R = fft_lines_ld<NF, true, NT, kXB3 / 2, false, kPlanInvZ>(A, B, NP, LZ, pz, ld);
  double mx = 0.0;
  const int which = (f < 3) ? f : -1;
  for (int idx = threadIdx.x; idx < NP * N; idx += blockDim.x) {
    const int m = idx / N, k = idx - m * N;
    const int xa = x0 + 2 * m, xb = xa + 1;
    const int zi = (k & 1) ? (N - 1 - (k >> 1)) : (k >> 1);
    const double2 z = R[m * LZ + zi];
    double* dst = phys + (((size_t)f * d.NYA + y) * d.NXA + xa) * N;
    if (xa < d.NXA) dst[k] = z.x;
    if (xb < d.NXA) dst[N + k] = z.y;
    if (which >= 0) {
      double s = (which == 2) ? 1.0 / wz[k] : 1.0;
      if (xa < d.NXA) mx = fmax(mx, fabs(z.x) * s);
      if (xb < d.NXA) mx = fmax(mx, fabs(z.y) * s);
    }
  }
  if (cfl_bits && which >= 0) {
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
      double m2 = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m2 = fmax(m2, red[w]);
      atomic_max_nonneg(cfl_bits + which, m2);
    }
  }
}

// ------------------------------------------------------------------------------
// forward transform, pass 1: pointwise products (marching.f90:279-291) + z REDFT10
// truncated to NZ (transforms.f90:243-249), for all quadratic variables of one
// pair of x columns; also partial volume averages for KE (output.f90:84-102)
// ------------------------------------------------------------------------------
template <int NF>
__global__ void __launch_bounds__(kThreads, kMinBlocksZ) k_fwd_z(Dims d, int nf, QuadDesc q, const double* phys, double* Q2,
                                                     FftPlan pz, const double2* dct_tw, const double* wz,
                                                     double* ke_partial) {
  extern __shared__ double2 sm[];
  __shared__ double red[3][kThreads / 32];
  const int x0 = blockIdx.x * 2, y = blockIdx.y;
  const int N = NF ? NF : d.NZA, nq = q.nq, nb = min(nq, kQC);
  double* P = reinterpret_cast<double*>(sm);  // [nf][2][N], z in Makhoul order
  double2* A = sm + nf * N;                    // nb lines
  double2* B = A + nb * N;                     // runtime plan only
  for (int idx = threadIdx.x; idx < nf * 2 * N; idx += blockDim.x) {
    const int fv = idx / (2 * N), r = idx - fv * 2 * N;
    const int c = r / N, z = r - c * N;
    const int m = (z & 1) ? (N - 1 - (z >> 1)) : (z >> 1);  // Makhoul position of z
    const int xc = x0 + c;
    P[idx - z + m] = (xc < d.NXA) ? phys[(((size_t)fv * d.NYA + y) * d.NXA + xc) * N + z] : 0.0;
  }
  __syncthreads();
  double ke[3] = {0.0, 0.0, 0.0};
  for (int q0 = 0; q0 < nq; q0 += kQC) {  // batches of kQC quadratic variables
    const int nc = min(kQC, nq - q0);
    for (int idx = threadIdx.x; idx < nc * N; idx += blockDim.x) {
      const int qi = idx / N, m = idx - qi * N, qg = q0 + qi;
      const int z = (m < N / 2) ? 2 * m : 2 * (N - 1 - m) + 1;  // Makhoul reordering
      const int v1 = q.v1[qg], v2 = q.v2[qg];
      double pa, pb;
      if (v1 < 0) { pa = P[(v2 * 2) * N + m]; pb = P[(v2 * 2 + 1) * N + m]; }
      else if (v2 < 0) { pa = P[(v1 * 2) * N + m]; pb = P[(v1 * 2 + 1) * N + m]; }
      else {
        pa = P[(v1 * 2) * N + m] * P[(v2 * 2) * N + m];
        pb = P[(v1 * 2 + 1) * N + m] * P[(v2 * 2 + 1) * N + m];
      }
      if (ke_partial) {
        for (int j = 0; j < 3; ++j)
          if (q.ke_q[j] == qg) ke[j] += wz[z] * (pa + ((x0 + 1 < d.NXA) ? pb : 0.0));
      }
      if (q.tau) {  // learned subgrid part of this quadratic variable
        const double* tq = q.tau + (((size_t)qg * d.NYA + y) * d.NXA + x0) * N + z;
        pa += tq[0];
        if (x0 + 1 < d.NXA) pb += tq[N];
      }
      A[qi * N + m] = make_double2(pa, pb);
    }
    __syncthreads();
    const double2* R = fft_lines_n<NF, false, kThreads, kQC, kPlanFZ>(A, B, nc, N, pz);
    for (int idx = threadIdx.x; idx < nc * d.NZ; idx += blockDim.x) {
      const int qi = idx / d.NZ, n = idx - qi * d.NZ;
      const double2 Z = R[qi * N + n];
      const double2 Zc = cconj(R[qi * N + ((N - n) % N)]);
      const double2 va = make_double2(0.5 * (Z.x + Zc.x), 0.5 * (Z.y + Zc.y));
      const double2 dd = csub(Z, Zc);
      const double2 vb = make_double2(0.5 * dd.y, -0.5 * dd.x);  // (Z - Zc) / 2i
      const double2 w = dct_tw[n];                                // exp(-i pi n / 2N)
      const double xa = 2.0 * (w.x * va.x - w.y * va.y);
      const double xb = 2.0 * (w.x * vb.x - w.y * vb.y);
      double* dst = Q2 + (((size_t)(q0 + qi) * d.NYA + y) * d.NXA + x0) * d.NZ;
      dst[n] = xa;
      if (x0 + 1 < d.NXA) dst[d.NZ + n] = xb;
    }
    __syncthreads();  // A is refilled by the next batch
  }
  if (ke_partial) {
    for (int j = 0; j < 3; ++j) {
      double v = ke[j];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if ((threadIdx.x & 31) == 0) red[j][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
      double s = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[threadIdx.x][w];
      ke_partial[((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 3 + threadIdx.x] = s;
    }
  }
}

// ------------------------------------------------------------------------------
// z passes of one stage fused: z REDFT01 of the full variables (transforms.f90:
// 216-223), the CFL maxima (marching.f90:219-238), the pointwise products
// (marching.f90:279-291), the KE partial averages (output.f90:84-102) and the z
// REDFT10 of the quadratic variables (transforms.f90:243-249), for one pair of
// x columns; the physical fields never leave shared memory.  The inverse
// transform leaves the physical values in Makhoul order (position m holds
// z = 2m, or 2(N-1-m)+1 for m >= N/2), which is the order the forward transform
// takes, so the products are formed position by position.
// ------------------------------------------------------------------------------

constexpr int kZPairs = 2;               // x-column pairs per CTA
constexpr int kZLines = 4 * kZPairs;     // lines per inverse FFT batch (4 full variables x 2 pairs)
// lines per forward FFT batch ((quadratic variable, pair) lines), the kernel's
// FB: 9 (two batches for 9 quadratic variables; 2 CTAs per SM at NZAA = 288) or
// 6 (three batches; shared memory and registers for 3 CTAs per SM)
constexpr int kZFwd = 9;
__host__ __device__ constexpr int z_threads_fused(int N, int fb) {
  return z_threads(N, kZLines) > z_threads(N, fb) ? z_threads(N, kZLines) : z_threads(N, fb);
}
__host__ __device__ constexpr int z_min_blocks(int N, int fb) {
  const int hot = hot_min_blocks(z_threads_fused(N, fb));
  return fb < kZFwd && hot > 3 ? 3 : hot;
}
#define kThreadsZF z_threads_fused(NF, FB)

template <int NF, int FB>
__global__ void __launch_bounds__(kThreadsZF, z_min_blocks(NF, FB)) k_z_fused(Dims d, int nf, QuadDesc q, const double* Y2,
                                                                       double* Q2, FftPlan pz, const double2* dct_tw,
                                                                       const double* wz, const double* wzinv,
                                                                       unsigned long long* cfl_bits, double* ke_partial,
                                                                       int y0) {
  constexpr int NT = kThreadsZF;
  extern __shared__ double2 sm[];
  __shared__ double red[3][(NT + 31) / 32];
  __shared__ int qv[2][kMaxQuad];
  const int x0 = blockIdx.x * 2 * kZPairs, y = y0 + blockIdx.y;
  const size_t cta = (size_t)y * gridDim.x + blockIdx.x;  // row of the KE and timeseries partial sums
  // compiled lengths: NZAA = 3 NZ / 2 (the launcher checks it)
  const int N = NF ? NF : d.NZA, NZ = NF ? 2 * NF / 3 : d.NZ;
  const int LZ = NF ? line_len(NF, kPlanHot, false) : N;  // line stride
  const int nq = q.nq;
  const size_t vstride = (size_t)d.NYA * d.NXA * NZ;  // between variables of Y2 / Q2
  const size_t col0 = ((size_t)y * d.NXA + x0) * NZ;  // column x0 of variable 0
  if (threadIdx.x < kMaxQuad) {
    qv[0][threadIdx.x] = q.v1[threadIdx.x];
    qv[1][threadIdx.x] = q.v2[threadIdx.x];
  }
  // compiled lengths: the FFT's pass tables and the DCT twiddles in shared memory
  constexpr int kTw = NF ? pass_tw_len(NF, kPlanHot) : 0;
  __shared__ double2 s_tw[kTw ? kTw : 1], s_dtw[NF ? NF : 1];
  FftPlan pzl = pz;
  const double2* dtw = dct_tw;
  if constexpr (NF != 0) {
    for (int i = threadIdx.x; i < kTw; i += blockDim.x) s_tw[i] = pz.tws[kPlanHot][i];
    for (int i = threadIdx.x; i < NF; i += blockDim.x) s_dtw[i] = dct_tw[i];
    pzl.tws[kPlanHot] = s_tw;
    dtw = s_dtw;
  }
  // line l of a batch: variable l / kZPairs, column pair l % kZPairs (columns
  // x0 + 2p (re) and x0 + 2p + 1 (im))
  auto col_ok = [&](int c) { return x0 + c < d.NXA; };
  double2* Fv = sm;                   // nf * kZPairs lines of the full variables
  double2* A = Fv + nf * kZPairs * LZ; // FB lines of quadratic variables
  double2* B = A + FB * LZ;           // runtime plan only (max(kZLines, FB) lines)
  // ---- inverse: X_n and X_{N-n} of both columns, twiddled, packed as va + i vb,
  //      produced inside the first FFT pass ----
  __syncthreads();  // qv
  for (int l0 = 0; l0 < nf * kZPairs; l0 += kZLines) {
    const int nl = min(kZLines, nf * kZPairs - l0);
    auto ld = [&](int line, int n) -> double2 {
      const int lg = l0 + line, f = lg / kZPairs, pr = lg - f * kZPairs;
      const bool ha = col_ok(2 * pr), hb = col_ok(2 * pr + 1);
      const double* sa = Y2 + f * vstride + col0 + (size_t)(2 * pr) * NZ;
      const double* sb = sa + NZ;
      const bool lo = n < NZ, hi = n > 0 && N - n < NZ;
      const double a0 = (lo && ha) ? sa[n] : 0.0, a1 = (hi && ha) ? sa[N - n] : 0.0;
      const double b0 = (lo && hb) ? sb[n] : 0.0, b1 = (hi && hb) ? sb[N - n] : 0.0;
      const double2 w = cconj(dtw[n]);  // exp(+i pi n / 2N)
      const double2 va = cmul(w, make_double2(a0, -a1));
      const double2 vb = cmul(w, make_double2(b0, -b1));
      return make_double2(va.x - vb.y, va.y + vb.x);
    };
    const double2* R = fft_lines_ld<NF, true, NT, kZLines, false, kPlanHot>(Fv + l0 * LZ, B, nl, LZ, pzl, ld);
    if (R != Fv + l0 * LZ) {  // runtime plan with the result in the scratch lines
      for (int idx = threadIdx.x; idx < nl * N; idx += blockDim.x) Fv[l0 * LZ + idx] = R[idx];
      __syncthreads();
    }
  }
  // full variables with given physical values replace their transforms
  if (q.st_n > 0) {
    for (int k = 0; k < q.st_n; ++k) {
      const double* src = q.st_src[k];
      const int f = q.st_var[k], prof = q.st_prof[k];
      for (int idx = threadIdx.x; idx < kZPairs * N; idx += blockDim.x) {
        const int pr = idx / N, m = idx - pr * N;
        const int z = (m < N / 2) ? 2 * m : 2 * (N - 1 - m) + 1;
        double a = 0.0, b = 0.0;
        if (prof) {
          a = b = src[z];
        } else {
          const size_t at = ((size_t)y * d.NXA + x0 + 2 * pr) * N + z;
          if (col_ok(2 * pr)) a = src[at];
          if (col_ok(2 * pr + 1)) b = src[at + N];
        }
        Fv[(f * kZPairs + pr) * LZ + m] = make_double2(a, b);
      }
    }
    __syncthreads();
  }
  // ---- CFL maxima of |u|, |v|, |w| / wz and the KE sums (z-weighted products
  //      of the quadratic variables uu, vv, ww) over all columns, from the
  //      physical values (Makhoul order: position m is grid point z) ----
  if (cfl_bits || ke_partial) {
    const int ncf = cfl_bits ? min(nf, 3) : 0;
    double mx[3] = {0.0, 0.0, 0.0}, ke[3] = {0.0, 0.0, 0.0};
    for (int idx = threadIdx.x; idx < kZPairs * N; idx += blockDim.x) {
      const int pr = idx / N, m = idx - pr * N;
      const bool oka = col_ok(2 * pr), okb = col_ok(2 * pr + 1);
      const int z = (m < N / 2) ? 2 * m : 2 * (N - 1 - m) + 1;
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (j < ncf) {
          const double2 v = Fv[(j * kZPairs + pr) * LZ + m];
          const double s = (j == 2) ? wzinv[z] : 1.0;
          double a = oka ? fabs(v.x) * s : 0.0;
          if (okb) a = fmax(a, fabs(v.y) * s);
          mx[j] = fmax(mx[j], a);
        }
      if (ke_partial) {
        const double w = wz[z];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const int qg = q.ke_q[j];
          if (qg < 0) continue;
          const int v1 = qv[0][qg], v2 = qv[1][qg];
          double pa, pb;
          if (v1 < 0 || v2 < 0) {
            const double2 f1 = Fv[((v1 < 0 ? v2 : v1) * kZPairs + pr) * LZ + m];
            pa = f1.x;
            pb = f1.y;
          } else {
            const double2 f1 = Fv[(v1 * kZPairs + pr) * LZ + m], f2 = Fv[(v2 * kZPairs + pr) * LZ + m];
            pa = f1.x * f2.x;
            pb = f1.y * f2.y;
          }
          ke[j] += w * ((oka ? pa : 0.0) + (okb ? pb : 0.0));
        }
      }
    }
    if (cfl_bits) {
      for (int j = 0; j < 3; ++j) {
        double v = mx[j];
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        if ((threadIdx.x & 31) == 0) red[j][threadIdx.x >> 5] = v;
      }
      __syncthreads();
      if (threadIdx.x < ncf) {
        double m2 = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m2 = fmax(m2, red[threadIdx.x][w]);
        atomic_max_nonneg(cfl_bits + threadIdx.x, m2);
      }
      __syncthreads();
    }
    if (ke_partial) {
      for (int j = 0; j < 3; ++j) {
        double v = ke[j];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) red[j][threadIdx.x >> 5] = v;
      }
      __syncthreads();
      if (threadIdx.x < 3) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[threadIdx.x][w];
        ke_partial[cta * 3 + threadIdx.x] = s;
      }
      __syncthreads();
    }
    // timeseries objects, one at a time (one accumulator register)
    if (ke_partial && q.ts_partial) {
      for (int o = 0; o < q.ts_n; ++o) {
        const int src = q.ts_src[o], zsel = q.ts_z[o];
        const int fa = src >= 0 ? src : qv[0][-1 - src], fb = src >= 0 ? -1 : qv[1][-1 - src];
        double acc = 0.0;
        for (int idx = threadIdx.x; idx < kZPairs * N; idx += blockDim.x) {
          const int pr = idx / N, m = idx - pr * N;
          const int z = (m < N / 2) ? 2 * m : 2 * (N - 1 - m) + 1;
          if (zsel >= 0 && z != zsel) continue;
          double pa, pb;
          if (fa < 0 || fb < 0) {
            const double2 f1 = Fv[((fa < 0 ? fb : fa) * kZPairs + pr) * LZ + m];
            pa = f1.x;
            pb = f1.y;
          } else {
            const double2 f1 = Fv[(fa * kZPairs + pr) * LZ + m], f2 = Fv[(fb * kZPairs + pr) * LZ + m];
            pa = f1.x * f2.x;
            pb = f1.y * f2.y;
          }
          const double w = zsel >= 0 ? 1.0 : wz[z];
          acc += w * ((col_ok(2 * pr) ? pa : 0.0) + (col_ok(2 * pr + 1) ? pb : 0.0));
        }
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
        if ((threadIdx.x & 31) == 0) red[0][threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
          double s = 0.0;
          for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[0][w];
          q.ts_partial[cta * kMaxTs + o] = s;
        }
        __syncthreads();
      }
    }
  }
  // ---- products and forward transforms, FB (quadratic variable, pair) lines a batch ----
  for (int l0 = 0; l0 < nq * kZPairs; l0 += FB) {
    const int nc = min(FB, nq * kZPairs - l0);
    // products formed inside the first FFT pass
    auto ld = [&](int line, int m) -> double2 {
      const int lg = l0 + line, qg = lg / kZPairs, pr = lg - qg * kZPairs;
      const int v1 = qv[0][qg], v2 = qv[1][qg];
      double pa, pb;
      if (v1 < 0 || v2 < 0) {
        const double2 f1 = Fv[((v1 < 0 ? v2 : v1) * kZPairs + pr) * LZ + m];
        pa = f1.x;
        pb = f1.y;
      } else {
        const double2 f1 = Fv[(v1 * kZPairs + pr) * LZ + m], f2 = Fv[(v2 * kZPairs + pr) * LZ + m];
        pa = f1.x * f2.x;
        pb = f1.y * f2.y;
      }
      return make_double2(pa, pb);
    };
    const double2* R = fft_lines_ld<NF, false, NT, FB, false, kPlanHot>(A, B, nc, LZ, pzl, ld);
    // coefficient n of the two packed columns from Z = R[n] and conj(R[N - n]);
    // coefficients n and N - n share those two loads: items n = 0 .. N/2 write
    // n (< NZ) and, for 0 < n < N/2, N - n when it is < NZ
    const int NH = N / 2 + 1;
    for (int idx = threadIdx.x; idx < nc * NH; idx += blockDim.x) {
      const int li = idx / NH, n = idx - li * NH;
      const int lg = l0 + li, qg = lg / kZPairs, pr = lg - qg * kZPairs;
      const int n2 = (n == 0) ? 0 : N - n;
      const double2 Z = R[li * LZ + n], W = R[li * LZ + n2];
      double* dst = Q2 + qg * vstride + col0 + (size_t)(2 * pr) * NZ;
      const bool oa = col_ok(2 * pr), ob = col_ok(2 * pr + 1);
      auto out = [&](int k, double2 P, double2 Pm) {  // coefficient k from R[k] = P, R[N - k] = Pm
        const double2 Pc = cconj(Pm);
        const double2 va = make_double2(0.5 * (P.x + Pc.x), 0.5 * (P.y + Pc.y));
        const double2 dd = csub(P, Pc);
        const double2 vb = make_double2(0.5 * dd.y, -0.5 * dd.x);  // (P - Pc) / 2i
        const double2 w = dtw[k];                                   // exp(-i pi k / 2N)
        if (oa) dst[k] = 2.0 * (w.x * va.x - w.y * va.y);
        if (ob) dst[NZ + k] = 2.0 * (w.x * vb.x - w.y * vb.y);
      };
      if (n < NZ) out(n, Z, W);
      if (n > 0 && n2 != n && n2 < NZ) out(n2, W, Z);
    }
    __syncthreads();  // A is refilled by the next batch
  }
}

// ------------------------------------------------------------------------------
// forward transform, pass 2: x r2c, keep kx < NX/2 (transforms.f90:255-267)
// ------------------------------------------------------------------------------
template <int NF, int PV>
__global__ void __launch_bounds__(kThreadsX, hot_min_blocks(kThreadsX)) k_fwd_x(Dims d, const double* Q2, double2* Q1, FftPlan px,
                                                                               int y0) {
  extern __shared__ double2 sm[];
  const int qi = blockIdx.x, n0 = blockIdx.y * kNB2, y = y0 + blockIdx.z;
  const int NXA = NF ? NF : d.NXA, NP = kNB2 / 2, LS = NF ? line_stride(NF, PV) : NXA + kPadRt;
  double2* A = sm;
  double2* B = sm + NP * LS;  // runtime plan only
  // rows na, na+1 of column x packed as one complex value, produced inside the
  // first FFT pass
  const double* src0 = Q2 + ((size_t)qi * d.NYA + y) * NXA * d.NZ;
  auto ld = [&](int m, int x) -> double2 {
    const int na = n0 + 2 * m;
    const double* src = src0 + (size_t)x * d.NZ;
    if (na + 1 < d.NZ && (d.NZ & 1) == 0) return *reinterpret_cast<const double2*>(src + na);  // 16-byte aligned
    return make_double2(na < d.NZ ? src[na] : 0.0, na + 1 < d.NZ ? src[na + 1] : 0.0);
  };
  const double2* R = fft_lines_ld<NF, false, kThreadsX, kNB2 / 2, true, PV>(A, B, NP, LS, px, ld);
  for (int idx = threadIdx.x; idx < NP * d.NXH; idx += blockDim.x) {
    const int m = idx % NP, kx = idx / NP, na = n0 + 2 * m;
    const double2 Z = R[m * LS + kx];
    const double2 Zc = cconj(R[m * LS + ((NXA - kx) % NXA)]);
    const double2 a = make_double2(0.5 * (Z.x + Zc.x), 0.5 * (Z.y + Zc.y));
    const double2 dd = csub(Z, Zc);
    const double2 b = make_double2(0.5 * dd.y, -0.5 * dd.x);
    double2* dst = Q1 + (((size_t)qi * d.NYA + y) * d.NXH + kx) * d.NZ;
    if (na + 1 < d.NZ && aligned32(dst + na)) {
      st32(dst + na, a, b);  // rows na, na + 1: one 32-byte store
    } else {
      if (na < d.NZ) dst[na] = a;
      if (na + 1 < d.NZ) dst[na + 1] = b;
    }
  }
}

// ------------------------------------------------------------------------------
// forward transform, pass 3: y c2c (e^{-i}), x0.5 on Chebyshev index 0 and the
// 1/(NXAA NYAA NZAA) normalisation (transforms.f90:280-296)
// ------------------------------------------------------------------------------
template <int NF>
__global__ void __launch_bounds__(kThreadsY, kMinBlocksY) k_fwd_y(Dims d, const double2* Q1, double2* qspec, double scale,
                                                     FftPlan py) {
  extern __shared__ double2 sm[];
  const int qi = blockIdx.x, n0 = blockIdx.y * kNB1, kx = blockIdx.z;
  const int NYA = NF ? NF : d.NYA, LS = NF ? line_stride(NF, kPlanY) : NYA + kPadRt;
  double2* A = sm;
  double2* B = sm + kNB1 * LS;  // runtime plan only
  // produced inside the first FFT pass
  auto ld = [&](int ln, int y) -> double2 {
    const int n = n0 + ln;
    double2 v = zero2();
    if (n < d.NZ) {
      v = Q1[(((size_t)qi * NYA + y) * d.NXH + kx) * d.NZ + n];
      if (n == 0) v = cscale(v, 0.5);
    }
    return v;
  };
  const double2* R = fft_lines_ld<NF, false, kThreadsY, kNB1, true, kPlanY>(A, B, kNB1, LS, py, ld);
  for (int idx = threadIdx.x; idx < kNB1 * NYA; idx += blockDim.x) {
    const int ln = idx % kNB1, ky = idx / kNB1, n = n0 + ln;
    if (n < d.NZ) qspec[(((size_t)qi * d.NXH + kx) * NYA + ky) * d.NZ + n] = cscale(R[ln * LS + ky], scale);
  }
}

// The same pass for compiled lengths as a persistent kernel: each CTA walks the
// tiles (quadratic variable, block of kNB1 Chebyshev rows, kx) with a stride of
// the grid size; the next tile's input is copied into a staging buffer with
// cp.async while the current tile's later FFT passes and stores run (the first
// pass reads the staging buffer and frees it).
template <int NF>
__global__ void __launch_bounds__(kThreadsYF, kMinBlocksYF) k_fwd_y_pipe(Dims d, int nq, const double2* Q1,
                                                                        double2* qspec, double scale, FftPlan py) {
  extern __shared__ double2 sm[];
  constexpr int NYA = NF;
  constexpr int LS = line_stride(NF, kPlanYF);
  double2* A = sm;                 // kNB1 lines, stride LS
  double2* stg = A + kNB1 * LS;    // staged input [y][kNB1]
  const int nnb = (d.NZ + kNB1 - 1) / kNB1;
  const int ntiles = nq * nnb * d.NXH;
  const size_t ystride = (size_t)d.NXH * d.NZ;
  auto issue = [&](int tile) {
    if (tile < ntiles) {
      const int qi = tile % nq, r = tile / nq, nb = r % nnb, kx = r / nnb, n0 = nb * kNB1;
      const double2* src = Q1 + ((size_t)qi * NYA * d.NXH + kx) * d.NZ + n0;
      for (int e = threadIdx.x; e < NYA * kNB1; e += blockDim.x) {
        const int y = e / kNB1, ln = e - y * kNB1;
        const bool ok = n0 + ln < d.NZ;
        cp_async16z(stg + e, ok ? src + y * ystride + ln : Q1, ok);
      }
    }
    cp_async_commit();
  };
  issue(blockIdx.x);
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int qi = tile % nq, r = tile / nq, nb = r % nnb, kx = r / nnb, n0 = nb * kNB1;
    cp_async_wait<0>();
    __syncthreads();
    auto ld = [&](int ln, int y) -> double2 {
      const double2 v = stg[y * kNB1 + ln];
      return (n0 + ln == 0) ? cscale(v, 0.5) : v;
    };
    fft_pass_first<NF, false, kThreadsYF, kNB1, true, kPlanYF>(A, kNB1, LS, py.tws[kPlanYF], ld);  // ends with a barrier
    issue(tile + gridDim.x);
    fft_passes<NF, 1, false, kThreadsYF, kNB1, kPlanYF, pad_every(NF, kPlanYF, true)>(A, kNB1, LS, py.tws[kPlanYF]);
    // two adjacent Chebyshev rows per thread: one 32-byte store
    for (int idx = threadIdx.x; idx < (kNB1 / 2) * NYA; idx += blockDim.x) {
      const int l0 = 2 * (idx % (kNB1 / 2)), ky = idx / (kNB1 / 2), n = n0 + l0;
      const double2 v0 = cscale(A[l0 * LS + ky], scale), v1 = cscale(A[(l0 + 1) * LS + ky], scale);
      double2* dst = qspec + (((size_t)qi * d.NXH + kx) * NYA + ky) * d.NZ + n;
      if (n + 1 < d.NZ && aligned32(dst)) {
        st32(dst, v0, v1);
      } else {
        if (n < d.NZ) dst[0] = v0;
        if (n + 1 < d.NZ) dst[1] = v1;
      }
    }
    __syncthreads();  // A is rewritten by the next tile's first pass
  }
  cp_async_wait<0>();
}

// remove_vertical_mean_of_quadratic_var (PL_IMEX_timestepping.f90:223-235)
__global__ void k_remove_zmean(Dims d, double2* qs) {
  const size_t col = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= (size_t)d.NXH * d.NYA) return;
  double2* s = qs + col * d.NZ;
  double2 acc = zero2();
  for (int q = 1; q <= d.NZ / 2 - 1; ++q) {
    const double c = 0.5 / (2.0 * q + 1.0) - 0.5 / (2.0 * q - 1.0);
    acc = csub(acc, cscale(s[2 * q], c));
  }
  s[0] = acc;
}

// ------------------------------------------------------------------------------
// NL assembly K_hat = sum_terms (i kx)^a (i ky)^b dsca trunc(I^Iz M^mz) qhat,
// inserted in the interleaved ordering (marching.f90:319-367); zero for dealiased
// modes and (0,0).  One warp per (kx,ky) system.
// ------------------------------------------------------------------------------
__global__ void __launch_bounds__(kWPB * 32) k_nl(NLArgs a) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sid = blockIdx.x * kWPB + warp;
  const int nsys = a.d.NXH * a.d.NYA;
  if (sid >= nsys) return;
  const int kx = sid / a.d.NYA, ky = sid - kx * a.d.NYA;
  const bool act = a.act_index[sid] >= 0;
  double2 coef[kMaxGroups];
#pragma unroll
  for (int g = 0; g < kMaxGroups; ++g)
    coef[g] = (g < a.NL.ngroups) ? cmul(ipow(a.kx[kx], a.NL.gkx[g]), ipow(a.ky[ky], a.NL.gky[g])) : zero2();
  double2* out = a.Khat + (size_t)sid * a.T;
  const int NZ = a.d.NZ;
  for (int t = lane; t < a.T; t += 32) {
    double2 acc = zero2();
    for (int k = 0; act && k < a.NL.width; ++k) {
      const double v = a.NL.v(t, k);
      if (v == 0.0) break;  // slots are filled in order; exact zeros are not stored
      const int c = a.NL.col(t, k);
      const int qv = c / NZ, n = c - qv * NZ;
      const double2 qh = a.qspec[(((size_t)qv * a.d.NXH + kx) * a.d.NYA + ky) * NZ + n];
      double2 cv = coef[0];
      const int g = a.NL.grp(t, k);
#pragma unroll
      for (int gg = 1; gg < kMaxGroups; ++gg)
        if (g == gg) cv = coef[gg];
      acc = cadd(acc, cmul(cv, make_double2(v * qh.x, v * qh.y)));
    }
    out[t] = acc;
  }
}

// ------------------------------------------------------------------------------
// stage update and banded solve, one warp per (kx,ky) system
//   rhs = M field + sum_{j<i} dt a(i,j) Kstd_j + dt ahat(i+1,j) Khat_j + dt ahat(i+1,i) Khat_i
//   aux = E^{-1} rhs  (E = identity for dealiased modes; (0,0): M is empty)
//   Kstd_i = L aux    (zero for dealiased modes and (0,0))
// (marching.f90:16-29, 53-171; PL_algebra_z_3D.f90:218-243 zgbtrs semantics)
// ------------------------------------------------------------------------------
constexpr int kPF = 8;  // factor columns prefetched ahead

__device__ __forceinline__ double2 ell_row(const DevEll& op, int t, const double2* coef, const double2* x) {
  double2 acc = zero2();
#pragma unroll 4
  for (int k = 0; k < op.width; ++k) {
    const int cg = op.cg[(size_t)k * op.rows + t];
    const double v = op.val[(size_t)k * op.rows + t];
    const double2 xv = x[cg & 0xFFFFFF];
    acc = cadd(acc, cmul(coef[cg >> 24], make_double2(v * xv.x, v * xv.y)));
  }
  return acc;
}

// WIDE: bands of kl <= 63, kl + ku <= 127 (each lane holds two multipliers and
// four U entries of a column); otherwise kl <= 31, kl + ku <= 64
template <bool WIDE>
__global__ void __launch_bounds__(kWPB * 32) k_solve(SolveArgs a) {
  extern __shared__ double2 sm[];
  __shared__ double2 coefs[kWPB][2][kMaxGroups];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sid = blockIdx.x * kWPB + warp;
  const int nsys = a.d.NXH * a.d.NYA;
  if (sid >= nsys) return;
  const int T = a.T;
  double2* b = sm + (size_t)warp * T;
  const int kx = sid / a.d.NYA, ky = sid - kx * a.d.NYA;
  const int act = a.act_index[sid];
  const bool origin = (kx == 0 && ky == 0);
  if (lane < kMaxGroups) {
    coefs[warp][0][lane] = (lane < a.M.ngroups) ? cmul(ipow(a.kx[kx], a.M.gkx[lane]), ipow(a.ky[ky], a.M.gky[lane])) : zero2();
    coefs[warp][1][lane] = (lane < a.L.ngroups) ? cmul(ipow(a.kx[kx], a.L.gkx[lane]), ipow(a.ky[ky], a.L.gky[lane])) : zero2();
  }
  __syncwarp();
  const double2* field = a.field + (size_t)sid * T;
  // ---- right-hand side
  for (int t = lane; t < T; t += 32) {
    double2 r = origin ? zero2() : ell_row(a.M, t, coefs[warp][0], field);
    for (int j = 0; j < a.nprev; ++j) {
      const double2 ks = a.Kstd[j][(size_t)sid * T + t];
      r = cadd(r, cscale(ks, a.ca[j]));
      const double2 kh = a.Khat[j][(size_t)sid * T + t];
      r = cadd(r, cscale(kh, a.ch[j]));
    }
    const double2 kh = a.Khat[a.nprev][(size_t)sid * T + t];
    r = cadd(r, cscale(kh, a.ch[a.nprev]));
    b[t] = r;
  }
  __syncwarp();
  if (act >= 0) {
    const int kl = a.kl, kv = a.kl + a.ku, ldab = a.ldab;
    const double2* ab = a.ab + (size_t)act * T * ldab;
    const unsigned char* dp = a.dpiv + (size_t)act * ((T + 7) & ~7);
    // ---- forward: apply row interchanges and L (zgbtrs, 'N', kl > 0)
    {
      double2 lr[kPF], lr2[WIDE ? kPF : 1];
#pragma unroll
      for (int q = 0; q < kPF; ++q) {
        lr[q] = (q < T - 1 && lane < kl) ? ab[(size_t)q * ldab + kv + 1 + lane] : zero2();
        if constexpr (WIDE) lr2[q] = (q < T - 1 && lane + 32 < kl) ? ab[(size_t)q * ldab + kv + 33 + lane] : zero2();
      }
      for (int j0 = 0; j0 < T - 1; j0 += kPF) {
#pragma unroll
        for (int q = 0; q < kPF; ++q) {
          const int j = j0 + q;
          if (j < T - 1) {
            const double2 l = lr[q];
            double2 l2 = zero2();
            const int jn = j + kPF;
            lr[q] = (jn < T - 1 && lane < kl) ? ab[(size_t)jn * ldab + kv + 1 + lane] : zero2();
            if constexpr (WIDE) {
              l2 = lr2[q];
              lr2[q] = (jn < T - 1 && lane + 32 < kl) ? ab[(size_t)jn * ldab + kv + 33 + lane] : zero2();
            }
            const int p = j + dp[j];
            if (p != j) {
              if (lane == 0) {
                double2 tmp = b[p];
                b[p] = b[j];
                b[j] = tmp;
              }
              __syncwarp();
            }
            const double2 bj = b[j];
            const int lm = min(kl, T - 1 - j);
            if (lane < lm) b[j + 1 + lane] = csub(b[j + 1 + lane], cmul(l, bj));
            if constexpr (WIDE)
              if (lane + 32 < lm) b[j + 33 + lane] = csub(b[j + 33 + lane], cmul(l2, bj));
            __syncwarp();
          }
        }
      }
    }
    // ---- backward: U x = y, U with kl+ku super-diagonals, diagonal stored as its reciprocal
    {
      constexpr int NU = WIDE ? 4 : 2;  // U entries per lane: offsets 1 + lane + 32 u
      double2 uu[NU][kPF], dg[kPF];
#pragma unroll
      for (int q = 0; q < kPF; ++q) {
        const int j = T - 1 - q;
        if (j >= 0) {
          const double2* col = ab + (size_t)j * ldab;
          dg[q] = col[kv];
#pragma unroll
          for (int u = 0; u < NU; ++u) uu[u][q] = (lane + 1 + 32 * u <= kv) ? col[kv - 1 - 32 * u - lane] : zero2();
        }
      }
      for (int j0 = T - 1; j0 >= 0; j0 -= kPF) {
#pragma unroll
        for (int q = 0; q < kPF; ++q) {
          const int j = j0 - q;
          if (j >= 0) {
            const double2 d = dg[q];
            double2 c[NU];
#pragma unroll
            for (int u = 0; u < NU; ++u) c[u] = uu[u][q];
            const int jn = j - kPF;
            if (jn >= 0) {
              const double2* col = ab + (size_t)jn * ldab;
              dg[q] = col[kv];
#pragma unroll
              for (int u = 0; u < NU; ++u) uu[u][q] = (lane + 1 + 32 * u <= kv) ? col[kv - 1 - 32 * u - lane] : zero2();
            }
            const double2 bj = cmul(b[j], d);
            __syncwarp();
            if (lane == 0) b[j] = bj;
#pragma unroll
            for (int u = 0; u < NU; ++u) {
              const int o = lane + 1 + 32 * u;
              if (o <= kv && j - o >= 0) b[j - o] = csub(b[j - o], cmul(c[u], bj));
            }
            __syncwarp();
          }
        }
      }
    }
  }
  // ---- outputs
  double2* out = a.out + (size_t)sid * T;
  bool bad = false;
  const bool zero_out = a.last_stage && (act < 0);
  for (int t = lane; t < T; t += 32) {
    const double2 v = zero_out ? zero2() : b[t];
    bad |= !(isfinite(v.x) && isfinite(v.y));
    out[t] = v;
  }
  if (a.Kstd_out) {
    double2* ko = a.Kstd_out + (size_t)sid * T;
    for (int t = lane; t < T; t += 32) ko[t] = (act >= 0) ? ell_row(a.L, t, coefs[warp][1], b) : zero2();
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.flags, 1u);
}

// ------------------------------------------------------------------------------
// factorisation of E = M + zsca L (zsca = -dt a11) with partial pivoting, one warp
// per active system, in place in LAPACK band storage (PL_IMEX_timestepping.f90:382-410;
// PL_algebra_z_3D.f90:245-276; the unblocked ZGBTF2 algorithm that ZGBTRF runs for
// kl < 32).  Pivot offsets are kept as bytes; U's diagonal is replaced by its reciprocal.
// ------------------------------------------------------------------------------
__device__ __forceinline__ double2 crecip(double2 p) {
  if (fabs(p.x) >= fabs(p.y)) {
    const double t = p.y / p.x, den = p.x + p.y * t;
    return make_double2(1.0 / den, -t / den);
  } else {
    const double t = p.x / p.y, den = p.y + p.x * t;
    return make_double2(t / den, -1.0 / den);
  }
}

// WIDE: kl <= 63 (two pivot candidates per lane); otherwise kl <= 31
template <bool WIDE>
__global__ void __launch_bounds__(kWPB * 32) k_factor(FactorArgs a) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sys = blockIdx.x * kWPB + warp;
  if (sys >= a.nact) return;
  const int T = a.T, kl = a.kl, ku = a.ku, kv = kl + ku, ldab = a.ldab;
  const int sid = a.act_list[sys];
  const int kx = sid / a.d.NYA, ky = sid - kx * a.d.NYA;
  double2 cm[kMaxGroups], cl[kMaxGroups];
#pragma unroll
  for (int g = 0; g < kMaxGroups; ++g) {
    cm[g] = (g < a.M.ngroups) ? cmul(ipow(a.kx[kx], a.M.gkx[g]), ipow(a.ky[ky], a.M.gky[g])) : zero2();
    cl[g] = (g < a.L.ngroups) ? cmul(ipow(a.kx[kx], a.L.gkx[g]), ipow(a.ky[ky], a.L.gky[g])) : zero2();
  }
  double2* ab = a.ab + (size_t)sys * T * ldab;
  for (size_t e = lane; e < (size_t)T * ldab; e += 32) ab[e] = zero2();
  __syncwarp();
  // E(t,c) = M(t,c) + zsca * L(t,c); lane owns rows t = lane mod 32 (no write conflicts)
  for (int t = lane; t < T; t += 32) {
    for (int k = 0; k < a.M.width; ++k) {
      const double v = a.M.v(t, k);
      if (v == 0.0) continue;  // empty slot
      const int c = a.M.col(t, k), g = a.M.grp(t, k);
      double2 cv = zero2();
#pragma unroll
      for (int gg = 0; gg < kMaxGroups; ++gg)
        if (g == gg) cv = cm[gg];
      double2& dst = ab[(size_t)c * ldab + kv + t - c];
      dst = cadd(dst, cscale(cv, v));
    }
    for (int k = 0; k < a.L.width; ++k) {
      const double v = a.L.v(t, k);
      if (v == 0.0) continue;
      const int c = a.L.col(t, k), g = a.L.grp(t, k);
      double2 cv = zero2();
#pragma unroll
      for (int gg = 0; gg < kMaxGroups; ++gg)
        if (g == gg) cv = cl[gg];
      double2& dst = ab[(size_t)c * ldab + kv + t - c];
      dst = cadd(dst, cscale(cscale(cv, v), a.zsca));
    }
  }
  __syncwarp();
  int ju = 0, info = 0;
  for (int j = 0; j < T; ++j) {
    const int km = min(kl, T - 1 - j);
    // pivot: first index of the largest |re|+|im| among rows j..j+km
    double mag = -1.0;
    int idx = 1 << 30;
    if (lane <= km) {
      const double2 v = ab[(size_t)j * ldab + kv + lane];
      mag = fabs(v.x) + fabs(v.y);
      idx = lane;
    }
    if constexpr (WIDE) {
      if (lane + 32 <= km) {  // the later row wins only when strictly larger (first maximum)
        const double2 v = ab[(size_t)j * ldab + kv + lane + 32];
        const double m2 = fabs(v.x) + fabs(v.y);
        if (m2 > mag) { mag = m2; idx = lane + 32; }
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double m2 = __shfl_xor_sync(0xffffffffu, mag, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, idx, o);
      if (m2 > mag || (m2 == mag && i2 < idx)) { mag = m2; idx = i2; }
    }
    const int jp = idx;
    if (lane == 0) a.dpiv[(size_t)sys * ((T + 7) & ~7) + j] = (unsigned char)jp;
    const double2 piv = ab[(size_t)j * ldab + kv + jp];
    if (piv.x == 0.0 && piv.y == 0.0) {
      if (info == 0) info = j + 1;
      continue;
    }
    ju = max(ju, min(j + ku + jp, T - 1));
    if (jp != 0) {
      for (int c = j + lane; c <= ju; c += 32) {
        double2* p1 = ab + (size_t)c * ldab + kv + j + jp - c;
        double2* p0 = ab + (size_t)c * ldab + kv + j - c;
        const double2 t0 = *p0;
        *p0 = *p1;
        *p1 = t0;
      }
      __syncwarp();
    }
    const double2 r = crecip(ab[(size_t)j * ldab + kv]);
    __syncwarp();
    if (km > 0) {
      for (int i = lane; i <= km; i += 32)
        if (i >= 1) {
          double2* m = ab + (size_t)j * ldab + kv + i;
          *m = cmul(*m, r);
        }
      __syncwarp();
      const int nc = ju - j;
      for (int e = lane; e < nc * km; e += 32) {
        const int c = j + 1 + e / km, i = 1 + e % km;
        const double2 mult = ab[(size_t)j * ldab + kv + i];
        const double2 rowv = ab[(size_t)c * ldab + kv + j - c];
        double2* dst = ab + (size_t)c * ldab + kv + j + i - c;
        *dst = csub(*dst, cmul(mult, rowv));
      }
    }
    __syncwarp();
    if (lane == 0) ab[(size_t)j * ldab + kv] = r;
    __syncwarp();
  }
  if (lane == 0) a.info[sys] = info;
}


// ------------------------------------------------------------------------------
// Real-scaled factorisation: E' = S_r E S_c with S_r = diag(-i on flagged
// equation rows), S_c = diag(+i on flagged variable columns) is real; the
// partial-pivoting choices equal those on E because |re|+|im| is unchanged by
// the +-i factors.  Real ZGBTF2-equivalent (DGBTF2), one warp per system, in place
// in LAPACK band storage; pivot offsets as bytes; U's diagonal as its reciprocal.
// ------------------------------------------------------------------------------
__device__ __forceinline__ double2 flip_row(double2 z, int f) { return f ? make_double2(z.y, -z.x) : z; }  // * (-i)
__device__ __forceinline__ double2 flip_col(double2 z, int f) { return f ? make_double2(-z.y, z.x) : z; }  // * (+i)

// With a class split (FactorArgs::ncls == 2) one warp factors one class of one
// system (blockIdx.y = class): the class's rows and columns in their original
// relative order, identity rows on padding positions, stored in the class's
// ldab rows of each column (column stride ncls * ldab).
__global__ void __launch_bounds__(kWPB * 32) k_factor_real(FactorArgs a) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sys = blockIdx.x * kWPB + warp;
  if (sys >= a.nact) return;
  const int cls = blockIdx.y;
  const int T = a.Tc, kl = a.kl, ku = a.ku, kv = kl + ku, ldab = a.ldab;
  const size_t cstr = (size_t)a.ncls * ldab;  // column stride
  const int sid = a.act_list[sys];
  const int kx = sid / a.d.NYA, ky = sid - kx * a.d.NYA;
  double2 cm[kMaxGroups], cl[kMaxGroups];
#pragma unroll
  for (int g = 0; g < kMaxGroups; ++g) {
    cm[g] = (g < a.M.ngroups) ? cmul(ipow(a.kx[kx], a.M.gkx[g]), ipow(a.ky[ky], a.M.gky[g])) : zero2();
    cl[g] = (g < a.L.ngroups) ? cmul(ipow(a.kx[kx], a.L.gkx[g]), ipow(a.ky[ky], a.L.gky[g])) : zero2();
  }
  double* ab = a.abr + (size_t)sys * T * cstr + (size_t)cls * ldab;
  for (size_t e = lane; e < (size_t)T * ldab; e += 32) ab[(e / ldab) * cstr + e % ldab] = 0.0;
  __syncwarp();
  for (int i = lane; i < T; i += 32) {
    const int t = a.cls_row ? a.cls_row[cls * T + i] : i;  // equation row of class position i
    if (t < 0) {
      ab[(size_t)i * cstr + kv] = 1.0;  // identity padding
      continue;
    }
    const int rf = a.rowflip[t];
    for (int pass = 0; pass < 2; ++pass) {
      const DevEll& op = pass ? a.L : a.M;
      for (int k = 0; k < op.width; ++k) {
        const double v = op.v(t, k);
        if (v == 0.0) continue;  // empty slot
        const int c = op.col(t, k), g = op.grp(t, k);
        const int jc = a.col_pos ? a.col_pos[c] - cls * T : c;  // column in the class
        double2 cv = zero2();
#pragma unroll
        for (int gg = 0; gg < kMaxGroups; ++gg)
          if (g == gg) cv = pass ? cl[gg] : cm[gg];
        double2 z = cscale(cv, v);
        if (pass) z = cscale(z, a.zsca);
        z = flip_col(flip_row(z, rf), a.colflip[c]);
        ab[(size_t)jc * cstr + kv + i - jc] += z.x;
      }
    }
  }
  __syncwarp();
  unsigned char* dpiv = a.dpiv + ((size_t)sys * a.ncls + cls) * ((T + 7) & ~7);  // rows padded to 8 bytes
  int ju = 0, info = 0;
  for (int j = 0; j < T; ++j) {
    const int km = min(kl, T - 1 - j);
    double mag = -1.0;
    int idx = 1 << 30;
    if (lane <= km) {
      mag = fabs(ab[(size_t)j * cstr + kv + lane]);
      idx = lane;
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double m2 = __shfl_xor_sync(0xffffffffu, mag, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, idx, o);
      if (m2 > mag || (m2 == mag && i2 < idx)) { mag = m2; idx = i2; }
    }
    const int jp = idx;
    if (lane == 0) dpiv[j] = (unsigned char)jp;
    const double piv = ab[(size_t)j * cstr + kv + jp];
    if (piv == 0.0) {
      if (info == 0) info = j + 1;
      continue;
    }
    ju = max(ju, min(j + ku + jp, T - 1));
    if (jp != 0) {
      for (int c = j + lane; c <= ju; c += 32) {
        double* p1 = ab + (size_t)c * cstr + kv + j + jp - c;
        double* p0 = ab + (size_t)c * cstr + kv + j - c;
        const double t0 = *p0;
        *p0 = *p1;
        *p1 = t0;
      }
      __syncwarp();
    }
    const double r = 1.0 / ab[(size_t)j * cstr + kv];
    __syncwarp();
    if (km > 0) {
      if (lane >= 1 && lane <= km) ab[(size_t)j * cstr + kv + lane] *= r;
      __syncwarp();
      const int nc = ju - j;
      for (int e = lane; e < nc * km; e += 32) {
        const int c = j + 1 + e / km, i = 1 + e % km;
        ab[(size_t)c * cstr + kv + j + i - c] -= ab[(size_t)j * cstr + kv + i] * ab[(size_t)c * cstr + kv + j - c];
      }
    }
    __syncwarp();
    if (lane == 0) ab[(size_t)j * cstr + kv] = r;
    __syncwarp();
  }
  if (lane == 0 && info) atomicMax(a.info + sys, info);
}

// ------------------------------------------------------------------------------
// Stage update + banded solve with real-scaled factors, one warp per system,
// no shared-memory vectors: the right-hand side and the intermediate solutions
// pass through the work array (L2-resident), while the active part of the
// band lives in registers, each lane owning the positions p = lane (mod 32):
//   forward  window [j, j+kl] (kl <= 31), one register per lane
//   backward window [j-kv, j] (kv <= 63), two registers per lane
// so a column step moves only the pivot value between lanes.  Factor columns
// reach the lanes through a per-warp shared-memory ring filled by cp.async.
// ------------------------------------------------------------------------------
constexpr int kWPBr = 4;   // warps per CTA
constexpr int kCW = 8;     // factor columns per ring chunk (divides 32)
constexpr int kNBUF = 4;   // ring chunks per warp

__device__ __forceinline__ double2 shfl2(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

__global__ void __launch_bounds__(kWPBr * 32) k_subst_real(SolveArgs a) {
  constexpr int H = 32, LH = 5;  // lanes, log2
  extern __shared__ double smr[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int act = blockIdx.x * kWPBr + warp;  // active systems only
  if (act >= a.nact) return;
  const int T = a.T;
  const int sid = a.act_list[act];
  double2* x = a.work + (size_t)sid * T;  // right-hand side in, solution out
  {
    const int kl = a.kl, kv = a.kl + a.ku, ldab = a.ldab;
    const double* ab = a.abr + (size_t)act * T * ldab;
    const unsigned char* dp = a.dpiv + (size_t)act * ((T + 7) & ~7);
    const unsigned char* cflip = a.colflip;
    // Factor columns stream through a per-warp shared-memory ring (kNBUF chunks
    // of kCW columns) with cp.async, kNBUF-1 chunks ahead of the sweep; the
    // forward sweep copies only the L rows of each column, the backward sweep
    // only the U rows.  (ldab is even, so both row ranges are 16-byte aligned.)
    double* ring = smr + (size_t)warp * kNBUF * kCW * a.ring_cols;
    const int u_rows = (kv + 2) & ~1;                 // rows [0, u_rows) hold U (+ maybe one L row)
    const int l_row0 = (kv + 1) & ~1;                 // rows [l_row0, l_row1) hold L
    const int l_rows = ((kv + 1 + kl + 1) & ~1) - l_row0;
    // ================= forward: P and L =================
    // lane l owns the positions p = l (mod 32); the active window is [j, j+kl].
    // Vector traffic moves in blocks of H columns: the owner of column j takes
    // the new position j+H (loaded one block ahead) and parks y_j until the
    // block's coalesced store.
    {
      const int nchunks = (T - 1 + kCW - 1) / kCW;
      auto issue = [&](int c) {  // columns [c*kCW, min(T-1, c*kCW+kCW)) of L
        if (c < nchunks) {
          const int j0 = c * kCW, nc = min(kCW, T - 1 - j0);
          double* dst = ring + (size_t)(c % kNBUF) * kCW * a.ring_cols;
          const int per = l_rows / 2;  // 16-byte pieces per column
          for (int e = lane; e < nc * per; e += 32) {
            const int q = e / per, r = e - q * per;
            cp_async16(dst + q * a.ring_cols + 2 * r, ab + (size_t)(j0 + q) * ldab + l_row0 + 2 * r);
          }
        }
        cp_async_commit();
      };
#pragma unroll
      for (int c = 0; c < kNBUF - 1; ++c) issue(c);
      double2 w = (lane < T) ? x[lane] : zero2();
      double2 incCur = (H + lane < T) ? x[H + lane] : zero2();
      double2 incNext = zero2(), ysave = zero2();
      // pivot offsets of a chunk as two 32-bit words, uniform over the warp (rows padded to 8 bytes)
      uint2 pw = *reinterpret_cast<const uint2*>(dp);
      for (int c = 0; c < nchunks; ++c) {
        const int j0 = c * kCW;
        if ((j0 & (H - 1)) == 0)  // new block of H columns: next block's incoming values
          incNext = (j0 + 2 * H + lane < T) ? x[j0 + 2 * H + lane] : zero2();
        const uint2 pwc = pw;
        if (c + 1 < nchunks) pw = *reinterpret_cast<const uint2*>(dp + j0 + kCW);
        __syncwarp();
        issue(c + kNBUF - 1);
        cp_async_wait<kNBUF - 1>();
        __syncwarp();
        const double* cb = ring + (size_t)(c % kNBUF) * kCW * a.ring_cols;
#pragma unroll
        for (int q = 0; q < kCW; ++q) {
          const int j = j0 + q;
          if (j < T - 1) {
            const int src = (j & (H - 1));
            const int i = (lane - j) & (H - 1);
            const int lm = min(kl, T - 1 - j);
            const double lv = (i >= 1 && i <= lm) ? cb[q * a.ring_cols + (kv + i - l_row0)] : 0.0;
            const int jp = ((q < 4 ? pwc.x : pwc.y) >> (8 * (q & 3))) & 0xFF;
            // Row interchange j <-> j+jp and broadcast of the pivot row in one shuffle:
            // the owner of row j+jp fetches row j (its new content), every other lane
            // fetches the pivot row; the owner of j+jp already holds the pivot value.
            const int r2 = ((j + jp) & (H - 1));
            const bool mine = (jp != 0 && lane == r2);
            const double2 got = shfl2(w, mine ? src : r2);
            const double2 bj = mine ? w : got;
            if (lane == src || mine) w = got;
            w.x -= lv * bj.x;  // zero multiplier outside rows j+1..j+lm
            w.y -= lv * bj.y;
            if (lane == src) {
              ysave = w;
              w = incCur;
            }
            if ((j & (H - 1)) == H - 1) {  // end of a block of H columns
              x[j - (H - 1) + lane] = ysave;
              incCur = incNext;
            }
          }
        }
      }
      cp_async_wait<0>();
      // the last (partial) block of y values and y[T-1]
      const int base = ((T - 1) >> LH) << LH;
      if ((T - 1) & (H - 1)) {
        if (base + lane <= T - 2) x[base + lane] = ysave;
      }
      if (lane == ((T - 1) & (H - 1))) x[T - 1] = w;
    }
    __syncwarp();
    // ================= backward: U (kl+ku super-diagonals, reciprocal diagonal) =================
    // lane l owns p = l (mod 32) in two registers: w0 for (p/H) even, w1 for odd.
    // Blocks of H columns j = T-1-H*b-s; the owner of j takes position j-2H.
    {
      double2 w0 = zero2(), w1 = zero2();
      {
        const int ih = (T - 1 - lane) & (H - 1), ph = T - 1 - ih, pl = ph - H;
        if (ph >= 0) { if ((ph >> LH) & 1) w1 = x[ph]; else w0 = x[ph]; }
        if (pl >= 0) { if ((pl >> LH) & 1) w1 = x[pl]; else w0 = x[pl]; }
      }
      const int nchunks = (T + kCW - 1) / kCW;  // chunk c: columns T-1-c*kCW-q, q < kCW
      auto issue = [&](int c) {
        if (c < nchunks) {
          const int jhi = T - 1 - c * kCW, jlo = max(0, jhi - kCW + 1), nc = jhi - jlo + 1;
          double* dst = ring + (size_t)(c % kNBUF) * kCW * a.ring_cols;
          const int per = u_rows / 2;
          for (int e = lane; e < nc * per; e += 32) {
            const int q = e / per, r = e - q * per;  // q counts down from jhi
            cp_async16(dst + q * a.ring_cols + 2 * r, ab + (size_t)(jhi - q) * ldab + 2 * r);
          }
        }
        cp_async_commit();
      };
      __syncwarp();
#pragma unroll
      for (int c = 0; c < kNBUF - 1; ++c) issue(c);
      auto own_col = [&](int b) {  // column of block b finished by this lane (may be < 0)
        const int top = T - 1 - H * b;
        return top - ((top - lane) & (H - 1));
      };
      int jl = own_col(0);
      double2 incCur = (jl - 2 * H >= 0) ? x[jl - 2 * H] : zero2();
      int cfCur = (jl >= 0) ? cflip[jl] : 0;
      double2 incNext = zero2(), xsave = zero2();
      int cfNext = 0, jn = jl;
      for (int c = 0; c < nchunks; ++c) {
        const int k0 = c * kCW;  // steps taken before this chunk
        if ((k0 & (H - 1)) == 0) {
          jn = own_col((k0 >> LH) + 1);
          incNext = (jn - 2 * H >= 0) ? x[jn - 2 * H] : zero2();
          cfNext = (jn >= 0) ? cflip[jn] : 0;
        }
        __syncwarp();
        issue(c + kNBUF - 1);
        cp_async_wait<kNBUF - 1>();
        __syncwarp();
        const double* cb = ring + (size_t)(c % kNBUF) * kCW * a.ring_cols;
#pragma unroll
        for (int q = 0; q < kCW; ++q) {
          const int k = k0 + q;
          const int j = T - 1 - k;
          if (j >= 0) {
            const int src = (j & (H - 1)), sel = (j >> LH) & 1;
            const double* col = cb + q * a.ring_cols;
            const int ih = (j - lane) & (H - 1), il = ih + H;
            const double h = (ih >= 1 && ih <= kv) ? col[kv - ih] : 0.0;
            const double l_ = (il <= kv) ? col[kv - il] : 0.0;
            const double d = col[kv];
            const double2 yj = shfl2(sel ? w1 : w0, src);
            const double2 xj = make_double2(yj.x * d, yj.y * d);
            const int hreg = ((j - ih) >> LH) & 1;
            if (hreg) { w1.x -= h * xj.x; w1.y -= h * xj.y; w0.x -= l_ * xj.x; w0.y -= l_ * xj.y; }
            else      { w0.x -= h * xj.x; w0.y -= h * xj.y; w1.x -= l_ * xj.x; w1.y -= l_ * xj.y; }
            if (lane == src) {
              xsave = flip_col(xj, cfCur);
              if (sel) w1 = incCur; else w0 = incCur;
            }
            if ((k & (H - 1)) == H - 1) {  // end of a block of H columns
              if (jl >= 0) x[jl] = xsave;
              jl = jn;
              incCur = incNext;
              cfCur = cfNext;
            }
          }
        }
      }
      cp_async_wait<0>();
      if ((T & (H - 1)) != 0 && jl >= 0) x[jl] = xsave;  // the last (partial) block
    }
  }
  __syncwarp();
}


// ------------------------------------------------------------------------------
// Block factorisation of the independent blocks (class split).  The block of
// unit u (one factorisation, of system act_list[u]) and one class is handled by
// one thread; the upw blocks of a group (one class) lie side by side in memory
// (abr[((G Tc + j) ldab + r) upw + lane], G = class * ngrp + u / upw), so the
// accesses of a warp in one step are contiguous rows.
// ------------------------------------------------------------------------------
constexpr int kTpbThreads = 128;

// thread b of the block kernels: class, unit, and its column of the group's
// factors and pivots; false for the padding lanes
struct TpbBlock {
  int cls, unit;
  double* F;
  unsigned char* P;
};
__device__ __forceinline__ bool tpb_block(const FactorArgs& a, int b, TpbBlock& t) {
  const int G = b / a.upw, lane = b - G * a.upw;
  if (G >= a.ncls * a.ngrp) return false;
  t.cls = G / a.ngrp;
  const int g = G - t.cls * a.ngrp;
  t.unit = g * a.upw + lane;
  t.F = a.abr + (size_t)G * a.Tc * a.ldab * a.upw + lane;
  t.P = a.dpiv + ((size_t)t.cls * a.ngrp + g) * a.Tc * a.upw + lane;
  return t.unit < a.nact;
}

// Rows i0 .. i1 - 1 of one block of M - dt a(0,0) L added to its zeroed interleaved
// band storage (M before L, slots in order).
// G: the monomial groups the coefficient registers hold (>= the operators' ngroups)
template <int G = kMaxGroups>
__device__ void assemble_tpb(const FactorArgs& a, const TpbBlock& tb, int i0, int i1) {
  const int cls = tb.cls;
  const int T = a.Tc, kv = a.kl + a.ku, ldab = a.ldab, RW = a.upw;
  const int sid = a.act_list[tb.unit];
  const int kx = sid / a.d.NYA, ky = sid - kx * a.d.NYA;
  double2 cm[G], cl[G];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    cm[g] = (g < a.M.ngroups) ? cmul(ipow(a.kx[kx], a.M.gkx[g]), ipow(a.ky[ky], a.M.gky[g])) : zero2();
    cl[g] = (g < a.L.ngroups) ? cmul(ipow(a.kx[kx], a.L.gkx[g]), ipow(a.ky[ky], a.L.gky[g])) : zero2();
  }
  double* F = tb.F;
  auto at = [&](int j, int r) -> double& { return F[((size_t)j * ldab + r) * RW]; };
  for (int i = i0; i < i1; ++i) {
    const int t = a.cls_row[cls * T + i];  // equation row of class position i
    if (t < 0) {
      at(i, kv) = 1.0;  // identity padding
      continue;
    }
    const int rf = a.rowflip[t];
    for (int pass = 0; pass < 2; ++pass) {
      const DevEll& op = pass ? a.L : a.M;
      for (int k = 0; k < op.width; ++k) {
        const double v = op.v(t, k);
        if (v == 0.0) continue;  // empty slot
        const int c = op.col(t, k), g = op.grp(t, k);
        const int jc = a.col_pos[c] - cls * T;  // column in the class
        double2 cv = zero2();
#pragma unroll
        for (int gg = 0; gg < G; ++gg)
          if (g == gg) cv = pass ? cl[gg] : cm[gg];
        double2 z = cscale(cv, v);
        if (pass) z = cscale(z, a.zsca);
        z = flip_col(flip_row(z, rf), a.colflip[c]);
        at(jc, kv + i - jc) += z.x;
      }
    }
  }
}

// One thread per block and kAsmRows rows: a row's entries have band places of their
// own, so the rows are independent (one thread per whole block, zero fill included:
// 1.88 ms at 96^2 x 48 of the toroidal-poloidal recipe; now 0.34 ms).
constexpr int kAsmRows = 8;
template <int G>
__global__ void __launch_bounds__(kTpbThreads) k_assemble_tpb(FactorArgs a) {
  TpbBlock tb;
  const int i0 = blockIdx.y * kAsmRows;
  if (tpb_block(a, blockIdx.x * blockDim.x + threadIdx.x, tb)) assemble_tpb<G>(a, tb, i0, min(a.Tc, i0 + kAsmRows));
}

// DGBTF2 on one block in place in global memory: the algorithm, pivot choice and
// update order of k_factor_real.

__global__ void __launch_bounds__(kTpbThreads) k_factor_tpb(FactorArgs a) {
  TpbBlock tb;
  if (!tpb_block(a, blockIdx.x * blockDim.x + threadIdx.x, tb)) return;
  assemble_tpb(a, tb, 0, a.Tc);
  const int sys = tb.unit, RW = a.upw;
  const int T = a.Tc, kl = a.kl, ku = a.ku, kv = kl + ku, ldab = a.ldab;
  double* F = tb.F;
  auto at = [&](int j, int r) -> double& { return F[((size_t)j * ldab + r) * RW]; };
  unsigned char* P = tb.P;
  int ju = 0, info = 0;
  for (int j = 0; j < T; ++j) {
    const int km = min(kl, T - 1 - j);
    int jp = 0;
    double mag = fabs(at(j, kv));
    for (int i = 1; i <= km; ++i) {
      const double m2 = fabs(at(j, kv + i));
      if (m2 > mag) { mag = m2; jp = i; }  // first maximum
    }
    P[(size_t)j * RW] = (unsigned char)jp;
    if (at(j, kv + jp) == 0.0) {
      if (info == 0) info = j + 1;
      continue;
    }
    ju = max(ju, min(j + ku + jp, T - 1));
    if (jp != 0) {
      for (int c = j; c <= ju; ++c) {
        double& p1 = at(c, kv + j + jp - c);
        double& p0 = at(c, kv + j - c);
        const double t0 = p0;
        p0 = p1;
        p1 = t0;
      }
    }
    const double r = 1.0 / at(j, kv);
    if (km > 0) {
      for (int i = 1; i <= km; ++i) at(j, kv + i) *= r;
      for (int c = j + 1; c <= ju; ++c) {
        const double u = at(c, kv + j - c);
        for (int i = 1; i <= km; ++i) at(c, kv + j + i - c) -= at(j, kv + i) * u;
      }
    }
    at(j, kv) = r;
  }
  if (info) atomicMax(a.info + sys, info);
}

// DGBTF2 on one block (after k_assemble_tpb) with its active part in shared memory:
// the algorithm, pivot choice and update order of k_factor_tpb (the same factors bit
// for bit), but every factor entry is read from and written to global memory once.
// At step j the active part is rows j .. j+kl by columns j .. j+kv: row j + kl + 1
// enters when row j, then final, leaves (its columns are exactly the next step's),
// column j + kv + 1 starts as fill.  Row and column slots are circular, each
// thread's entries in its own column of shared memory (stride 32: conflict-free).
// Bound by the latency of a step (one warp issues it), so what counts is how many
// warps an SM holds: 1.9 KB a thread for the band (9, 23), 3 warps (a window of kv + 2
// whole band columns took 6.8 KB, 1 warp), and how many loads are ahead of a store:
// two columns' (2.58 ms at 128^2 x 96 with one column's, now 1.29; 2.39 with the
// whole-column window).  At 384^2 x 192 the whole factorisation takes 28.9 ms (54.0).
constexpr int kFacKl = 15, kFacKv = 31;
template <int KL, int KV>
__global__ void __launch_bounds__(32) k_factor_win(FactorArgs a) {
  extern __shared__ double fwin[];
  constexpr int NT = 32;
  TpbBlock tb;
  if (!tpb_block(a, blockIdx.x * NT + threadIdx.x, tb)) return;  // no barriers below
  const int RW = a.upw, T = a.Tc, kl = a.kl, kv = a.kl + a.ku, ldab = a.ldab, NR = kl + 1, NC = kv + 1;
  double* F = tb.F;
  unsigned char* P = tb.P;
  double* w = fwin + threadIdx.x;
  auto band = [&](int r, int c) -> double& { return F[((size_t)c * ldab + kv + r - c) * RW]; };
  int r0 = 0, c0 = 0;  // slots of row j and column j
  auto row = [&](int i) {  // offset of row j + i's slot
    const int q = r0 + i;
    return (q >= NR ? q - NR : q) * NC * NT;
  };
  auto col = [&](int i) {
    const int q = c0 + i;
    return (q >= NC ? q - NC : q) * NT;
  };
  for (int r = 0; r <= kl && r < T; ++r)
    for (int c = 0; c <= kv && c < T; ++c) w[row(r) + col(c)] = band(r, c);
  const size_t diag = (size_t)(ldab - 1) * RW;  // along a row of the band
  double* Fj = F + (size_t)kv * RW;              // entry (j, j)
  int ju = 0, info = 0;
  for (int j = 0; j < T; ++j) {
    double in[KV + 1];  // row j + kl + 1, columns j + 1 ..
    {
      const double* src = Fj + (size_t)ldab * RW + (size_t)kl * RW;
      const int n = j + kl + 1 < T ? min(kv, T - 2 - j) : -1;
#pragma unroll
      for (int q = 0; q <= KV; ++q) in[q] = q <= n ? src[q * diag] : 0.0;
    }
    const int km = min(kl, T - 1 - j), cj = col(0), rj = row(0);
    int ro[KL];  // rows j + 1 ..
#pragma unroll
    for (int i = 0; i < KL; ++i) ro[i] = i < kl ? row(1 + i) : rj;
    double m[KL];
    const double d0 = w[rj + cj];
    double piv = d0, mag = fabs(d0);
    int jp = 0, rp = rj;
#pragma unroll
    for (int i = 0; i < KL; ++i) m[i] = i < km ? w[ro[i] + cj] : 0.0;
#pragma unroll
    for (int i = 0; i < KL; ++i)
      if (i < km && fabs(m[i]) > mag) {  // first maximum
        mag = fabs(m[i]);
        piv = m[i];
        jp = i + 1;
        rp = ro[i];
      }
    P[(size_t)j * RW] = (unsigned char)jp;
    double dout = piv;
    double* dst = Fj;
    if (piv == 0.0) {
      if (info == 0) info = j + 1;
      for (int c = 1; c <= kv && j + c < T; ++c) Fj[c * diag] = w[rj + col(c)];
    } else {
      ju = max(ju, min(j + a.ku + jp, T - 1));
      const double r = 1.0 / piv;
      dout = r;
      // row j + jp comes up, row j goes down; multipliers
#pragma unroll
      for (int i = 0; i < KL; ++i)
        if (i < km) {
          if (i + 1 == jp) m[i] = d0;
          m[i] *= r;
        }
      // two columns at a time, loads first
      int cc = col(1);
#pragma unroll 1
      for (int c = 1; j + c <= ju; c += 2) {
        const int c1 = cc, c2 = cc + NT == NC * NT ? 0 : cc + NT;
        cc = c2 + NT == NC * NT ? 0 : c2 + NT;
        const bool two = j + c < ju;
        const double xp1 = w[rp + c1], xj1 = w[rj + c1], xp2 = w[rp + c2], xj2 = w[rj + c2];
        double v1[KL], v2[KL];
#pragma unroll
        for (int i = 0; i < KL; ++i) {
          v1[i] = w[ro[i] + c1];
          v2[i] = w[ro[i] + c2];
        }
#pragma unroll
        for (int i = 0; i < KL; ++i)
          if (i < km) {
            const double x1 = i + 1 == jp ? xj1 : v1[i], x2 = i + 1 == jp ? xj2 : v2[i];
            w[ro[i] + c1] = x1 - m[i] * xp1;
            if (two) w[ro[i] + c2] = x2 - m[i] * xp2;
          }
        dst += diag;
        *dst = xp1;
        dst += diag;
        if (two) *dst = xp2;
      }
    }
    *Fj = dout;
#pragma unroll
    for (int i = 0; i < KL; ++i)
      if (i < km) {
        Fj[(1 + i) * RW] = m[i];
        w[ro[i] + cj] = 0.0;  // column j + kv + 1: fill
      }
    // the next row in row j's slot
    {
      int cn = cj;
#pragma unroll
      for (int q = 0; q <= KV; ++q)
        if (q <= kv) {
          cn = cn + NT == NC * NT ? 0 : cn + NT;
          w[rj + cn] = in[q];
        }
    }
    Fj += (size_t)ldab * RW;
    r0 = r0 + 1 == NR ? 0 : r0 + 1;
    c0 = c0 + 1 == NC ? 0 : c0 + 1;
  }
  if (info) atomicMax(a.info + tb.unit, info);
}

// Band rows that are nonzero in any unit, per class and column: one warp per
// (group, column) tests the units of its group row by row (padding lanes count
// as zero).
__global__ void __launch_bounds__(256) k_mask_cols(FactorArgs a) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int G = blockIdx.x, j = blockIdx.y * 8 + w;
  const int T = a.Tc, ldab = a.ldab;
  if (j >= T) return;
  const int cls = G / a.ngrp, u0 = (G - cls * a.ngrp) * a.upw;
  const bool ok = lane < a.upw && u0 + lane < a.nact;
  const double* F = a.abr + ((size_t)G * T + j) * ldab * a.upw + (ok ? lane : 0);
  unsigned long long bits = 0;
  for (int r = 0; r < ldab; ++r) {
    const double v = ok ? F[(size_t)r * a.upw] : 0.0;
    if (__any_sync(0xffffffffu, v != 0.0)) bits |= 1ull << r;
  }
  if (lane == 0 && bits) atomicOr(a.cmask + (size_t)cls * T + j, bits);
}
// The records of the substitution from cmask, one warp per class.  A factor row
// is upw doubles (one entry of every unit of a group).  A group's rows: first its L
// records, forward, column j's being its L rows i (band row kl+ku+1+i) that are
// nonzero in some unit; then its U records, step k of the backward sweep handling
// row j = Tc-1-k: the reciprocal diagonal (row 0) and the entries (j, j+i) (row i)
// that are nonzero in some unit.  Rows in increasing i.
//   finfo[k] = first row (of the L records), mask of the rows held
//   binfo[k] = first row (of the U records), mask of the rows held, variable column (-1 = padding),
//              bit 0 colflip, bit 1 col_neg
// ptot: rows per group.
__global__ void __launch_bounds__(32) k_pack_info(FactorArgs a) {
  const int lane = threadIdx.x, cls = blockIdx.x;
  const int T = a.Tc, kl = a.kl, kv = a.kl + a.ku;
  const unsigned long long* cm = a.cmask + (size_t)cls * T;
  int base[2] = {0, 0};
  for (int k0 = 0; k0 < T; k0 += 32) {
    const int k = k0 + lane;
    unsigned lm = 0, um = 0;
    if (k < T) {
      lm = (unsigned)((cm[k] >> (kv + 1)) & ((1ull << kl) - 1));
      const int j = T - 1 - k;
      um = 1u;
      for (int i = 1; i <= kv; ++i)
        if (j + i < T && ((cm[j + i] >> (kv - i)) & 1ull)) um |= 1u << i;
    }
    const int n[2] = {__popc(lm), __popc(um)};
    int off[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      int inc = n[q];
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += up;
      }
      off[q] = base[q] + inc - n[q];
      base[q] += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (k < T) {
      const size_t at = (size_t)cls * T + k;
      a.finfo[at] = make_uint4((unsigned)off[0], lm, 0u, 0u);
      const int t = a.cls_col[(size_t)cls * T + T - 1 - k];
      const unsigned fl = t >= 0 ? (a.colflip[t] ? 1u : 0u) | (a.col_neg[t] ? 2u : 0u) : 0u;
      a.binfo[at] = make_uint4((unsigned)off[1], um, (unsigned)t, fl);
    }
  }
  if (lane == 0) {
    a.ptot[cls] = base[0];
    a.ptot[2 + cls] = base[1];
  }
}
// first row of group G's L (q = 0) or U (q = 1) records: a group starts where its
// factors do in abr (Tc ldab rows, more than all of its records)
__device__ __forceinline__ size_t pack_base(const int* ptot, int q, int cls, size_t G, int Tc, int ldab) {
  return G * Tc * ldab + (q ? ptot[cls] : 0);
}
// The band factors of the groups g0 .. g0 + gn - 1 of each class copied into records in
// out (group cls gn + g - g0 there): one warp per (group, column).  The substitution
// then reads two linear streams that hold only what it needs.
__global__ void __launch_bounds__(256) k_pack(FactorArgs a, double* out, int g0, int gn) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int k = blockIdx.y * 8 + w;
  const int T = a.Tc, kv = a.kl + a.ku, ldab = a.ldab, RW = a.upw;
  if (k >= T) return;
  const int cls = blockIdx.x / gn, g = g0 + blockIdx.x - cls * gn;
  const double* F = a.abr + ((size_t)cls * a.ngrp + g) * T * ldab * RW;
  const int half = lane / RW, ln = lane - half * RW, per = 32 / RW;  // rows a warp copies at a time
  {
    const uint4 fi = a.finfo[(size_t)cls * T + k];
    double* dst = out + (pack_base(a.ptot, 0, cls, blockIdx.x, T, ldab) + fi.x) * RW;
    const int n = __popc(fi.y);
    for (int r = half; r < n; r += per) {
      const int i = __fns(fi.y, 0, r + 1);  // the (r + 1)-th set bit
      dst[(size_t)r * RW + ln] = F[((size_t)k * ldab + kv + 1 + i) * RW + ln];
    }
  }
  {
    const uint4 bi = a.binfo[(size_t)cls * T + k];
    double* dst = out + (pack_base(a.ptot, 1, cls, blockIdx.x, T, ldab) + bi.x) * RW;
    const int j = T - 1 - k, n = __popc(bi.y);
    for (int r = half; r < n; r += per) {
      const int i = __fns(bi.y, 0, r + 1);
      dst[(size_t)r * RW + ln] = F[((size_t)(j + i) * ldab + kv - i) * RW + ln];
    }
  }
}
// The staged records of those groups over their factors; blockIdx.y takes a part of a
// group's rows.
__global__ void __launch_bounds__(256) k_pack_back(FactorArgs a, int g0, int gn) {
  const int cls = blockIdx.x / gn, g = g0 + blockIdx.x - cls * gn;
  const size_t group = (size_t)a.Tc * a.ldab * a.upw / 2;  // in 16-byte words
  const int n = (a.ptot[cls] + a.ptot[2 + cls]) * a.upw / 2;
  const double2* src = reinterpret_cast<const double2*>(a.stage) + blockIdx.x * group;
  double2* dst = reinterpret_cast<double2*>(a.abr) + ((size_t)cls * a.ngrp + g) * group;
  for (int e = blockIdx.y * 256 + threadIdx.x; e < n; e += gridDim.y * 256) dst[e] = src[e];
}

// ------------------------------------------------------------------------------
// Band substitutions of one group by one warp: forward (P, L: the column sweep
// with the row interchanges interleaved, as the reference's band solve) then
// backward (U, row form: each x_j subtracts the known x_{j+i} in decreasing
// column order, the order in which the column sweep reaches it); the solution,
// scaled back, goes straight into the stage output.
//
// What bounds it: the factor and vector streams on large grids; on small ones the 2 Tc
// column steps one after the other, each of them one warp's own instructions (128^2 x
// 192: 3.4 warps an SM, a scheduler issues in 38% of the cycles, its warp stalls on
// fixed latencies, 1.1 cycles an instruction, and hardly on memory, 0.3).  So (a) the systems (kx, ky) and
// (kx, -ky) share one factorisation where the recipe's mirror symmetry allows: 16
// units a warp, two right-hand sides each, half the factor bytes; (b) the factors
// come as linear streams of the entries that are nonzero in some unit (k_pack);
// (c) both streams, the right-hand sides and the intermediate vector are copied
// with cp.async into a ring in shared memory DF (forward) or DB (backward)
// columns ahead, so that a column step waits for shared memory only.  Against
// one thread per system that loads its factors one column ahead, no-slip
// convection, per launch: 384^2 x 192 3.83 -> 2.41 ms (11.65 GB, 6.2 of them the
// streams, 4.84 TB/s, 0.74 of the copy rate; before, 20.1 GB, 14.7 of factors),
// 128^2 x 192 1.26 -> 0.39 ms, 64^2 x 48 0.318 -> 0.099 ms; without the symmetry
// (rotating, 192^2 x 96) 0.72 -> 0.49 ms.
//
// The window of the vector (rows j .. j+KL, x_{j+1} .. x_{j+KV}) is in registers:
// U column steps are unrolled, so that every row has a fixed register, and the
// window moves by U rows after them; the row interchange is a chain of selects.
// (With the window in shared memory the kernel was bound by that memory's
// accesses, 75% of the LSU's peak at 256^2 x 96, 1.76 ms per step.)  The ring
// holds a record's rows at fixed places (holes zero-filled by the copies), the
// rows that most records hold are handled without a test, a step's factors are
// read from the ring one step ahead, and the record descriptions come in blocks of
// 32, one per lane.
// ------------------------------------------------------------------------------
template <int KL, int KV, int UPW>
struct SubstShape {
  static constexpr int DF = 6, DB = UPW == 16 ? 5 : 4;        // columns copied ahead
  static constexpr int kLBytes = KL * UPW * 8;
  static constexpr int kFSlot = kLBytes + UPW + 512;          // L rows, pivot bytes, row j + KL of the vector
  static constexpr int kUBytes = (KV + 1) * UPW * 8;
  static constexpr int kBSlot = kUBytes + 512;                // U rows, row j of the vector
  static constexpr int kRingF = (DF + 1) * kFSlot, kRingB = (DB + 1) * kBSlot;
  static constexpr int kBytes = kRingF > kRingB ? kRingF : kRingB;
  static_assert(kFSlot % 16 == 0 && kBSlot % 16 == 0, "16-byte copies");
};
__device__ __forceinline__ void cp_async16s(unsigned sa, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
// One warp copies a record (the rows of mask m, contiguous at src) to rows i =
// 0 .. ROWS-1 at dst, zeros where m has no bit.  Rows from HARD on are left alone
// where no row of their group of kRowGroup is held.
constexpr int kRowGroup = 4;
template <int ROWS, int HARD, int UPW>
__device__ __forceinline__ void record_copy(unsigned dst, const char* src, unsigned m, int lane) {
  constexpr int GPR = UPW / 2, RPC = 32 / GPR;  // 16-byte granules per row, rows per 512-byte piece
  const int il = lane / GPR, w = (lane % GPR) * 16;
#pragma unroll
  for (int q = 0; q * RPC < ROWS; ++q) {
    const int i = q * RPC + il;
    if (q * RPC < HARD || ((m >> (q * RPC / kRowGroup * kRowGroup)) & ((1u << kRowGroup) - 1))) {
      const unsigned sa = dst + q * 512 + lane * 16;
      const char* p = src + __popc(m & ((1u << i) - 1)) * (UPW * 8) + w;
      const int n = (m >> i) & 1u ? 16 : 0;
      if (i < ROWS) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(p), "r"(n) : "memory");
    }
  }
}
// Descriptions of consecutive records k = 0 .. n-1, one per lane for a block of 32
// and the next block: rec(k) for k in the current or the next block, col(k) for k
// in the current one; next(k) after record k.
struct RecordBlock {
  const uint4* src;
  int n, base, lane;
  uint4 cur, nxt;
  __device__ __forceinline__ uint4 load(int k) const {
    return k < n ? __ldg(src + k) : make_uint4(0u, 0u, 0u, 0u);
  }
  __device__ __forceinline__ RecordBlock(const uint4* s, int count, int ln) : src(s), n(count), base(0), lane(ln) {
    cur = load(lane);
    nxt = load(32 + lane);
  }
  __device__ __forceinline__ uint2 rec(int k) const {  // first row, mask
    const int i = k - base;
    const unsigned a = i < 32 ? cur.x : nxt.x, b = i < 32 ? cur.y : nxt.y;
    return make_uint2(__shfl_sync(0xffffffffu, a, i & 31), __shfl_sync(0xffffffffu, b, i & 31));
  }
  __device__ __forceinline__ uint2 col(int k) const {  // variable column, signs
    return make_uint2(__shfl_sync(0xffffffffu, cur.z, k & 31), __shfl_sync(0xffffffffu, cur.w, k & 31));
  }
  __device__ __forceinline__ void next(int k) {
    if ((k & 31) == 31) {
      base += 32;
      cur = nxt;
      nxt = load(base + 32 + lane);
    }
  }
};

// b = 2 g + class: the two classes of a group's systems run side by side, so that
// their interleaved entries of the stage output meet in L2 (class after class:
// 3.24 instead of 2.42 ms at 384^2 x 192)
template <int KL, int KV, int UPW>
__device__ __forceinline__ void subst_group(const SolveArgs& a, int b, unsigned char* ring) {
  using S = SubstShape<KL, KV, UPW>;
  constexpr int DF = S::DF, DB = S::DB;
  constexpr int RB = UPW * 8;  // bytes of a factor row
  const int lane = threadIdx.x & 31, unit = lane & (UPW - 1);
  const int T = a.Tc, cls = b & 1, g = b >> 1, G = cls * a.ngrp + g;
  const int sid = a.lane_sid[g * 32 + lane];
  const unsigned ring_s = (unsigned)__cvta_generic_to_shared(ring);
  double2* X = a.work2 + (size_t)G * T * 32 + lane;
  // ---- forward: rows j .. j+KL at r[s .. s+KL] in step s of the unrolled ones ----
  {
    constexpr int U = 4;
    constexpr int NA = KL < 6 ? KL : 6;       // L rows handled without a test
    const char* L = reinterpret_cast<const char*>(a.pack + pack_base(a.ptot, 0, cls, G, T, a.ldab) * UPW);
    const unsigned char* P = a.dpiv + (size_t)G * T * UPW;
    const int nc = T - 1;  // columns
    RecordBlock info(a.finfo + (size_t)cls * T, nc, lane);
    auto issue = [&](int c, int slot, uint2 rec) {  // column c and row c + KL
      const unsigned dst = ring_s + slot * S::kFSlot;
      if (c < nc) {
        record_copy<KL, KL, UPW>(dst, L + (size_t)rec.x * RB, rec.y, lane);
        if (lane < UPW / 16) cp_async16s(dst + S::kLBytes + lane * 16, P + (size_t)c * UPW + lane * 16);
        if (c + KL < T) cp_async16s(dst + S::kLBytes + UPW + lane * 16, X + (size_t)(c + KL) * 32);
      }
    };
#pragma unroll
    for (int c = 0; c < DF; ++c) {
      issue(c, c, info.rec(c));
      cp_async_commit();
    }
    uint2 recn = info.rec(DF);
    double2 r[KL + U + 1];
#pragma unroll
    for (int p = 0; p < KL; ++p) r[p] = p < T ? X[(size_t)p * 32] : zero2();
    int sw = DF, sr = 0;  // ring slots of columns j + DF and j
    // a column's pivot, L rows and incoming row, read one step ahead (of a column
    // past the last: stale, unused)
    int jp;
    double l[KL];
    double2 rin;
    auto read = [&](int slot, int& piv, double (&lv)[KL], double2& row) {
      const unsigned char* b = ring + slot * S::kFSlot;
      piv = b[S::kLBytes + unit];
#pragma unroll
      for (int i = 0; i < KL; ++i) lv[i] = reinterpret_cast<const double*>(b)[i * UPW + unit];
      row = *reinterpret_cast<const double2*>(b + S::kLBytes + UPW + lane * 16);
    };
    cp_async_wait<DF - 1>();
    __syncwarp();
    read(0, jp, l, rin);
    for (int j0 = 0; j0 < nc; j0 += U) {
#pragma unroll
      for (int s = 0; s < U; ++s) {
        const int j = j0 + s;
        if (j < nc) {
          const unsigned m = info.rec(j).y;
          cp_async_wait<DF - 2>();  // column j + 1's record is in
          __syncwarp();             // for every lane; and every lane is done with column j - 1's slot
          issue(j + DF, sw, recn);
          cp_async_commit();
          recn = info.rec(j + DF + 1);
          int jpn;
          double ln[KL];
          double2 rinn;
          sr = sr == DF ? 0 : sr + 1;
          sw = sw == DF ? 0 : sw + 1;
          read(sr, jpn, ln, rinn);
          r[s + KL] = rin;
          // row j + jp comes up, row j goes down
          double2 bj = r[s];
          const double2 x0 = r[s];
#pragma unroll
          for (int i = 1; i <= NA; ++i)
            if (jp == i) {
              bj = r[s + i];
              r[s + i] = x0;
            }
          const bool far = KL > NA && ((m >> NA) || __any_sync(0xffffffffu, jp > NA));
          if (far) {
#pragma unroll
            for (int i = NA + 1; i <= KL; ++i)
              if (jp == i) {
                bj = r[s + i];
                r[s + i] = x0;
              }
          }
#pragma unroll
          for (int i = 0; i < NA; ++i) {
            r[s + 1 + i].x -= l[i] * bj.x;
            r[s + 1 + i].y -= l[i] * bj.y;
          }
          if (far) {
#pragma unroll
            for (int i = NA; i < KL; ++i) {
              r[s + 1 + i].x -= l[i] * bj.x;
              r[s + 1 + i].y -= l[i] * bj.y;
            }
          }
          X[(size_t)j * 32] = bj;
          jp = jpn;
          rin = rinn;
#pragma unroll
          for (int i = 0; i < KL; ++i) l[i] = ln[i];
          info.next(j);
          if (j == nc - 1) X[(size_t)nc * 32] = r[s + 1];
        }
      }
#pragma unroll
      for (int p = 0; p < KL; ++p) r[p] = r[p + U];
    }
    cp_async_wait<0>();
    __threadfence();  // the copies below read the intermediate vector back
    __syncwarp();
  }
  // ---- backward: x_{j+i} at r[U-1-s+i] in step s of the unrolled ones ----
  {
    constexpr int U = KV > 24 ? 2 : 4;
    constexpr int NA = 12;   // U rows handled without a test (row 0 the diagonal)
    constexpr int CB = kRowGroup;
    static_assert(NA % CB == 0 && NA <= KV, "groups");
    const char* Up = reinterpret_cast<const char*>(a.pack + pack_base(a.ptot, 1, cls, G, T, a.ldab) * UPW);
    double2* out = a.out + (size_t)(sid >= 0 ? sid : 0) * a.T;
    bool bad = false;
    RecordBlock info(a.binfo + (size_t)cls * T, T, lane);
    auto issue = [&](int k, int slot, uint2 rec) {
      if (k < T) {
        const unsigned dst = ring_s + slot * S::kBSlot;
        record_copy<KV + 1, NA, UPW>(dst, Up + (size_t)rec.x * RB, rec.y, lane);
        cp_async16s(dst + S::kUBytes + lane * 16, X + (size_t)(T - 1 - k) * 32);
      }
    };
#pragma unroll
    for (int c = 0; c < DB; ++c) {
      issue(c, c, info.rec(c));
      cp_async_commit();
    }
    uint2 recn = info.rec(DB);
    double2 r[KV + U];
#pragma unroll
    for (int p = 0; p < KV + U; ++p) r[p] = zero2();
    int sw = DB, sr = 0;
    double u[NA];
    double2 y;
    auto read = [&](int slot, double (&uv)[NA], double2& row) {
      const unsigned char* b = ring + slot * S::kBSlot;
      row = *reinterpret_cast<const double2*>(b + S::kUBytes + lane * 16);
#pragma unroll
      for (int i = 0; i < NA; ++i) uv[i] = reinterpret_cast<const double*>(b)[i * UPW + unit];
    };
    cp_async_wait<DB - 1>();
    __syncwarp();
    read(0, u, y);
    for (int k0 = 0; k0 < T; k0 += U) {
#pragma unroll
      for (int s = 0; s < U; ++s) {
        const int k = k0 + s;
        if (k < T) {
          const unsigned m = info.rec(k).y;
          const uint2 col = info.col(k);
          cp_async_wait<DB - 2>();
          __syncwarp();
          issue(k + DB, sw, recn);
          cp_async_commit();
          recn = info.rec(k + DB + 1);
          const double* slot = reinterpret_cast<const double*>(ring + sr * S::kBSlot) + unit;
          sr = sr == DB ? 0 : sr + 1;
          sw = sw == DB ? 0 : sw + 1;
          double un[NA];
          double2 yn;
          read(sr, un, yn);
          // (one sum in the reference's order: the operators' conditioning turns
          // another order's rounding into 1e-9 of the pressure)
          double2 acc = y;
          if (m >> NA) {
#pragma unroll
            for (int i0 = (KV - NA) / CB * CB + NA; i0 >= NA; i0 -= CB) {
              if ((m >> i0) & ((1u << CB) - 1)) {
#pragma unroll
                for (int i = i0 + CB - 1; i >= i0; --i)
                  if (i <= KV) {
                    const double ui = slot[i * UPW];
                    acc.x -= ui * r[U - 1 - s + i].x;
                    acc.y -= ui * r[U - 1 - s + i].y;
                  }
              }
            }
          }
#pragma unroll
          for (int i = NA - 1; i >= 1; --i) {
            acc.x -= u[i] * r[U - 1 - s + i].x;
            acc.y -= u[i] * r[U - 1 - s + i].y;
          }
          const double2 xj = make_double2(acc.x * u[0], acc.y * u[0]);  // the diagonal is stored as its reciprocal
          r[U - 1 - s] = xj;
          const int t = (int)col.x;
          if (t >= 0 && sid >= 0) {
            double2 xo = flip_col(xj, col.y & 1u);
            if (UPW == 16 && lane >= 16 && (col.y & 2u)) xo = make_double2(-xo.x, -xo.y);
            bad |= !(isfinite(xo.x) && isfinite(xo.y));
            out[t] = xo;
          }
          y = yn;
#pragma unroll
          for (int i = 0; i < NA; ++i) u[i] = un[i];
          info.next(k);
        }
      }
#pragma unroll
      for (int i = KV; i >= 1; --i) r[U - 1 + i] = r[i - 1];
    }
    cp_async_wait<0>();
    if (bad) atomicOr(a.flags, 1u);
  }
}

template <int KL, int KV, int UPW>
__global__ void __launch_bounds__(32) k_subst_block(const __grid_constant__ SolveArgs a) {
  extern __shared__ __align__(16) unsigned char sbuf[];
  subst_group<KL, KV, UPW>(a, blockIdx.x, sbuf);
}

// The substitutions of many systems (the members of an ensemble) in one launch:
// CTA b takes group b of the members' concatenated groups (member m owns groups
// [prefix[m], prefix[m+1])); each group runs exactly the arithmetic of k_subst_block.
template <int KL, int KV>
__global__ void __launch_bounds__(32) k_subst_block_multi(const SolveArgs* args, const int* prefix, int nmem) {
  extern __shared__ __align__(16) unsigned char sbuf[];
  const int b = blockIdx.x;
  int lo = 0, hi = nmem - 1;  // member m with prefix[m] <= b < prefix[m+1]
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (prefix[mid] <= b) lo = mid;
    else hi = mid - 1;
  }
  const SolveArgs& a = args[lo];
  if (a.upw == 16) subst_group<KL, KV, 16>(a, b - prefix[lo], sbuf);
  else subst_group<KL, KV, 32>(a, b - prefix[lo], sbuf);
}

// ------------------------------------------------------------------------------
// Stage right-hand side with the NL assembly fused in, one CTA per (kx,ky) system
// (marching.f90:16-21, 93-125, 319-367):
//   Khat_i = sum_terms (i kx)^a (i ky)^b dsca trunc(I^Iz M^mz) qhat    (0 for inactive)
//   rhs    = M field + sum_{j<i} (dt a(i,j) Kstd_j + dt ahat(i+1,j) Khat_j) + dt ahat(i+1,i) Khat_i
// The system's quadratic-variable coefficients and state are first staged in
// shared memory with coalesced loads, so the row gathers run from shared memory.
// Active systems: rows flagged in rowflip are multiplied by -i for the real-scaled
// solve and the right-hand side goes to the solve's work layout.  Inactive systems
// (E = I): the right-hand side is the stage output itself (zero in the last
// stage), K_std_i = 0.
// ------------------------------------------------------------------------------
constexpr int kRhsThreads = 256;

// entry pc of class c of the system with slot word sl into the block layout
__device__ __forceinline__ void store_block_rhs(const SolveArgs& a, int sl, int c, int pc, unsigned char neg, double2 v) {
  if ((sl & kMirrorBit) && neg) v = make_double2(-v.x, -v.y);
  sl &= kMirrorBit - 1;
  a.work2[((size_t)(c * a.ngrp + (sl >> 5)) * a.Tc + pc) * 32 + (sl & 31)] = v;
}

// slots k0 .. k0 + 3 of row t.  Slots are filled in order and exact zeros are not
// stored, so a zero ends the row: a loop over batches that stops after the first
// batch with one leaves out nothing but further zero terms.
__device__ __forceinline__ void load_slots(const DevEll& op, int k0, int t, int (&cg)[4], double (&v)[4]) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const bool ok = k0 + u < op.width;
    cg[u] = ok ? op.cg[(size_t)(k0 + u) * op.rows + t] : 0;
    v[u] = ok ? op.val[(size_t)(k0 + u) * op.rows + t] : 0.0;
  }
}

// S consecutive systems per CTA, so that an operator entry is loaded once for S
// systems.  Bound by the loads of operator entries and the shared-memory gathers they
// address (2.5 k instructions a warp, half the cycles without an eligible warp): 143 us
// at 96^2 x 48 of the toroidal-poloidal recipe with one system, 127 with two.
template <int S>
__global__ void __launch_bounds__(kRhsThreads) k_rhs_nl(SolveArgs a, NLArgs n) {
  extern __shared__ double2 shr[];
  __shared__ double2 cms[S][kMaxGroups], cns[S][kMaxGroups];
  const int T = a.T, NZ = a.d.NZ, nsys = a.d.NXH * a.d.NYA, sid0 = blockIdx.x * S;
  const int nqz = n.nq * NZ, str = nqz + T;  // per system: [quad][n], then its state
  bool act[S], any = false;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    act[s] = sid0 + s < nsys && a.act_index[sid0 + s] >= 0;
    any |= act[s];
  }
  for (int e = threadIdx.x; e < S * kMaxGroups; e += blockDim.x) {
    const int s = e / kMaxGroups, g = e - s * kMaxGroups, sid = min(sid0 + s, nsys - 1);
    const int kx = sid / a.d.NYA, ky = sid - kx * a.d.NYA;
    cms[s][g] = (g < a.M.ngroups) ? cmul(ipow(a.kx[kx], a.M.gkx[g]), ipow(a.ky[ky], a.M.gky[g])) : zero2();
    cns[s][g] = (g < n.NL.ngroups) ? cmul(ipow(a.kx[kx], n.NL.gkx[g]), ipow(a.ky[ky], n.NL.gky[g])) : zero2();
  }
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int sid = sid0 + s;
    const size_t qstride = (size_t)nsys * NZ;  // between quad vars
    double2* qs = shr + s * str;
    if (act[s]) {
      // flat index idx = q NZ + nn, advanced without a division per element
      int q = threadIdx.x / NZ, nn = threadIdx.x - q * NZ;
      for (int idx = threadIdx.x; idx < nqz; idx += blockDim.x) {
        qs[idx] = n.qspec[q * qstride + (size_t)sid * NZ + nn];
        nn += blockDim.x;
        while (nn >= NZ) { nn -= NZ; ++q; }
      }
    }
    if (sid < nsys) {
      const double2* field = a.field + (size_t)sid * T;
      for (int t = threadIdx.x; t < T; t += blockDim.x) qs[nqz + t] = field[t];
    }
  }
  __syncthreads();
  bool bad = false;
  for (int t = threadIdx.x; t < T; t += blockDim.x) {
    double2 kh[S], r[S];
#pragma unroll
    for (int s = 0; s < S; ++s) kh[s] = r[s] = zero2();
    if (any) {
      // slots in batches of 4 independent loads; slots are filled in order and
      // exact zeros are not stored, so a zero ends the row
      for (int k0 = 0; k0 < n.NL.width; k0 += 4) {
        int cg[4];
        double v[4];
        load_slots(n.NL, k0, t, cg, v);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (v[u] != 0.0) {
#pragma unroll
            for (int s = 0; s < S; ++s)
              if (act[s]) {
                const double2 qh = shr[s * str + (cg[u] & 0xFFFFFF)];  // column = quad * NZ + n
                kh[s] = cadd(kh[s], cmul(cns[s][cg[u] >> 24], make_double2(v[u] * qh.x, v[u] * qh.y)));
              }
          }
        }
        if (v[3] == 0.0) break;
      }
    }
    for (int k0 = 0; k0 < a.M.width; k0 += 4) {
      int cg[4];
      double v[4];
      load_slots(a.M, k0, t, cg, v);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (k0 + u >= a.M.width) break;
#pragma unroll
        for (int s = 0; s < S; ++s)
          if (sid0 + s > 0 && sid0 + s < nsys) {  // not the origin
            const double2 xv = shr[s * str + nqz + (cg[u] & 0xFFFFFF)];
            r[s] = cadd(r[s], cmul(cms[s][cg[u] >> 24], make_double2(v[u] * xv.x, v[u] * xv.y)));
          }
      }
      if (v[3] == 0.0) break;
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int sid = sid0 + s;
      if (sid >= nsys) break;
      const size_t base = (size_t)sid * T;
      // K_hat of the last stage is used only here, from the register (the next step
      // starts from K_hat_0)
      if (!a.last_stage) n.Khat[base + t] = kh[s];
      double2 b = r[s];
#pragma unroll
      for (int j = 0; j < kMaxStages - 1; ++j) {  // static indices into the argument arrays
        if (j < a.nprev) {
          b = cadd(b, cscale(a.Kstd[j][base + t], a.ca[j]));
          b = cadd(b, cscale(a.Khat[j][base + t], a.ch[j]));
        }
      }
      b = cadd(b, cscale(kh[s], a.ch[a.nprev]));
      if (act[s]) {
        if (a.rowflip) b = flip_row(b, a.rowflip[t]);
        if (a.work2) {  // block layout, class order
          const int pos = a.row_pos[t], c = pos >= a.Tc ? 1 : 0;
          store_block_rhs(a, a.slot[sid], c, pos - c * a.Tc, a.row_neg[t], b);
        } else {
          a.work[(size_t)sid * T + t] = b;
        }
      } else {
        const double2 v = a.last_stage ? zero2() : b;
        bad |= !(isfinite(v.x) && isfinite(v.y));
        a.out[base + t] = v;
        if (a.Kstd_out) a.Kstd_out[base + t] = zero2();
      }
    }
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(a.flags, 1u);
}

// ------------------------------------------------------------------------------
// After the substitutions, one CTA per active system: the solution is staged in
// shared memory (from the solve's layout), then K_std_i = L x (S systems a CTA, a row
// ending at its first zero: 82 us -> 71 at 96^2 x 48, toroidal-poloidal), the stage output
// (the new state in the last stage) and the non-finite check.
// ------------------------------------------------------------------------------
template <int S>
__global__ void __launch_bounds__(kRhsThreads) k_kstd_out(SolveArgs a) {
  extern __shared__ double2 xs[];
  __shared__ double2 cls[S][kMaxGroups];
  const int a0 = blockIdx.x * S, ns = min(S, a.nact - a0), T = a.T;
  // block solve: the solution is already in out, original order, and
  // only K_std remains (L with its original columns); whole-system solve: the
  // solution is in work (class order = original order), copied to out here
  const bool in_out = a.work2 != nullptr;
  const DevEll& L = a.L;
  for (int e = threadIdx.x; e < ns * kMaxGroups; e += blockDim.x) {
    const int s = e / kMaxGroups, g = e - s * kMaxGroups, sid = a.act_list[a0 + s];
    const int kx = sid / a.d.NYA, ky = sid - kx * a.d.NYA;
    cls[s][g] = (g < L.ngroups) ? cmul(ipow(a.kx[kx], L.gkx[g]), ipow(a.ky[ky], L.gky[g])) : zero2();
  }
  for (int s = 0; s < ns; ++s) {
    const int sid = a.act_list[a0 + s];
    const double2* x = in_out ? a.out + (size_t)sid * T : a.work + (size_t)sid * T;
    for (int p = threadIdx.x; p < T; p += blockDim.x) xs[s * T + p] = x[p];
  }
  __syncthreads();
  bool bad = false;
  for (int t = threadIdx.x; t < T; t += blockDim.x) {
    if (!in_out) {
      for (int s = 0; s < ns; ++s) {
        const double2 v = xs[s * T + t];
        bad |= !(isfinite(v.x) && isfinite(v.y));
        if (a.out != a.work) a.out[(size_t)a.act_list[a0 + s] * T + t] = v;
      }
    }
    if (a.Kstd_out) {
      double2 ks[S];
#pragma unroll
      for (int s = 0; s < S; ++s) ks[s] = zero2();
      for (int k0 = 0; k0 < L.width; k0 += 4) {
        int cg[4];
        double v[4];
        load_slots(L, k0, t, cg, v);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (k0 + u >= L.width) break;
#pragma unroll
          for (int s = 0; s < S; ++s)
            if (s < ns) {
              const double2 xv = xs[s * T + (cg[u] & 0xFFFFFF)];
              ks[s] = cadd(ks[s], cmul(cls[s][cg[u] >> 24], make_double2(v[u] * xv.x, v[u] * xv.y)));
            }
        }
        if (v[3] == 0.0) break;
      }
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (s < ns) a.Kstd_out[(size_t)a.act_list[a0 + s] * T + t] = ks[s];
    }
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(a.flags, 1u);
}

// ------------------------------------------------------------------------------
// Operator-stationary K_std: a CTA takes one tile of kTileRows rows and kTileSys
// active systems.  Each thread keeps its row of L in grouped form (columns
// relative to the tile's solution window) in registers; the CTA first copies the
// windows of all its systems into shared memory (cp.async from the stage
// output), then evaluates its row for the systems one after the other: per
// monomial group a real sum, then one complex multiply by the group coefficient.
// ------------------------------------------------------------------------------
constexpr int kTileSys = 8;  // systems per CTA
constexpr int kLW = kGSlots;  // register slots of an L row (wider grouped L takes k_kstd_out)

// coefficient of group g of a grouped operator at (kx, ky)
__device__ __forceinline__ double2 gcoef(const DevGEll& G, int g, double kx, double ky) {
  double2 c = zero2();
  for (int m = 0; m < G.nmono[g]; ++m) c = cadd(c, cmul(ipow(kx, G.mkx[g][m]), ipow(ky, G.mky[g][m])));
  return c;
}
// one grouped row (slots in registers) applied to x: real sums per group, one
// complex multiply by the group coefficient c[g] per group
template <int RW>
__device__ __forceinline__ double2 grow(const DevGEll& G, const int* col, const double* val, const double2* x,
                                        const double2* c) {
  double2 r = zero2(), acc = zero2();
  int lg = 0;
#pragma unroll
  for (int k = 0; k < RW; ++k) {
    if (k < G.width) {
      if (k > 0 && G.slot_grp[k] != lg) {
        r = cadd(r, cmul(c[lg], acc));
        acc = zero2();
      }
      lg = G.slot_grp[k];
      if (val[k] != 0.0) {
        const double2 xv = x[col[k]];
        acc.x += val[k] * xv.x;
        acc.y += val[k] * xv.y;
      }
    }
  }
  if (G.width > 0) r = cadd(r, cmul(c[lg], acc));
  return r;
}

// G0..G3 > 0: the grouped L's slot ranges compiled (no run-time group test)
template <int G0 = 0, int G1 = 0, int G2 = 0, int G3 = 0>
__global__ void __launch_bounds__(kTileRows, 4) k_kstd_tiles(SolveArgs a) {
  extern __shared__ double2 xw[];
  __shared__ double2 cls[kTileSys][kMaxGroups];
  const int T = a.T;
  const int tile = blockIdx.x, t = tile * kTileRows + threadIdx.x;
  const bool row_ok = t < T;
  const int llo = a.tile_win[2 * tile], lw = a.tile_win[2 * tile + 1];
  const int a0 = blockIdx.y * kTileSys;
  const int ns = min(kTileSys, a.nact - a0);
  if (threadIdx.x < kTileSys * kMaxGroups) {
    const int u = threadIdx.x / kMaxGroups, g = threadIdx.x - u * kMaxGroups;
    const int sid = a.act_list[a0 + (u < ns ? u : 0)];
    const int kx = sid / a.d.NYA, ky = sid - kx * a.d.NYA;
    cls[u][g] = (g < a.Lw.ngroups) ? gcoef(a.Lw, g, a.kx[kx], a.ky[ky]) : zero2();
  }
  for (int u = 0; u < ns; ++u) {  // cp.async: no register round trip per system
    const double2* x = a.out + (size_t)a.act_list[a0 + u] * T + llo;
    for (int i = threadIdx.x; i < lw; i += kTileRows) cp_async16(xw + u * lw + i, x + i);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (!row_ok) return;
  int lc[kLW];
  double lv[kLW];
#pragma unroll
  for (int k = 0; k < kLW; ++k) {
    const bool ok = k < a.Lw.width;
    lc[k] = ok ? a.Lw.col[k * a.Lw.rows + t] : 0;
    lv[k] = ok ? a.Lw.val[k * a.Lw.rows + t] : 0.0;
  }
  for (int u = 0; u < ns; ++u) {
    double2 ks;
    if constexpr (G0 > 0) {
      constexpr int W = G0 + G1 + G2 + G3;
      static_assert(W <= kLW, "grouped L slots");
      const double2* x = xw + u * lw;
      double2 acc[4] = {zero2(), zero2(), zero2(), zero2()};
#pragma unroll
      for (int k = 0; k < W; ++k) {
        const int g = k < G0 ? 0 : (k < G0 + G1 ? 1 : (k < G0 + G1 + G2 ? 2 : 3));
        if (lv[k] != 0.0) {
          const double2 xv = x[lc[k]];
          acc[g].x += lv[k] * xv.x;
          acc[g].y += lv[k] * xv.y;
        }
      }
      ks = cmul(cls[u][0], acc[0]);
      if (G1 > 0) ks = cadd(ks, cmul(cls[u][1], acc[1]));
      if (G2 > 0) ks = cadd(ks, cmul(cls[u][2], acc[2]));
      if (G3 > 0) ks = cadd(ks, cmul(cls[u][3], acc[3]));
    } else {
      ks = grow<kLW>(a.Lw, lc, lv, xw + u * lw, cls[u]);
    }
    a.Kstd_out[(size_t)a.act_list[a0 + u] * T + t] = ks;
  }
}

// ------------------------------------------------------------------------------
// Operator-stationary right-hand side: a CTA takes one tile of kTileRows rows
// and kRhsSys consecutive systems (active or not).  Each thread keeps its row of
// M and of the NL operator (columns relative to the tile's windows) in
// registers; the CTA copies the state window and the quadratic-variable windows
// of its systems into shared memory with cp.async, then evaluates its row: first
// K_hat and M x of every system from shared memory, then the earlier stages' K
// arrays (loads of all systems in flight together), then the stores.  Same
// arithmetic and order as k_rhs_nl.
// ------------------------------------------------------------------------------
constexpr int kRhsSys = 4;  // systems per CTA
constexpr int kRhsStg = 4;  // window entries per thread with precomputed offsets (wider: plain loops)

// G0, G1, G2 > 0: the NL operator in grouped form (SolveArgs::NLg) with slot
// ranges of these widths per monomial group, compiled: per group a real sum,
// then one complex multiply by the group coefficient (RN = G0 + G1 + G2)
template <int RM, int RN, int G0 = 0, int G1 = 0, int G2 = 0>
__global__ void __launch_bounds__(kTileRows, 6) k_rhs_tiles(SolveArgs a, NLArgs n) {
  extern __shared__ double2 win[];
  __shared__ double2 cms[kRhsSys][kMaxGroups], cns[kRhsSys][kMaxGroups];
  const int T = a.T, NZ = a.d.NZ, nsys = a.d.NXH * a.d.NYA;
  const int tile = blockIdx.y, t = tile * kTileRows + threadIdx.x;
  const int* rw = a.rhs_win + tile * kRhsWin;
  const int mlo = rw[0], mw = rw[1], nlo = rw[2], nw = rw[3], nqt = rw[4];
  const int ws = mw + nqt * nw;  // window entries per system
  const int s0 = blockIdx.x * kRhsSys, ns = min(kRhsSys, nsys - s0);
  const size_t qstride = (size_t)nsys * NZ;  // between quadratic variables of qspec
  if (ws <= kRhsStg * kTileRows) {
    // window entry e = threadIdx.x + j kTileRows: the same source offset for every
    // system (plus the system's base), computed once
    size_t off[kRhsStg];
#pragma unroll
    for (int j = 0; j < kRhsStg; ++j) {
      const int e = threadIdx.x + j * kTileRows;
      if (e < mw) {
        off[j] = (size_t)(mlo + e);
      } else {
        const int i = e - mw, sl = i / nw, k = i - sl * nw;
        off[j] = e < ws ? rw[5 + sl] * qstride + nlo + k : 0;
      }
    }
    for (int u = 0; u < ns; ++u) {
      const int sid = s0 + u;
      const bool act = a.act_index[sid] >= 0;
      double2* w = win + u * ws;
      const double2* f = a.field + (size_t)sid * T;
      const double2* qb = n.qspec + (size_t)sid * NZ;
#pragma unroll
      for (int j = 0; j < kRhsStg; ++j) {
        const int e = threadIdx.x + j * kTileRows;
        if (e < mw) cp_async16(w + e, f + off[j]);
        else if (e < ws && act) cp_async16(w + e, qb + off[j]);
      }
    }
  } else {
    for (int u = 0; u < ns; ++u) {
      const int sid = s0 + u;
      double2* w = win + u * ws;
      const double2* f = a.field + (size_t)sid * T + mlo;
      for (int i = threadIdx.x; i < mw; i += kTileRows) cp_async16(w + i, f + i);
      if (a.act_index[sid] >= 0)
        for (int i = threadIdx.x; i < nqt * nw; i += kTileRows) {
          const int sl = i / nw, k = i - sl * nw;
          cp_async16(w + mw + i, n.qspec + rw[5 + sl] * qstride + (size_t)sid * NZ + nlo + k);
        }
    }
  }
  cp_async_commit();
  for (int i = threadIdx.x; i < kRhsSys * kMaxGroups; i += kTileRows) {
    const int u = i / kMaxGroups, g = i - u * kMaxGroups;
    const int sid = s0 + (u < ns ? u : 0);
    const int kx = sid / a.d.NYA, ky = sid - kx * a.d.NYA;
    cms[u][g] = (g < a.Mw.ngroups) ? cmul(ipow(a.kx[kx], a.Mw.gkx[g]), ipow(a.ky[ky], a.Mw.gky[g])) : zero2();
    if constexpr (G0 > 0)
      cns[u][g] = (g < a.NLg.ngroups) ? gcoef(a.NLg, g, a.kx[kx], a.ky[ky]) : zero2();
    else
      cns[u][g] = (g < a.NLw.ngroups) ? cmul(ipow(a.kx[kx], a.NLw.gkx[g]), ipow(a.ky[ky], a.NLw.gky[g])) : zero2();
  }
  const bool row_ok = t < T;
  const int tr = row_ok ? t : 0;
  int mcg[RM], ncg[RN];
  double mv[RM], nv[RN];
#pragma unroll
  for (int k = 0; k < RM; ++k) {
    const bool ok = k < a.Mw.width;
    mcg[k] = ok ? a.Mw.cg[(size_t)k * a.Mw.rows + tr] : 0;
    mv[k] = ok ? a.Mw.val[(size_t)k * a.Mw.rows + tr] : 0.0;
  }
  constexpr bool kGrouped = G0 > 0;
  static_assert(!kGrouped || G0 + G1 + G2 == RN, "grouped NL slots");
#pragma unroll
  for (int k = 0; k < RN; ++k) {
    if constexpr (kGrouped) {
      ncg[k] = a.NLg.col[(size_t)k * a.NLg.rows + tr];
      nv[k] = a.NLg.val[(size_t)k * a.NLg.rows + tr];
    } else {
      const bool ok = k < a.NLw.width;
      ncg[k] = ok ? a.NLw.cg[(size_t)k * a.NLw.rows + tr] : 0;
      nv[k] = ok ? a.NLw.val[(size_t)k * a.NLw.rows + tr] : 0.0;
    }
  }
  // shared-memory index and group of every slot
  int nix[RN], ngr[RN], mix[RM], mgr[RM];
#pragma unroll
  for (int k = 0; k < RN; ++k) {
    nix[k] = mw + (ncg[k] & 0xFFFFFF);
    ngr[k] = kGrouped ? 0 : ncg[k] >> 24;
  }
#pragma unroll
  for (int k = 0; k < RM; ++k) {
    mix[k] = mcg[k] & 0xFFFFFF;
    mgr[k] = mcg[k] >> 24;
  }
  // M with the single monomial 1 (every recipe here): its coefficient is exactly
  // 1 and the complex multiply is skipped (identical for finite values)
  const bool m_unit = a.Mw.ngroups == 1 && a.Mw.gkx[0] == 0 && a.Mw.gky[0] == 0;
  int ai[kRhsSys];  // slot words, -1: inactive
#pragma unroll
  for (int u = 0; u < kRhsSys; ++u) ai[u] = u < ns ? a.slot[s0 + u] : -1;
  cp_async_wait<0>();
  __syncthreads();
  if (!row_ok) return;  // no barrier below
  // phase 1 (shared memory only): K_hat and M x of every system
  double2 kh[kRhsSys], r[kRhsSys];
#pragma unroll
  for (int u = 0; u < kRhsSys; ++u) {
    kh[u] = zero2();
    r[u] = zero2();
    if (u < ns) {
      const double2* w = win + u * ws;
      if (ai[u] >= 0) {
        if constexpr (kGrouped) {
          double2 acc[3] = {zero2(), zero2(), zero2()};
#pragma unroll
          for (int k = 0; k < RN; ++k) {
            const int g = k < G0 ? 0 : (k < G0 + G1 ? 1 : 2);
            if (nv[k] != 0.0) {
              const double2 qh = w[nix[k]];
              acc[g].x += nv[k] * qh.x;
              acc[g].y += nv[k] * qh.y;
            }
          }
          kh[u] = cmul(cns[u][0], acc[0]);
          if (G1 > 0) kh[u] = cadd(kh[u], cmul(cns[u][1], acc[1]));
          if (G2 > 0) kh[u] = cadd(kh[u], cmul(cns[u][2], acc[2]));
        } else {
#pragma unroll
          for (int k = 0; k < RN; ++k)
            if (nv[k] != 0.0) {
              const double2 qh = w[nix[k]];
              kh[u] = cadd(kh[u], cmul(cns[u][ngr[k]], make_double2(nv[k] * qh.x, nv[k] * qh.y)));
            }
        }
      }
      if (s0 + u != 0) {
#pragma unroll
        for (int k = 0; k < RM; ++k)
          if (k < a.Mw.width) {
            const double2 xv = w[mix[k]];
            const double2 p = make_double2(mv[k] * xv.x, mv[k] * xv.y);
            r[u] = cadd(r[u], m_unit ? p : cmul(cms[u][mgr[k]], p));
          }
      }
    }
  }
  // phase 2: the earlier stages' K arrays (no store in between: the loads of all
  // systems can be in flight together)
#pragma unroll
  for (int j = 0; j < kMaxStages - 1; ++j) {  // static indices into the argument arrays
    if (j < a.nprev) {
#pragma unroll
      for (int u = 0; u < kRhsSys; ++u)
        if (u < ns) {
          const size_t base = (size_t)(s0 + u) * T + t;
          r[u] = cadd(r[u], cscale(a.Kstd[j][base], a.ca[j]));
          r[u] = cadd(r[u], cscale(a.Khat[j][base], a.ch[j]));
        }
    }
  }
  // phase 3: stores
  const int pos = a.row_pos[t], c = pos >= a.Tc ? 1 : 0, pc = pos - c * a.Tc;
  const unsigned char rf = a.rowflip ? a.rowflip[t] : 0, rn = a.row_neg[t];
  bool bad = false;
#pragma unroll
  for (int u = 0; u < kRhsSys; ++u) {
    if (u >= ns) break;
    const size_t base = (size_t)(s0 + u) * T;
    // K_hat of the last stage is used only here, from the register
    if (!a.last_stage) n.Khat[base + t] = kh[u];
    double2 v = cadd(r[u], cscale(kh[u], a.ch[a.nprev]));
    if (ai[u] >= 0) {
      if (a.rowflip) v = flip_row(v, rf);
      store_block_rhs(a, ai[u], c, pc, rn, v);
    } else {
      if (a.last_stage) v = zero2();
      bad |= !(isfinite(v.x) && isfinite(v.y));
      a.out[base + t] = v;
      if (a.Kstd_out) a.Kstd_out[base + t] = zero2();
    }
  }
  if (bad) atomicOr(a.flags, 1u);
}

// ------------------------------------------------------------------------------
// mean (kx = ky = 0) systems: real arithmetic, one warp per system
// ------------------------------------------------------------------------------
__device__ double ell_row_real(const DevEll& op, int t, const double* x) {
  double acc = 0.0;
  for (int k = 0; k < op.width; ++k) acc += op.v(t, k) * x[op.col(t, k)];
  return acc;
}

__global__ void k_zero_step(ZeroArgs a) {
  extern __shared__ double smd[];
  const int lane = threadIdx.x;
  const int s = blockIdx.x;
  if (s >= a.nsys) return;
  const ZeroSysDev& z = a.sys[s];
  const int T = z.T, i = a.stage;
  double* b = smd;
  double* kh = a.sys[s].Khat[i];
  // NL: K_hat_i from the real part of the (0,0) Chebyshev coefficients (marching.f90:372-397)
  for (int t = lane; t < T; t += 32) {
    double acc = 0.0;
    for (int k = 0; k < z.NL.width; ++k) {
      const int c = z.NL.col(t, k);
      const int qv = c / a.d.NZ, n = c - qv * a.d.NZ;
      acc += z.NL.v(t, k) * a.qspec[(size_t)qv * a.d.NXH * a.d.NYA * a.d.NZ + n].x;
    }
    if (z.src) acc += z.src[t];
    kh[t] = acc;
  }
  __syncwarp();
  for (int t = lane; t < T; t += 32) {
    double r = ell_row_real(z.M, t, z.field);
    for (int j = 0; j < i; ++j) {
      r = r + a.ca[j] * z.Kstd[j][t];
      r = r + a.ch[j] * z.Khat[j][t];
    }
    r = r + a.ch[i] * kh[t];
    b[t] = r;
  }
  // band solve with the factors staged in shared memory; the updates of one
  // column run across the lanes (each entry sees the same sequence of updates)
  const int kl = z.kl, kv = z.kl + z.ku, ldab = z.ldab;
  double* fab = smd + T;
  for (int e = lane; e < T * ldab; e += 32) fab[e] = z.ab[e];
  __syncwarp();
  for (int j = 0; j < T - 1; ++j) {
    const int p = j + z.dpiv[j];
    if (lane == 0 && p != j) { const double tmp = b[p]; b[p] = b[j]; b[j] = tmp; }
    __syncwarp();
    const double bj = b[j];
    const int lm = min(kl, T - 1 - j);
    for (int q = 1 + lane; q <= lm; q += 32) b[j + q] -= fab[j * ldab + kv + q] * bj;
    __syncwarp();
  }
  for (int j = T - 1; j >= 0; --j) {
    const double bj = b[j] * fab[j * ldab + kv];
    __syncwarp();
    if (lane == 0) b[j] = bj;
    for (int q = 1 + lane; q <= kv && j - q >= 0; q += 32) b[j - q] -= fab[j * ldab + kv - q] * bj;
    __syncwarp();
  }
  double* out = a.last_stage ? z.field : z.aux;
  if (!a.last_stage)
    for (int t = lane; t < T; t += 32) z.Kstd[i][t] = ell_row_real(z.L, t, b);
  __syncwarp();
  for (int t = lane; t < T; t += 32) out[t] = b[t];
}

// Factorisation of the mean systems (DGBTF2), one warp per system, in shared memory
// when the bands fit (smem_ok), else in place: lanes own the rows of the assembly
// and share a column's updates.  (One thread, in place:
// 0.41 ms at NZ 48; now 0.10 ms.)
__global__ void __launch_bounds__(32) k_zero_factor(ZeroArgs a, int smem_ok) {
  extern __shared__ double smd[];
  const int s = blockIdx.x, lane = threadIdx.x;
  if (s >= a.nsys) return;
  const ZeroSysDev& z = a.sys[s];
  const int T = z.T, kl = z.kl, ku = z.ku, kv = kl + ku, ldab = z.ldab;
  double* ab = smem_ok ? smd : z.ab;
  for (int e = lane; e < T * ldab; e += 32) ab[e] = 0.0;
  __syncwarp();
  for (int t = lane; t < T; t += 32) {
    for (int k = 0; k < z.M.width; ++k) {
      const double v = z.M.v(t, k);
      if (v == 0.0) continue;
      const int c = z.M.col(t, k);
      ab[(size_t)c * ldab + kv + t - c] += v;
    }
    for (int k = 0; k < z.L.width; ++k) {
      const double v = z.L.v(t, k);
      if (v == 0.0) continue;
      const int c = z.L.col(t, k);
      ab[(size_t)c * ldab + kv + t - c] += a.zsca * v;
    }
  }
  __syncwarp();
  int ju = 0, info = 0;
  for (int j = 0; j < T; ++j) {
    const int km = min(kl, T - 1 - j);
    double* cj = ab + (size_t)j * ldab + kv;
    double best = -1.0;
    int jp = 0;
    for (int q = lane; q <= km; q += 32) {
      const double v = fabs(cj[q]);
      if (v > best) { best = v; jp = q; }
    }
    for (int o = 16; o > 0; o >>= 1) {  // first maximum
      const double b2 = __shfl_xor_sync(0xffffffffu, best, o);
      const int q2 = __shfl_xor_sync(0xffffffffu, jp, o);
      if (b2 > best || (b2 == best && q2 < jp)) { best = b2; jp = q2; }
    }
    if (lane == 0) z.dpiv[j] = (unsigned char)jp;
    // (from the register all lanes share: lane 0 overwrites cj[jp] below)
    if (best == 0.0) { if (!info) info = j + 1; continue; }
    ju = max(ju, min(j + ku + jp, T - 1));
    __syncwarp();  // every lane has read the column
    if (jp != 0) {
      for (int c = j + lane; c <= ju; c += 32) {
        double* p1 = ab + (size_t)c * ldab + kv + j + jp - c;
        double* p0 = ab + (size_t)c * ldab + kv + j - c;
        const double t0 = *p0;
        *p0 = *p1;
        *p1 = t0;
      }
      __syncwarp();
    }
    const double r = 1.0 / cj[0];
    __syncwarp();
    for (int q = 1 + lane; q <= km; q += 32) cj[q] *= r;
    __syncwarp();
    const int nc = ju - j;
    for (int e = lane; e < nc * km; e += 32) {
      const int c = j + 1 + e / km, q = 1 + e % km;
      ab[(size_t)c * ldab + kv + j + q - c] -= cj[q] * ab[(size_t)c * ldab + kv + j - c];
    }
    if (lane == 0) cj[0] = r;
    __syncwarp();
  }
  if (smem_ok)
    for (int e = lane; e < T * ldab; e += 32) z.ab[e] = ab[e];
  if (lane == 0) a.info[s] = info;
}

// ------------------------------------------------------------------------------
// QuickSave / checkpoint helpers
// ------------------------------------------------------------------------------
__global__ void k_transpose_xy(Dims d, const double* in, double* out, int to_file) {
  const size_t n = (size_t)d.NXA * d.NYA * d.NZA;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const int z = (int)(e % d.NZA);
    const size_t r = e / d.NZA;
    // e indexes the output array
    if (to_file) {  // out[x][y][z] <- in[y][x][z]
      const int y = (int)(r % d.NYA), x = (int)(r / d.NYA);
      out[e] = in[((size_t)y * d.NXA + x) * d.NZA + z];
    } else {        // out[y][x][z] <- in[x][y][z]
      const int x = (int)(r % d.NXA), y = (int)(r / d.NXA);
      out[e] = in[((size_t)x * d.NYA + y) * d.NZA + z];
    }
  }
}

// ------------------------------------------------------------------------------
// User outputs (coral.usrOutput, PL_equations.f90:322-427) of one physical field
// phys[y][x][z], in the reference's file order (transforms.f90:53-105,772-866):
//   kind 1 ZSlice at z index k:  out[x][y] = phys(z = k)
//   kind 2 YSlice at y index k:  out[x][z] = phys(y = k)
//   kind 3 XSlice at x index k:  out[y][z] = phys(x = k)
//   kind 4 Zsummed:              out[x][y] = sum_z w(z) phys, z in grid order
// (indices 0-based here).  Profiles: k_usr_profile.
// ------------------------------------------------------------------------------
__global__ void k_usr_slice(Dims d, const double* phys, int kind, int k, const double* wz, double* out) {
  const size_t n = kind == 1 || kind == 4 ? (size_t)d.NXA * d.NYA
                   : kind == 2          ? (size_t)d.NXA * d.NZA
                                        : (size_t)d.NYA * d.NZA;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    double v;
    if (kind == 1 || kind == 4) {
      const int y = (int)(e % d.NYA), x = (int)(e / d.NYA);
      const double* col = phys + ((size_t)y * d.NXA + x) * d.NZA;
      if (kind == 1) {
        v = col[k];
      } else {
        v = 0.0;
        for (int z = 0; z < d.NZA; ++z) v += col[z] * wz[z];
      }
    } else if (kind == 2) {
      const int z = (int)(e % d.NZA), x = (int)(e / d.NZA);
      v = phys[((size_t)k * d.NXA + x) * d.NZA + z];
    } else {
      const int z = (int)(e % d.NZA), y = (int)(e / d.NZA);
      v = phys[((size_t)y * d.NXA + k) * d.NZA + z];
    }
    out[e] = v;
  }
}

// Horizontal average profile (export_Profile_fftw_mpi, PL_IMEX_timestepping_output.f90:
// 489-581): one CTA per z level, sum over x and y, then / NXAA / NYAA.
__global__ void __launch_bounds__(256) k_usr_profile(Dims d, const double* phys, double* out) {
  __shared__ double red[8];
  const int z = blockIdx.x;
  double s = 0.0;
  for (size_t e = threadIdx.x; e < (size_t)d.NXA * d.NYA; e += blockDim.x) s += phys[e * d.NZA + z];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[w];
    out[z] = t / d.NXA / d.NYA;
  }
}

// product of two physical fields (a quadratic variable), or a copy when b is null
__global__ void k_phys_product(size_t n, const double* a, const double* b, double* out) {
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    out[e] = b ? a[e] * b[e] : a[e];
}

// ------------------------------------------------------------------------------
// z derivatives in full-variable builds (compute_full_variables_in_physical_space,
// marching.f90:455-466, with differentiate_kxky, PL_IMEX_timestepping.f90:276-319):
// per (kx, ky) column, the Chebyshev coefficients of one kxky variable (its
// Galerkin stencil applied to the state) times dsca, differentiated `order`
// times -- the coefficients shifted down by one and back-substituted against
// the Chebyshev integration operator trunc(I)[rows 2..NZ, cols 1..NZ-1] (upper
// triangular: diagonal gap/2 at n = 0, gap/(4(n+1)) beyond; second
// super-diagonal -gap/(4(n+1)); prepare_chebyshev_integration, :488-505), the
// last coefficient zero -- into out[kx][ky][n].
// A column's back substitution is two serial chains (n even, n odd: d(n) needs
// d(n + 2)) of NZ / 2 divides each, so their latency bounds it: a CTA takes cols
// columns in shared memory, builds and writes them coalesced, and 4 threads a
// column run the chains (parity, component).  Each chain reads its next c(n + 1)
// before the step's d(n) overwrite the place.  (One thread a column in global
// memory: 70 us at 96^2 x 48, now 14.)
// ------------------------------------------------------------------------------
constexpr int kDzThreads = 128, kDzCols = 8;
// column stride in shared memory: 4 columns' places in different banks
__host__ __device__ inline int dz_stride(int NZ) { return NZ + ((2 - NZ) & 7); }

__global__ void __launch_bounds__(kDzThreads) k_full_dz(Dims d, const double2* state, int T, const int* tab_t,
                                                        const double* tab_v, double dsca, int order, double gap,
                                                        double2* out, int cols) {
  extern __shared__ double2 shd[];
  const int NZ = d.NZ, ld = dz_stride(NZ);
  double* piv = reinterpret_cast<double*>(shd + (size_t)cols * ld);  // gap / (4 (n + 1))
  const size_t ncol = (size_t)d.NXH * d.NYA, col0 = (size_t)blockIdx.x * cols;
  const int nc = (int)(ncol - col0 < (size_t)cols ? ncol - col0 : cols);
  for (int n = threadIdx.x; n < NZ; n += kDzThreads) piv[n] = gap / (4.0 * (n + 1));
  for (int e = threadIdx.x; e < nc * NZ; e += kDzThreads) {
    const int c = e / NZ, n = e - c * NZ;
    const double2* sv = state + (col0 + c) * T;
    double2 x = zero2();
    for (int k = 0; k < kTabW; ++k) {
      const int tt = tab_t[n * kTabW + k];
      if (tt >= 0) {
        const double w = tab_v[n * kTabW + k];
        const double2 f = sv[tt];
        x.x += w * f.x;
        x.y += w * f.y;
      }
    }
    shd[c * ld + n] = cscale(x, dsca);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int c = threadIdx.x >> 2, par = (threadIdx.x >> 1) & 1, comp = threadIdx.x & 1;
    const bool on = c < nc;
    double* o = reinterpret_cast<double*>(shd + (on ? c : 0) * ld) + comp;
    for (int r = 0; r < order; ++r) {
      int n = NZ - 2 - par;
      double chi = n >= 0 ? o[2 * (n + 1)] : 0.0, dp2 = 0.0;  // c(n + 1), d(n + 2)
      for (int k = 0; k < NZ / 2; ++k, n -= 2) {
        const double cn = n >= 1 ? o[2 * (n - 1)] : 0.0;
        __syncwarp();
        if (n >= 0) {
          const double diag = (n == 0) ? 0.5 * gap : piv[n];
          const double sup = -piv[n];
          const double v = (n + 2 <= NZ - 2) ? chi - sup * dp2 : chi;
          const double dn = v / diag;
          if (on) o[2 * n] = dn;
          dp2 = dn;
        }
        chi = cn;
      }
      __syncwarp();
      if (on && par == 0) o[2 * (NZ - 1)] = 0.0;
      __syncwarp();
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nc * NZ; e += kDzThreads) {
    const int c = e / NZ, n = e - c * NZ;
    out[(col0 + c) * NZ + n] = shd[c * ld + n];
  }
}

// The same for a mean variable (differentiate_zero, PL_IMEX_timestepping.f90:
// 321-360): one real profile, one thread.
__global__ void k_zero_dz(int NZ, const double* state, const int* tab_t, const double* tab_v, double dsca,
                          int order, double gap, double* out) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  for (int n = 0; n < NZ; ++n) {
    double c = 0.0;
    for (int k = 0; k < kTabW; ++k) {
      const int tt = tab_t[n * kTabW + k];
      if (tt >= 0) c += tab_v[n * kTabW + k] * state[tt];
    }
    out[n] = c * dsca;
  }
  for (int r = 0; r < order; ++r) {
    double chi = out[NZ - 1], dp1 = 0.0, dp2 = 0.0;
    for (int n = NZ - 2; n >= 0; --n) {
      const double cn = out[n];
      const double diag = (n == 0) ? 0.5 * gap : gap / (4.0 * (n + 1));
      const double sup = -gap / (4.0 * (n + 1));
      const double v = (n + 2 <= NZ - 2) ? chi - sup * dp2 : chi;
      const double dn = v / diag;
      out[n] = dn;
      chi = cn;
      dp2 = dp1;
      dp1 = dn;
    }
    out[NZ - 1] = 0.0;
  }
}

// Projection of Chebyshev coefficients onto one variable's Galerkin basis
// (square-stencil solve of import_quicksave, PL_IMEX_timestepping_output.f90:343-355).
// The square stencil is lower triangular, so a forward substitution solves it;
// the caller has zeroed the state, so the result is written into the slots.
__global__ void k_galerkin_insert(Dims d, const double2* spec, int T, const int* var_pos, int nc,
                                  const double* sq, const int* sq_col, double2* field) {
  const size_t col = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= (size_t)d.NXH * d.NYA) return;
  const double2* c = spec + col * d.NZ;
  double2* f = field + col * T;
  for (int r = 0; r < nc; ++r) {
    double2 acc = c[r];
    double diag = 1.0;
    for (int k = 0; k < kTabW; ++k) {
      const int cc = sq_col[r * kTabW + k];
      if (cc < 0) continue;
      const double v = sq[r * kTabW + k];
      if (cc == r) diag = v;
      else if (cc < r) acc = csub(acc, cscale(f[var_pos[cc]], v));
    }
    f[var_pos[r]] = make_double2(acc.x / diag, acc.y / diag);
  }
}

__global__ void k_cheb_extract(Dims d, const double2* field, int T, const int* tab_t, const double* tab_v,
                               double2* spec) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t n_all = (size_t)d.NXH * d.NYA * d.NZ;
  if (e >= n_all) return;
  const int n = (int)(e % d.NZ);
  const size_t col = e / d.NZ;
  const double2* f = field + col * T;
  double2 s = zero2();
  for (int k = 0; k < kTabW; ++k) {
    const int tt = tab_t[n * kTabW + k];
    if (tt >= 0) s = cadd(s, cscale(f[tt], tab_v[n * kTabW + k]));
  }
  spec[e] = s;
}

__global__ void k_check_finite(const double2* x, size_t n, unsigned int* flags) {
  bool bad = false;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    bad |= !(isfinite(x[e].x) && isfinite(x[e].y));
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flags, 1u);
}

int grid1d(size_t n, int bs) { return (int)((n + bs - 1) / bs); }

// Raise a kernel's dynamic shared-memory limit when its static plus dynamic
// shared memory exceeds the default 48 KB (a launch above it without the
// attribute is an invalid argument); a refused attribute is reported with the
// kernel and the size (instead of surfacing later as a generic launch failure).
template <typename K>
void set_smem_named(const char* name, K kernel, size_t bytes) {
  size_t stat = 0;
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, kernel) == cudaSuccess) stat = fa.sharedSizeBytes;
  else cudaGetLastError();
  if (bytes + stat <= 48 * 1024) return;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();  // the refusal is reported here, not left for the next launch check
    throw CoralError(CORAL_ECUDA, std::string("cudaFuncSetAttribute(") + name + ", dynamic shared memory " +
                                      std::to_string(bytes) + " bytes): " + cudaGetErrorString(e));
  }
}
// (variadic so that template argument lists pass through; the text names the call)
#define set_smem(...) set_smem_named(#__VA_ARGS__, __VA_ARGS__)
// CTAs with that much dynamic shared memory that an SM's shared memory holds (0: refused)
template <typename K>
int resident_by_smem(K kernel, size_t bytes) {
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  int dev = 0, optin = 0, sm = 0, reserved = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
  const size_t total = fa.sharedSizeBytes + bytes;
  return total > (size_t)optin ? 0 : (int)((size_t)sm / (total + reserved));
}

}  // namespace

// ---- launchers ----------------------------------------------------------------
template <template <int> class L, typename... Args>
void dispatch_len(int n, Args&&... args) {
  switch (n) {
#define CORAL_CASE(v) \
  case v:             \
    L<v>::run(args...); \
    return;
    CORAL_FFT_LENGTHS(CORAL_CASE)
#undef CORAL_CASE
    default:
      L<0>::run(args...);
  }
}

// CTAs of a persistent kernel: as many as fit on the device at once
template <class K>
int persistent_ctas(K kernel, int threads, size_t smem) {
  int dev = 0, nsm = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem);
  return std::max(1, nsm * std::max(per, 1));
}

template <int NF>
struct InvY {
  static void run(const Dims& d, int nf, const FullVarDev* fv, StateSet st, const double2* plain_spec,
                  const double* kx, const double* ky, double2* Y1, const FftPlan& py, int single, cudaStream_t s) {
    size_t sm = (NF ? 1 : 2) * kNB1 * (size_t)(NF ? line_stride(NF, kPlanY) : d.NYA + kPadRt) * sizeof(double2);
    dim3 g(nf, (d.NZ + kNB1 - 1) / kNB1, d.NXH);
    if (single && !plain_spec) {
      set_smem(k_inv_y1<NF>, sm);
      k_inv_y1<NF><<<g, kThreadsY, sm, s>>>(d, fv, st, kx, ky, Y1, py);
      return;
    }
    set_smem(k_inv_y<NF>, sm);
    k_inv_y<NF><<<g, kThreadsY, sm, s>>>(d, fv, st, plain_spec, kx, ky, Y1, py);
  }
};
template <int NF>
struct InvX {
  template <int PV>
  static void go(const Dims& d, int nf, const double2* Y1, double* Y2, const FftPlan& px, cudaStream_t s) {
    go<PV>(d, nf, Y1, Y2, px, 0, d.NYA, s);
  }
  template <int PV>
  static void go(const Dims& d, int nf, const double2* Y1, double* Y2, const FftPlan& px, int y0, int ny,
                 cudaStream_t s) {
    size_t sm = (NF ? 1 : 2) * (kNB2 / 2) * (size_t)(NF ? line_stride(NF, PV) : d.NXA + kPadRt) * sizeof(double2);
    set_smem(k_inv_x<NF, PV>, sm);
    dim3 g(nf, (d.NZ + kNB2 - 1) / kNB2, ny);
    k_inv_x<NF, PV><<<g, kThreadsX, sm, s>>>(d, Y1, Y2, px, y0);
  }
  static void rows(const Dims& d, int nf, const double2* Y1, double* Y2, const FftPlan& px, int pv, int y0, int ny,
                   cudaStream_t s) {
    if (pv) go<1>(d, nf, Y1, Y2, px, y0, ny, s);
    else go<0>(d, nf, Y1, Y2, px, y0, ny, s);
  }
  static void run(const Dims& d, int nf, const double2* Y1, double* Y2, const FftPlan& px, int pv, int tiles,
                  cudaStream_t s) {
    if constexpr (NF != 0 && plan_of(NF, 1).nst == 2) {
      if (pv && !tiles) {
        // persistent pipelined kernel: as many CTAs as fit on the device at once
        const size_t sm = ((kNB2 / 2) * (size_t)line_stride(NF, 1) + (size_t)d.NXH * kStgX) * sizeof(double2);
        set_smem(k_inv_x_pipe<NF>, sm);
        static int nct = 0;
        if (!nct) nct = persistent_ctas(k_inv_x_pipe<NF>, kThreadsXP, sm);
        const int ntiles = nf * ((d.NZ + kNB2 - 1) / kNB2) * d.NYA;
        k_inv_x_pipe<NF><<<std::min(nct, ntiles), kThreadsXP, sm, s>>>(d, nf, Y1, Y2, px);
        return;
      }
    }
    if (pv) go<1>(d, nf, Y1, Y2, px, s);
    else go<0>(d, nf, Y1, Y2, px, s);
  }
};
template <int NF>
struct InvZ {
  static void run(const Dims& d, int nf, const double* Y2, double* phys, const FftPlan& pz, const double2* dct_tw,
                  const double* wz, unsigned long long* cfl_bits, cudaStream_t s) {
    size_t sm = (NF ? 1 : 2) * (kXB3 / 2) * (size_t)(NF ? line_len(NF, kPlanInvZ, false) : d.NZA) * sizeof(double2);
    set_smem(k_inv_z<NF>, sm);
    dim3 g(nf, (d.NXA + kXB3 - 1) / kXB3, d.NYA);
    k_inv_z<NF><<<g, kThreadsIZ, sm, s>>>(d, Y2, phys, pz, dct_tw, wz, cfl_bits);
  }
};
template <int NF>
struct FwdZ {
  static void run(const Dims& d, int nf, const QuadDesc& q, const double* phys, double* Q2, const FftPlan& pz,
                  const double2* dct_tw, const double* wz, double* ke_partial, cudaStream_t s) {
    // one variable of 432 points: few of the threads have a butterfly, and the run-time
    // plan's smaller ones are faster (73 us, compiled 92 us)
    if constexpr (NF == 432) {
      if (q.nq == 1) return FwdZ<0>::run(d, nf, q, phys, Q2, pz, dct_tw, wz, ke_partial, s);
    }
    size_t sm = (size_t)nf * d.NZA * sizeof(double2) + (NF ? 1 : 2) * (size_t)std::min(q.nq, kQC) * d.NZA * sizeof(double2);
    set_smem(k_fwd_z<NF>, sm);
    dim3 g((d.NXA + 1) / 2, d.NYA);
    k_fwd_z<NF><<<g, kThreads, sm, s>>>(d, nf, q, phys, Q2, pz, dct_tw, wz, ke_partial);
  }
};
template <int NF>
struct ZFused {
  template <int FB>
  static size_t bytes(int nf, const Dims& d) {
    const size_t lines = (size_t)nf * kZPairs + FB + (NF ? 0 : std::max(kZLines, FB));
    return lines * (NF ? line_len(NF, kPlanHot, false) : d.NZA) * sizeof(double2);
  }
  // CTAs that an SM's shared memory holds
  template <int FB>
  static int resident(int nf, const Dims& d) {
    return resident_by_smem(k_z_fused<NF, FB>, bytes<FB>(nf, d));
  }
  template <int FB>
  static void go(const Dims& d, int nf, const QuadDesc& q, const double* Y2, double* Q2, const FftPlan& pz,
                 const double2* dct_tw, const double* wz, const double* wzinv, unsigned long long* cfl_bits,
                 double* ke_partial, int y0, int ny, cudaStream_t s) {
    const size_t sm = bytes<FB>(nf, d);
    set_smem(k_z_fused<NF, FB>, sm);
    dim3 g((d.NXA + 2 * kZPairs - 1) / (2 * kZPairs), ny);
    k_z_fused<NF, FB><<<g, z_threads_fused(NF, FB), sm, s>>>(d, nf, q, Y2, Q2, pz, dct_tw, wz, wzinv, cfl_bits,
                                                               ke_partial, y0);
  }
  static void run(const Dims& d, int nf, const QuadDesc& q, const double* Y2, double* Q2, const FftPlan& pz,
                  const double2* dct_tw, const double* wz, const double* wzinv, unsigned long long* cfl_bits,
                  double* ke_partial, int batch6, int y0, int ny, cudaStream_t s) {
    if (NF != 0 && 3 * d.NZ != 2 * NF) {  // compiled lengths assume NZAA = 3 NZ / 2
      ZFused<0>::run(d, nf, q, Y2, Q2, pz, dct_tw, wz, wzinv, cfl_bits, ke_partial, batch6, y0, ny, s);
      return;
    }
    // Up to 4 full variables batches of 6 lines (unless the variant asks for 9); above
    // that of 9, but of 6 where an SM's shared memory then holds two CTAs and not one (ms
    // a step with 9 | 6 lines: 7 variables at 96^2 x 192 9.06 | 8.57, 5 at 64^2 x 256
    // 2.88 | 2.70), or one and not none (7 or 8 variables at NZ 384).
    const bool six = batch6 && (nf <= 4 || (resident<kZFwd>(nf, d) < 2 && resident<6>(nf, d) > resident<kZFwd>(nf, d)));
    if (six || resident<kZFwd>(nf, d) < 1)
      go<6>(d, nf, q, Y2, Q2, pz, dct_tw, wz, wzinv, cfl_bits, ke_partial, y0, ny, s);
    else
      go<kZFwd>(d, nf, q, Y2, Q2, pz, dct_tw, wz, wzinv, cfl_bits, ke_partial, y0, ny, s);
  }
};
template <int NF>
struct FwdX {
  template <int PV>
  static void go(const Dims& d, int nq, const double* Q2, double2* Q1, const FftPlan& px, int y0, int ny,
                 cudaStream_t s) {
    size_t sm = (NF ? 1 : 2) * (kNB2 / 2) * (size_t)(NF ? line_stride(NF, PV) : d.NXA + kPadRt) * sizeof(double2);
    set_smem(k_fwd_x<NF, PV>, sm);
    dim3 g(nq, (d.NZ + kNB2 - 1) / kNB2, ny);
    k_fwd_x<NF, PV><<<g, kThreadsX, sm, s>>>(d, Q2, Q1, px, y0);
  }
  static void run(const Dims& d, int nq, const double* Q2, double2* Q1, const FftPlan& px, int pv, int y0, int ny,
                  cudaStream_t s) {
    if (pv) go<1>(d, nq, Q2, Q1, px, y0, ny, s);
    else go<0>(d, nq, Q2, Q1, px, y0, ny, s);
  }
};
template <int NF>
struct FwdY {
  static void run(const Dims& d, int nq, const double2* Q1, double2* qspec, double scale, const FftPlan& py,
                  int grid_variant, cudaStream_t s) {
    if constexpr (NF != 0) {
      if (!grid_variant) {
      // persistent pipelined kernel: as many CTAs as fit on the device at once
      const size_t sm = (kNB1 * (size_t)line_stride(NF, kPlanYF) + (size_t)NF * kNB1) * sizeof(double2);
      set_smem(k_fwd_y_pipe<NF>, sm);
      static int nct = 0;
      if (!nct) nct = persistent_ctas(k_fwd_y_pipe<NF>, kThreadsYF, sm);
      const int ntiles = nq * ((d.NZ + kNB1 - 1) / kNB1) * d.NXH;
      k_fwd_y_pipe<NF><<<std::min(nct, ntiles), kThreadsYF, sm, s>>>(d, nq, Q1, qspec, scale, py);
      return;
    }
    }
    size_t sm = (NF ? 1 : 2) * kNB1 * (size_t)(NF ? line_stride(NF, kPlanY) : d.NYA + kPadRt) * sizeof(double2);
    set_smem(k_fwd_y<NF>, sm);
    dim3 g(nq, (d.NZ + kNB1 - 1) / kNB1, d.NXH);
    k_fwd_y<NF><<<g, kThreadsY, sm, s>>>(d, Q1, qspec, scale, py);
  }
};

void launch_inv_y(const Dims& d, int nf, const FullVarDev* fv, StateSet st, const double2* plain_spec,
                  const double* kx, const double* ky, double2* Y1, const FftPlan& py, cudaStream_t s, int single) {
  dispatch_len<InvY>(d.NYA, d, nf, fv, st, plain_spec, kx, ky, Y1, py, single, s);
}
void launch_z_fused(const Dims& d, int nf, const QuadDesc& q, const double* Y2, double* Q2, const FftPlan& pz,
                    const double2* dct_tw, const double* wz, const double* wzinv, unsigned long long* cfl_bits,
                    double* ke_partial, cudaStream_t s, int batch6, int y0, int ny) {
  if (ny < 0) ny = d.NYA - y0;
  dispatch_len<ZFused>(d.NZA, d, nf, q, Y2, Q2, pz, dct_tw, wz, wzinv, cfl_bits, ke_partial, batch6, y0, ny, s);
}
template <int NF>
struct InvXRows {
  static void run(const Dims& d, int nf, const double2* Y1, double* Y2, const FftPlan& px, int pv, int y0, int ny,
                  cudaStream_t s) {
    InvX<NF>::rows(d, nf, Y1, Y2, px, pv, y0, ny, s);
  }
};
void launch_inv_x_rows(const Dims& d, int nf, const double2* Y1, double* Y2, const FftPlan& px, int pv, int y0, int ny,
                       cudaStream_t s) {
  dispatch_len<InvXRows>(d.NXA, d, nf, Y1, Y2, px, pv, y0, ny, s);
}
void launch_inv_x(const Dims& d, int nf, const double2* Y1, double* Y2, const FftPlan& px, cudaStream_t s, int pv,
                  int tiles) {
  dispatch_len<InvX>(d.NXA, d, nf, Y1, Y2, px, pv, tiles, s);
}
void launch_inv_z(const Dims& d, int nf, const double* Y2, double* phys, const FftPlan& pz,
                  const double2* dct_tw, const double* wz, unsigned long long* cfl_bits, cudaStream_t s) {
  dispatch_len<InvZ>(d.NZA, d, nf, Y2, phys, pz, dct_tw, wz, cfl_bits, s);
}
void launch_fwd_z(const Dims& d, int nf, const QuadDesc& q, const double* phys, double* Q2, const FftPlan& pz,
                  const double2* dct_tw, const double* wz, double* ke_partial, cudaStream_t s) {
  dispatch_len<FwdZ>(d.NZA, d, nf, q, phys, Q2, pz, dct_tw, wz, ke_partial, s);
}
void launch_fwd_x(const Dims& d, int nq, const double* Q2, double2* Q1, const FftPlan& px, cudaStream_t s, int pv,
                  int y0, int ny) {
  if (ny < 0) ny = d.NYA - y0;
  dispatch_len<FwdX>(d.NXA, d, nq, Q2, Q1, px, pv, y0, ny, s);
}
void launch_fwd_y(const Dims& d, int nq, const double2* Q1, double2* qspec, double scale, const FftPlan& py,
                  cudaStream_t s, int grid_variant) {
  dispatch_len<FwdY>(d.NYA, d, nq, Q1, qspec, scale, py, grid_variant, s);
}
// total of the KE partial sums written by the z kernels: one CTA, each thread a
// strided sum, then a fixed-order tree
__global__ void __launch_bounds__(1024) k_ke_sum(const double* part, size_t n, double* out) {
  __shared__ double red[32];
  double v = 0.0;
  for (size_t i = threadIdx.x; i < n; i += blockDim.x) v += part[i];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) *out = v;
  }
}
size_t z_fused_ctas(const Dims& d) { return (size_t)((d.NXA + 2 * kZPairs - 1) / (2 * kZPairs)) * d.NYA; }
void launch_ke_sum(const double* part, size_t n, double* out, cudaStream_t s) {
  k_ke_sum<<<1, 1024, 0, s>>>(part, n, out);
}
void launch_remove_zmean(const Dims& d, double2* qspec_q, cudaStream_t s) {
  k_remove_zmean<<<grid1d((size_t)d.NXH * d.NYA, 128), 128, 0, s>>>(d, qspec_q);
}

// ------------------------------------------------------------------------------
// full variables that are not plain transforms (marching.f90:505-575)
// ------------------------------------------------------------------------------
namespace {

// z operations of one CTA on kZfCols consecutive x columns of one y row, whose
// Chebyshev coefficients are contiguous in Y2: the tile is staged in shared
// memory and each column runs the reference's loops in its order.  Y2 holds
// c_0 and c_n / 2 (n >= 1; the inverse y pass folds the x padding's 0.5 and
// the REDFT01 convention in), so every c_n (n >= 1) read into c_0 is 2 Y2[n]
// (exact).
constexpr int kZfCols = 16;
__global__ void k_zfilter(Dims d, double* Y2v, int extract, int decomp, int y0) {
  extern __shared__ double tile[];
  const int NZ = d.NZ, y = y0 + blockIdx.y, xc0 = blockIdx.x * kZfCols;
  const int nc = min(kZfCols, d.NXA - xc0);
  double* base = Y2v + ((size_t)y * d.NXA + xc0) * NZ;
  for (int i = threadIdx.x; i < nc * NZ; i += blockDim.x) tile[i] = base[i];
  __syncthreads();
  if ((int)threadIdx.x < nc) {
    double* c = tile + threadIdx.x * NZ;
    if (extract == 1) {  // bottom surface: T_n(-1) = (-1)^n
      for (int iz = 2; iz <= NZ; ++iz) {
        c[0] = c[0] - (2.0 * c[iz - 1]) * ((iz & 1) ? -1.0 : 1.0);
        c[iz - 1] = 0.0;
      }
    } else if (extract == 2) {  // top surface: T_n(1) = 1
      for (int iz = 2; iz <= NZ; ++iz) {
        c[0] = c[0] + 2.0 * c[iz - 1];
        c[iz - 1] = 0.0;
      }
    }
    if (decomp == 2) {  // baroclinic: the vertical mean removed (PL_IMEX_timestepping.f90:238-250)
      c[0] = 0.0;
      for (int q = 1; q < NZ / 2; ++q)
        c[0] = c[0] - (2.0 * c[2 * q]) * (0.5 / (2.0 * q + 1.0) - 0.5 / (2.0 * q - 1.0));
    } else if (decomp == 1) {  // barotropic: the vertical fluctuations removed (:252-274)
      for (int q = 1; q < NZ / 2; ++q) {
        c[0] = c[0] + (2.0 * c[2 * q]) * (0.5 / (2.0 * q + 1.0) - 0.5 / (2.0 * q - 1.0));
        c[2 * q - 1] = 0.0;
        c[2 * q] = 0.0;
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nc * NZ; i += blockDim.x) base[i] = tile[i];
}

__global__ void k_static_phys(Dims d, QuadDesc q, double* phys) {
  const size_t n = (size_t)d.NYA * d.NXA * d.NZA;
  for (int k = 0; k < q.st_n; ++k) {
    double* dst = phys + (size_t)q.st_var[k] * n;
    const double* src = q.st_src[k];
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
      dst[i] = q.st_prof[k] ? src[i % d.NZA] : src[i];
  }
}

struct SmagoVars {
  int n;
  int v[4];
};
// part[y][z]: the sum over x of the squares of the variables at (y, z); one CTA
// per y row, threads along z (contiguous in phys)
__global__ void k_smago_rows(Dims d, const double* phys, SmagoVars sv, double* part) {
  const int y = blockIdx.x;
  const size_t n = (size_t)d.NYA * d.NXA * d.NZA;
  for (int z = threadIdx.x; z < d.NZA; z += blockDim.x) {
    double acc = 0.0;
    for (int x = 0; x < d.NXA; ++x) {
      const size_t at = ((size_t)y * d.NXA + x) * d.NZA + z;
      double s = 0.0;
      for (int k = 0; k < sv.n; ++k) {
        const double v = phys[(size_t)sv.v[k] * n + at];
        s += v * v;
      }
      acc += s;
    }
    part[(size_t)y * d.NZA + z] = acc;
  }
}
// prof[z] = c sqrt(prof[z] + sum_y part[y][z] / NXA / NYA); the maximum to cfl_max
__global__ void k_smago_final(Dims d, const double* part, double c, double* prof, unsigned long long* cfl_max) {
  __shared__ double red[32];
  double mx = 0.0;
  for (int z = threadIdx.x; z < d.NZA; z += blockDim.x) {
    double s = 0.0;
    for (int y = 0; y < d.NYA; ++y) s += part[(size_t)y * d.NZA + z];
    const double p = c * sqrt(prof[z] + s / d.NXA / d.NYA);
    prof[z] = p;
    mx = fmax(mx, p);
  }
  if (!cfl_max) return;
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m2 = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m2 = fmax(m2, red[w]);
    atomic_max_nonneg(cfl_max, m2);
  }
}

// PL_user_penalisation_mask.f90 as the reference ships it: two masks, the
// larger taken; grid labels x = (i + 2) Lx / NXAA, y = (j + 2) Ly / NYAA
// (PL_geometry.f90:138-145 with phys_iStart = 1); pi, 0.9 and 0.1 are
// single-precision literals there
__global__ void k_penal_default(Dims d, double Lx, double Ly, const double* zgrid, double* mask) {
  const size_t n = (size_t)d.NYA * d.NXA * d.NZA;
  const double pi = (double)3.14159265358979311599796346854f, c09 = (double)0.9f, c01 = (double)0.1f;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int k = (int)(i % d.NZA);
    const size_t r = i / d.NZA;
    const int ix = (int)(r % d.NXA), iy = (int)(r / d.NXA);
    const double x = (double)(ix + 2) * Lx / d.NXA, y = (double)(iy + 2) * Ly / d.NYA, z = zgrid[k];
    const double m1 = z - (c09 + c01 * cos(5.0 * (x + y) * 2.0 * pi / Lx));
    const double cx = 6.0 + cos(2.0 * pi * x / Lx);
    const double m2 = (0.4 * exp(-(cx * cx)) / exp(-25.0)) - z;
    mask[i] = fmax(m1, m2);
  }
}
// init_penalisation (marching.f90:812-816)
__global__ void k_penal_field(size_t n, const double* mask, double strength, double width, double* out) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    double pm = tanh(width * mask[i]);
    pm = (1.0 + pm) / 2.0;
    out[i] = strength * pm;
  }
}

}  // namespace

void launch_zfilter(const Dims& d, double* Y2_var, int extract, int decomp, int y0, int ny, cudaStream_t s) {
  if (ny <= 0 || (!extract && !decomp)) return;
  const size_t sm = (size_t)kZfCols * d.NZ * sizeof(double);
  set_smem(k_zfilter, sm);
  k_zfilter<<<dim3((d.NXA + kZfCols - 1) / kZfCols, ny), 128, sm, s>>>(d, Y2_var, extract, decomp, y0);
}
void launch_static_phys(const Dims& d, const QuadDesc& q, double* phys, cudaStream_t s) {
  if (q.st_n <= 0) return;
  k_static_phys<<<4 * 148, 256, 0, s>>>(d, q, phys);
}
void launch_smago(const Dims& d, const double* phys, const int* vars, int nvars, double c, double* part, double* prof,
                  unsigned long long* cfl_max, cudaStream_t s) {
  SmagoVars sv{};
  sv.n = nvars < 4 ? nvars : 4;
  for (int k = 0; k < sv.n; ++k) sv.v[k] = vars[k];
  const int bz = d.NZA < 128 ? 128 : (d.NZA >= 512 ? 512 : (d.NZA + 31) / 32 * 32);
  k_smago_rows<<<d.NYA, bz, 0, s>>>(d, phys, sv, part);
  k_smago_final<<<1, bz, 0, s>>>(d, part, c, prof, cfl_max);
}
void launch_penal_default(const Dims& d, double Lx, double Ly, const double* zgrid, double* mask, cudaStream_t s) {
  k_penal_default<<<4 * 148, 256, 0, s>>>(d, Lx, Ly, zgrid, mask);
}
void launch_penal_field(size_t n, const double* mask, double strength, double width, double* out, cudaStream_t s) {
  k_penal_field<<<4 * 148, 256, 0, s>>>(n, mask, strength, width, out);
}
void launch_nl(const NLArgs& a, cudaStream_t s) {
  const int nsys = a.d.NXH * a.d.NYA;
  k_nl<<<(nsys + kWPB - 1) / kWPB, kWPB * 32, 0, s>>>(a);
}
void launch_solve(const SolveArgs& a, cudaStream_t s) {
  const int nsys = a.d.NXH * a.d.NYA;
  size_t sm = (size_t)kWPB * a.T * sizeof(double2);
  if (a.kl > 31 || a.kl + a.ku > 64) {
    set_smem(k_solve<true>, sm);
    k_solve<true><<<(nsys + kWPB - 1) / kWPB, kWPB * 32, sm, s>>>(a);
  } else {
    set_smem(k_solve<false>, sm);
    k_solve<false><<<(nsys + kWPB - 1) / kWPB, kWPB * 32, sm, s>>>(a);
  }
}
void launch_factor(const FactorArgs& a, cudaStream_t s) {
  if (a.nact <= 0) return;
  if (a.kl > 31) k_factor<true><<<(a.nact + kWPB - 1) / kWPB, kWPB * 32, 0, s>>>(a);
  else k_factor<false><<<(a.nact + kWPB - 1) / kWPB, kWPB * 32, 0, s>>>(a);
}
template <int RM, int RN, int G0 = 0, int G1 = 0, int G2 = 0>
static void launch_rhs_tiles(const SolveArgs& a, const NLArgs& n, cudaStream_t s) {
  const int nsys = a.d.NXH * a.d.NYA;
  const size_t sm = (size_t)kRhsSys * a.rhs_win_max * sizeof(double2);
  set_smem(k_rhs_tiles<RM, RN, G0, G1, G2>, sm);
  const dim3 g((nsys + kRhsSys - 1) / kRhsSys, (a.T + kTileRows - 1) / kTileRows);
  k_rhs_tiles<RM, RN, G0, G1, G2><<<g, kTileRows, sm, s>>>(a, n);
}
// slot widths of the groups of a grouped operator (0 past its last group)
static void group_widths(const DevGEll& G, int w[3]) {
  w[0] = w[1] = w[2] = 0;
  for (int k = 0; k < G.width; ++k)
    if (G.slot_grp[k] < 3) ++w[G.slot_grp[k]];
}
// threads of a one-CTA-per-system kernel: one per row up to kRhsThreads (a
// system of 64 rows takes 2 warps, not 8 of which 6 would idle)
static int rows_threads(int T) { return std::min(kRhsThreads, std::max(32, (T + 31) / 32 * 32)); }
// Systems a CTA of k_rhs_nl and k_kstd_out: two from 8 an SM on while their rows fit in
// kPairBytes, below that one (the CTAs no longer fill the chip and a pair only makes
// each longer).  Toroidal-poloidal recipe, us a step with one | two: 32^2 x 48
// 302 | 308, 48^2 x 48 404 | 387, 96^2 x 96 1828 | 1793, 128^3 3837 | 3681; four:
// 96^2 x 48 slower than one.
constexpr int kPairSys = 8 * 148;
constexpr size_t kPairBytes = 100 * 1024;
static bool pair_systems(const SolveArgs& a, size_t bytes_per_system) {
  return a.d.NXH * a.d.NYA >= kPairSys && 2 * bytes_per_system <= kPairBytes;
}
void launch_rhs_nl(const SolveArgs& a, const NLArgs& n, cudaStream_t s) {
  if (a.work2 && a.rhs_win && a.row_pos) {
    if (!a.generic_tiles && a.NLg.valid && a.NLg.ngroups == 3 && a.Mw.width <= 4) {
      int w[3];
      group_widths(a.NLg, w);
      // the plane-layer recipes' NL operator: groups i kx, i ky, 1 of widths 3, 3, 2;
      // with a penalisation drag (- Iz.Iz.Gu beside - Iz.uw) 3, 3, 5; with a
      // second flux in each derivative group (an eddy-viscosity term) 6, 6, 2
      if (w[0] == 3 && w[1] == 3 && w[2] == 2) return launch_rhs_tiles<4, 8, 3, 3, 2>(a, n, s);
      if (w[0] == 3 && w[1] == 3 && w[2] == 5) return launch_rhs_tiles<4, 11, 3, 3, 5>(a, n, s);
      if (w[0] == 6 && w[1] == 6 && w[2] == 2) return launch_rhs_tiles<4, 14, 6, 6, 2>(a, n, s);
    }
    if (a.Mw.width <= 4 && a.NLw.width <= 8) return launch_rhs_tiles<4, 8>(a, n, s);
    if (a.Mw.width <= 8 && a.NLw.width <= 16) return launch_rhs_tiles<8, 16>(a, n, s);
  }
  const int nsys = a.d.NXH * a.d.NYA;
  const size_t sm = ((size_t)n.nq * a.d.NZ + a.T) * sizeof(double2);
  if (pair_systems(a, sm)) {
    set_smem(k_rhs_nl<2>, 2 * sm);
    k_rhs_nl<2><<<(nsys + 1) / 2, rows_threads(a.T), 2 * sm, s>>>(a, n);
  } else {
    set_smem(k_rhs_nl<1>, sm);
    k_rhs_nl<1><<<nsys, rows_threads(a.T), sm, s>>>(a, n);
  }
}
template <int KL, int KV, int UPW>
static void launch_subst_block(const SolveArgs& a, cudaStream_t s) {
  const size_t sm = SubstShape<KL, KV, UPW>::kBytes;
  set_smem(k_subst_block<KL, KV, UPW>, sm);
  k_subst_block<KL, KV, UPW><<<a.ncls * a.ngrp, 32, sm, s>>>(a);
}
void launch_subst(const SolveArgs& a, cudaStream_t s) {
  if (a.nact <= 0) return;
  if (a.work2) {
    // the band (kl, kl+ku) = (9, 23) of the plane-layer recipes compiled, any
    // other band within (15, 31) through the wider instance
    const bool plane = !a.subst_rt && a.kl == 9 && a.kl + a.ku == 23;
    if (a.upw == 16) {
      if (plane) launch_subst_block<9, 23, 16>(a, s);
      else launch_subst_block<15, 31, 16>(a, s);
    } else {
      if (plane) launch_subst_block<9, 23, 32>(a, s);
      else launch_subst_block<15, 31, 32>(a, s);
    }
    return;
  }
  // whole systems (no class split): one warp per system
  const size_t sm = (size_t)kWPBr * kNBUF * kCW * a.ring_cols * sizeof(double);
  set_smem(k_subst_real, sm);
  k_subst_real<<<(a.nact + kWPBr - 1) / kWPBr, kWPBr * 32, sm, s>>>(a);
}
bool subst_multi_supported(const SolveArgs& a) {
  return a.work2 && a.ngrp > 0 && a.kl == 9 && a.kl + a.ku == 23;
}
void launch_subst_multi(const SolveArgs* d_args, const int* d_prefix, int nmem, int total, bool wide, cudaStream_t s) {
  if (total <= 0) return;
  const size_t sm = wide ? SubstShape<9, 23, 32>::kBytes : SubstShape<9, 23, 16>::kBytes;
  set_smem(k_subst_block_multi<9, 23>, sm);
  k_subst_block_multi<9, 23><<<total, 32, sm, s>>>(d_args, d_prefix, nmem);
}
void launch_kstd_out(const SolveArgs& a, cudaStream_t s) {
  if (a.nact <= 0) return;
  if (a.work2 && !a.Kstd_out) return;  // solution already in out, no K_std in the last stage
  if (a.work2 && a.tile_win && a.Lw.valid && a.Lw.width <= kLW) {
    const size_t sm = (size_t)kTileSys * a.tile_lwin_max * sizeof(double2);
    const dim3 g((a.T + kTileRows - 1) / kTileRows, (a.nact + kTileSys - 1) / kTileSys);
    int w[4] = {0, 0, 0, 0};
    for (int k = 0; k < a.Lw.width; ++k)
      if (a.Lw.slot_grp[k] < 4) ++w[a.Lw.slot_grp[k]];
    if (!a.generic_tiles && a.Lw.ngroups == 4 && w[0] == 4 && w[1] == 6 && w[2] == 3 && w[3] == 3) {
      // the plane-layer recipes' L: (kx^2 + ky^2), 1, kx, ky groups
      set_smem(k_kstd_tiles<4, 6, 3, 3>, sm);
      k_kstd_tiles<4, 6, 3, 3><<<g, kTileRows, sm, s>>>(a);
      return;
    }
    set_smem(k_kstd_tiles<>, sm);
    k_kstd_tiles<><<<g, kTileRows, sm, s>>>(a);
    return;
  }
  const size_t smx = (size_t)a.T * sizeof(double2);
  if (pair_systems(a, smx)) {
    set_smem(k_kstd_out<2>, 2 * smx);
    k_kstd_out<2><<<(a.nact + 1) / 2, rows_threads(a.T), 2 * smx, s>>>(a);
  } else {
    set_smem(k_kstd_out<1>, smx);
    k_kstd_out<1><<<a.nact, rows_threads(a.T), smx, s>>>(a);
  }
}
void launch_solve_real(const SolveArgs& a, const NLArgs& n, cudaStream_t s) {
  launch_rhs_nl(a, n, s);
  launch_subst(a, s);
  launch_kstd_out(a, s);
}
// Block layout: the union masks need every group's factors before any is packed.
static void launch_factor_blocks(const FactorArgs& a, cudaStream_t s) {
  const int nb = a.ncls * a.ngrp * a.upw;
  const size_t sm = (size_t)(a.kl + 1) * (a.kl + a.ku + 1) * 32 * sizeof(double);
  cudaMemsetAsync(a.abr, 0, (size_t)nb * a.Tc * a.ldab * sizeof(double), s);
  if (a.window && a.kl <= kFacKl && a.kl + a.ku <= kFacKv) {
    const dim3 g((nb + kTpbThreads - 1) / kTpbThreads, (a.Tc + kAsmRows - 1) / kAsmRows);
    if (a.M.ngroups <= 8 && a.L.ngroups <= 8) k_assemble_tpb<8><<<g, kTpbThreads, 0, s>>>(a);
    else k_assemble_tpb<kMaxGroups><<<g, kTpbThreads, 0, s>>>(a);
    if (a.kl <= 9 && a.kl + a.ku <= 23) {
      set_smem(k_factor_win<9, 23>, sm);
      k_factor_win<9, 23><<<(nb + 31) / 32, 32, sm, s>>>(a);
    } else {
      set_smem(k_factor_win<kFacKl, kFacKv>, sm);
      k_factor_win<kFacKl, kFacKv><<<(nb + 31) / 32, 32, sm, s>>>(a);
    }
  } else {
    k_factor_tpb<<<(nb + kTpbThreads - 1) / kTpbThreads, kTpbThreads, 0, s>>>(a);
  }
  const auto cols = [&](int gn) { return dim3(a.ncls * gn, (a.Tc + 7) / 8); };
  cudaMemsetAsync(a.cmask, 0, (size_t)a.ncls * a.Tc * sizeof(unsigned long long), s);
  k_mask_cols<<<cols(a.ngrp), 256, 0, s>>>(a);
  k_pack_info<<<a.ncls, 32, 0, s>>>(a);
  if (!a.stage) {
    k_pack<<<cols(a.ngrp), 256, 0, s>>>(a, a.pack, 0, a.ngrp);
    return;
  }
  for (int g0 = 0; g0 < a.ngrp; g0 += a.nstage) {
    const int gn = std::min(a.nstage, a.ngrp - g0);
    k_pack<<<cols(gn), 256, 0, s>>>(a, a.stage, g0, gn);
    // as many CTAs as hold the chip, at least one a group
    k_pack_back<<<dim3(a.ncls * gn, std::max(1, 8 * 148 / (a.ncls * gn))), 256, 0, s>>>(a, g0, gn);
  }
}
void launch_factor_real(const FactorArgs& a, cudaStream_t s) {
  if (a.nact <= 0) return;
  if (a.tpb) {
    launch_factor_blocks(a, s);
    return;
  }
  k_factor_real<<<dim3((a.nact + kWPB - 1) / kWPB, a.ncls), kWPB * 32, 0, s>>>(a);
}
void launch_zero_step(const ZeroArgs& a, cudaStream_t s) {
  if (a.nsys <= 0) return;
  size_t sm = 8;
  for (int i = 0; i < a.nsys; ++i) sm = std::max(sm, (size_t)a.sys[i].T * (1 + a.sys[i].ldab) * sizeof(double));
  set_smem(k_zero_step, sm);
  k_zero_step<<<a.nsys, 32, sm, s>>>(a);
}
void launch_zero_factor(const ZeroArgs& a, cudaStream_t s) {
  if (a.nsys <= 0) return;
  size_t sm = 8;
  for (int i = 0; i < a.nsys; ++i) sm = std::max(sm, (size_t)a.sys[i].T * a.sys[i].ldab * sizeof(double));
  int dev = 0, smax = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const bool fits = sm <= (size_t)smax;
  if (fits) set_smem(k_zero_factor, sm);
  k_zero_factor<<<a.nsys, 32, fits ? sm : 0, s>>>(a, fits ? 1 : 0);
}
void launch_full_dz(const Dims& d, const double2* state, int T, const int* tab_t, const double* tab_v, double dsca,
                    int order, double gap, double2* out, cudaStream_t s) {
  // columns a CTA: kDzCols, fewer where that many do not fit in 48 KB (any length
  // whose transforms run fits with one)
  const size_t colb = dz_stride(d.NZ) * sizeof(double2), tabb = d.NZ * sizeof(double);
  const int cols = (int)std::max<size_t>(1, std::min<size_t>(kDzCols, (48 * 1024 - std::min<size_t>(tabb, 48 * 1024)) / colb));
  const size_t sm = cols * colb + tabb, ncol = (size_t)d.NXH * d.NYA;
  set_smem(k_full_dz, sm);
  k_full_dz<<<(unsigned)((ncol + cols - 1) / cols), kDzThreads, sm, s>>>(d, state, T, tab_t, tab_v, dsca, order, gap, out,
                                                                         cols);
}
void launch_zero_dz(int NZ, const double* state, const int* tab_t, const double* tab_v, double dsca, int order,
                    double gap, double* out, cudaStream_t s) {
  k_zero_dz<<<1, 32, 0, s>>>(NZ, state, tab_t, tab_v, dsca, order, gap, out);
}
void launch_usr_slice(const Dims& d, const double* phys, int kind, int k, const double* wz, double* out,
                      cudaStream_t s) {
  k_usr_slice<<<1024, 256, 0, s>>>(d, phys, kind, k, wz, out);
}
void launch_usr_profile(const Dims& d, const double* phys, double* out, cudaStream_t s) {
  k_usr_profile<<<d.NZA, 256, 0, s>>>(d, phys, out);
}
void launch_phys_product(size_t n, const double* a, const double* b, double* out, cudaStream_t s) {
  k_phys_product<<<1024, 256, 0, s>>>(n, a, b, out);
}
void launch_transpose_xy(const Dims& d, const double* in, double* out, int to_file, cudaStream_t s) {
  k_transpose_xy<<<1024, 256, 0, s>>>(d, in, out, to_file);
}
void launch_galerkin_insert(const Dims& d, const double2* spec, int T, const int* var_pos, int nc, const double* sq,
                            const int* sq_col, double2* field, cudaStream_t s) {
  k_galerkin_insert<<<grid1d((size_t)d.NXH * d.NYA, 128), 128, 0, s>>>(d, spec, T, var_pos, nc, sq, sq_col, field);
}
void launch_cheb_extract(const Dims& d, const double2* field, int T, const int* tab_t, const double* tab_v,
                         double2* spec, cudaStream_t s) {
  k_cheb_extract<<<grid1d((size_t)d.NXH * d.NYA * d.NZ, 256), 256, 0, s>>>(d, field, T, tab_t, tab_v, spec);
}
void launch_check_finite(const double2* x, size_t n, unsigned int* flags, cudaStream_t s) {
  k_check_finite<<<1024, 256, 0, s>>>(x, n, flags);
}

}  // namespace coral
