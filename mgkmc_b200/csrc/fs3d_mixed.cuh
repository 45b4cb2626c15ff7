// Krylov kernels of the finite-strain solver's mixed form: FP32 matvecs on
// FP32 CG vectors held as 9 real fields.
//
// The FP64 form's vectors are potentials in Fourier space (fs3d.cu), which
// takes half of the time; this form keeps the real fields and every rounding of
// the passes below, its FP64 right-hand sides included.  With F_p the tangent as
// the reference applies it is not symmetric and Newton converges linearly: a
// solve ends some 1e-6 (of the stress) from its limit wherever the increments
// reach the tolerance, and CG in FP32 carries a changed last bit into that.  The
// 128^3 load step on FP32 potentials (54 instead of 106 ms) ended 8e-8 from the
// FP64 result, this one 1e-6; right-hand sides that differ in the last bits of
// FP64 alone moved it by 3e-8.
#pragma once
#include "fs3d_dev.cuh"

namespace mgk {
namespace fs32 {

struct Fs32Args {
  int nx, ny, nz, nzh, ld, tc;
  long long N;
  int has_fp, model;
  FftLen fx, fy, fz;
  const double* Fpi;
  const double* P;
  double *r, *st64;
  double2* spec;
  double* part;
  FsScalars* sc;
  FftLen fx32, fy32, fz32;
  const float* Fpi32;
  float *p32, *q32, *r32, *x32, *st32;
};

// Tangent state planes: Fe (9), S_ref (6: 00 11 22 12 02 01), C^-1 (6, same
// order; Neo-Hookean only), lambda, c (mu - lambda ln Je for Neo-Hookean, mu
// for SVK), F_p flag (1 where F_p^-1 is not the identity).
constexpr int kState = 24;

// the planes and FFT tables that precision T reads
template <typename T> struct FsP;
template <> struct FsP<double> {
  static __device__ __forceinline__ const double* Fpi(const Fs32Args& a) { return a.Fpi; }
  static __device__ __forceinline__ double* st(const Fs32Args& a) { return a.st64; }
  static __device__ __forceinline__ double2* spec(const Fs32Args& a) { return a.spec; }
  static __device__ __forceinline__ const FftLen& fx(const Fs32Args& a) { return a.fx; }
  static __device__ __forceinline__ const FftLen& fy(const Fs32Args& a) { return a.fy; }
  static __device__ __forceinline__ const FftLen& fz(const Fs32Args& a) { return a.fz; }
};
template <> struct FsP<float> {
  static __device__ __forceinline__ const float* Fpi(const Fs32Args& a) { return a.Fpi32; }
  static __device__ __forceinline__ float* st(const Fs32Args& a) { return a.st32; }
  static __device__ __forceinline__ float2* spec(const Fs32Args& a) { return reinterpret_cast<float2*>(a.spec); }
  static __device__ __forceinline__ const FftLen& fx(const Fs32Args& a) { return a.fx32; }
  static __device__ __forceinline__ const FftLen& fy(const Fs32Args& a) { return a.fy32; }
  static __device__ __forceinline__ const FftLen& fz(const Fs32Args& a) { return a.fz32; }
};

// symmetric 3x3 from its 6 stored components (00 11 22 12 02 01)
template <typename T> __device__ __forceinline__ void sym_load(const T* st, long long N, int off, long long i, T* M) {
  const T a00 = st[(off + 0) * N + i], a11 = st[(off + 1) * N + i], a22 = st[(off + 2) * N + i];
  const T a12 = st[(off + 3) * N + i], a02 = st[(off + 4) * N + i], a01 = st[(off + 5) * N + i];
  M[0] = a00; M[1] = a01; M[2] = a02;
  M[3] = a01; M[4] = a11; M[5] = a12;
  M[6] = a02; M[7] = a12; M[8] = a22;
}

// trans2(K4 : trans2(d)) from the tangent state (the kdf of VoxelLaw with
// Fe, S_ref, C^-1 precomputed; F_p^-1 read only where the flag is set).
template <typename T>
__device__ __forceinline__ void kdf_state(const Fs32Args& a, long long i, const T* d, T* out) {
  const long long N = a.N;
  const T* st = FsP<T>::st(a);
  T Fe[9], Sref[9], X[9], Tm[9], Y[9];
  for (int q = 0; q < 9; ++q) Fe[q] = st[q * N + i];
  sym_load(st, N, 9, i, Sref);
  const T lam = st[21 * N + i], c = st[22 * N + i];
  const bool fp = a.has_fp && st[23 * N + i] != T(0);
  T Fpi[9];
  if (fp) {
    const T* fpp = FsP<T>::Fpi(a);
    for (int q = 0; q < 9; ++q) Fpi[q] = fpp[q * N + i];
  }
  mtm(Fe, d, Tm);
  if (fp) mm(Tm, Fpi, X);
  else for (int q = 0; q < 9; ++q) X[q] = Tm[q];
  if (a.model == 0) {
    const T tr = X[0] + X[4] + X[8];
    for (int r = 0; r < 3; ++r)
      for (int s2 = 0; s2 < 3; ++s2) Y[3 * r + s2] = c * (X[3 * r + s2] + X[3 * s2 + r]) + (r == s2 ? lam * tr : T(0));
  } else {
    T Ci[9], CX[9], Xs[9], U[9];
    sym_load(st, N, 15, i, Ci);
    mm(Ci, X, CX);
    const T tr = CX[0] + CX[4] + CX[8];
    for (int r = 0; r < 3; ++r)
      for (int s2 = 0; s2 < 3; ++s2) Xs[3 * r + s2] = X[3 * r + s2] + X[3 * s2 + r];
    mm(Ci, Xs, U);
    mm(U, Ci, Xs);
    for (int q = 0; q < 9; ++q) Y[q] = lam * tr * Ci[q] + c * Xs[q];
  }
  T A[9], B[9];
  mmt(Sref, d, A);  // S_ref d^T
  if (fp) { mm(Fpi, Y, Tm); mmt(Tm, Fe, B); }
  else mmt(Y, Fe, B);
  if (a.has_fp) {
    for (int q = 0; q < 9; ++q) out[q] = A[q] + B[q];
  } else {
    for (int r = 0; r < 3; ++r)
      for (int s2 = 0; s2 < 3; ++s2) out[3 * r + s2] = A[3 * s2 + r] + B[3 * s2 + r];
  }
}

// z-line forward: MODE 0 CG (p = r + beta p, or p = r when beta = 0; A = K:p),
// 1 uniform (A = K:dbar), 2 residual (A = P).  R2C along z of pairs of
// z-lines, 9 components, in precision T (MODEs 1 and 2 are FP64 only).
template <int MODE, typename T>
__global__ void __launch_bounds__(256) fs_zfwd_kernel(Fs32Args a) {
  using C = C_t<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nz = a.nz, nzh = a.nzh, ld = a.ld;
  const long long N = a.N;
  const long long l0 = 2LL * blockIdx.x;
  const long long plane = (long long)a.nx * a.ny * ld;
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 9 * nz;
  const double beta = MODE == 0 ? a.sc->beta : 0.0;
  float* pp = a.p32;
  const float* rr = a.r32;
  for (int z = threadIdx.x; z < nz; z += blockDim.x) {
    T out[2][9];
    for (int h = 0; h < 2; ++h) {
      const long long i = (l0 + h) * nz + z;
      if (MODE == 2) {
        for (int q = 0; q < 9; ++q) out[h][q] = (T)a.P[q * N + i];
      } else {
        T d[9];
        if (MODE == 0) {
          for (int q = 0; q < 9; ++q) {
            const double rv = (double)rr[q * N + i];
            const float pn = beta == 0.0 ? (float)rv : (float)(rv + beta * (double)pp[q * N + i]);
            pp[q * N + i] = pn;
            d[q] = pn;
          }
        } else {
          for (int q = 0; q < 9; ++q) d[q] = (T)a.sc->dbar[q];
        }
        kdf_state<T>(a, i, d, out[h]);
      }
    }
    for (int q = 0; q < 9; ++q) bufA[q * nz + z] = mk<C>(out[0][q], out[1][q]);
  }
  __syncthreads();
  C* Z = fft_any<-1>(bufA, bufB, 9, nz, FsP<T>::fz(a));
  C* spec = FsP<T>::spec(a);
  for (int e = threadIdx.x; e < 9 * nzh; e += blockDim.x) {
    const int c = e / nzh, k = e - c * nzh;
    const C z = Z[c * nz + k];
    const C w = Z[c * nz + (k == 0 ? 0 : nz - k)];
    C* ra = spec + c * plane + l0 * ld;
    ra[k] = mk<C>(T(0.5) * (z.x + w.x), T(0.5) * (z.y - w.y));
    ra[ld + k] = mk<C>(T(0.5) * (z.y + w.y), T(-0.5) * (z.x - w.x));
  }
}

// z-line inverse: C2R along z.  MODE 0: q = result, partial p.q (FP64 sums).
// MODE 1 (FP64): r = -result (right-hand side), x = 0, partial r.r.
template <int MODE, typename T>
__global__ void __launch_bounds__(256) fs_zinv_kernel(Fs32Args a) {
  using C = C_t<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  const int nz = a.nz, ld = a.ld;
  const long long N = a.N;
  const long long l0 = 2LL * blockIdx.x;
  const long long plane = (long long)a.nx * a.ny * ld;
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 9 * nz;
  const C* spec = FsP<T>::spec(a);
  for (int e = threadIdx.x; e < 9 * nz; e += blockDim.x) {
    const int c = e / nz, k = e - c * nz;
    const int ks = (2 * k <= nz) ? k : nz - k;
    const C* ra = spec + c * plane + l0 * ld;
    C av = ra[ks], bv = ra[ld + ks];
    C z;
    if (2 * k <= nz) {
      if (k == 0 || 2 * k == nz) { av.y = 0; bv.y = 0; }
      z = mk<C>(av.x - bv.y, av.y + bv.x);
    } else {
      z = mk<C>(av.x + bv.y, bv.x - av.y);
    }
    bufA[e] = z;
  }
  __syncthreads();
  C* R = fft_any<+1>(bufA, bufB, 9, nz, FsP<T>::fz(a));
  float* qq = a.q32;
  const float* pp = a.p32;
  double acc = 0;
  for (int e = threadIdx.x; e < 9 * nz; e += blockDim.x) {
    const int c = e / nz, z = e - c * nz;
    const C v = R[e];
    for (int h = 0; h < 2; ++h) {
      const long long i = (l0 + h) * nz + z;
      const T val = h == 0 ? v.x : v.y;
      if (MODE == 0) {
        qq[c * N + i] = val;
        acc += (double)pp[c * N + i] * (double)val;
      } else {
        a.r[c * N + i] = -(double)val;
        acc += (double)val * (double)val;
      }
    }
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) a.part[blockIdx.x] = acc;
}

// y-axis pass over tiles of tc kz columns (9 components)
template <int SIGN, typename T>
__global__ void __launch_bounds__(256) fs_ypass_kernel(Fs32Args a) {
  using C = C_t<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nx = a.nx, ny = a.ny, nzh = a.nzh, ld = a.ld, tc = a.tc;
  const int ntile = (nzh + tc - 1) / tc;
  const int o = blockIdx.x / ntile;  // x
  const int k0 = (blockIdx.x - o * ntile) * tc;
  const int tcw = min(tc, nzh - k0);
  const long long plane = (long long)nx * ny * ld;
  const long long obase = (long long)o * ny * ld;
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 9 * tc * ny;
  C* spec = FsP<T>::spec(a);
  const int tot = 9 * tcw * ny;
  for (int e = threadIdx.x; e < tot; e += blockDim.x) {
    const int c = e / (tcw * ny), rem = e - c * tcw * ny, j = rem / tcw, t = rem - j * tcw;
    bufA[(c * tc + t) * ny + j] = spec[c * plane + obase + (long long)j * ld + k0 + t];
  }
  __syncthreads();
  C* F = fft_any<SIGN>(bufA, bufB, 9 * tc, ny, FsP<T>::fy(a));
  for (int e = threadIdx.x; e < tot; e += blockDim.x) {
    const int c = e / (tcw * ny), rem = e - c * tcw * ny, j = rem / tcw, t = rem - j * tcw;
    spec[c * plane + obase + (long long)j * ld + k0 + t] = F[(c * tc + t) * ny + j];
  }
}

// x pass: FFT along x, G, IFFT along x (with the 1/N of the transform pair)
template <typename T>
__global__ void __launch_bounds__(256) fs_xg_kernel(Fs32Args a) {
  using C = C_t<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nx = a.nx, ny = a.ny, nz = a.nz, nzh = a.nzh, ld = a.ld, tc = a.tc;
  const int ntile = (nzh + tc - 1) / tc;
  const int o = blockIdx.x / ntile;  // y
  const int k0 = (blockIdx.x - o * ntile) * tc;
  const int tcw = min(tc, nzh - k0);
  const long long plane = (long long)nx * ny * ld;
  const long long lstride = (long long)ny * ld;
  const long long obase = (long long)o * ld;
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 9 * tc * nx;
  C* spec = FsP<T>::spec(a);
  const int tot = 9 * tcw * nx;
  for (int e = threadIdx.x; e < tot; e += blockDim.x) {
    const int c = e / (tcw * nx), rem = e - c * tcw * nx, j = rem / tcw, t = rem - j * tcw;
    bufA[(c * tc + t) * nx + j] = spec[c * plane + obase + j * lstride + k0 + t];
  }
  __syncthreads();
  C* G = fft_any<-1>(bufA, bufB, 9 * tc, nx, FsP<T>::fx(a));
  const T scale = (T)(1.0 / (double)a.N);
  const int ky = o;
  const double uy = (double)ffq(ky, ny) / ny;
  const bool nqy = (ny & 1) == 0 && 2 * ky == ny;
  for (int e = threadIdx.x; e < tcw * nx; e += blockDim.x) {
    const int t = e / nx, kx = e - t * nx;
    const int kz = k0 + t;
    const bool nqx = (nx & 1) == 0 && 2 * kx == nx, nqz = (nz & 1) == 0 && 2 * kz == nz;
    if ((kx == 0 && ky == 0 && kz == 0) || nqx || nqy || nqz) {
      for (int c = 0; c < 9; ++c) G[(c * tc + t) * nx + kx] = mk<C>(T(0), T(0));
      continue;
    }
    const double ux = (double)ffq(kx, nx) / nx, uz = (double)ffq(kz, nz) / nz;
    const double inv = 1.0 / sqrt(ux * ux + uy * uy + uz * uz);
    const T n[3] = {(T)(ux * inv), (T)(uy * inv), (T)(uz * inv)};
    C A[9];
    for (int c = 0; c < 9; ++c) A[c] = G[(c * tc + t) * nx + kx];
    for (int i = 0; i < 3; ++i) {
      T vx = 0, vy = 0;
      for (int l = 0; l < 3; ++l) { vx += A[3 * i + l].x * n[l]; vy += A[3 * i + l].y * n[l]; }
      for (int j = 0; j < 3; ++j) G[((3 * i + j) * tc + t) * nx + kx] = mk<C>(vx * n[j] * scale, vy * n[j] * scale);
    }
  }
  __syncthreads();
  C* H = (G == bufA) ? bufB : bufA;
  C* Rz = fft_any<+1>(G, H, 9 * tc, nx, FsP<T>::fx(a));
  for (int e = threadIdx.x; e < tot; e += blockDim.x) {
    const int c = e / (tcw * nx), rem = e - c * tcw * nx, j = rem / tcw, t = rem - j * tcw;
    spec[c * plane + obase + j * lstride + k0 + t] = Rz[(c * tc + t) * nx + j];
  }
}

// CG update: x += alpha p; r -= alpha q (the Krylov vectors in the matvec
// precision, FP64 arithmetic and sums); partial r.r
__global__ void __launch_bounds__(256) fs_update_kernel(Fs32Args a) {
  __shared__ double red[32];
  const double alpha = a.sc->alpha;
  const long long n9 = 9 * a.N;
  const float* pp = a.p32;
  const float* qq = a.q32;
  float* xx = a.x32;
  float* rr = a.r32;
  double acc = 0;
  long long start = 0;
  {
    // FP32 vectors: four elements per access (16-byte aligned planes)
    const bool vec = ((reinterpret_cast<uintptr_t>(pp) | reinterpret_cast<uintptr_t>(qq) |
                       reinterpret_cast<uintptr_t>(xx) | reinterpret_cast<uintptr_t>(rr)) & 15) == 0;
    if (vec) {
      const long long n4 = n9 / 4;
      const float4* p4 = reinterpret_cast<const float4*>(pp);
      const float4* q4 = reinterpret_cast<const float4*>(qq);
      float4* x4 = reinterpret_cast<float4*>(xx);
      float4* r4 = reinterpret_cast<float4*>(rr);
      for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4;
           i += (long long)gridDim.x * blockDim.x) {
        const float4 pv = p4[i], qv = q4[i];
        float4 xv = x4[i], rv = r4[i];
        xv.x = (float)((double)xv.x + alpha * (double)pv.x);
        xv.y = (float)((double)xv.y + alpha * (double)pv.y);
        xv.z = (float)((double)xv.z + alpha * (double)pv.z);
        xv.w = (float)((double)xv.w + alpha * (double)pv.w);
        rv.x = (float)((double)rv.x - alpha * (double)qv.x);
        rv.y = (float)((double)rv.y - alpha * (double)qv.y);
        rv.z = (float)((double)rv.z - alpha * (double)qv.z);
        rv.w = (float)((double)rv.w - alpha * (double)qv.w);
        x4[i] = xv;
        r4[i] = rv;
        acc += (double)rv.x * rv.x + (double)rv.y * rv.y + (double)rv.z * rv.z + (double)rv.w * rv.w;
      }
      start = 4 * n4;
    }
  }
  for (long long i = start + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n9;
       i += (long long)gridDim.x * blockDim.x) {
    xx[i] = (float)((double)xx[i] + alpha * (double)pp[i]);
    const float rn = (float)((double)rr[i] - alpha * (double)qq[i]);
    rr[i] = rn;
    acc += (double)rn * (double)rn;
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) a.part[blockIdx.x] = acc;
}

// fixed-order sum of nb partials; MODE 0: pq -> alpha; 1: r.r -> beta, rr,
// one more Krylov iteration counted; 2: right-hand side -> rr = bb, beta = 0,
// iteration count reset.  MODEs 1 and 2 decide, when use_cond, whether the
// device-side Krylov loop runs another iteration: rr > tol^2 bb, finite, and
// below the iteration cap.
template <int MODE>
__global__ void fs_scalar_kernel(Fs32Args a, int nb, cudaGraphConditionalHandle cond, int use_cond) {
  __shared__ double red[32];
  double s = 0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) s += a.part[i];
  s = block_sum(s, red);
  if (threadIdx.x != 0) return;
  FsScalars& S = *a.sc;
  if (MODE == 0) {
    S.pq = s;
    S.alpha = (s != 0.0) ? S.rr / s : 0.0;
  } else if (MODE == 1) {
    S.beta = (S.rr != 0.0) ? s / S.rr : 0.0;
    S.rr = s;
    S.kcount += 1.0;
  } else {
    S.rr = s;
    S.bb = s;
    S.beta = 0.0;
    S.kcount = 0.0;
  }
  if (MODE != 0 && use_cond) {
    const bool go = isfinite(S.rr) && S.rr > S.tol2 * S.bb && S.kcount < S.kmax;
    cudaGraphSetConditional(cond, go ? 1u : 0u);
  }
}

// Krylov direction and tangent product, per voxel: p = r + beta p (p = r
// when beta = 0), A = K:p from the tangent state, A written to the q planes
// (free until the inverse z pass writes q).  Elementwise at full occupancy;
// the z forward pass (MODE 3) then only transforms A.
__global__ void __launch_bounds__(256) fs_kp_kernel(Fs32Args a) {
  const long long N = a.N;
  const double beta = a.sc->beta;
  float* pp = a.p32;
  const float* rr = a.r32;
  float* qq = a.q32;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    float d[9], out[9];
    for (int q = 0; q < 9; ++q) {
      const double rv = (double)rr[q * N + i];
      const float pn = beta == 0.0 ? (float)rv : (float)(rv + beta * (double)pp[q * N + i]);
      pp[q * N + i] = pn;
      d[q] = pn;
    }
    kdf_state<float>(a, i, d, out);
    for (int q = 0; q < 9; ++q) qq[q * N + i] = out[q];
  }
}

// ------------------------------------------------- warp-line 3D passes ---
// The same five matvec stages for grids whose sides are 64, 96 or 128 (the
// served and benchmark sizes): lines sit in padded shared memory and
// each warp transforms its own lines with warp-local passes.
//   axis kernels: CTA of NC warps per tile of kFsTile kz columns at one x (y
//     pass) or one y (x pass); warp c transforms component c0 + c's lines.  The
//     x pass applies G between the forward and inverse transforms (CTA
//     barrier); G couples the three components of a row of the tensor only.
//     FP64 CTAs hold 3 components (one row; three CTAs per tile: 5 resident
//     CTAs of 3 warps per SM instead of one of 9 at the registers an FP64 line
//     pair needs), FP32 CTAs all 9.
//   z kernels: CTA of 3 warps per pair of z-lines; the per-voxel stage (K:p or
//     P, or q and the p.q sums) uses all threads, warp w transforms the lines
//     of components 3w..3w+2.
constexpr int kFsTile = 4;

__host__ __device__ constexpr bool fs_fast_len(int n) { return n == 64 || n == 96 || n == 128; }
__host__ __device__ constexpr int fs_pl(int n, int csz) {
  return csz == 16 ? n + n / 8 + 1 : ((n + n / 16 + 2) & ~1);
}

template <int SIGN, typename T, int NL, bool XG, int NC>
__device__ __forceinline__ void fs_axis_body(const Fs32Args& a, int o, int k0, int c0, long long obase,
                                             long long jstride, unsigned char* smem) {
  using C = C_t<T>;
  constexpr int PL = padded_len<C>(NL);
  constexpr int TC = kFsTile;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nzh = a.nzh;
  const int tcw = min(TC, nzh - k0);
  const long long plane = (long long)a.nx * a.ny * a.ld;
  C* lines = reinterpret_cast<C*>(smem);  // line (c * TC + t), c relative to c0
  C* spec = FsP<T>::spec(a) + c0 * plane;
  constexpr int TOT = NC * NL * TC;
  for (int e = threadIdx.x; e < TOT; e += NC * 32) {
    const int c = e / (NL * TC);
    const int rem = e - c * NL * TC;
    const int j = rem / TC, t = rem - j * TC;
    if (t < tcw)
      cp_async_elem(&lines[(c * TC + t) * PL + pidx<C>(j)], &spec[c * plane + o * obase + j * jstride + k0 + t]);
  }
  cp_async_wait_all();
  __syncthreads();
  const C* tw = reinterpret_cast<const C*>((XG ? FsP<T>::fx(a) : FsP<T>::fy(a)).tw);
  C* l0 = lines + warp * TC * PL;  // warp = component
  warp_fft<NL, XG ? -1 : SIGN, 2>(l0, PL, tw, lane);
  warp_fft<NL, XG ? -1 : SIGN, 2>(l0 + 2 * PL, PL, tw, lane);
  if constexpr (XG) {
    __syncthreads();
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const T scale = (T)(1.0 / (double)a.N);
    const int ky = o;
    const double uy = (double)ffq(ky, ny) / ny;
    const bool nqy = (ny & 1) == 0 && 2 * ky == ny;
    for (int e = threadIdx.x; e < tcw * NL; e += NC * 32) {
      const int t = e / NL, kx = e - t * NL;
      const int kz = k0 + t;
      const int pk = pidx<C>(kx);
      const bool nqx = (nx & 1) == 0 && 2 * kx == nx, nqz = (nz & 1) == 0 && 2 * kz == nz;
      if ((kx == 0 && ky == 0 && kz == 0) || nqx || nqy || nqz) {
        for (int c = 0; c < NC; ++c) lines[(c * TC + t) * PL + pk] = mk<C>(T(0), T(0));
        continue;
      }
      const double ux = (double)ffq(kx, nx) / nx, uz = (double)ffq(kz, nz) / nz;
      const double inv = 1.0 / sqrt(ux * ux + uy * uy + uz * uz);
      const T n[3] = {(T)(ux * inv), (T)(uy * inv), (T)(uz * inv)};
      // (G:A)_ij = (A_il n_l) n_j couples the three components of a row of A
      // only: the CTA's NC components are NC / 3 whole rows
      C A[NC];
      for (int c = 0; c < NC; ++c) A[c] = lines[(c * TC + t) * PL + pk];
      for (int i = 0; i < NC / 3; ++i) {
        T vx = 0, vy = 0;
        for (int l = 0; l < 3; ++l) { vx += A[3 * i + l].x * n[l]; vy += A[3 * i + l].y * n[l]; }
        for (int j = 0; j < 3; ++j)
          lines[((3 * i + j) * TC + t) * PL + pk] = mk<C>(vx * n[j] * scale, vy * n[j] * scale);
      }
    }
    __syncthreads();
    warp_fft<NL, +1, 2>(l0, PL, tw, lane);
    warp_fft<NL, +1, 2>(l0 + 2 * PL, PL, tw, lane);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < TOT; e += NC * 32) {
    const int c = e / (NL * TC);
    const int rem = e - c * NL * TC;
    const int j = rem / TC, t = rem - j * TC;
    if (t < tcw) spec[c * plane + o * obase + j * jstride + k0 + t] = lines[(c * TC + t) * PL + pidx<C>(j)];
  }
}

// components per CTA of the axis kernels (FP32 keeps 9: measured faster at
// 128^3), and resident-CTA targets for the register allocator
__host__ __device__ constexpr int fs_axis_nc(bool, int tsz) { return tsz == 4 ? 9 : 3; }
__host__ __device__ constexpr int fs_axis_minb(bool xg, int tsz) { return fs_axis_nc(xg, tsz) == 3 ? 5 : (tsz == 8 ? 1 : 3); }

// y pass (XG = false) or x pass with G (XG = true); grid = (nx or ny) * ntile
// * (9 / NC), the component group fastest
template <int SIGN, typename T, bool XG>
__global__ void __launch_bounds__(fs_axis_nc(XG, sizeof(T)) * 32, fs_axis_minb(XG, sizeof(T)))
    fs_axis_fast_kernel(Fs32Args a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NC = fs_axis_nc(XG, sizeof(T));
  const int ntile = (a.nzh + kFsTile - 1) / kFsTile;
  const int cg = blockIdx.x % (9 / NC);
  const int item = blockIdx.x / (9 / NC);
  const int o = item / ntile;
  const int k0 = (item - o * ntile) * kFsTile;
  const long long obase = XG ? (long long)a.ld : (long long)a.ny * a.ld;
  const long long jstride = XG ? (long long)a.ny * a.ld : (long long)a.ld;
  const int nl = XG ? a.nx : a.ny;
#define MGK_AX_CASE(n) case n: fs_axis_body<SIGN, T, n, XG, NC>(a, o, k0, cg * NC, obase, jstride, smem_raw); break;
  switch (nl) {
    MGK_AX_CASE(64) MGK_AX_CASE(96) MGK_AX_CASE(128)
    default: break;
  }
#undef MGK_AX_CASE
}

// z forward: per-voxel stage (MODE 0: p = r + beta p and K:p; 1: K:dbar;
// 2: P; 3: A from the q planes, written by fs_kp_kernel), R2C along z of the
// pair of z-lines, 9 components.
template <int MODE, typename T, int NZ>
__device__ __forceinline__ void fs_zfwd_body(const Fs32Args& a, unsigned char* smem) {
  using C = C_t<T>;
  constexpr int PL = padded_len<C>(NZ);
  constexpr int NZH = NZ / 2 + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long N = a.N;
  const long long l0 = 2LL * blockIdx.x;
  const long long plane = (long long)a.nx * a.ny * a.ld;
  const int ld = a.ld;
  C* lines = reinterpret_cast<C*>(smem);
  for (int z = threadIdx.x; z < NZ; z += 3 * 32) {
    T out[2][9];
    for (int h = 0; h < 2; ++h) {
      const long long i = (l0 + h) * NZ + z;
      if (MODE == 2) {
        for (int q = 0; q < 9; ++q) out[h][q] = (T)a.P[q * N + i];
      } else if (MODE == 3) {
        const float* qq = a.q32;
        for (int q = 0; q < 9; ++q) out[h][q] = qq[q * N + i];
      } else {
        T d[9];
        for (int q = 0; q < 9; ++q) d[q] = (T)a.sc->dbar[q];
        kdf_state<T>(a, i, d, out[h]);
      }
    }
    const int pz = pidx<C>(z);
    for (int q = 0; q < 9; ++q) lines[q * PL + pz] = mk<C>(out[0][q], out[1][q]);
  }
  __syncthreads();
  const C* tw = reinterpret_cast<const C*>(FsP<T>::fz(a).tw);
  C* lw = lines + 3 * warp * PL;
  warp_fft<NZ, -1, 3>(lw, PL, tw, lane);
  C* spec = FsP<T>::spec(a);
  for (int cc = 0; cc < 3; ++cc) {
    const int c = 3 * warp + cc;
    const C* ln = lines + c * PL;
    C* ra = spec + c * plane + l0 * ld;
    for (int k = lane; k < NZH; k += 32) {
      const C zz = ln[pidx<C>(k)];
      const C w = ln[pidx<C>(k == 0 ? 0 : NZ - k)];
      ra[k] = mk<C>(T(0.5) * (zz.x + w.x), T(0.5) * (zz.y - w.y));
      ra[ld + k] = mk<C>(T(0.5) * (zz.y + w.y), T(-0.5) * (zz.x - w.x));
    }
  }
}

template <int MODE, typename T>
__global__ void __launch_bounds__(3 * 32) fs_zfwd_fast_kernel(Fs32Args a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
#define MGK_ZF_CASE(n) case n: fs_zfwd_body<MODE, T, n>(a, smem_raw); break;
  switch (a.nz) {
    MGK_ZF_CASE(64) MGK_ZF_CASE(96) MGK_ZF_CASE(128)
    default: break;
  }
#undef MGK_ZF_CASE
}

// z inverse: C2R along z of the pair of z-lines; MODE 0: q and the p.q
// partial; MODE 1 (FP64): r = -result, x = 0, the r.r partial.
template <int MODE, typename T, int NZ>
__device__ __forceinline__ void fs_zinv_body(const Fs32Args& a, unsigned char* smem, double* red) {
  using C = C_t<T>;
  constexpr int PL = padded_len<C>(NZ);
  constexpr int NZH = NZ / 2 + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long N = a.N;
  const long long l0 = 2LL * blockIdx.x;
  const long long plane = (long long)a.nx * a.ny * a.ld;
  const int ld = a.ld;
  C* lines = reinterpret_cast<C*>(smem);
  const C* spec = FsP<T>::spec(a);
  constexpr int U = (NZH + 31) / 32;
  for (int cc = 0; cc < 3; ++cc) {
    const int c = 3 * warp + cc;
    C* ln = lines + c * PL;
    const C* ra = spec + c * plane + l0 * ld;
    // the component's half-spectrum rows into registers first: one memory
    // round trip, not one per strided step behind the shared-memory stores
    C av[U], bv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = lane + 32 * u;
      if (k < NZH) { av[u] = ra[k]; bv[u] = ra[ld + k]; }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = lane + 32 * u;
      if (k < NZH) {
        C x = av[u], y = bv[u];
        if (k == 0 || 2 * k == NZ) { x.y = 0; y.y = 0; }
        ln[pidx<C>(k)] = mk<C>(x.x - y.y, x.y + y.x);
        if (k > 0 && 2 * k < NZ) ln[pidx<C>(NZ - k)] = mk<C>(x.x + y.y, y.x - x.y);
      }
    }
  }
  __syncwarp();
  const C* tw = reinterpret_cast<const C*>(FsP<T>::fz(a).tw);
  warp_fft<NZ, +1, 3>(lines + 3 * warp * PL, PL, tw, lane);
  __syncthreads();
  float* qq = a.q32;
  const float* pp = a.p32;
  double acc = 0;
  for (int z = threadIdx.x; z < NZ; z += 3 * 32) {
    const int pz = pidx<C>(z);
    for (int c = 0; c < 9; ++c) {
      const C v = lines[c * PL + pz];
      for (int h = 0; h < 2; ++h) {
        const long long i = (l0 + h) * NZ + z;
        const T val = h == 0 ? v.x : v.y;
        if (MODE == 0) {
          qq[c * N + i] = val;
          acc += (double)pp[c * N + i] * (double)val;
        } else {
          a.r[c * N + i] = -(double)val;
          acc += (double)val * (double)val;
        }
      }
    }
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) a.part[blockIdx.x] = acc;
}

template <int MODE, typename T>
__device__ __forceinline__ void fs_zinv_fast_entry(const Fs32Args& a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
#define MGK_ZI_CASE(n) case n: fs_zinv_body<MODE, T, n>(a, smem_raw, red); break;
  switch (a.nz) {
    MGK_ZI_CASE(64) MGK_ZI_CASE(96) MGK_ZI_CASE(128)
    default: break;
  }
#undef MGK_ZI_CASE
}

// FP32 kernel (the compiler's own register target), and the FP64 kernel with
// a register target of 5 resident CTAs per SM (measured faster than 4 at
// 128^3 despite a few spilled registers; the forward z pass is not)
template <int MODE, typename T>
__global__ void __launch_bounds__(3 * 32) fs_zinv_fast_kernel(Fs32Args a) { fs_zinv_fast_entry<MODE, T>(a); }
template <int MODE>
__global__ void __launch_bounds__(3 * 32, 5) fs_zinv_fast64_kernel(Fs32Args a) { fs_zinv_fast_entry<MODE, double>(a); }
template <int MODE, typename T> static void* fs_zinv_fast_fn() {
  if constexpr (sizeof(T) == 8) return (void*)fs_zinv_fast64_kernel<MODE>;
  else return (void*)fs_zinv_fast_kernel<MODE, T>;
}

// FP32 copies of n doubles
__global__ void fs_to_f32_kernel(long long n, const double* __restrict__ src, float* __restrict__ dst) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = (float)src[i];
}

}  // namespace fs32
}  // namespace mgk
