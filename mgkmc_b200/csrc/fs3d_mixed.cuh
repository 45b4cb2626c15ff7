// Kernels of the mixed form (fs3d_mixed_dev.cuh): the CTA-wide FP32 passes for
// lengths without a register FFT (fs3d_mixed_line.cuh), the FP64 right-hand
// side's passes, the CG update and scalars.
#pragma once
#include "fs3d_mixed_dev.cuh"

namespace mgk {
namespace fs32 {

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
// device-side Krylov loop runs another iteration (fs_go()).
template <int MODE>
__global__ void fs_scalar_kernel(Fs32Args a, int nb, cudaGraphConditionalHandle cond, int use_cond) {
  __shared__ double red[32];
  double s = 0;
  // sixteen loads in flight, added in order (one CTA sums a partial of every pair
  // of z-lines: 17 us at 128^3 one load after the other)
  int i = threadIdx.x;
  for (; i + 15 * (int)blockDim.x < nb; i += 16 * blockDim.x) {
    double v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = a.part[i + k * blockDim.x];
#pragma unroll
    for (int k = 0; k < 16; ++k) s += v[k];
  }
  for (; i < nb; i += blockDim.x) s += a.part[i];
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
  if (MODE != 0 && use_cond) cudaGraphSetConditional(cond, fs_go(S) ? 1u : 0u);
}

// ------------------------------------------------- warp-line 3D passes ---
// The FP64 right-hand side's stages for grids whose sides are 64, 96 or 128:
// lines sit in padded shared memory and each warp transforms its own lines with
// warp-local passes.
//   axis kernels: CTA of 3 warps (one tensor row: G couples its three components
//     only) per tile of kFsTile kz columns at one x (y pass) or one y (x pass,
//     with G between the transforms); a warp transforms a component's lines.
//   z kernels: CTA of 3 warps per pair of z-lines; the per-voxel stage uses all
//     threads, warp w transforms the lines of components 3w..3w+2.
constexpr int kFsTile = 4;

__host__ __device__ constexpr bool fs_fast_len(int n) { return n == 64 || n == 96 || n == 128; }
__host__ __device__ constexpr int fs_pl(int n) { return n + n / 8 + 1; }

template <int SIGN, int NL, bool XG>
__device__ __forceinline__ void fs_axis_body(const Fs32Args& a, int o, int k0, int c0, long long obase,
                                             long long jstride, unsigned char* smem) {
  using T = double;
  using C = double2;
  constexpr int PL = padded_len<C>(NL);
  constexpr int TC = kFsTile, NC = 3;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nzh = a.nzh;
  const int tcw = min(TC, nzh - k0);
  const long long plane = (long long)a.nx * a.ny * a.ld;
  C* lines = reinterpret_cast<C*>(smem);  // line (c * TC + t), c relative to c0
  C* spec = a.spec + c0 * plane;
  constexpr int TOT = NC * NL * TC;
  for (int e = threadIdx.x; e < TOT; e += NC * 32) {
    const int c = e / (NL * TC);
    const int rem = e - c * NL * TC;
    const int j = rem / TC, t = rem - j * TC;
    if (t < tcw)
      cp_async16(&lines[(c * TC + t) * PL + pidx<C>(j)], &spec[c * plane + o * obase + j * jstride + k0 + t]);
  }
  cp_async_wait_all();
  __syncthreads();
  const C* tw = reinterpret_cast<const C*>((XG ? a.fx : a.fy).tw);
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

// y pass (XG = false) or x pass with G (XG = true); grid = (nx or ny) * ntile
// * 3, the component group fastest
template <int SIGN, bool XG>
__global__ void __launch_bounds__(3 * 32, 5)
    fs_axis_fast_kernel(Fs32Args a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NC = 3;
  const int ntile = (a.nzh + kFsTile - 1) / kFsTile;
  const int cg = blockIdx.x % (9 / NC);
  const int item = blockIdx.x / (9 / NC);
  const int o = item / ntile;
  const int k0 = (item - o * ntile) * kFsTile;
  const long long obase = XG ? (long long)a.ld : (long long)a.ny * a.ld;
  const long long jstride = XG ? (long long)a.ny * a.ld : (long long)a.ld;
  const int nl = XG ? a.nx : a.ny;
#define MGK_AX_CASE(n) case n: fs_axis_body<SIGN, n, XG>(a, o, k0, cg * NC, obase, jstride, smem_raw); break;
  switch (nl) {
    MGK_AX_CASE(64) MGK_AX_CASE(96) MGK_AX_CASE(128)
    default: break;
  }
#undef MGK_AX_CASE
}

// z forward: per-voxel stage (MODE 1: K:dbar; 2: P), R2C along z of the pair of
// z-lines, 9 components.
template <int MODE, int NZ>
__device__ __forceinline__ void fs_zfwd_body(const Fs32Args& a, unsigned char* smem) {
  using T = double;
  using C = double2;
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
  const C* tw = reinterpret_cast<const C*>(a.fz.tw);
  C* lw = lines + 3 * warp * PL;
  warp_fft<NZ, -1, 3>(lw, PL, tw, lane);
  C* spec = a.spec;
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

template <int MODE>
__global__ void __launch_bounds__(3 * 32) fs_zfwd_fast_kernel(Fs32Args a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
#define MGK_ZF_CASE(n) case n: fs_zfwd_body<MODE, n>(a, smem_raw); break;
  switch (a.nz) {
    MGK_ZF_CASE(64) MGK_ZF_CASE(96) MGK_ZF_CASE(128)
    default: break;
  }
#undef MGK_ZF_CASE
}

// z inverse: C2R along z of the pair of z-lines; r = -result, the r.r partial
template <int NZ>
__device__ __forceinline__ void fs_zinv_body(const Fs32Args& a, unsigned char* smem, double* red) {
  using T = double;
  using C = double2;
  constexpr int PL = padded_len<C>(NZ);
  constexpr int NZH = NZ / 2 + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long N = a.N;
  const long long l0 = 2LL * blockIdx.x;
  const long long plane = (long long)a.nx * a.ny * a.ld;
  const int ld = a.ld;
  C* lines = reinterpret_cast<C*>(smem);
  const C* spec = a.spec;
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
  const C* tw = reinterpret_cast<const C*>(a.fz.tw);
  warp_fft<NZ, +1, 3>(lines + 3 * warp * PL, PL, tw, lane);
  __syncthreads();
  double acc = 0;
  for (int z = threadIdx.x; z < NZ; z += 3 * 32) {
    const int pz = pidx<C>(z);
    for (int c = 0; c < 9; ++c) {
      const C v = lines[c * PL + pz];
      for (int h = 0; h < 2; ++h) {
        const long long i = (l0 + h) * NZ + z;
        const T val = h == 0 ? v.x : v.y;
        a.r[c * N + i] = -(double)val;
        acc += (double)val * (double)val;
      }
    }
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) a.part[blockIdx.x] = acc;
}

__global__ void __launch_bounds__(3 * 32, 5) fs_zinv_fast64_kernel(Fs32Args a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
#define MGK_ZI_CASE(n) case n: fs_zinv_body<n>(a, smem_raw, red); break;
  switch (a.nz) {
    MGK_ZI_CASE(64) MGK_ZI_CASE(96) MGK_ZI_CASE(128)
    default: break;
  }
#undef MGK_ZI_CASE
}

// FP32 copies of n doubles
__global__ void fs_to_f32_kernel(long long n, const double* __restrict__ src, float* __restrict__ dst) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = (float)src[i];
}

}  // namespace fs32
}  // namespace mgk
