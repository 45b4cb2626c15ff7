// 3D small-strain Lippmann-Schwinger solver (FP64), batched over replicas.
//
// Restates mgkmc/linear_elastic_simulator.py:274-376 (spectral_solver_3d) and
// the 3D Green operator of mgkmc/elasticity.py:70-105, applied on the fly:
//   tau = C:(eps - eps_p) - C0:eps;  eps_new = eps_bar - IFFT(Gamma0 : FFT(tau));
//   diff = ||eps_new - eps|| / (||eps|| + 1e-20).
//
// HBM layout per replica, N = nx*ny*nz (C order, z fastest):
//   mu, lam           2 planes
//   eps[6]            symmetric components xx, yy, zz, yz, xz, xy
//   ep[6]             eigenstrain, symmetric components
//   epa[6]            its off-diagonal entries as given (only when given; output)
//   spec[6]           half spectrum [c][x][y][kz], kz < nz/2+1
// The antisymmetric part of eps is uniform after the first iteration and is
// carried as three scalars.
//
// One iteration = four kernels:
//   zline  (CTA per pair of z-lines): C2R along z of the previous spectrum,
//          eps update, diff/norm partials (+ device convergence decision),
//          tau, R2C along z;
//   axis   FFT along y (forward);
//   xgamma FFT along x, eps~^ = -Gamma0_sym : tau^ / N, IFFT along x;
//   axis   IFFT along y.
// Nyquist handling and the device-driven CUDA-graph loop are as in the 2D
// solver (ls2d.cu): Gamma_sym averages Gamma over q and its mirror in the
// Nyquist components, with numpy's fftfreq signs.
#include <math.h>
#include <stddef.h>
#include <stdlib.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "fft.cuh"
#include "ls3d_dev.cuh"
#include "ls3d_line.cuh"

namespace mgk {

const void* twiddles(int n, int prec);

const Ls3Line* ls3_line_a(int n, int prec);
const Ls3Line* ls3_line_b(int n, int prec);
const Ls3Line* ls3_line_c(int n, int prec);
const Ls3Line* ls3_line_d(int n, int prec);
const Ls3Line* ls3_line(int n, int prec) {
  for (auto f : {ls3_line_a, ls3_line_b, ls3_line_c, ls3_line_d})
    if (const Ls3Line* k = f(n, prec)) return k;
  return nullptr;
}

// -------------------------------------------------------------- kernels ---

constexpr int kT3 = 256;
// per-voxel kernels: at most 4 CTAs per SM (they loop over tiles of kT3)
constexpr int kG3 = 592;


// Block sums of K values per thread in a fixed order: warp trees, then one
// warp per value; value q of the block to out[q].
template <int K> __device__ __forceinline__ void block_sums(const double* v, double* out) {
  __shared__ double w[kT3 / 32][K];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const double t = warp_sum(v[q]);
    if (lane == 0) w[wid][q] = t;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double t = 0;
#pragma unroll
    for (int k = 0; k < kT3 / 32; ++k) t += w[k][threadIdx.x];
    out[threadIdx.x] = t;
  }
}

// kT3 voxels' 3x3 tensors between the caller's interleaved layout and one
// thread per voxel, through shared memory: the warp's accesses are contiguous
// (a thread's own nine doubles would be 72 bytes apart from its neighbour's).
// m: voxels in this tile.
__device__ __forceinline__ void tile_load9(const double* __restrict__ src, int m, double* buf, double* v) {
  __syncthreads();
  for (int i = threadIdx.x; i < 9 * m; i += kT3) buf[i] = __ldcs(src + i);
  __syncthreads();
  if ((int)threadIdx.x < m)
#pragma unroll
    for (int q = 0; q < 9; ++q) v[q] = buf[9 * threadIdx.x + q];
}
__device__ __forceinline__ void tile_store9(double* __restrict__ dst, int m, double* buf, const double* v) {
  __syncthreads();
  if ((int)threadIdx.x < m)
#pragma unroll
    for (int q = 0; q < 9; ++q) buf[9 * threadIdx.x + q] = v[q];
  __syncthreads();
  for (int i = threadIdx.x; i < 9 * m; i += kT3) __stcs(dst + i, buf[i]);
}

// Moduli and eigenstrain planes of one replica, per-CTA partial sums of the
// two moduli inputs.  HBM-bound: 25 planes per voxel with an eigenstrain.
__global__ void __launch_bounds__(kT3, 3) ls3d_material_kernel(const Ls3dRep* reps, int rep,
                                                               const double* __restrict__ E,
                                                               const double* __restrict__ nu,
                                                               const double* __restrict__ epsp, int set_moduli,
                                                               double* partials) {
  __shared__ double buf[9 * kT3];
  const Ls3dRep& R = reps[rep];
  const long long N = R.N;
  double sm[2] = {0, 0};
  for (long long i0 = blockIdx.x * (long long)kT3; i0 < N; i0 += (long long)gridDim.x * kT3) {
    const int m = (int)min((long long)kT3, N - i0);
    const long long i = i0 + threadIdx.x;
    const bool in = (int)threadIdx.x < m;
    double p[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    double e = 0, v = 0;
    if (set_moduli && in) { e = E[i]; v = nu[i]; }
    if (epsp) tile_load9(epsp + 9 * i0, m, buf, p);
    if (!in) continue;
    if (set_moduli) {
      // elasticity.py:55-59 (set_moduli 1); set_moduli 2: E holds lambda and
      // nu holds mu, as the secant solver takes them
      const double mu = set_moduli == 2 ? v : e / (2 * (1 + v));
      const double lam = set_moduli == 2 ? e : e * v / ((1 + v) * (1 - 2 * v));
      R.mu[i] = mu;
      R.lam[i] = lam;
      if (R.mu32) { R.mu32[i] = (float)mu; R.lam32[i] = (float)lam; }
      sm[0] += e;
      sm[1] += v;
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      constexpr int kI[6] = {0, 1, 2, 1, 0, 0}, kJ[6] = {0, 1, 2, 2, 2, 1};
      const int a = 3 * kI[c] + kJ[c], b = 3 * kJ[c] + kI[c];
      const double sy = (p[a] == p[b]) ? p[a] : 0.5 * (p[a] + p[b]);
      R.ep[c * N + i] = sy;
      if (R.ep32) R.ep32[c * N + i] = (float)sy;
      // the off-diagonal entries as given (the output stress uses them)
      if (c >= 3 && R.epa) {
        R.epa[(c - 3) * N + i] = p[a];
        R.epa[c * N + i] = p[b];
      }
    }
  }
  if (set_moduli) block_sums<2>(sm, partials + 2 * blockIdx.x);
}

// reference medium from the means of E and nu (linear_elastic_simulator.py:
// 284-289), or of lambda and mu (lame_in; the secant solver, :783-784)
__global__ void ls3d_medium_kernel(const Ls3dRep* reps, Ls3dState* st, int rep, const double* partials, int nb,
                                   int lame_in) {
  __shared__ double red[32];
  double a = 0, b = 0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) { a += partials[2 * i]; b += partials[2 * i + 1]; }
  a = block_sum(a, red);
  b = block_sum(b, red);
  if (threadIdx.x == 0) {
    const double N = (double)reps[rep].N;
    const double E = a / N, v = b / N;
    const double mu0 = lame_in ? v : E / (2 * (1 + v));
    const double lam0 = lame_in ? E : E * v / ((1 + v) * (1 - 2 * v));
    Ls3dState& S = st[rep];
    S.mu0 = mu0;
    S.lam0 = lam0;
    S.Bc = (lam0 + mu0) / (mu0 * (lam0 + 2 * mu0));
    S.inv2mu0 = 1.0 / (2 * mu0);
  }
}

// per-CTA partials of the 9 components of the warm-start field; grid (G, nsel)
__global__ void __launch_bounds__(kT3, 4) ls3d_means_kernel(const Ls3dRep* reps, const int* sel, double* partials) {
  __shared__ double buf[9 * kT3];
  const Ls3dRep& R = reps[sel[blockIdx.y]];
  if (!R.init) return;
  double s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (long long i0 = blockIdx.x * (long long)kT3; i0 < R.N; i0 += (long long)gridDim.x * kT3) {
    double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    tile_load9(R.init + 9 * i0, (int)min((long long)kT3, R.N - i0), buf, v);
#pragma unroll
    for (int q = 0; q < 9; ++q) s[q] += v[q];
  }
  block_sums<9>(s, partials + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 18);
}

// fixed-order sums (stride 18 per CTA slot), one warp per value; mode 0:
// means of every replica, 1: means for warm-started replicas, 2: plain sums
// for warm-started replicas
__global__ void ls3d_finalize_kernel(const Ls3dRep* reps, Ls3dState* st, const int* sel, const double* partials,
                                     int G, int off, int mode) {
  const int r = sel[blockIdx.x], q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (mode && !reps[r].init) return;
  double* out = reinterpret_cast<double*>(reinterpret_cast<char*>(&st[r]) + off);
  double a = 0;
#pragma unroll 4
  for (int i = lane; i < G; i += 32) a += partials[((size_t)blockIdx.x * G + i) * 18 + q];
  a = warp_sum(a);
  if (lane == 0) out[q] = a * (mode == 2 ? 1.0 : 1.0 / (double)reps[r].N);
}

// initial field (linear_elastic_simulator.py:302-313); grid (G, nsel).  arrivals:
// the z-line kernels' counters, which start at zero whatever the call before left (a
// CTA whose copy wait gave up does not arrive)
__global__ void __launch_bounds__(kT3, 3) ls3d_begin_kernel(const Ls3dRep* reps, Ls3dState* st, const int* sel,
                                                            double* partials, unsigned int* arrivals) {
  __shared__ double buf[9 * kT3];
  const int r = sel[blockIdx.y];
  const Ls3dRep& R = reps[r];
  Ls3dState& S = st[r];
  const long long N = R.N;
  const double* eb = R.eb;
  double ab[3] = {0.5 * (eb[1] - eb[3]), 0.5 * (eb[2] - eb[6]), 0.5 * (eb[5] - eb[7])};
  double sb[6];
  for (int c = 0; c < 6; ++c) {
    const int a = 3 * kSymI[c] + kSymJ[c], b = 3 * kSymJ[c] + kSymI[c];
    sb[c] = (eb[a] == eb[b]) ? eb[a] : 0.5 * (eb[a] + eb[b]);
  }
  double dn[2] = {0, 0};
  for (long long i0 = blockIdx.x * (long long)kT3; i0 < N; i0 += (long long)gridDim.x * kT3) {
    const int m = (int)min((long long)kT3, N - i0);
    const long long i = i0 + threadIdx.x;
    if (R.init) {
      double v[9];
      tile_load9(R.init + 9 * i0, m, buf, v);
      if ((int)threadIdx.x >= m) continue;
#pragma unroll
      for (int q = 0; q < 9; ++q) v[q] += eb[q] - S.means[q];
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        constexpr int kI[6] = {0, 1, 2, 1, 0, 0}, kJ[6] = {0, 1, 2, 2, 2, 1};
        const int a = 3 * kI[c] + kJ[c], b = 3 * kJ[c] + kI[c];
        const double sy = (v[a] == v[b]) ? v[a] : 0.5 * (v[a] + v[b]);
        R.eps[c * N + i] = sy;
        if (R.eps32) R.eps32[c * N + i] = (float)sy;
      }
      const double a0[3] = {0.5 * (v[1] - v[3]), 0.5 * (v[2] - v[6]), 0.5 * (v[5] - v[7])};
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        dn[0] += 2 * (ab[q] - a0[q]) * (ab[q] - a0[q]);
        dn[1] += 2 * a0[q] * a0[q];
      }
    } else if ((int)threadIdx.x < m) {
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        R.eps[c * N + i] = sb[c];
        if (R.eps32) R.eps32[c * N + i] = (float)sb[c];
      }
    }
  }
  if (R.init) block_sums<2>(dn, partials + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 18);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    for (int c = 0; c < 6; ++c) S.ebar[c] = sb[c];
    for (int q = 0; q < 3; ++q) S.abar[q] = ab[q];
    S.iter = 0;
    S.phase_iter = 0;
    S.done = R.max_iter <= 0 ? 2 : 0;
    S.status = MGK_OK;
    S.diff = 0;
    arrivals[r] = 0;
    if (!R.init) {
      S.extra_d0 = 0;
      S.extra_n0 = 2.0 * (double)N * (ab[0] * ab[0] + ab[1] * ab[1] + ab[2] * ab[2]);
    }
  }
}

// z-line kernel: pairs of z-lines (flattened (x, y) index 2p, 2p+1)
template <bool IN_SPEC>
__global__ void __launch_bounds__(256) ls3d_zline_kernel(const Ls3dRep* __restrict__ reps, Ls3dState* st,
                                                        const int* __restrict__ map, const int* __restrict__ loc,
                                                        double* partials, unsigned int* rep_counter, Ls3dCtl* ctl,
                                                        cudaGraphConditionalHandle cond, int use_cond,
                                                        int guard_cap) {
  using C = double2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  __shared__ int s_last;
  const int item = blockIdx.x;
  const int r = map[item];
  const Ls3dRep& R = reps[r];
  Ls3dState& S = st[r];
  if (IN_SPEC && use_cond && item == 0 && threadIdx.x == 0) {
    const unsigned int b = atomicAdd(&ctl->bodies, 1u) + 1u;
    if (ctl->n_active == 0 || b > (unsigned int)guard_cap || *(volatile int*)&ctl->error != 0) {
      ctl->any = 0;
      cudaGraphSetConditional(cond, 0u);
    }
  }
  if (S.done != 0) return;
  const int nz = R.nz, nzh = R.nzh, ld = R.ld;
  const long long N = R.N;
  const long long l0 = 2LL * loc[item];  // first line (flattened x*ny + y)
  const long long plane = (long long)R.nx * R.ny * ld;  // complex elements per component
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 6 * nz;
  C* spec = R.spec;
  double d2 = 0, n2 = 0;
  C* cur = bufA;
  if (IN_SPEC) {
    const int tot = 6 * nz;
    for (int e = threadIdx.x; e < tot; e += blockDim.x) {
      const int c = e / nz, k = e - c * nz;
      const int ks = (2 * k <= nz) ? k : nz - k;
      const C* ra = spec + c * plane + l0 * ld;
      C a = ra[ks], b = ra[ld + ks];
      C z;
      if (2 * k <= nz) {
        if (k == 0 || 2 * k == nz) { a.y = 0; b.y = 0; }
        z = make_double2(a.x - b.y, a.y + b.x);
      } else {
        z = make_double2(a.x + b.y, b.x - a.y);
      }
      bufA[e] = z;
    }
    __syncthreads();
    cur = fft_any<+1>(bufA, bufB, 6, nz, R.fz);
  }
  C* out = (IN_SPEC && cur == bufA) ? bufB : bufA;
  const double mu0 = S.mu0, lam0 = S.lam0;
  for (int z = threadIdx.x; z < nz; z += blockDim.x) {
    double tr[2][6];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long i = (l0 + h) * nz + z;
      double e[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        const double o = R.eps[c * N + i];
        if (IN_SPEC) {
          const C zz = cur[c * nz + z];
          const double nw = S.ebar[c] + (h == 0 ? zz.x : zz.y);
          const double dd = nw - o;
          const double w = c < 3 ? 1.0 : 2.0;
          d2 += w * dd * dd;
          n2 += w * o * o;
          R.eps[c * N + i] = nw;
          e[c] = nw;
        } else {
          e[c] = o;
        }
      }
      double m = R.mu[i];
      const double l = R.lam[i];
      double d[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) d[c] = e[c] - R.ep[c * N + i];
      if (R.law == 1) m = secant_mu3(m, d[0], d[1], d[2], d[3], d[4], d[5], R.law_a, R.law_b);
      const double trd = d[0] + d[1] + d[2], tre = e[0] + e[1] + e[2];
      if (R.law == 3) {
        double sg[6];
        landau_sigma3(m, l, d, R.lp, sg);
#pragma unroll
        for (int c = 0; c < 3; ++c) tr[h][c] = sg[c] - (2 * mu0 * e[c] + lam0 * tre);
#pragma unroll
        for (int c = 3; c < 6; ++c) tr[h][c] = sg[c] - 2 * mu0 * e[c];
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) tr[h][c] = (2 * m * d[c] + l * trd) - (2 * mu0 * e[c] + lam0 * tre);
#pragma unroll
        for (int c = 3; c < 6; ++c) tr[h][c] = 2 * m * d[c] - 2 * mu0 * e[c];
      }
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) out[c * nz + z] = make_double2(tr[0][c], tr[1][c]);
  }
  __syncthreads();
  C* scratch = (out == bufA) ? bufB : bufA;
  C* Z = fft_any<-1>(out, scratch, 6, nz, R.fz);
  for (int e = threadIdx.x; e < 6 * nzh; e += blockDim.x) {
    const int c = e / nzh, k = e - c * nzh;
    const C z = Z[c * nz + k];
    const C w = Z[c * nz + (k == 0 ? 0 : nz - k)];
    C* ra = spec + c * plane + l0 * ld;
    ra[k] = make_double2(0.5 * (z.x + w.x), 0.5 * (z.y - w.y));
    ra[ld + k] = make_double2(0.5 * (z.y + w.y), -0.5 * (z.x - w.x));
  }
  if (!IN_SPEC) return;
  ls3d_decide<true>(R, S, r, item, d2, n2, partials, rep_counter, ctl, cond, use_cond, guard_cap, red, &s_last);
}

// Strided-axis pass over tiles of tc consecutive kz columns.
// AXIS = 1: FFT along y (SIGN given); AXIS = 0: FFT along x, Gamma0_sym,
// IFFT along x.
template <int AXIS, int SIGN>
__global__ void __launch_bounds__(256) ls3d_axis_kernel(const Ls3dRep* __restrict__ reps,
                                                       const Ls3dState* __restrict__ st,
                                                       const int* __restrict__ map, const int* __restrict__ loc) {
  using C = double2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int item = blockIdx.x;
  const int r = map[item];
  const Ls3dRep& R = reps[r];
  const Ls3dState& S = st[r];
  if (S.done != 0) return;
  const int nx = R.nx, ny = R.ny, nz = R.nz, nzh = R.nzh, ld = R.ld, tc = R.tc;
  const int ntile = (nzh + tc - 1) / tc;
  const int o = loc[item] / ntile;          // x (AXIS 1) or y (AXIS 0)
  const int k0 = (loc[item] - o * ntile) * tc;
  const int tcw = min(tc, nzh - k0);
  const int n = AXIS == 1 ? ny : nx;
  const FftLen& f = AXIS == 1 ? R.fy : R.fx;
  const long long plane = (long long)nx * ny * ld;
  const long long lstride = AXIS == 1 ? ld : (long long)ny * ld;
  const long long obase = AXIS == 1 ? (long long)o * ny * ld : (long long)o * ld;
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 6 * tc * n;
  C* spec = R.spec;
  const int tot = 6 * tcw * n;
  for (int e0 = threadIdx.x; e0 < tot; e0 += 4 * blockDim.x) {
    C v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * blockDim.x;
      if (e < tot) {
        const int c = e / (tcw * n), rem = e - c * tcw * n, j = rem / tcw, t = rem - j * tcw;
        v[u] = spec[c * plane + obase + j * lstride + k0 + t];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * blockDim.x;
      if (e < tot) {
        const int c = e / (tcw * n), rem = e - c * tcw * n, j = rem / tcw, t = rem - j * tcw;
        bufA[(c * tc + t) * n + j] = v[u];
      }
    }
  }
  __syncthreads();
  C* F;
  if (AXIS == 1) {
    F = fft_any<SIGN>(bufA, bufB, 6 * tc, n, f);
  } else {
    C* G = fft_any<-1>(bufA, bufB, 6 * tc, n, f);
    const double scale = 1.0 / (double)R.N;
    const int ky = o;
    const double uy = (double)fftfreq3(ky, ny) / ny;
    const bool nqy = (ny & 1) == 0 && 2 * ky == ny;
    for (int e = threadIdx.x; e < tcw * n; e += blockDim.x) {
      const int t = e / n, kx = e - t * n;
      const int kz = k0 + t;
      C tv[6], ev[6];
      for (int c = 0; c < 6; ++c) tv[c] = G[(c * tc + t) * n + kx];
      if (kx == 0 && ky == 0 && kz == 0) {
        for (int c = 0; c < 6; ++c) G[(c * tc + t) * n + kx] = make_double2(0.0, 0.0);
        continue;
      }
      const double ux = (double)fftfreq3(kx, nx) / nx, uz = (double)fftfreq3(kz, nz) / nz;
      const double inv = 1.0 / sqrt(ux * ux + uy * uy + uz * uz);
      const double n0 = ux * inv, n1 = uy * inv, n2 = uz * inv;
      gamma3d_apply(tv, n0, n1, n2, S.inv2mu0, S.Bc, ev);
      const bool nqx = (nx & 1) == 0 && 2 * kx == nx, nqz = (nz & 1) == 0 && 2 * kz == nz;
      if (nqx || nqy || nqz) {
        C fv[6];
        gamma3d_apply(tv, nqx ? -n0 : n0, nqy ? -n1 : n1, nqz ? -n2 : n2, S.inv2mu0, S.Bc, fv);
        for (int c = 0; c < 6; ++c) ev[c] = make_double2(0.5 * (ev[c].x + fv[c].x), 0.5 * (ev[c].y + fv[c].y));
      }
      for (int c = 0; c < 6; ++c) G[(c * tc + t) * n + kx] = make_double2(ev[c].x * scale, ev[c].y * scale);
    }
    __syncthreads();
    C* H = (G == bufA) ? bufB : bufA;
    F = fft_any<+1>(G, H, 6 * tc, n, f);
  }
  for (int e = threadIdx.x; e < tot; e += blockDim.x) {
    const int c = e / (tcw * n), rem = e - c * tcw * n, j = rem / tcw, t = rem - j * tcw;
    spec[c * plane + obase + j * lstride + k0 + t] = F[(c * tc + t) * n + j];
  }
}

// Mixed plans, between the phases: FP64 field from the FP32 one; grid (G, nsel)
__global__ void ls3d_promote_kernel(const Ls3dRep* reps, const int* sel) {
  const int r = sel[blockIdx.y];
  const Ls3dRep& R = reps[r];
  const long long n6 = 6 * R.N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n6; i += (long long)gridDim.x * blockDim.x)
    R.eps[i] = (double)R.eps32[i];
}

// replicas that finished phase 1 re-enter for phase 2; resets the control block
__global__ void ls3d_phase2_kernel(Ls3dState* st, const int* sel, int nsel, Ls3dCtl* ctl) {
  if (threadIdx.x != 0) return;
  unsigned int n = 0;
  for (int q = 0; q < nsel; ++q) {
    Ls3dState& S = st[sel[q]];
    if (S.done == 1) { S.done = 0; S.phase_iter = 0; ++n; }
  }
  ctl->n_active = n;
  ctl->decided = 0;
  ctl->still = 0;
  ctl->bodies = 0;
  ctl->any = n > 0;
}

// outputs (nx,ny,nz,3,3) and partial sums for the means; grid (G, nsel)
// Stores through shared memory (tile_store9): written one double per
// thread at a time the 18 output planes' sectors are touched four times each,
// and the pass took 239 us at 128^3 with 256 CTAs; 96 us so (705 MB).
template <int LAW = 0>  // 1: the secant law, 3: the Landau law
__global__ void __launch_bounds__(kT3, 2) ls3d_output_kernel(const Ls3dRep* reps, const Ls3dState* st, const int* sel,
                                                             double* partials) {
  __shared__ double buf[9 * kT3];
  const int r = sel[blockIdx.y];
  const Ls3dRep& R = reps[r];
  const Ls3dState& S = st[r];
  const long long N = R.N;
  const double ab[3] = {S.abar[0], S.abar[1], S.abar[2]};
  double s[18];
#pragma unroll
  for (int q = 0; q < 18; ++q) s[q] = 0;
  for (long long i0 = blockIdx.x * (long long)kT3; i0 < N; i0 += (long long)gridDim.x * kT3) {
    const int m = (int)min((long long)kT3, N - i0);
    const long long i = i0 + min((int)threadIdx.x, m - 1);  // idle threads of the last tile repeat its last voxel
    double e[9], p[9];
    const double sxx = R.eps[i], syy = R.eps[N + i], szz = R.eps[2 * N + i];
    const double syz = R.eps[3 * N + i], sxz = R.eps[4 * N + i], sxy = R.eps[5 * N + i];
    p[0] = R.ep[i]; p[4] = R.ep[N + i]; p[8] = R.ep[2 * N + i];
    if (R.epa) {
      p[5] = R.epa[i]; p[2] = R.epa[N + i]; p[1] = R.epa[2 * N + i];
      p[7] = R.epa[3 * N + i]; p[6] = R.epa[4 * N + i]; p[3] = R.epa[5 * N + i];
    } else {
      p[5] = p[7] = R.ep[3 * N + i];
      p[2] = p[6] = R.ep[4 * N + i];
      p[1] = p[3] = R.ep[5 * N + i];
    }
    double mu = R.mu[i];
    const double lam = R.lam[i];
    e[0] = sxx; e[4] = syy; e[8] = szz;
    e[1] = ab[0] == 0 ? sxy : sxy + ab[0];
    e[3] = ab[0] == 0 ? sxy : sxy - ab[0];
    e[2] = ab[1] == 0 ? sxz : sxz + ab[1];
    e[6] = ab[1] == 0 ? sxz : sxz - ab[1];
    e[5] = ab[2] == 0 ? syz : syz + ab[2];
    e[7] = ab[2] == 0 ? syz : syz - ab[2];
    double d[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) d[q] = e[q] - p[q];
    if constexpr (LAW == 1)
      mu = secant_mu3(mu, d[0], d[4], d[8], 0.5 * (d[5] + d[7]), 0.5 * (d[2] + d[6]), 0.5 * (d[1] + d[3]),
                      R.law_a, R.law_b);
    const double tr = d[0] + d[4] + d[8];
    double sg[9];
    if constexpr (LAW == 3) {
      // symmetric strains (the Landau solver takes symmetric tensors)
      const double a6[6] = {d[0], d[4], d[8], d[5], d[2], d[1]};
      double s6[6];
      landau_sigma3(mu, lam, a6, R.lp, s6);
      sg[0] = s6[0]; sg[4] = s6[1]; sg[8] = s6[2];
      sg[5] = sg[7] = s6[3];
      sg[2] = sg[6] = s6[4];
      sg[1] = sg[3] = s6[5];
    } else {
#pragma unroll
      for (int q = 0; q < 9; ++q) sg[q] = 2 * mu * d[q] + ((q % 4) == 0 ? lam * tr : 0.0);
    }
    if (R.out_eps) tile_store9(R.out_eps + 9 * i0, m, buf, e);
    if (R.out_sig) tile_store9(R.out_sig + 9 * i0, m, buf, sg);
    if ((int)threadIdx.x < m) {
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        s[q] += e[q];
        s[9 + q] += sg[q];
      }
    }
  }
  block_sums<18>(s, partials + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 18);
}

}  // namespace mgk

// ================================================================== plan ===
using namespace mgk;

namespace {
int g3(long long N) {
  long long b = (N + kT3 - 1) / kT3;
  return (int)std::max(1LL, std::min((long long)kG3, b));
}
int tc3(int n) {
  int tc = 8;
  while (tc > 1 && 2 * 6 * (size_t)tc * n * sizeof(double2) > 64 * 1024) tc >>= 1;
  return tc;
}
}  // namespace

struct mgk_ls3d_plan {
  int nrep = 0;
  long long maxN = 0;
  size_t zl_smem = 0, ax_smem = 0;  // CTA-wide passes
  std::vector<char> line;           // replicas on the register-FFT kernels (every side has one)
  bool mixed_ok = false;            // every side of every replica 64, 96 or 128
  int prec = MGK_FP64;
  std::vector<Ls3dRep> reps;
  std::vector<char> has_material;
  std::vector<void*> allocations;
  Ls3dRep* h_reps = nullptr;
  int* h_maps = nullptr;
  Ls3dCtl* h_ctl = nullptr;
  Ls3dState* h_state = nullptr;
  cudaEvent_t staged = nullptr;
  bool staged_pending = false;
  Ls3dRep* d_reps = nullptr;
  Ls3dState* d_st = nullptr;
  Ls3dCtl* d_ctl = nullptr;
  int* d_maps = nullptr;
  unsigned int* d_repctr = nullptr;
  double* d_part = nullptr;
  double* d_mat_part = nullptr;
  int tot_zl = 0, tot_y = 0, tot_x = 0;
  // instantiated loop graphs by the selection's shapes (its signature)
  struct GraphEntry {
    std::vector<int> sig;
    int cap;
    cudaGraph_t g;
    cudaGraphExec_t x;
  };
  std::vector<GraphEntry> gcache;
  int graph_mode = 1;  // 0: host-driven loop
  int law = 0;  // 1: secant degradation law (mgk_ls3d_set_secant)
};

static int a3(mgk_ls3d_t p, void** ptr, size_t bytes) {
  if (cudaMalloc(ptr, bytes) != cudaSuccess) {
    cudaGetLastError();
    set_error("mgk_ls3d: cudaMalloc of %zu bytes failed", bytes);
    return MGK_OOM;
  }
  p->allocations.push_back(*ptr);
  return MGK_OK;
}

static int wait3(mgk_ls3d_t p);

static void drop_graphs3(mgk_ls3d_t p) {
  for (auto& e : p->gcache) {
    cudaGraphExecDestroy(e.x);
    cudaGraphDestroy(e.g);
  }
  p->gcache.clear();
}

// Precision form (sides 64, 96 and 128): MGK_MIXED runs FP32 iterations
// (FP32 fields, spectra and Gamma0) until the update norm is below
// max(tol, 2e-6), then FP64 iterations from that field to tol.
extern "C" int mgk_ls3d_set_precision(mgk_ls3d_t p, int precision) {
  MGK_REQUIRE(p, "mgk_ls3d_set_precision: null plan");
  MGK_REQUIRE(precision == MGK_FP64 || precision == MGK_MIXED, "mgk_ls3d_set_precision: bad precision");
  MGK_REQUIRE(precision == MGK_FP64 || p->mixed_ok,
              "mgk_ls3d_set_precision: the mixed form needs every side in {64, 96, 128}");
  if (precision == MGK_MIXED && !p->reps[0].mu32) {
    for (int r = 0; r < p->nrep; ++r) {
      Ls3dRep& R = p->reps[r];
      void* f = nullptr;
      int st = a3(p, &f, sizeof(float) * R.N * 14);
      if (st) return st;
      float* fl = reinterpret_cast<float*>(f);
      R.mu32 = fl; R.lam32 = fl + R.N; R.eps32 = fl + 2 * R.N; R.ep32 = fl + 8 * R.N;
      const int n[3] = {R.nx, R.ny, R.nz};
      for (int q = 0; q < 3; ++q) {
        R.rtw32[q] = reinterpret_cast<const float2*>(twiddles_reg(n[q], 1));
        if (!R.rtw32[q]) return MGK_OOM;
      }
      p->has_material[r] = 0;  // the FP32 copies come with the next set_material
    }
    // the staged records too: a solve uploads all of them, those of replicas that it
    // leaves out as they were staged last
    int st = wait3(p);
    if (st) return st;
    memcpy(p->h_reps, p->reps.data(), sizeof(Ls3dRep) * p->nrep);
    MGK_CUDA(cudaMemcpy(p->d_reps, p->h_reps, sizeof(Ls3dRep) * p->nrep, cudaMemcpyHostToDevice));
  }
  p->prec = precision;
  return MGK_OK;
}

extern "C" int mgk_ls3d_destroy(mgk_ls3d_t p) {
  if (!p) return MGK_OK;
  drop_graphs3(p);
  if (p->staged) cudaEventDestroy(p->staged);
  for (void* a : p->allocations) cudaFree(a);
  if (p->h_reps) cudaFreeHost(p->h_reps);
  if (p->h_maps) cudaFreeHost(p->h_maps);
  if (p->h_ctl) cudaFreeHost(p->h_ctl);
  if (p->h_state) cudaFreeHost(p->h_state);
  delete p;
  return MGK_OK;
}

extern "C" int mgk_ls3d_create_batch(int nrep, const int* nxs, const int* nys, const int* nzs, mgk_ls3d_t* out) {
  MGK_REQUIRE(out, "mgk_ls3d_create: null output handle");
  *out = nullptr;
  MGK_REQUIRE(nrep >= 1 && nrep <= 4096 && nxs && nys && nzs, "mgk_ls3d_create: bad replica count");
  for (int r = 0; r < nrep; ++r) {
    FftLen f;
    MGK_REQUIRE(fft_schedule(nxs[r], &f) && fft_schedule(nys[r], &f) && fft_schedule(nzs[r], &f),
                "mgk_ls3d_create: grid %dx%dx%d unsupported (each side 2^a 3^b up to 4096)", nxs[r], nys[r],
                nzs[r]);
    MGK_REQUIRE(((long long)nxs[r] * nys[r]) % 2 == 0 /* z-lines are transformed in pairs */ && 2 * 6 * (size_t)nzs[r] * sizeof(double2) <= 220 * 1024 &&
                    2 * 6 * (size_t)tc3(std::max(nxs[r], nys[r])) * std::max(nxs[r], nys[r]) * sizeof(double2) <=
                        220 * 1024,
                "mgk_ls3d_create: grid too large for the shared-memory FFT");
  }
  mgk_ls3d_t p = new mgk_ls3d_plan();
  auto fail = [&](int s) { mgk_ls3d_destroy(p); return s; };
  p->nrep = nrep;
  p->reps.resize(nrep);
  p->has_material.assign(nrep, 0);
  const char* env = getenv("MGK_FAST");
  const bool use_line = !(env && env[0] == '0');
  p->mixed_ok = use_line;
  p->line.assign(nrep, 0);
  for (int r = 0; r < nrep; ++r) {
    Ls3dRep& R = p->reps[r];
    memset(&R, 0, sizeof(R));
    R.nx = nxs[r]; R.ny = nys[r]; R.nz = nzs[r];
    R.nzh = R.nz / 2 + 1;
    const int side[3] = {R.nx, R.ny, R.nz};
    bool line = use_line;
    for (int n : side) {
      line = line && ls3_line(n, MGK_FP64);
      p->mixed_ok = p->mixed_ok && (n == 64 || n == 96 || n == 128);
    }
    p->line[r] = line;
    R.ld = line ? ls3_ld(R.nz) : R.nzh;  // register-FFT tiles read rows of 64 aligned bytes
    R.N = (long long)R.nx * R.ny * R.nz;
    R.tc = tc3(std::max(R.nx, R.ny));
    const int ntile = (R.nzh + R.tc - 1) / R.tc;
    R.zl_items = line ? (R.nx * R.ny / 2 + ls3_line(R.nz, MGK_FP64)->zp - 1) / ls3_line(R.nz, MGK_FP64)->zp
                      : R.nx * R.ny / 2;
    R.y_items = R.nx * ntile;
    R.x_items = R.ny * ntile;
    fft_schedule(R.nx, &R.fx); fft_schedule(R.ny, &R.fy); fft_schedule(R.nz, &R.fz);
    R.fx.tw = twiddles(R.nx, MGK_FP64); R.fy.tw = twiddles(R.ny, MGK_FP64); R.fz.tw = twiddles(R.nz, MGK_FP64);
    if (!R.fx.tw || !R.fy.tw || !R.fz.tw) return fail(MGK_OOM);
    if (line) {
      for (int q = 0; q < 3; ++q) {
        R.rtw[q] = reinterpret_cast<const double2*>(twiddles_reg(side[q], MGK_FP64));
        if (!R.rtw[q]) return fail(MGK_OOM);
      }
    } else {
      p->zl_smem = std::max(p->zl_smem, 2 * 6 * (size_t)R.nz * sizeof(double2));
      p->ax_smem = std::max(p->ax_smem, 2 * 6 * (size_t)R.tc * std::max(R.nx, R.ny) * sizeof(double2));
    }
    p->maxN = std::max(p->maxN, R.N);
    p->tot_zl += R.zl_items; p->tot_y += R.y_items; p->tot_x += R.x_items;
    void* f = nullptr;
    int st = a3(p, &f, sizeof(double) * R.N * 20);
    if (st) return fail(st);
    double* d = reinterpret_cast<double*>(f);
    R.mu = d; R.lam = d + R.N; R.eps = d + 2 * R.N; R.ep = d + 8 * R.N; R.epa = nullptr;
    void* sp = nullptr;
    st = a3(p, &sp, 6 * (size_t)R.nx * R.ny * R.ld * sizeof(double2));
    if (st) return fail(st);
    R.spec = reinterpret_cast<double2*>(sp);
  }
  int st;
  const int G = g3(p->maxN);
  const size_t part = std::max((size_t)2 * p->tot_zl, (size_t)nrep * G * 18);
  void* v = nullptr;
  if ((st = a3(p, &v, sizeof(double) * part))) return fail(st);
  p->d_part = reinterpret_cast<double*>(v);
  if ((st = a3(p, &v, sizeof(double) * 2 * kG3))) return fail(st);
  p->d_mat_part = reinterpret_cast<double*>(v);
  if ((st = a3(p, &v, sizeof(Ls3dRep) * nrep))) return fail(st);
  p->d_reps = reinterpret_cast<Ls3dRep*>(v);
  if ((st = a3(p, &v, sizeof(Ls3dState) * nrep))) return fail(st);
  p->d_st = reinterpret_cast<Ls3dState*>(v);
  if ((st = a3(p, &v, sizeof(Ls3dCtl)))) return fail(st);
  p->d_ctl = reinterpret_cast<Ls3dCtl*>(v);
  const size_t nm = 2 * (size_t)(p->tot_zl + p->tot_y + p->tot_x) + nrep;
  if ((st = a3(p, &v, sizeof(int) * nm))) return fail(st);
  p->d_maps = reinterpret_cast<int*>(v);
  if ((st = a3(p, &v, sizeof(unsigned int) * nrep))) return fail(st);
  p->d_repctr = reinterpret_cast<unsigned int*>(v);
  if (cudaMemset(p->d_repctr, 0, sizeof(unsigned int) * nrep) || cudaMemset(p->d_st, 0, sizeof(Ls3dState) * nrep) ||
      cudaMemset(p->d_ctl, 0, sizeof(Ls3dCtl)))
    return fail(MGK_CUDA_ERROR);
  if (cudaMallocHost(&p->h_reps, sizeof(Ls3dRep) * nrep) || cudaMallocHost(&p->h_maps, sizeof(int) * nm) ||
      cudaMallocHost(&p->h_ctl, sizeof(Ls3dCtl)) || cudaMallocHost(&p->h_state, sizeof(Ls3dState) * nrep))
    return fail(MGK_OOM);
  if (cudaEventCreateWithFlags(&p->staged, cudaEventDisableTiming)) return fail(MGK_CUDA_ERROR);
  memcpy(p->h_reps, p->reps.data(), sizeof(Ls3dRep) * nrep);
  if (cudaMemcpy(p->d_reps, p->h_reps, sizeof(Ls3dRep) * nrep, cudaMemcpyHostToDevice)) return fail(MGK_CUDA_ERROR);
  *out = p;
  return MGK_OK;
}

extern "C" int mgk_ls3d_create(int nx, int ny, int nz, mgk_ls3d_t* out) {
  return mgk_ls3d_create_batch(1, &nx, &ny, &nz, out);
}

static int wait3(mgk_ls3d_t p) {
  if (p->staged_pending) {
    MGK_CUDA(cudaEventSynchronize(p->staged));
    p->staged_pending = false;
  }
  return MGK_OK;
}

static int set3(mgk_ls3d_t p, int rep, const double* E, const double* nu, const double* epsp, int set_moduli,
                cudaStream_t s) {
  Ls3dRep& R = p->reps[rep];
  const bool want = epsp != nullptr;
  if (want != (R.epa != nullptr)) {
    R.epa = want ? R.mu + 14 * R.N : nullptr;
    int st = wait3(p);
    if (st) return st;
    p->h_reps[rep] = R;
    MGK_CUDA(cudaMemcpyAsync(&p->d_reps[rep], &p->h_reps[rep], sizeof(Ls3dRep), cudaMemcpyHostToDevice, s));
    MGK_CUDA(cudaEventRecord(p->staged, s));
    p->staged_pending = true;
  }
  const int G = g3(R.N);
  ls3d_material_kernel<<<G, kT3, 0, s>>>(p->d_reps, rep, E, nu, epsp, set_moduli, p->d_mat_part);
  MGK_CUDA(cudaGetLastError());
  if (set_moduli) {
    ls3d_medium_kernel<<<1, kT3, 0, s>>>(p->d_reps, p->d_st, rep, p->d_mat_part, G, set_moduli == 2);
    MGK_CUDA(cudaGetLastError());
  }
  return MGK_OK;
}

extern "C" int mgk_ls3d_set_material_rep(mgk_ls3d_t p, int rep, const double* E, const double* nu,
                                         const double* epsp, mgk_stream_t stream) {
  MGK_REQUIRE(p && E && nu && rep >= 0 && rep < p->nrep, "mgk_ls3d_set_material: bad argument");
  int st = set3(p, rep, E, nu, epsp, 1, (cudaStream_t)stream);
  if (st == MGK_OK) p->has_material[rep] = 1;
  return st;
}

extern "C" int mgk_ls3d_set_lame_rep(mgk_ls3d_t p, int rep, const double* lam, const double* mu,
                                     const double* epsp, mgk_stream_t stream) {
  MGK_REQUIRE(p && lam && mu && rep >= 0 && rep < p->nrep, "mgk_ls3d_set_lame: bad argument");
  int st = set3(p, rep, lam, mu, epsp, 2, (cudaStream_t)stream);
  if (st == MGK_OK) p->has_material[rep] = 1;
  return st;
}

// every replica to the secant law (d > 0) or back to the linear law; cached
// loop graphs hold the previous law's z-line kernel and are dropped
extern "C" int mgk_ls3d_set_secant(mgk_ls3d_t p, double d, double k) {
  MGK_REQUIRE(p, "mgk_ls3d_set_secant: null plan");
  MGK_REQUIRE(d >= 0.0 && d <= 1.0 && k >= 0.0 && isfinite(k), "mgk_ls3d_set_secant: need 0 <= d <= 1, k >= 0");
  MGK_REQUIRE(d == 0.0 || p->prec == MGK_FP64, "mgk_ls3d_set_secant: the secant law runs in FP64 plans only");
  const int law = d != 0.0 ? 1 : 0;
  for (auto& R : p->reps) { R.law = law; R.law_a = d; R.law_b = k; }
  if (law != p->law) {
    drop_graphs3(p);
    p->law = law;
  }
  return MGK_OK;
}

// every replica to the Landau law (spectral_solver_landau_3d); cached loop
// graphs hold the previous law's z-line kernel and are dropped
extern "C" int mgk_ls3d_set_landau(mgk_ls3d_t p, const double* v, int capping, double e_cap, double tangent_ratio,
                                   double smooth_power) {
  MGK_REQUIRE(p && v, "mgk_ls3d_set_landau: null argument");
  MGK_REQUIRE(p->prec == MGK_FP64, "mgk_ls3d_set_landau: the Landau law runs in FP64 plans only");
  MGK_REQUIRE(capping >= 0 && capping <= 2, "mgk_ls3d_set_landau: capping must be 0, 1 or 2");
  MGK_REQUIRE(capping == 0 || (e_cap > 0.0 && (capping != 2 || smooth_power > 0.0)),
              "mgk_ls3d_set_landau: need e_cap > 0 (and smooth_power > 0 for smooth capping)");
  for (int q = 0; q < 7; ++q) MGK_REQUIRE(isfinite(v[q]), "mgk_ls3d_set_landau: non-finite coefficient");
  for (auto& R : p->reps) {
    R.law = 3;
    for (int q = 0; q < 7; ++q) R.lp[q] = v[q];
    R.lp[7] = capping;
    R.lp[8] = e_cap;
    R.lp[9] = tangent_ratio;
    R.lp[10] = smooth_power;
  }
  if (p->law != 3) {
    drop_graphs3(p);
    p->law = 3;
  }
  return MGK_OK;
}

extern "C" int mgk_ls3d_set_eigenstrain_rep(mgk_ls3d_t p, int rep, const double* epsp, mgk_stream_t stream) {
  MGK_REQUIRE(p && rep >= 0 && rep < p->nrep && p->has_material[rep], "mgk_ls3d_set_eigenstrain: no material");
  return set3(p, rep, nullptr, nullptr, epsp, 0, (cudaStream_t)stream);
}

// One launch group of a solve: the selected replicas of one shape on the
// register-FFT kernels (kx, ky, kz), or every other replica on the CTA-wide
// passes (kz null), which find their replica in work maps.
struct Grp3 {
  const Ls3Line *kx = nullptr, *ky = nullptr, *kz = nullptr;
  const Ls3Line *kx32 = nullptr, *ky32 = nullptr, *kz32 = nullptr;
  const int* sel = nullptr;  // the group's slice of the selection (device)
  int n = 0;                 // replicas
  int nx = 0, ny = 0, nzh = 0, zl_items = 0;  // of one replica
  // CTA-wide group: maps and item counts over its replicas
  const int *zm = nullptr, *zl = nullptr, *ym = nullptr, *yl = nullptr, *xm = nullptr, *xl = nullptr;
  int czl = 0, cy = 0, cx = 0;
  int lead = 0;  // counts the loop bodies
};

struct Loop3 {
  const Ls3dRep* reps;
  Ls3dState* st;
  double* part;
  unsigned int* ctr;
  Ls3dCtl* ctl;
  size_t zs, as;  // shared memory of the CTA-wide passes
  const int* sel;
  int nsel, G, law;
  std::vector<Grp3> grp;
};

// The stages of one iteration of a group: 0 y forward, 1 x with Gamma0, 2 y
// inverse, 3 z-lines; 4: the first z-line pass of a phase.
struct Launch3 {
  const void* fn;
  dim3 grid, block;
  size_t smem;
};
static Launch3 stage3(const Loop3& a, const Grp3& g, int stage, bool f32) {
  if (!g.kz) {
    switch (stage) {
      case 0: return {(const void*)ls3d_axis_kernel<1, -1>, dim3(g.cy), dim3(kT3), a.as};
      case 1: return {(const void*)ls3d_axis_kernel<0, 0>, dim3(g.cx), dim3(kT3), a.as};
      case 2: return {(const void*)ls3d_axis_kernel<1, 1>, dim3(g.cy), dim3(kT3), a.as};
      case 3: return {(const void*)ls3d_zline_kernel<true>, dim3(g.czl), dim3(kT3), a.zs};
      default: return {(const void*)ls3d_zline_kernel<false>, dim3(g.czl), dim3(kT3), a.zs};
    }
  }
  const Ls3Line *kx = f32 ? g.kx32 : g.kx, *ky = f32 ? g.ky32 : g.ky, *kz = f32 ? g.kz32 : g.kz;
  if (stage >= 3)
    return {kz->zline[f32 ? 0 : a.law], dim3(g.n * g.zl_items), dim3(kz->z_threads), (size_t)kz->z_bytes};
  if (stage == 1)
    return {kx->x, dim3(g.n * g.ny * ceil_div(g.nzh, kx->tile)), dim3(kx->x_threads), (size_t)kx->x_bytes};
  return {ky->y[stage == 0 ? 0 : 1], dim3(2 * g.n * g.nx * ceil_div(g.nzh, ky->tile)), dim3(ky->y_threads),
          (size_t)ky->y_bytes};
}

// Calls f(fn, grid, block, smem, args) with a stage's launch and arguments.
template <typename F>
static cudaError_t with_stage3(Loop3& a, Grp3& g, int stage, bool f32, cudaGraphConditionalHandle h, int use, int cap,
                               F f) {
  const Launch3 L = stage3(a, g, stage, f32);
  if (g.kz) {
    int first = stage == 4;
    if (stage >= 3) {
      void* z[] = {&a.reps, &a.st, &g.sel, &a.part, &a.ctr, &a.ctl, &h, &use, &cap, &g.lead, &first};
      return f(L, z);
    }
    void* x[] = {&a.reps, &a.st, &g.sel};
    return f(L, x);
  }
  if (stage >= 3) {
    void* z[] = {&a.reps, &a.st, &g.zm, &g.zl, &a.part, &a.ctr, &a.ctl, &h, &use, &cap};
    return f(L, z);
  }
  void* x[] = {&a.reps, &a.st, stage == 1 ? &g.xm : &g.ym, stage == 1 ? &g.xl : &g.yl};
  return f(L, x);
}

static int launch3(Loop3& a, int stage, bool f32, cudaStream_t s) {
  for (Grp3& g : a.grp)
    MGK_CUDA(with_stage3(a, g, stage, f32, 0, 0, 0, [&](const Launch3& L, void** args) {
      return cudaLaunchKernel(L.fn, L.grid, L.block, args, L.smem, s);
    }));
  return MGK_OK;
}

static cudaError_t add_node3(cudaGraph_t g, cudaGraphNode_t* node, const cudaGraphNode_t* dep, int ndep,
                             const Launch3& L, void** args) {
  cudaKernelNodeParams k;
  memset(&k, 0, sizeof(k));
  k.func = const_cast<void*>(L.fn);
  k.gridDim = L.grid;
  k.blockDim = L.block;
  k.sharedMemBytes = (unsigned)L.smem;
  k.kernelParams = args;
  return cudaGraphAddKernelNode(node, g, dep, ndep, &k);
}

// One while node running iterations of the FP32 (phase 1) or FP64 kernels;
// the groups' stages are independent chains of the body.
static int add_while3(cudaGraph_t g, const cudaGraphNode_t* dep, int ndep, Loop3& a, bool f32, int cap,
                      cudaGraphNode_t* out) {
  cudaGraphConditionalHandle h;
  if (cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault)) return MGK_CUDA_ERROR;
  alignas(cudaGraphNodeParams) unsigned char raw[sizeof(cudaGraphNodeParams)];
  memset(raw, 0, sizeof(raw));
  cudaGraphNodeParams& cp = *reinterpret_cast<cudaGraphNodeParams*>(raw);
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  if (cudaGraphAddNode(out, g, dep, ndep, &cp)) return MGK_CUDA_ERROR;
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  for (Grp3& gr : a.grp) {
    cudaGraphNode_t prev = nullptr;
    for (int stage = 0; stage < 4; ++stage) {
      cudaGraphNode_t node;
      if (with_stage3(a, gr, stage, f32, h, 1, cap, [&](const Launch3& L, void** args) {
            return add_node3(body, &node, prev ? &prev : nullptr, prev ? 1 : 0, L, args);
          }))
        return MGK_CUDA_ERROR;
      prev = node;
    }
  }
  return MGK_OK;
}

// Loop graph: FP64 plans one while node; mixed plans [FP32 while, promote,
// phase-2 set-up, first FP64 z-line pass, FP64 while].
static int graph3(mgk_ls3d_t p, Loop3& a, int cap, cudaGraph_t* gout, cudaGraphExec_t* xout) {
  cudaGraph_t g;
  MGK_CUDA(cudaGraphCreate(&g, 0));
  int rc = MGK_OK;
  cudaGraphNode_t last;
  if (p->prec == MGK_MIXED) {
    cudaGraphNode_t w1, np, n2;
    std::vector<cudaGraphNode_t> nz0(a.grp.size());
    rc = add_while3(g, nullptr, 0, a, true, cap, &w1);
    if (rc == MGK_OK) {
      void* ap[] = {&a.reps, &a.sel};
      if (add_node3(g, &np, &w1, 1, {(const void*)ls3d_promote_kernel, dim3(a.G, a.nsel), dim3(kT3), 0}, ap))
        rc = MGK_CUDA_ERROR;
    }
    if (rc == MGK_OK) {
      void* ap[] = {&a.st, &a.sel, &a.nsel, &a.ctl};
      if (add_node3(g, &n2, &np, 1, {(const void*)ls3d_phase2_kernel, dim3(1), dim3(32), 0}, ap)) rc = MGK_CUDA_ERROR;
    }
    for (size_t i = 0; i < a.grp.size() && rc == MGK_OK; ++i)
      if (with_stage3(a, a.grp[i], 4, false, 0, 0, 0, [&](const Launch3& L, void** args) {
            return add_node3(g, &nz0[i], &n2, 1, L, args);
          }))
        rc = MGK_CUDA_ERROR;
    if (rc == MGK_OK) rc = add_while3(g, nz0.data(), (int)nz0.size(), a, false, cap, &last);
  } else {
    rc = add_while3(g, nullptr, 0, a, false, cap, &last);
  }
  cudaGraphExec_t x = nullptr;
  if (rc == MGK_OK && cudaGraphInstantiate(&x, g, 0)) rc = MGK_CUDA_ERROR;
  if (rc) { cudaGraphDestroy(g); cudaGetLastError(); return MGK_CUDA_ERROR; }
  *gout = g;
  *xout = x;
  return MGK_OK;
}

extern "C" int mgk_ls3d_solve_batch(mgk_ls3d_t p, int nsel, const int* sel, const double* eps_bar,
                                    const double* const* eps_init, double* const* eps_out, double* const* sig_out,
                                    int max_iter, double tol, mgk_ls_info3* infos, mgk_stream_t stream) {
  MGK_REQUIRE(p && eps_bar && nsel >= 1 && nsel <= p->nrep, "mgk_ls3d_solve_batch: bad argument");
  MGK_REQUIRE(max_iter >= 0 && max_iter <= 1000000, "mgk_ls3d_solve: max_iter out of range");
  cudaStream_t s = (cudaStream_t)stream;
  std::vector<int> selv(nsel);
  std::vector<char> seen(p->nrep, 0);
  for (int q = 0; q < nsel; ++q) {
    const int r = sel ? sel[q] : q;
    MGK_REQUIRE(r >= 0 && r < p->nrep && !seen[r], "mgk_ls3d_solve_batch: bad or repeated replica index");
    MGK_REQUIRE(p->has_material[r], "mgk_ls3d_solve: replica %d has no material", r);
    seen[r] = 1;
    selv[q] = r;
  }
  int rc = wait3(p);
  if (rc) return rc;
  // shared-memory limits are raised below as the kernels are taken up, not in the
  // constructor: the first one named of a translation unit loads it (a 72x54x48 plan,
  // created first: 8 .. 15 -> 4 ms)
  Loop3 a{p->d_reps, p->d_st, p->d_part, p->d_repctr, p->d_ctl, p->zl_smem, p->ax_smem, p->d_maps, nsel,
          g3(p->maxN), p->law, {}};
  // the selection by groups: the CTA-wide replicas first, then each shape
  std::vector<int> order, sig{p->law, p->prec};
  order.reserve(nsel);
  {
    Grp3 g;
    for (int r : selv)
      if (!p->line[r]) {
        order.push_back(r);
        ++g.n;
        g.czl += p->reps[r].zl_items; g.cy += p->reps[r].y_items; g.cx += p->reps[r].x_items;
      }
    const int* m = p->d_maps + nsel;
    g.zm = m; g.zl = g.zm + g.czl; g.ym = g.zl + g.czl; g.yl = g.ym + g.cy; g.xm = g.yl + g.cy; g.xl = g.xm + g.cx;
    sig.insert(sig.end(), {nsel, g.n, g.czl, g.cy, g.cx});
    if (g.n) {
      MGK_CUDA(raise_smem((const void*)ls3d_zline_kernel<true>, p->zl_smem));
      MGK_CUDA(raise_smem((const void*)ls3d_zline_kernel<false>, p->zl_smem));
      MGK_CUDA(raise_smem((const void*)ls3d_axis_kernel<1, -1>, p->ax_smem));
      MGK_CUDA(raise_smem((const void*)ls3d_axis_kernel<1, 1>, p->ax_smem));
      MGK_CUDA(raise_smem((const void*)ls3d_axis_kernel<0, 0>, p->ax_smem));
      a.grp.push_back(g);
    }
  }
  std::vector<char> placed(p->nrep, 0);
  for (int q = 0; q < nsel; ++q) {
    const Ls3dRep& R = p->reps[selv[q]];
    if (!p->line[selv[q]] || placed[selv[q]]) continue;
    Grp3 g;
    g.kx = ls3_line(R.nx, MGK_FP64); g.ky = ls3_line(R.ny, MGK_FP64); g.kz = ls3_line(R.nz, MGK_FP64);
    if (p->prec == MGK_MIXED) {
      g.kx32 = ls3_line(R.nx, MGK_MIXED); g.ky32 = ls3_line(R.ny, MGK_MIXED); g.kz32 = ls3_line(R.nz, MGK_MIXED);
    }
    g.nx = R.nx; g.ny = R.ny; g.nzh = R.nzh; g.zl_items = R.zl_items;
    g.sel = p->d_maps + order.size();
    for (int w = q; w < nsel; ++w) {
      const int r = selv[w];
      const Ls3dRep& O = p->reps[r];
      if (!p->line[r] || placed[r] || O.nx != R.nx || O.ny != R.ny || O.nz != R.nz) continue;
      placed[r] = 1;
      order.push_back(r);
      ++g.n;
    }
    sig.insert(sig.end(), {R.nx, R.ny, R.nz, g.n});
    for (int stage = 0; stage < 4; ++stage)
      for (int f32 = 0; f32 <= (g.kx32 ? 1 : 0); ++f32) {
        const Launch3 l = stage3(a, g, stage, f32 != 0);
        MGK_CUDA(raise_smem(l.fn, l.smem));
      }
    a.grp.push_back(g);
  }
  a.grp[0].lead = 1;
  // per-call records, the selection and the CTA-wide group's maps
  const Grp3& cg = a.grp[0];
  int* zm = p->h_maps + nsel; int* zl = zm + cg.czl; int* ym = zl + cg.czl; int* yl = ym + cg.cy;
  int* xm = yl + cg.cy; int* xl = xm + cg.cx;
  std::vector<int> at(p->nrep, 0);
  for (int q = 0; q < nsel; ++q) at[selv[q]] = q;
  int zfirst = 0, zi = 0, yi = 0, xi = 0;
  for (int k = 0; k < nsel; ++k) {
    const int r = order[k], q = at[r];
    Ls3dRep& H = p->h_reps[r];
    H = p->reps[r];
    H.init = eps_init ? eps_init[q] : nullptr;
    H.out_eps = eps_out ? eps_out[q] : nullptr;
    H.out_sig = sig_out ? sig_out[q] : nullptr;
    for (int c = 0; c < 9; ++c) H.eb[c] = eps_bar[9 * q + c];
    H.tol = tol;
    H.max_iter = max_iter;
    H.zl_first = zfirst;
    zfirst += H.zl_items;
    p->h_maps[k] = r;
    if (p->line[r]) continue;
    for (int i = 0; i < H.zl_items; ++i) { zm[zi] = r; zl[zi] = i; ++zi; }
    for (int i = 0; i < H.y_items; ++i) { ym[yi] = r; yl[yi] = i; ++yi; }
    for (int i = 0; i < H.x_items; ++i) { xm[xi] = r; xl[xi] = i; ++xi; }
  }
  const int n_active = max_iter > 0 ? nsel : 0;
  *p->h_ctl = Ls3dCtl{(unsigned int)n_active, 0u, 0u, 0u, n_active > 0, 0};
  const size_t nm = nsel + 2 * (size_t)(zi + yi + xi);
  MGK_CUDA(cudaMemcpyAsync(p->d_maps, p->h_maps, sizeof(int) * nm, cudaMemcpyHostToDevice, s));
  MGK_CUDA(cudaMemcpyAsync(p->d_reps, p->h_reps, sizeof(Ls3dRep) * p->nrep, cudaMemcpyHostToDevice, s));
  MGK_CUDA(cudaMemcpyAsync(p->d_ctl, p->h_ctl, sizeof(Ls3dCtl), cudaMemcpyHostToDevice, s));
  MGK_CUDA(cudaEventRecord(p->staged, s));
  p->staged_pending = true;
  const int* d_sel = a.sel;
  const int G = a.G;
  bool any_init = false;
  for (int q = 0; q < nsel && eps_init; ++q) any_init |= eps_init[q] != nullptr;
  if (any_init) {
    ls3d_means_kernel<<<dim3(G, nsel), kT3, 0, s>>>(p->d_reps, d_sel, p->d_part);
    ls3d_finalize_kernel<<<nsel, 32 * 9, 0, s>>>(p->d_reps, p->d_st, d_sel, p->d_part, G,
                                              (int)offsetof(Ls3dState, means), 1);
    MGK_CUDA(cudaGetLastError());
  }
  ls3d_begin_kernel<<<dim3(G, nsel), kT3, 0, s>>>(p->d_reps, p->d_st, d_sel, p->d_part, p->d_repctr);
  MGK_CUDA(cudaGetLastError());
  if (any_init) {
    ls3d_finalize_kernel<<<nsel, 32 * 2, 0, s>>>(p->d_reps, p->d_st, d_sel, p->d_part, G,
                                              (int)offsetof(Ls3dState, extra_d0), 2);
    MGK_CUDA(cudaGetLastError());
  }
  if (n_active > 0) {
    const bool mixed = p->prec == MGK_MIXED;
    rc = launch3(a, 4, mixed, s);
    if (rc) return rc;
    const int cap = max_iter + 2 > 1000 ? max_iter + 2 : 1000;
    const char* env = getenv("MGK_NO_GRAPH_WHILE");
    if (env && env[0] == '1') p->graph_mode = 0;
    cudaGraphExec_t exec = nullptr;
    if (p->graph_mode == 1) {
      for (auto& e : p->gcache)
        if (e.cap >= cap && e.sig == sig) exec = e.x;
      if (!exec) {
        cudaGraph_t g;
        if (graph3(p, a, cap, &g, &exec) == MGK_OK) {
          constexpr size_t kMaxGraphs3 = 16;
          if (p->gcache.size() >= kMaxGraphs3) {
            cudaGraphExecDestroy(p->gcache.front().x);
            cudaGraphDestroy(p->gcache.front().g);
            p->gcache.erase(p->gcache.begin());
          }
          p->gcache.push_back({sig, cap, g, exec});
        } else {
          p->graph_mode = 0;
        }
      }
    }
    if (p->graph_mode == 1) {
      MGK_CUDA(cudaGraphLaunch(exec, s));
    } else {
      for (int phase = mixed ? 1 : 2; phase <= 2; ++phase) {
        if (phase == 2 && mixed) {
          ls3d_promote_kernel<<<dim3(G, nsel), kT3, 0, s>>>(p->d_reps, d_sel);
          ls3d_phase2_kernel<<<1, 32, 0, s>>>(p->d_st, d_sel, nsel, p->d_ctl);
          if ((rc = launch3(a, 4, false, s))) return rc;
        }
        for (int it = 0; it < max_iter; ++it) {
          for (int stage = 0; stage < 4; ++stage)
            if ((rc = launch3(a, stage, phase == 1, s))) return rc;
          Ls3dCtl hc;
          MGK_CUDA(cudaMemcpyAsync(&hc, p->d_ctl, sizeof(Ls3dCtl), cudaMemcpyDeviceToHost, s));
          MGK_CUDA(cudaStreamSynchronize(s));
          if (!hc.any) break;
        }
      }
    }
  }
  if (p->law == 1)
    ls3d_output_kernel<1><<<dim3(G, nsel), kT3, 0, s>>>(p->d_reps, p->d_st, d_sel, p->d_part);
  else if (p->law == 3)
    ls3d_output_kernel<3><<<dim3(G, nsel), kT3, 0, s>>>(p->d_reps, p->d_st, d_sel, p->d_part);
  else
    ls3d_output_kernel<0><<<dim3(G, nsel), kT3, 0, s>>>(p->d_reps, p->d_st, d_sel, p->d_part);
  MGK_CUDA(cudaGetLastError());
  ls3d_finalize_kernel<<<nsel, 32 * 18, 0, s>>>(p->d_reps, p->d_st, d_sel, p->d_part, G,
                                            (int)offsetof(Ls3dState, out_eps_mean), 0);
  MGK_CUDA(cudaGetLastError());
  if (infos) {
    MGK_CUDA(cudaMemcpyAsync(p->h_state, p->d_st, sizeof(Ls3dState) * p->nrep, cudaMemcpyDeviceToHost, s));
    Ls3dCtl hc3;
    MGK_CUDA(cudaMemcpyAsync(&hc3, p->d_ctl, sizeof(Ls3dCtl), cudaMemcpyDeviceToHost, s));
    MGK_CUDA(cudaStreamSynchronize(s));
    if (hc3.error) {
      set_error("mgk_ls3d_solve: a device wait gave up");
      return MGK_TIMEOUT;
    }
    int worst = MGK_OK;
    for (int q = 0; q < nsel; ++q) {
      const Ls3dState& S = p->h_state[selv[q]];
      infos[q].iterations = S.iter;
      infos[q].status = S.status;
      infos[q].final_diff = S.diff;
      for (int k = 0; k < 9; ++k) { infos[q].eps_mean[k] = S.out_eps_mean[k]; infos[q].sig_mean[k] = S.out_sig_mean[k]; }
      if (S.status == MGK_NONFINITE) worst = MGK_NONFINITE;
    }
    if (worst) { set_error("mgk_ls3d_solve: non-finite residual"); return worst; }
  }
  return MGK_OK;
}

extern "C" int mgk_ls3d_leave_arrivals(mgk_ls3d_t p, int rep, int count, mgk_stream_t stream) {
  MGK_REQUIRE(p && rep >= 0 && rep < p->nrep && count >= 0 && count < p->reps[rep].zl_items && count < 256,
              "mgk_ls3d_leave_arrivals: bad argument");
  MGK_CUDA(cudaMemsetAsync(p->d_repctr + rep, count, 1, (cudaStream_t)stream));  // the low byte; the others are zero
  return MGK_OK;
}
