// 3D finite-strain de Geus Newton-Krylov solver (FP64), matrix-free.
//
// Restates finite_strain_solver_step_3d (mgkmc/finite_strain_simulator.py:
// 2967-3168) with solver="newton_cg": the macro mixed-BC loop, the Newton
// loop with the alpha-halving line search, and the Krylov solve of
//     G : K(F) : dF = rhs,   rhs = -G:K:DbarF (first iteration) or -G:P,
// where G is the de Geus projection (build_ghat4_3d :1121-1167, applied as
// (G:A)_ij = (A^ xi)_i xi_j / |xi|^2, zero at DC and on Nyquist planes) and
// K(F) is applied per voxel from F, F_p^-1 and the moduli without forming
// the 81-component tangent:
//   with F_p:    K:dF = S_ref dF^T + Fp^-1 Y Fe^T,  Y = C_eff : sym(Fe^T dF Fp^-1)
//   without F_p: K:dF = dF S + Fe Y',               Y' = C_eff : sym(Fe^T dF)
// (the two branches of the reference's tangent, :1849-1871).  Materials:
// SVK (the reference's 3D law) and Neo-Hookean (the reference's plane-strain
// law restated in 3D: S = mu I + (lam ln Je - mu) C^-1).  The Krylov solver
// is CG (the operator is symmetric on the range of G); every inner product
// and norm is FP64.
//
// Layout: tensor-first planes like the reference API, F[i][j] is plane
// 3*i+j of N = nx*ny*nz doubles (C order, z fastest).
//
// The FP64 form's CG vectors stay in Fourier space.  Every one of them lies in the range
// of G, where a field's nine spectra are v_i u_j of three potentials v_i (u the
// wave vector), so a vector is 3 planes of half spectra instead of 9 real
// fields, the inner products are sums of |u|^2 conj(a_i) b_i, and the increment
// and its stress exist in shared memory only.  One iteration:
//   x inverse  p = r + beta p; per tensor row i the lines ux p_i and p_i transformed
//   y inverse  the row's two lines to three: as is, uy times the second, the second
//   z          uz times the third; C2R, K:p per voxel, R2C, the third times uz
//   y forward  A_x as is, B = uy A_y + uz A_z: three lines to two
//   x forward  q_i = (ux X_i + B_i) / (N |u|^2), p.q, alpha
//   update     x += alpha p, r -= alpha q, r.r, beta and the loop's decision
// What bounds it: memory.  In numbers of one real value per voxel an iteration
// moves 15 + 15 + 30 + 15 + 12 + 18 = 105 (12 of them the tangent state); with
// real CG vectors, 9 spectra in the x passes and a state of 24 planes it moved
// 213.  A Neo-Hookean FP64 load step of 152 .. 156 iterations: 64^3 30.1 -> 11.9
// ms, 96^3 87 -> 40 ms, 128^3 180 -> 77 ms (0.57 of the measured copy rate over an
// iteration's 1.76 GB); 72^3, which had no warp-line kernels, 68 -> 18 ms.  Host
// reads are one per Newton iteration: the trial state is evaluated behind the
// Krylov loop, writes the next tangent state and is accepted by a swap.
//
// The mixed form (fs3d_mixed.cuh) keeps FP32 real fields and their kernels.
#include <math.h>
#include <stddef.h>
#include <stdlib.h>

#include <algorithm>
#include <vector>

#include "fs3d_dev.cuh"
#include "fs3d_line.cuh"
#include "fs3d_mixed.cuh"
#include "fs3d_mixed_line.cuh"

namespace mgk {

const void* twiddles(int n, int prec);
const void* twiddles_reg(int n, int prec);

const FsLine* fs_line_a(int n);
const FsLine* fs_line_b(int n);
const FsLine* fs_line_c(int n);
const FsLine* fs_line(int n) {
  for (auto f : {fs_line_a, fs_line_b, fs_line_c})
    if (const FsLine* k = f(n)) return k;
  return nullptr;
}

namespace fs32 {
const MixedLine* mixed_line_0(int n);
const MixedLine* mixed_line_1b(int n);
const MixedLine* mixed_line_1c(int n);
const MixedLine* mixed_line(int n, int alt) {
  if (!alt) return mixed_line_0(n);
  const MixedLine* k = mixed_line_1b(n);
  return k ? k : mixed_line_1c(n);
}
}  // namespace fs32

template <typename T> __device__ __forceinline__ T det3(const T* A) {
  return A[0] * (A[4] * A[8] - A[5] * A[7]) - A[1] * (A[3] * A[8] - A[5] * A[6]) + A[2] * (A[3] * A[7] - A[4] * A[6]);
}
template <typename T> __device__ __forceinline__ void inv3(const T* A, T* B) {
  const T d = det3(A);
  const T s = T(1) / d;
  B[0] = (A[4] * A[8] - A[5] * A[7]) * s;
  B[1] = -(A[1] * A[8] - A[2] * A[7]) * s;
  B[2] = (A[1] * A[5] - A[2] * A[4]) * s;
  B[3] = -(A[3] * A[8] - A[5] * A[6]) * s;
  B[4] = (A[0] * A[8] - A[2] * A[6]) * s;
  B[5] = -(A[0] * A[5] - A[2] * A[3]) * s;
  B[6] = (A[3] * A[7] - A[4] * A[6]) * s;
  B[7] = -(A[0] * A[7] - A[1] * A[6]) * s;
  B[8] = (A[0] * A[4] - A[1] * A[3]) * s;
}

// Per-voxel material state at F: Fe, S and what the tangent needs.
struct VoxelLaw {
  using T = double;
  T Fe[9], Fpi[9], S[9], Ci[9];
  T lam, mu, c, Je;
  T f33;  // out-of-plane stretch of a plane-stress plan (1 otherwise)
  int model, has_fp;

  __device__ void init(const FsArgs& a, long long i, const T* F, T alpha, const T* dX) {
    model = a.model;
    has_fp = a.has_fp;
    lam = a.lam[i];
    mu = a.mu[i];
    T Fv[9];
    for (int q = 0; q < 9; ++q) Fv[q] = F[q] + (dX ? alpha * dX[q] : T(0));
    if (has_fp && a.fpf[i] != 0) {
      for (int q = 0; q < 9; ++q) Fpi[q] = a.Fpi[q * a.N + i];
    } else {
      for (int q = 0; q < 9; ++q) Fpi[q] = (q % 4 == 0) ? T(1) : T(0);
    }
    mm(Fv, Fpi, Fe);
    T C[9];
    mtm(Fe, Fe, C);
    Je = det3(Fe);
    f33 = T(1);
    if (model == 0) {
      T Eg[9];
      for (int q = 0; q < 9; ++q) Eg[q] = T(0.5) * (C[q] - ((q % 4 == 0) ? T(1) : T(0)));
      const T tr = Eg[0] + Eg[4] + Eg[8];
      for (int q = 0; q < 9; ++q) S[q] = 2 * mu * Eg[q] + ((q % 4 == 0) ? lam * tr : T(0));
      if (a.plane_stress) {
        // :1042-1049: E33 = -(lam / (2 mu)) tr E of the in-plane strain (x, z)
        const T e33 = -(lam / (T(2) * mu)) * (Eg[0] + Eg[8]);
        f33 = sqrt(fmax(T(1e-12), T(1) + T(2) * e33));
      }
    } else if (a.plane_stress) {
      // plane-stress Neo-Hookean (:631-684): lam is the plane-stress lambda,
      // lam_3d = 2 mu lam / (2 mu - lam); x = F33^2 from the Newton solve of
      // mu x + lam_3d/2 ln x = mu - lam_3d ln Je (Je of the in-plane Fe, at
      // most 10 steps, until the step is below 1e-12); S = mu I - mu x C^-1;
      // the tangent's lam* = 2 lam_3d mu x / (lam_3d + 2 mu x), c = mu x
      const T lam3 = (T(2) * mu * lam) / fmax(T(1e-14), T(2) * mu - lam);
      const T target = mu - lam3 * log(fmax(T(1e-14), Je));
      T x = T(1);
#pragma unroll 1
      for (int it = 0; it < 10; ++it) {
        const T fx = mu * x + T(0.5) * lam3 * log(x) - target;
        const T dx = -fx / (mu + T(0.5) * lam3 / x);
        x = fmax(T(1e-10), x + dx);
        if (fabs(dx) < T(1e-12)) break;
      }
      f33 = sqrt(fmax(T(1e-12), x));
      inv3(C, Ci);
      c = mu * x;
      for (int q = 0; q < 9; ++q) S[q] = -c * Ci[q] + ((q % 4 == 0) ? mu : T(0));
      lam = (T(2) * lam3 * c) / fmax(T(1e-14), lam3 + T(2) * c);
    } else {
      const T lnJ = log(fmax(T(1e-14), Je));
      inv3(C, Ci);
      c = mu - lam * lnJ;
      const T k = lam * lnJ - mu;
      for (int q = 0; q < 9; ++q) S[q] = k * Ci[q] + ((q % 4 == 0) ? mu : T(0));
    }
  }

  // tangent state (see kFsState)
  __device__ void store(double* st, long long N, long long i) const {
    T M[9];
    if (model == 1) {
      inv3(Fe, M);
    } else {
      for (int q = 0; q < 9; ++q) M[q] = Fe[q] - ((q % 4 == 0) ? T(1) : T(0));
    }
    for (int q = 0; q < 9; ++q) st[q * N + i] = M[q];
    st[9 * N + i] = lam;
    st[10 * N + i] = mu;
    if (model == 1) st[11 * N + i] = c;
  }

  // the mixed form's (see fs32::kState)
  template <typename O> __device__ void store32(O* st, long long N, long long i, bool fp) const {
    T Tm[9], Sref[9];
    mm(Fpi, S, Tm);
    mmt(Tm, Fpi, Sref);
    for (int q = 0; q < 9; ++q) st[q * N + i] = (O)Fe[q];
    const int sidx[6] = {0, 4, 8, 5, 2, 1};
    for (int k = 0; k < 6; ++k) st[(9 + k) * N + i] = (O)Sref[sidx[k]];
    if (model == 1)
      for (int k = 0; k < 6; ++k) st[(15 + k) * N + i] = (O)Ci[sidx[k]];
    st[21 * N + i] = (O)lam;
    st[22 * N + i] = (O)(model == 1 ? c : mu);
    st[23 * N + i] = (O)(fp ? 1 : 0);
  }

  // P = Fe S Fp^-T
  __device__ void stress(T* P) const {
    T Tm[9];
    mm(Fe, S, Tm);
    mmt(Tm, Fpi, P);
  }
};

// ------------------------------------------------- general matvec stages ---
// The same stages for any supported side (fft_any: whole lines ping-pong in
// shared memory).

// z stage of one pair of z-lines; modes as fs_zline_reg
template <int MODE, int MODEL>
__global__ void __launch_bounds__(256) fs_z_kernel(FsArgs a) {
  using C = double2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nz = a.nz, nzh = a.nzh, ld = a.ld;
  const long long N = a.N;
  const long long l0 = 2LL * blockIdx.x;
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 9 * nz;
  C* spec = a.spec + l0 * ld;
  if constexpr (MODE == 0 || MODE == 3) {
    for (int e = threadIdx.x; e < 9 * nz; e += blockDim.x) {
      const int c = e / nz, k = e - c * nz;
      const int ks = (2 * k <= nz) ? k : nz - k;
      const C* ra = spec + c * a.plane;
      C x = ra[ks], y = ra[ld + ks];
      if (k == 0 || 2 * k == nz) { x.y = 0; y.y = 0; }
      C z = 2 * k <= nz ? mk<C>(x.x - y.y, x.y + y.x) : mk<C>(x.x + y.y, y.x - x.y);
      if (c % 3 == 2) {
        const double u = fs_u(ks, a.iz);
        z.x *= u;
        z.y *= u;
      }
      bufA[e] = z;
    }
    __syncthreads();
    C* R = fft_any<+1>(bufA, bufB, 9, nz, a.fz);
    if constexpr (MODE == 3) {
      for (int e = threadIdx.x; e < 9 * nz; e += blockDim.x) {
        const int c = e / nz, z = e - c * nz;
        double* X = a.X + c * N + l0 * nz + z;
        X[0] = R[e].x;
        X[nz] = R[e].y;
      }
      return;
    }
    bufB = R == bufA ? bufB : bufA;
    bufA = R;
  }
  for (int e = threadIdx.x; e < 2 * nz; e += blockDim.x) {
    const int h = e & 1, z = e >> 1;
    const long long i = (l0 + h) * nz + z;
    double* vx = reinterpret_cast<double*>(bufA + z) + h;
    double d[9], out[9];
    if constexpr (MODE == 2) {
      for (int q = 0; q < 9; ++q) out[q] = a.P[q * N + i];
    } else {
      for (int q = 0; q < 9; ++q) d[q] = MODE == 0 ? vx[q * 2 * nz] : a.sc->dbar[q];
      fs_kdf<MODEL>(a, i, d, out);
    }
    for (int q = 0; q < 9; ++q) vx[q * 2 * nz] = out[q];
  }
  __syncthreads();
  C* Z = fft_any<-1>(bufA, bufB, 9, nz, a.fz);
  for (int e = threadIdx.x; e < 9 * nzh; e += blockDim.x) {
    const int c = e / nzh, k = e - c * nzh;
    const C z = Z[c * nz + k];
    const C w = Z[c * nz + (k == 0 ? 0 : nz - k)];
    C* ra = spec + c * a.plane;
    const double f = c % 3 == 2 ? 0.5 * fs_u(k, a.iz) : 0.5;
    ra[k] = mk<C>(f * (z.x + w.x), f * (z.y - w.y));
    ra[ld + k] = mk<C>(f * (z.y + w.y), -f * (z.x - w.x));
  }
}

// y stage of one tensor row over a tile of kz columns; see fs_yline_reg
template <int SIGN>
__global__ void __launch_bounds__(256) fs_y_kernel(FsArgs a) {
  using C = double2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ny = a.ny, nzh = a.nzh, ld = a.ld, tc = a.tcy;
  const int ntile = (nzh + tc - 1) / tc;
  const int row = blockIdx.x % 3, item = blockIdx.x / 3;
  const int o = item / ntile, k0 = (item - o * ntile) * tc;
  const int tcw = min(tc, nzh - k0);
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 3 * tc * ny;
  C* spec = a.spec + 3 * row * a.plane + (long long)o * ny * ld + k0;
  for (int e = threadIdx.x; e < tcw * ny; e += blockDim.x) {
    const int j = e / tcw, t = e - j * tcw;
    const C* g = spec + (long long)j * ld + t;
    C v0 = g[0], v1 = g[a.plane], v2;
    if (SIGN < 0) {
      v2 = g[2 * a.plane];
    } else {
      const double u = fs_u(ffq(j, ny), a.iy);
      v2 = v1;
      v1 = mk<C>(u * v1.x, u * v1.y);
    }
    bufA[t * ny + j] = v0;
    bufA[(tc + t) * ny + j] = v1;
    bufA[(2 * tc + t) * ny + j] = v2;
  }
  __syncthreads();
  const C* F = fft_any<SIGN>(bufA, bufB, 3 * tc, ny, a.fy);
  for (int e = threadIdx.x; e < tcw * ny; e += blockDim.x) {
    const int j = e / tcw, t = e - j * tcw;
    C* g = spec + (long long)j * ld + t;
    const C v1 = F[(tc + t) * ny + j], v2 = F[(2 * tc + t) * ny + j];
    g[0] = F[t * ny + j];
    if (SIGN < 0) {
      const double u = fs_u(ffq(j, ny), a.iy);
      g[a.plane] = mk<C>(u * v1.x + v2.x, u * v1.y + v2.y);
    } else {
      g[a.plane] = v1;
      g[2 * a.plane] = v2;
    }
  }
}

// forward x stage with G's contraction
template <bool RHS>
__global__ void __launch_bounds__(256) fs_xfwd_kernel(FsArgs a) {
  using C = double2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  const int nx = a.nx, ld = a.ld, tc = a.tcx;
  const int ntile = (a.nzh + tc - 1) / tc;
  const int o = blockIdx.x / ntile, k0 = (blockIdx.x - o * ntile) * tc;
  const int tcw = min(tc, a.nzh - k0);
  const long long js = (long long)a.ny * ld, base = (long long)o * ld + k0;
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 6 * tc * nx;
  const C* spec = a.spec;
  for (int e = threadIdx.x; e < 6 * tcw * nx; e += blockDim.x) {
    const int c = e / (tcw * nx), rem = e - c * tcw * nx, j = rem / tcw, t = rem - j * tcw;
    bufA[(c * tc + t) * nx + j] = spec[(3 * (c >> 1) + (c & 1)) * a.plane + j * js + base + t];
  }
  __syncthreads();
  const C* F = fft_any<-1>(bufA, bufB, 6 * tc, nx, a.fx);
  double s = 0;
  for (int e = threadIdx.x; e < tcw * nx; e += blockDim.x) {
    const int kx = e / tcw, t = e - kx * tcw;
    C xv[3], bv[3];
    for (int i = 0; i < 3; ++i) { xv[i] = F[(2 * i * tc + t) * nx + kx]; bv[i] = F[((2 * i + 1) * tc + t) * nx + kx]; }
    s += fs_contract<RHS>(a, kx, o, k0 + t, xv, bv);
  }
  fs_finish(a, s, red, [&](double v) { fs_after_x<RHS>(a, v); });
}

// inverse x stage from the direction (or, FINAL, x)
template <bool FINAL>
__global__ void __launch_bounds__(256) fs_xinv_kernel(FsArgs a) {
  using C = double2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nx = a.nx, ld = a.ld, tc = a.tcx;
  const int ntile = (a.nzh + tc - 1) / tc;
  const int o = blockIdx.x / ntile, k0 = (blockIdx.x - o * ntile) * tc;
  const int tcw = min(tc, a.nzh - k0);
  const long long js = (long long)a.ny * ld, base = (long long)o * ld + k0;
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 6 * tc * nx;
  C* spec = a.spec;
  const double beta = a.sc->beta;
  for (int e = threadIdx.x; e < tcw * nx; e += blockDim.x) {
    const int kx = e / tcw, t = e - kx * tcw;
    const double u = fs_u(ffq(kx, nx), a.ix);
    for (int i = 0; i < 3; ++i) {
      const C v = fs_direction<FINAL>(a, beta, i * a.plane + kx * js + base + t);
      bufA[(2 * i * tc + t) * nx + kx] = mk<C>(u * v.x, u * v.y);
      bufA[((2 * i + 1) * tc + t) * nx + kx] = v;
    }
  }
  __syncthreads();
  const C* F = fft_any<+1>(bufA, bufB, 6 * tc, nx, a.fx);
  for (int e = threadIdx.x; e < 6 * tcw * nx; e += blockDim.x) {
    const int c = e / (tcw * nx), rem = e - c * tcw * nx, j = rem / tcw, t = rem - j * tcw;
    spec[(3 * (c >> 1) + (c & 1)) * a.plane + j * js + base + t] = F[(c * tc + t) * nx + j];
  }
}

// ------------------------------------------------------------ CG scalars ---
__global__ void fs_loop_head(FsArgs a, cudaGraphConditionalHandle cond) {
  cudaGraphSetConditional(cond, fs_go(*a.sc) ? 1u : 0u);
}

// CG update: x += alpha p, r -= alpha q, r.r, beta, and the loop's decision; the
// three components of a frequency together for their |u|^2.
__global__ void __launch_bounds__(256) fs_update_kernel(FsArgs a, cudaGraphConditionalHandle cond, int use_cond) {
  __shared__ double red[32];
  const double alpha = a.sc->alpha;
  const int ld = a.ld, tot = (int)a.plane;
  double acc = 0;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += gridDim.x * blockDim.x) {
    const int row = e / ld, kz = e - row * ld;
    if (kz >= a.nzh) continue;
    double2 p[3], q[3], x[3], r[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const long long at = i * a.plane + e;
      p[i] = a.vp[at]; q[i] = a.vq[at]; x[i] = a.vx[at]; r[i] = a.vr[at];
    }
    double s = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const long long at = i * a.plane + e;
      a.vx[at] = make_double2(x[i].x + alpha * p[i].x, x[i].y + alpha * p[i].y);
      const double2 v = make_double2(r[i].x - alpha * q[i].x, r[i].y - alpha * q[i].y);
      a.vr[at] = v;
      s += v.x * v.x + v.y * v.y;
    }
    acc += s * fs_u2(a, row / a.ny, row % a.ny, kz) * (kz > 0 ? 2.0 : 1.0);
  }
  fs_finish(a, acc, red, [&](double v) {
    FsScalars& S = *a.sc;
    S.beta = S.rr != 0.0 ? v / S.rr : 0.0;
    S.rr = v;
    S.kcount += 1.0;
    if (use_cond) cudaGraphSetConditional(cond, fs_go(S) ? 1u : 0u);
  });
}

// Sums of K values over the CTA (the tree of block_sum(), for all of them at
// once: 2 barriers, not 3 K, which took 0.5 ms of a 64^3 load step): out[k] for
// every thread.
template <int K> __device__ __forceinline__ void block_sums(const double* v, double (*red)[32], double* out) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double s = warp_sum(v[k]);
    if (lane == 0) red[k][wid] = s;
  }
  __syncthreads();
  for (int k = wid; k < K; k += nw) {
    const double s = warp_sum(lane < nw ? red[k][lane] : 0.0);
    if (lane == 0) out[k] = s;
  }
  __syncthreads();
}

// Constitutive evaluation at F + alpha (x + dbar) (at F without use_x): writes
// Fout, Pout and the tangent state there; min Je, NaN count, sum F^2, sum x^2 and the Cauchy stress means (cauchy_from_P_3d) are
// reduced by the CTA that arrives last.  16 values per CTA.
// x32, st32: the mixed form's increment and tangent state (null: FP64).  Two CTAs
// per SM (128 registers, 158 without being asked): 485 -> 290 us at 128^3, mixed.
__global__ void __launch_bounds__(256, 2) fs_constitutive_kernel(FsArgs a, double alpha, int use_dbar, int use_x, const float* __restrict__ x32,
                                       float* __restrict__ st32) {
  __shared__ double red[12][32], sum[12];
  const long long N = a.N;
  double mnJ = INFINITY, nan = 0, FF = 0, xx = 0;
  double sg[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    double F[9], dX[9];
    for (int q = 0; q < 9; ++q) {
      F[q] = a.F[q * N + i];
      const double xv = !use_x ? 0.0 : x32 ? (double)x32[q * N + i] : a.X[q * N + i];
      dX[q] = xv + (use_dbar ? a.sc->dbar[q] : 0.0);
      xx += xv * xv;
    }
    VoxelLaw law;
    law.init(a, i, F, alpha, dX);
    double Ft[9], P[9];
    for (int q = 0; q < 9; ++q) Ft[q] = F[q] + alpha * dX[q];
    law.stress(P);
    if (st32) law.store32(st32, N, i, law.has_fp && a.fpf[i] != 0);
    else law.store(a.st, N, i);
    if (!(law.Je == law.Je)) nan += 1;
    mnJ = fmin(mnJ, law.Je);
    double J = det3(Ft);
    if (a.plane_stress) J *= law.f33;
    if (fabs(J) < 1e-14) J = 1e-14;
    double PF[9];
    mmt(P, Ft, PF);
    for (int q = 0; q < 9; ++q) {
      if (!(P[q] == P[q])) nan += 1;
      a.Fout[q * N + i] = Ft[q];
      a.Pout[q * N + i] = P[q];
      FF += Ft[q] * Ft[q];
      sg[q] += PF[q] / J;
    }
  }
  // min via block reduction on -x with max semantics
  double v[13] = {0};
  v[0] = nan; v[1] = FF; v[2] = xx;
  for (int q = 0; q < 9; ++q) v[3 + q] = sg[q];
  block_sums<12>(v, red, sum);
  if (threadIdx.x < 12) {
    a.part[(size_t)blockIdx.x * 16 + threadIdx.x] = sum[threadIdx.x];
    __threadfence();
  }
  // min Je
  __shared__ double mn[32];
  double m = mnJ;
  for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) mn[threadIdx.x >> 5] = m;
  __syncthreads();
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    double r = INFINITY;
    for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w) r = fmin(r, mn[w]);
    a.part[(size_t)blockIdx.x * 16 + 12] = r;
    __threadfence();
    s_last = atomicInc(a.counter, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int nb = gridDim.x;
  for (int q = 0; q < 12; ++q) v[q] = 0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x)
    for (int q = 0; q < 12; ++q) v[q] += __ldcg(&a.part[(size_t)i * 16 + q]);
  block_sums<12>(v, red, sum);
  m = INFINITY;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) m = fmin(m, __ldcg(&a.part[(size_t)i * 16 + 12]));
  for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) mn[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    FsScalars& S = *a.sc;
    double r = INFINITY;
    for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w) r = fmin(r, mn[w]);
    S.nan = sum[0];
    S.FF = sum[1];
    S.xx = sum[2];
    for (int q = 0; q < 9; ++q) S.sig[q] = sum[3 + q] / (double)a.N;
    S.minJe = r;
  }
}

// Start of a Newton solve: dbar = F_bar - mean(F), and the Krylov loop's
// tolerance and iteration cap; 16 values per CTA, the last CTA sums.
struct FsBegin {
  double F_bar[9], tol2, kmax;
};
__global__ void fs_begin_kernel(FsArgs a, FsBegin b) {
  __shared__ double red[9][32], sum[9];
  __shared__ int s_last;
  double s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.N; i += (long long)gridDim.x * blockDim.x)
    for (int q = 0; q < 9; ++q) s[q] += a.F[q * a.N + i];
  block_sums<9>(s, red, sum);
  if (threadIdx.x < 9) {
    a.part[(size_t)blockIdx.x * 16 + threadIdx.x] = sum[threadIdx.x];
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicInc(a.counter, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int q = 0; q < 9; ++q) s[q] = 0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x)
    for (int q = 0; q < 9; ++q) s[q] += __ldcg(&a.part[(size_t)i * 16 + q]);
  block_sums<9>(s, red, sum);
  if (threadIdx.x == 0) {
    for (int q = 0; q < 9; ++q) a.sc->dbar[q] = b.F_bar[q] - sum[q] / (double)a.N;
    a.sc->tol2 = b.tol2;
    a.sc->kmax = b.kmax;
    a.sc->err = 0.0;
  }
}

// FP64 tangent state at F for the mixed form's first right-hand side
__global__ void fs_tangent_kernel(FsArgs a, double* __restrict__ st) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.N; i += (long long)gridDim.x * blockDim.x) {
    double F[9];
    for (int q = 0; q < 9; ++q) F[q] = a.F[q * a.N + i];
    VoxelLaw law;
    law.init(a, i, F, 0.0, nullptr);
    law.store32(st, a.N, i, law.has_fp && a.fpf[i] != 0);
  }
}

// Cauchy stress field (cauchy_from_P_3d; cauchy_from_P with F33 for plane
// stress), tensor-first
__global__ void fs_cauchy_kernel(FsArgs a, double* sig) {
  const long long N = a.N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    double Pv[9], Fv[9], PF[9];
    for (int q = 0; q < 9; ++q) { Pv[q] = a.P[q * N + i]; Fv[q] = a.F[q * N + i]; }
    double J = det3(Fv);
    if (a.plane_stress) {
      VoxelLaw law;
      law.init(a, i, Fv, 0.0, nullptr);
      J *= law.f33;
    }
    if (fabs(J) < 1e-14) J = 1e-14;
    mmt(Pv, Fv, PF);
    for (int q = 0; q < 9; ++q) sig[q * N + i] = PF[q] / J;
  }
}

// material: lam, mu planes, Fp^-1 (plain inverse of F_p, as _invert_Fp_3d) and
// where it is not the identity
__global__ void fs_material_kernel(long long N, const double* __restrict__ lam_in, const double* __restrict__ mu_in,
                                   const double* __restrict__ Fp, double* lam, double* mu, double* Fpi,
                                   unsigned char* fpf) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    lam[i] = lam_in[i];
    mu[i] = mu_in[i];
    if (Fp) {
      double A[9], B[9];
      for (int q = 0; q < 9; ++q) A[q] = Fp[q * N + i];
      double d = det3(A);
      if (fabs(d) < 1e-14) d = 1e-14;
      const double s = 1.0 / d;
      B[0] = (A[4] * A[8] - A[5] * A[7]) * s;
      B[1] = -(A[1] * A[8] - A[2] * A[7]) * s;
      B[2] = (A[1] * A[5] - A[2] * A[4]) * s;
      B[3] = -(A[3] * A[8] - A[5] * A[6]) * s;
      B[4] = (A[0] * A[8] - A[2] * A[6]) * s;
      B[5] = -(A[0] * A[5] - A[2] * A[3]) * s;
      B[6] = (A[3] * A[7] - A[4] * A[6]) * s;
      B[7] = -(A[0] * A[7] - A[1] * A[6]) * s;
      B[8] = (A[0] * A[4] - A[1] * A[3]) * s;
      bool ident = true;
      for (int q = 0; q < 9; ++q) {
        Fpi[q * N + i] = B[q];
        ident = ident && B[q] == ((q % 4 == 0) ? 1.0 : 0.0);
      }
      fpf[i] = ident ? 0 : 1;
    }
  }
}

}  // namespace mgk

// ================================================================== plan ===
using namespace mgk;

struct mgk_fs3d_plan {
  int nx, ny, nz, nzh, ld, tc, tcx, tcy, model;
  long long N, plane;
  int has_fp = 0, has_material = 0;
  FftLen fft[3];
  const double2* rtw[3];  // register-FFT twiddles (null: no such length)
  const FsLine* line[3];
  double* fields = nullptr;  // F, Ftr, P, Ptr, X, Fpi, lam, mu
  double *F, *Ftr, *P, *Ptr, *X, *Fpi, *lam, *mu;
  unsigned char* fpf = nullptr;
  double2* spec = nullptr;  // 9 spectrum planes, then the Krylov vectors (4 x 3)
  double* st64 = nullptr;   // tangent state planes
  double* part = nullptr;
  unsigned int* counter = nullptr;
  FsScalars* sc = nullptr;
  FsScalars* h_sc = nullptr;  // pinned
  size_t zsmem = 0, ysmem = 0, xsmem = 0;
  int nblk = 0, ublk = 0;
  int stat_newton = 0, stat_krylov = 0, stat_macro = 0;
  // precision form: MGK_FP64, or MGK_MIXED (FP32 Krylov loop)
  int prec = MGK_FP64;
  float* f32 = nullptr;  // p, q, r, x, F_p^-1, and the FP64 tangent state of its right-hand sides
  FftLen fft32[3];
  const void* rtw32[3];
  const fs32::MixedLine* line32[3];
  // device-side Krylov loop graphs, one per precision (0 FP64, 1 FP32)
  cudaGraph_t cg_graph[2] = {nullptr, nullptr};
  cudaGraphExec_t cg_exec[2] = {nullptr, nullptr};
  int graph_mode = -1;  // -1 untried, 1 graphs, 0 host-driven loop
  int fast = 1;         // register-FFT kernels on the axes that have them
  // plane strain embedded as (nx, 1, ny): the out-of-plane F_yy = 1 adds N
  // to ||F||^2, which the 2D solver's Newton norm does not contain
  double ff_offset = 0.0;
  int plane_stress = 0;  // 2D plane stress on the (nx, 1, ny) plan
};

static FsArgs fs_args(mgk_fs3d_t p) {
  FsArgs a;
  memset(&a, 0, sizeof(a));
  a.nx = p->nx; a.ny = p->ny; a.nz = p->nz; a.nzh = p->nzh; a.ld = p->ld; a.tcx = p->tcx; a.tcy = p->tcy;
  a.N = p->N; a.plane = p->plane;
  a.ix = 1.0 / p->nx; a.iy = 1.0 / p->ny; a.iz = 1.0 / p->nz;
  a.has_fp = p->has_fp; a.model = p->model; a.plane_stress = p->plane_stress;
  a.fx = p->fft[0]; a.fy = p->fft[1]; a.fz = p->fft[2];
  for (int q = 0; q < 3; ++q) a.rtw[q] = p->rtw[q];
  a.F = p->F; a.Fpi = p->Fpi; a.mu = p->mu; a.lam = p->lam; a.P = p->P; a.fpf = p->fpf;
  a.X = p->X; a.Fout = p->Ftr; a.Pout = p->Ptr;
  a.spec = p->spec;
  double2* v = p->spec + 9 * p->plane;
  a.vr = v; a.vp = v + 3 * p->plane; a.vx = v + 6 * p->plane; a.vq = v + 9 * p->plane;
  a.st = p->st64;
  a.part = p->part; a.counter = p->counter; a.sc = p->sc;
  return a;
}

static fs32::Fs32Args fs32_args(mgk_fs3d_t p) {
  fs32::Fs32Args a;
  memset(&a, 0, sizeof(a));
  a.nx = p->nx; a.ny = p->ny; a.nz = p->nz; a.nzh = p->nzh; a.ld = p->ld; a.tc = p->tc;
  a.N = p->N; a.has_fp = p->has_fp; a.model = p->model;
  a.fx = p->fft[0]; a.fy = p->fft[1]; a.fz = p->fft[2];
  a.fx32 = p->fft32[0]; a.fy32 = p->fft32[1]; a.fz32 = p->fft32[2];
  for (int q = 0; q < 3; ++q) a.rtw32[q] = p->rtw32[q];
  a.Fpi = p->Fpi; a.P = p->P; a.r = p->X;
  float* f = p->f32;
  a.p32 = f; a.q32 = f + 9 * p->N; a.r32 = f + 18 * p->N; a.x32 = f + 27 * p->N; a.Fpi32 = f + 36 * p->N;
  a.st64 = reinterpret_cast<double*>(f + 46 * p->N);
  a.st32 = reinterpret_cast<float*>(p->st64);  // 12 planes of doubles that the FP64 loop alone reads
  a.spec = p->spec;
  a.part = p->part; a.sc = p->sc;
  return a;
}
// whether the right-hand side takes the warp-line passes (and the FP32 passes
// their roundings)
static bool fs32_fast(mgk_fs3d_t p) {
  return p->fast && fs32::fs_fast_len(p->nx) && fs32::fs_fast_len(p->ny) && fs32::fs_fast_len(p->nz);
}

extern "C" int mgk_fs3d_destroy(mgk_fs3d_t p) {
  if (!p) return MGK_OK;
  for (int k = 0; k < 2; ++k) {
    if (p->cg_exec[k]) cudaGraphExecDestroy(p->cg_exec[k]);
    if (p->cg_graph[k]) cudaGraphDestroy(p->cg_graph[k]);
  }
  cudaFree(p->f32);
  cudaFree(p->st64);
  cudaFree(p->fields);
  cudaFree(p->fpf);
  cudaFree(p->spec);
  cudaFree(p->part);
  cudaFree(p->counter);
  cudaFree(p->sc);
  if (p->h_sc) cudaFreeHost(p->h_sc);
  delete p;
  return MGK_OK;
}

// One kernel launch; the FP64 CG update also takes the loop's handle.
struct FsLaunch {
  const void* fn;
  int grid, block;
  size_t smem;
};
static const FsLine* fs_kernels(mgk_fs3d_t p, int axis) { return p->fast ? p->line[axis] : nullptr; }

// z stage; modes as fs_zline_reg
static FsLaunch fs_z_launch(mgk_fs3d_t p, int mode) {
  const int pairs = (int)(p->N / p->nz / 2);
  if (const FsLine* k = fs_kernels(p, 2))
    return {k->z[p->model][mode], pairs, k->z_threads, (size_t)k->z_bytes};
  const void* fn = mode == 0   ? (p->model ? (const void*)fs_z_kernel<0, 1> : (const void*)fs_z_kernel<0, 0>)
                   : mode == 1 ? (p->model ? (const void*)fs_z_kernel<1, 1> : (const void*)fs_z_kernel<1, 0>)
                   : mode == 2 ? (const void*)fs_z_kernel<2, 0>
                               : (const void*)fs_z_kernel<3, 0>;
  return {fn, pairs, 256, p->zsmem};
}
static FsLaunch fs_y_launch(mgk_fs3d_t p, int inverse) {
  if (const FsLine* k = fs_kernels(p, 1))
    return {k->y[inverse], 3 * p->nx * ((p->nzh + k->tile - 1) / k->tile), k->y_threads, (size_t)k->y_bytes};
  return {inverse ? (const void*)fs_y_kernel<1> : (const void*)fs_y_kernel<-1>,
          3 * p->nx * ((p->nzh + p->tcy - 1) / p->tcy), 256, p->ysmem};
}
// forward x stage: kind 0 matvec, 1 right-hand side; inverse: 0 direction, 1 x
static FsLaunch fs_x_launch(mgk_fs3d_t p, int inverse, int kind) {
  if (const FsLine* k = fs_kernels(p, 0))
    return {inverse ? k->xi[kind] : k->xf[kind], p->ny * ((p->nzh + k->tile - 1) / k->tile), k->x_threads, (size_t)k->x_bytes};
  const void* fn = inverse ? (kind ? (const void*)fs_xinv_kernel<true> : (const void*)fs_xinv_kernel<false>)
                           : (kind ? (const void*)fs_xfwd_kernel<true> : (const void*)fs_xfwd_kernel<false>);
  return {fn, p->ny * ((p->nzh + p->tcx - 1) / p->tcx), 256, p->xsmem};
}

// The CTA-wide passes' launches (T float: the matvec's; double: a right-hand
// side's, mode 1 uniform, 2 P): z forward, y, x with G, y inverse, z inverse.
template <typename T> static void fs32_general(mgk_fs3d_t p, int mode, FsLaunch L[5]) {
  using namespace fs32;
  constexpr int zm = sizeof(T) == 8 ? 1 : 0;  // z inverse: q and p.q, or r and r.r
  const int zl = (int)(p->N / p->nz / 2), ntile = (p->nzh + p->tc - 1) / p->tc;
  const size_t zs = p->zsmem * sizeof(T) / 8, ys = 2 * 9 * (size_t)p->tc * p->ny * 2 * sizeof(T),
               xs = 2 * 9 * (size_t)p->tc * p->nx * 2 * sizeof(T);
  if constexpr (zm == 0) L[0] = {(const void*)fs_zfwd_kernel<0, T>, zl, 256, zs};
  else L[0] = {mode == 1 ? (const void*)fs_zfwd_kernel<1, T> : (const void*)fs_zfwd_kernel<2, T>, zl, 256, zs};
  L[1] = {(const void*)fs_ypass_kernel<-1, T>, p->nx * ntile, 256, ys};
  L[2] = {(const void*)fs_xg_kernel<T>, p->ny * ntile, 256, xs};
  L[3] = {(const void*)fs_ypass_kernel<1, T>, p->nx * ntile, 256, ys};
  L[4] = {(const void*)fs_zinv_kernel<zm, T>, zl, 256, zs};
}
static void fs32_rhs(mgk_fs3d_t p, int mode, FsLaunch L[5]) {
  using namespace fs32;
  if (!fs32_fast(p)) return fs32_general<double>(p, mode, L);
  const int zl = (int)(p->N / p->nz / 2), ntile = 3 * ((p->nzh + kFsTile - 1) / kFsTile);
  const size_t zs = 9 * (size_t)fs_pl(p->nz) * 16, ys = 3 * (size_t)kFsTile * fs_pl(p->ny) * 16,
               xs = 3 * (size_t)kFsTile * fs_pl(p->nx) * 16;
  L[0] = {mode == 1 ? (const void*)fs_zfwd_fast_kernel<1> : (const void*)fs_zfwd_fast_kernel<2>, zl, 96, zs};
  L[1] = {(const void*)fs_axis_fast_kernel<-1, false>, p->nx * ntile, 96, ys};
  L[2] = {(const void*)fs_axis_fast_kernel<-1, true>, p->ny * ntile, 96, xs};
  L[3] = {(const void*)fs_axis_fast_kernel<1, false>, p->nx * ntile, 96, ys};
  L[4] = {(const void*)fs_zinv_fast64_kernel, zl, 96, zs};
}
// the matvec's launches: register FFTs on the axes that have one
static void fs32_matvec(mgk_fs3d_t p, FsLaunch L[5]) {
  fs32_general<float>(p, 0, L);
  if (!p->fast) return;
  const int zl = (int)(p->N / p->nz / 2);
  if (const fs32::MixedLine* k = p->line32[2]) {
    L[0] = {k->zfwd, zl, k->zf_threads, (size_t)k->zf_bytes};
    L[4] = {k->zinv, zl, k->zi_threads, (size_t)k->zi_bytes};
  }
  if (const fs32::MixedLine* k = p->line32[1])
    for (int inv = 0; inv < 2; ++inv)
      L[inv ? 3 : 1] = {k->y[inv], 3 * p->nx * ((p->nzh + k->yw - 1) / k->yw), k->y_threads, (size_t)k->y_bytes};
  if (const fs32::MixedLine* k = p->line32[0])
    L[2] = {k->x, p->ny * ((p->nzh + k->xw - 1) / k->xw), k->x_threads, (size_t)k->x_bytes};
}

// Raise the shared-memory limits of the kernels that the plan launches in its
// family and precision, where they need it.
static int fs_raise(mgk_fs3d_t p) {
  cudaError_t e = cudaSuccess;
  auto up = [&](const FsLaunch& l) { if (e == cudaSuccess) e = raise_smem(l.fn, l.smem); };
  if (p->prec == MGK_MIXED) {
    FsLaunch L[5];
    fs32_matvec(p, L);
    for (const FsLaunch& l : L) up(l);
    for (int m = 1; m < 3; ++m) {
      fs32_rhs(p, m, L);
      for (const FsLaunch& l : L) up(l);
    }
  }
  // a mixed plan's FP64 kernels run under the profiler
  for (int m = 0; m < 4; ++m) up(fs_z_launch(p, m));
  for (int k = 0; k < 2; ++k) { up(fs_y_launch(p, k)); up(fs_x_launch(p, 0, k)); up(fs_x_launch(p, 1, k)); }
  if (e != cudaSuccess) { cudaGetLastError(); set_error("mgk_fs3d: cudaFuncSetAttribute failed"); return MGK_CUDA_ERROR; }
  return MGK_OK;
}

extern "C" int mgk_fs3d_create(int nx, int ny, int nz, int model, mgk_fs3d_t* out) {
  MGK_REQUIRE(out, "mgk_fs3d_create: null output handle");
  *out = nullptr;
  MGK_REQUIRE(model == 0 || model == 1, "mgk_fs3d_create: model must be 0 (SVK) or 1 (Neo-Hookean)");
  FftLen fx, fy, fz;
  MGK_REQUIRE(fft_schedule(nx, &fx) && fft_schedule(ny, &fy) && fft_schedule(nz, &fz) && ((long long)nx * ny) % 2 == 0,
              "mgk_fs3d_create: grid %dx%dx%d unsupported (sides 2^a 3^b up to 4096, nx*ny even)", nx, ny, nz);
  // the shared memory of whole lines of all nine components decides which
  // grids are taken
  int tc = 4;
  while (tc > 1 && 2 * 9 * (size_t)tc * std::max(nx, ny) * sizeof(double2) > 96 * 1024) tc >>= 1;
  const size_t zsmem = 2 * 9 * (size_t)nz * sizeof(double2);
  MGK_REQUIRE(zsmem <= 220 * 1024 && 2 * 9 * (size_t)tc * std::max(nx, ny) * sizeof(double2) <= 220 * 1024,
              "mgk_fs3d_create: grid too large for the shared-memory FFT");
  mgk_fs3d_t p = new mgk_fs3d_plan();
  auto fail = [&](int s) { mgk_fs3d_destroy(p); return s; };
  p->nx = nx; p->ny = ny; p->nz = nz; p->nzh = nz / 2 + 1; p->ld = fs_ld(nz); p->model = model;
  p->tc = tc;
  p->N = (long long)nx * ny * nz;
  p->plane = (long long)nx * ny * p->ld;
  // kz columns per CTA of the general axis passes: as above, more on short
  // lines (y has one point in a 2D plan), where a CTA of four would idle
  auto tile = [&](int n, int lines) {
    int t = tc;
    while (t < 64 && t < p->nzh && 2 * lines * 2 * (size_t)t * n * sizeof(double2) <= 24 * 1024) t *= 2;
    return t;
  };
  p->tcy = tile(ny, 3);
  p->tcx = tile(nx, 6);
  p->zsmem = zsmem;
  p->ysmem = 2 * 3 * (size_t)p->tcy * ny * sizeof(double2);
  p->xsmem = 2 * 6 * (size_t)p->tcx * nx * sizeof(double2);
  p->fft[0] = fx; p->fft[1] = fy; p->fft[2] = fz;
  const int n[3] = {nx, ny, nz};
  for (int q = 0; q < 3; ++q) {
    p->fft32[q] = p->fft[q];
    p->line[q] = fs_line(n[q]);
    p->rtw[q] = p->line[q] ? reinterpret_cast<const double2*>(twiddles_reg(n[q], MGK_FP64)) : nullptr;
    if (!(p->fft[q].tw = twiddles(n[q], MGK_FP64)) || (p->line[q] && !p->rtw[q])) return fail(MGK_OOM);
  }
  const long long N = p->N;
  auto alloc = [&](auto** d, size_t n) {
    if (cudaMalloc((void**)d, n * sizeof(**d)) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
  };
  p->nblk = (int)std::max(1LL, std::min(1024LL, (N + 255) / 256));
  p->ublk = (int)std::max(1LL, std::min(1184LL, (p->plane + 255) / 256));  // <= 16 nblk
  const size_t npart = std::max((size_t)16 * p->nblk, (size_t)std::max((long long)nx * ny / 2, (long long)ny * p->nzh));
  if (!alloc(&p->fields, (size_t)N * (9 * 6 + 2)) || !alloc(&p->fpf, (size_t)N) || !alloc(&p->spec, 21 * (size_t)p->plane) ||
      !alloc(&p->st64, (size_t)kFsState * N) || !alloc(&p->part, npart) || !alloc(&p->counter, 1) || !alloc(&p->sc, 1))
    return fail(MGK_OOM);
  double* f = p->fields;
  p->F = f; p->Ftr = f + 9 * N; p->P = f + 18 * N; p->Ptr = f + 27 * N; p->X = f + 36 * N; p->Fpi = f + 45 * N;
  p->lam = f + 54 * N; p->mu = f + 55 * N;
  if (cudaMallocHost(&p->h_sc, sizeof(FsScalars)) != cudaSuccess) return fail(MGK_OOM);
  // The memsets run on the legacy stream and do not hold the host up; the caller's
  // stream need not wait for that one, so the plan leaves here with them done.
  // (The spectra and Krylov vectors start unset: every entry is written before it is read.)
  if (cudaMemset(p->fields, 0, sizeof(double) * N * (9 * 6 + 2)) != cudaSuccess ||
      cudaMemset(p->counter, 0, sizeof(unsigned int)) != cudaSuccess || cudaMemset(p->sc, 0, sizeof(FsScalars)) != cudaSuccess ||
      cudaStreamSynchronize(0) != cudaSuccess)
    return fail(MGK_CUDA_ERROR);
  const char* env = getenv("MGK_FS_FAST");
  p->fast = !(env && env[0] == '0');
  if (int rc = fs_raise(p)) return fail(rc);
  *out = p;
  return MGK_OK;
}

static void fs_drop_graphs(mgk_fs3d_t p) {
  for (int k = 0; k < 2; ++k) {
    if (p->cg_exec[k]) cudaGraphExecDestroy(p->cg_exec[k]);
    if (p->cg_graph[k]) cudaGraphDestroy(p->cg_graph[k]);
    p->cg_exec[k] = nullptr;
    p->cg_graph[k] = nullptr;
  }
}

// FP32 copy of F_p^-1 for the mixed form's matvecs
static int fs_refresh_f32(mgk_fs3d_t p, cudaStream_t s) {
  if (p->prec != MGK_MIXED || !p->has_fp) return MGK_OK;
  fs32::fs_to_f32_kernel<<<p->nblk, 256, 0, s>>>(9 * p->N, p->Fpi, p->f32 + 36 * p->N);
  MGK_CUDA(cudaGetLastError());
  return MGK_OK;
}

extern "C" int mgk_fs3d_set_precision(mgk_fs3d_t p, int precision) {
  MGK_REQUIRE(p, "mgk_fs3d_set_precision: null plan");
  MGK_REQUIRE(precision == MGK_FP64 || precision == MGK_MIXED, "mgk_fs3d_set_precision: bad precision");
  if (precision == MGK_MIXED && !p->f32) {
    const int n[3] = {p->nx, p->ny, p->nz};
    const bool alt = !fs32_fast(p);
    for (int q = 0; q < 3; ++q) {
      p->line32[q] = fs32::mixed_line(n[q], alt);
      p->rtw32[q] = p->line32[q] ? twiddles_reg(n[q], MGK_MIXED) : nullptr;
      if (!(p->fft32[q].tw = twiddles(n[q], 1)) || (p->line32[q] && !p->rtw32[q])) return MGK_OOM;
    }
    // one allocation: the FP32 planes (an even number of floats), the FP64 state
    if (cudaMalloc(&p->f32, sizeof(float) * p->N * 46 + sizeof(double) * p->N * fs32::kState) != cudaSuccess) {
      cudaGetLastError();
      p->f32 = nullptr;
      set_error("mgk_fs3d_set_precision: cudaMalloc of the FP32 planes failed");
      return MGK_OOM;
    }
  }
  if (precision != p->prec) fs_drop_graphs(p);  // the graphs capture the plane set
  p->prec = precision;
  if (int rc = fs_raise(p)) return rc;
  if (precision == MGK_MIXED && p->has_material) {
    MGK_CUDA(cudaDeviceSynchronize());
    int rc = fs_refresh_f32(p, 0);
    if (rc) return rc;
    MGK_CUDA(cudaDeviceSynchronize());
  }
  return MGK_OK;
}

extern "C" int mgk_fs3d_set_material(mgk_fs3d_t p, const double* lam, const double* mu, const double* Fp,
                                     mgk_stream_t stream) {
  MGK_REQUIRE(p && lam && mu, "mgk_fs3d_set_material: null argument");
  cudaStream_t s = (cudaStream_t)stream;
  fs_material_kernel<<<p->nblk, 256, 0, s>>>(p->N, lam, mu, Fp, p->lam, p->mu, p->Fpi, p->fpf);
  MGK_CUDA(cudaGetLastError());
  if ((Fp ? 1 : 0) != p->has_fp) fs_drop_graphs(p);  // the graphs capture has_fp
  p->has_fp = Fp ? 1 : 0;
  p->has_material = 1;
  return fs_refresh_f32(p, s);
}

extern "C" int mgk_fs3d_set_F(mgk_fs3d_t p, const double* F, mgk_stream_t stream) {
  MGK_REQUIRE(p && F, "mgk_fs3d_set_F: null argument");
  MGK_CUDA(cudaMemcpyAsync(p->F, F, sizeof(double) * 9 * p->N, cudaMemcpyDeviceToDevice, (cudaStream_t)stream));
  return MGK_OK;
}

extern "C" int mgk_fs3d_get(mgk_fs3d_t p, double* F_out, double* P_out, double* sig_out, mgk_stream_t stream) {
  MGK_REQUIRE(p, "mgk_fs3d_get: null plan");
  cudaStream_t s = (cudaStream_t)stream;
  if (F_out) MGK_CUDA(cudaMemcpyAsync(F_out, p->F, sizeof(double) * 9 * p->N, cudaMemcpyDeviceToDevice, s));
  if (P_out) MGK_CUDA(cudaMemcpyAsync(P_out, p->P, sizeof(double) * 9 * p->N, cudaMemcpyDeviceToDevice, s));
  if (sig_out) {
    fs_cauchy_kernel<<<p->nblk, 256, 0, s>>>(fs_args(p), sig_out);
    MGK_CUDA(cudaGetLastError());
  }
  return MGK_OK;
}

template <typename A> static int fs_run(const FsLaunch& l, A& a, cudaStream_t s) {
  void* args[] = {&a};
  MGK_CUDA(cudaLaunchKernel(l.fn, dim3(l.grid), dim3(l.block), args, l.smem, s));
  return MGK_OK;
}

// right-hand side -G:K:dbar (uniform) or -G:P into r, always in FP64; x = 0.
// The mixed form: r as a real field, its FP32 copy, and the partials of r.r.
static int fs_rhs(mgk_fs3d_t p, bool uniform, cudaStream_t s) {
  if (p->prec == MGK_MIXED) {
    fs32::Fs32Args b = fs32_args(p);
    FsLaunch l[5];
    fs32_rhs(p, uniform ? 1 : 2, l);
    for (const FsLaunch& k : l)
      if (int rc = fs_run(k, b, s)) return rc;
    fs32::fs_to_f32_kernel<<<p->nblk, 256, 0, s>>>(9 * p->N, b.r, b.r32);
    MGK_CUDA(cudaGetLastError());
    MGK_CUDA(cudaMemsetAsync(b.x32, 0, sizeof(float) * 9 * p->N, s));
    return MGK_OK;
  }
  FsArgs a = fs_args(p);
  const FsLaunch l[3] = {fs_z_launch(p, uniform ? 1 : 2), fs_y_launch(p, 0), fs_x_launch(p, 0, 1)};
  for (const FsLaunch& k : l)
    if (int rc = fs_run(k, a, s)) return rc;
  return MGK_OK;
}

// the increment as a real field X
static int fs_field(mgk_fs3d_t p, cudaStream_t s) {
  FsArgs a = fs_args(p);
  const FsLaunch l[3] = {fs_x_launch(p, 1, 1), fs_y_launch(p, 1), fs_z_launch(p, 3)};
  for (const FsLaunch& k : l)
    if (int rc = fs_run(k, a, s)) return rc;
  return MGK_OK;
}

// the FP64 matvec's five launches, up to the CG update
static void fs_matvec(mgk_fs3d_t p, FsLaunch l[5]) {
  l[0] = fs_x_launch(p, 1, 0);
  l[1] = fs_y_launch(p, 1);
  l[2] = fs_z_launch(p, 0);
  l[3] = fs_y_launch(p, 0);
  l[4] = fs_x_launch(p, 0, 0);
}

static int fs_read_scalars(mgk_fs3d_t p, cudaStream_t s) {
  MGK_CUDA(cudaMemcpyAsync(p->h_sc, p->sc, sizeof(FsScalars), cudaMemcpyDeviceToHost, s));
  MGK_CUDA(cudaStreamSynchronize(s));
  return MGK_OK;
}

// constitutive at F + alpha (x + dbar), and the tangent state there; results in
// Ftr/Ptr and the scalars
static int fs_trial(mgk_fs3d_t p, double alpha, bool use_dbar, bool use_x, cudaStream_t s) {
  const bool mixed = p->prec == MGK_MIXED;
  fs_constitutive_kernel<<<p->nblk, 256, 0, s>>>(fs_args(p), alpha, use_dbar, use_x, mixed ? p->f32 + 27 * p->N : nullptr,
                                                 mixed ? reinterpret_cast<float*>(p->st64) : nullptr);
  MGK_CUDA(cudaGetLastError());
  return MGK_OK;
}

// accept the trial state (the Krylov graphs read neither F nor P)
static void fs_accept(mgk_fs3d_t p) {
  std::swap(p->F, p->Ftr);
  std::swap(p->P, p->Ptr);
}

// The Krylov loop of either precision as launches: the head, and the body that
// the last launch decides to repeat.
struct FsLoop {
  FsArgs a;
  fs32::Fs32Args b;
  cudaGraphConditionalHandle h{};
  int use_cond = 0, n = 0, nb, zl;
  void *a1[1], *b1[1], *ah[3], *bz[4], *bn[4];
  struct Node {
    FsLaunch l;
    void** args;
  } head, body[8];
};
static void fs_loop(mgk_fs3d_t p, int f, FsLoop& L) {
  L.a = fs_args(p);
  L.b = fs32_args(p);
  L.nb = p->nblk;
  L.zl = (int)(p->N / p->nz / 2);
  L.a1[0] = &L.a;
  L.b1[0] = &L.b;
  L.ah[0] = &L.a; L.ah[1] = &L.h; L.ah[2] = &L.use_cond;
  L.bz[0] = &L.b; L.bz[1] = &L.zl; L.bz[2] = &L.h; L.bz[3] = &L.use_cond;
  L.bn[0] = &L.b; L.bn[1] = &L.nb; L.bn[2] = &L.h; L.bn[3] = &L.use_cond;
  FsLaunch l[5];
  if (f) fs32_matvec(p, l);
  else fs_matvec(p, l);
  for (const FsLaunch& k : l) L.body[L.n++] = {k, f ? L.b1 : L.a1};
  if (f) {
    L.head = {{(const void*)fs32::fs_scalar_kernel<2>, 1, 256, 0}, L.bz};
    L.body[L.n++] = {{(const void*)fs32::fs_scalar_kernel<0>, 1, 256, 0}, L.bz};
    L.body[L.n++] = {{(const void*)fs32::fs_update_kernel, p->nblk, 256, 0}, L.b1};
    L.body[L.n++] = {{(const void*)fs32::fs_scalar_kernel<1>, 1, 256, 0}, L.bn};
  } else {
    L.head = {{(const void*)fs_loop_head, 1, 1, 0}, L.ah};
    L.body[L.n++] = {{(const void*)fs_update_kernel, p->ublk, 256, 0}, L.ah};
  }
}
static int fs_run(const FsLoop::Node& k, cudaStream_t s) {
  MGK_CUDA(cudaLaunchKernel(k.l.fn, dim3(k.l.grid), dim3(k.l.block), k.args, k.l.smem, s));
  return MGK_OK;
}

// Krylov loop graph: head, then while (condition) body.
static int fs_build_graph(mgk_fs3d_t p, int f) {
  cudaGraph_t g = nullptr;
  MGK_CUDA(cudaGraphCreate(&g, 0));
  int rc = MGK_OK;
  FsLoop L;
  fs_loop(p, f, L);
  L.use_cond = 1;
  auto add = [&](cudaGraph_t gr, cudaGraphNode_t* node, const cudaGraphNode_t* dep, const FsLoop::Node& n) {
    cudaKernelNodeParams k;
    memset(&k, 0, sizeof(k));
    k.func = const_cast<void*>(n.l.fn);
    k.gridDim = dim3(n.l.grid);
    k.blockDim = dim3(n.l.block);
    k.sharedMemBytes = (unsigned)n.l.smem;
    k.kernelParams = n.args;
    if (rc == MGK_OK && cudaGraphAddKernelNode(node, gr, dep, dep ? 1 : 0, &k) != cudaSuccess) rc = MGK_CUDA_ERROR;
  };
  if (cudaGraphConditionalHandleCreate(&L.h, g, 0, cudaGraphCondAssignDefault) != cudaSuccess) rc = MGK_CUDA_ERROR;
  cudaGraphNode_t n0 = nullptr, wn = nullptr;
  add(g, &n0, nullptr, L.head);
  cudaGraph_t body = nullptr;
  if (rc == MGK_OK) {
    alignas(cudaGraphNodeParams) unsigned char raw[sizeof(cudaGraphNodeParams)];
    memset(raw, 0, sizeof(raw));
    cudaGraphNodeParams& cp = *reinterpret_cast<cudaGraphNodeParams*>(raw);
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = L.h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    if (cudaGraphAddNode(&wn, g, &n0, 1, &cp) != cudaSuccess) rc = MGK_CUDA_ERROR;
    else body = cp.conditional.phGraph_out[0];
  }
  cudaGraphNode_t kn[8];
  for (int k = 0; k < L.n; ++k) add(body, &kn[k], k ? &kn[k - 1] : nullptr, L.body[k]);
  cudaGraphExec_t x = nullptr;
  if (rc == MGK_OK && cudaGraphInstantiate(&x, g, 0) != cudaSuccess) rc = MGK_CUDA_ERROR;
  if (rc != MGK_OK) {
    cudaGraphDestroy(g);
    cudaGetLastError();
    return rc;
  }
  p->cg_graph[f] = g;
  p->cg_exec[f] = x;
  return MGK_OK;
}

static int fs_krylov_status(mgk_fs3d_t p) {
  if (p->h_sc->err != 0.0) { set_error("mgk_fs3d_step: a bulk copy wait gave up (device timeout)"); return MGK_TIMEOUT; }
  if (!isfinite(p->h_sc->rr)) { set_error("mgk_fs3d_step: non-finite Krylov residual"); return MGK_NONFINITE; }
  return MGK_OK;
}

// Krylov solve of G:K:dx = r (r holds the right-hand side, x = 0): on the
// device through the graph, without a host read, or host-driven (one scalar
// read per iteration) when conditional graphs are unavailable.
static int fs_krylov(mgk_fs3d_t p, double tol_CG, int max_cg, cudaStream_t s) {
  const int f = p->prec == MGK_MIXED ? 1 : 0;
  int rc;
  if (p->graph_mode < 0) {
    const char* env = getenv("MGK_NO_GRAPH_WHILE");
    p->graph_mode = (env && env[0] == '1') ? 0 : 1;
  }
  if (p->graph_mode == 1 && !p->cg_exec[f] && fs_build_graph(p, f) != MGK_OK) p->graph_mode = 0;
  if (p->graph_mode == 1) {
    MGK_CUDA(cudaGraphLaunch(p->cg_exec[f], s));
    return MGK_OK;
  }
  FsLoop L;
  fs_loop(p, f, L);
  if (f && (rc = fs_run(L.head, s))) return rc;
  if ((rc = fs_read_scalars(p, s))) return rc;
  const FsScalars& S = *p->h_sc;
  while (isfinite(S.rr) && S.rr > tol_CG * tol_CG * S.bb && S.kcount < max_cg && S.err == 0.0) {
    for (int k = 0; k < L.n; ++k)
      if ((rc = fs_run(L.body[k], s))) return rc;
    if ((rc = fs_read_scalars(p, s))) return rc;
  }
  return MGK_OK;
}

// Newton branch (:3046-3119).  F holds F_start on entry, F_curr on exit.
// fresh: the stress and tangent at F are not those of the last accepted trial.
static int fs_newton(mgk_fs3d_t p, const double* F_bar, double tol_NW, double tol_CG, int max_NW, int max_cg, bool fresh,
                     cudaStream_t s) {
  FsBegin b;
  for (int q = 0; q < 9; ++q) b.F_bar[q] = F_bar[q];
  b.tol2 = tol_CG * tol_CG;
  b.kmax = (double)max_cg;
  fs_begin_kernel<<<p->nblk, 256, 0, s>>>(fs_args(p), b);
  MGK_CUDA(cudaGetLastError());
  int rc;
  if (fresh) {
    // P, K at F_start
    if ((rc = fs_trial(p, 0.0, false, false, s))) return rc;
    fs_accept(p);
  }
  for (int it = 0; it < max_NW; ++it) {
    if (it == 0 && p->prec == MGK_MIXED) {
      fs_tangent_kernel<<<p->nblk, 256, 0, s>>>(fs_args(p), fs32_args(p).st64);
      MGK_CUDA(cudaGetLastError());
    }
    if ((rc = fs_rhs(p, it == 0, s))) return rc;
    if ((rc = fs_krylov(p, tol_CG, max_cg, s))) return rc;
    if (p->prec != MGK_MIXED && (rc = fs_field(p, s))) return rc;
    // line search (:3088-3114)
    double alpha = 1.0;
    bool ok = false;
    for (int t = 0; t < 16; ++t) {
      if ((rc = fs_trial(p, alpha, it == 0, true, s)) || (rc = fs_read_scalars(p, s))) return rc;
      const FsScalars& S = *p->h_sc;
      if (t == 0) {
        p->stat_krylov += (int)S.kcount;
        if ((rc = fs_krylov_status(p))) return rc;
      }
      if (!(S.minJe > 1e-4) || S.nan != 0) { alpha *= 0.5; continue; }
      ok = true;
      break;
    }
    if (!ok) { set_error("Newton-CG line search failed to find a valid step."); return MGK_NOT_CONVERGED; }
    fs_accept(p);
    ++p->stat_newton;
    const double res = sqrt(p->h_sc->xx) / (sqrt(std::max(0.0, p->h_sc->FF - p->ff_offset)) + 1e-20);
    if (res < tol_NW && it > 0) return MGK_OK;
  }
  set_error("Newton-CG inner solver did not converge within %d iterations.", max_NW);
  return MGK_NOT_CONVERGED;
}

// Timing hook: mean duration (ms, CUDA events on `stream`) of each kernel
// of one Krylov iteration in the plan's kernel family.  FP64: [0] z stage (C2R,
// K:p, R2C), [1] forward y, [2] forward x with G and p.q, [3] inverse y, [4]
// inverse x with the direction, [5] CG update.  fp32 = 1, the mixed form's FP32
// kernels: [0] z forward with K:p, [1] y, [2] x with G, [3] inverse y, [4] z
// inverse with p.q, [5] CG update.  Runs `reps` iterations on the current state
// and leaves the Krylov vectors in an unspecified state.
extern "C" int mgk_fs3d_profile(mgk_fs3d_t p, int fp32, int reps, float* ms_out, mgk_stream_t stream) {
  MGK_REQUIRE(p && ms_out && reps >= 1 && p->has_material, "mgk_fs3d_profile: bad argument");
  MGK_REQUIRE(!fp32 || p->prec == MGK_MIXED, "mgk_fs3d_profile: fp32 needs a mixed-precision plan");
  cudaStream_t s = (cudaStream_t)stream;
  const int f = fp32 ? 1 : 0;
  FsLoop L;
  fs_loop(p, f, L);
  // output of each launch: FP64 {x inv, y inv, z, y, x, update}; FP32 {z, y, x, y
  // inv, z inv, scalars, update, scalars}
  int slot[8];
  static const int slot64[6] = {4, 3, 0, 1, 2, 5};
  for (int k = 0; k < L.n; ++k) slot[k] = f ? std::min(k, 5) : slot64[k];
  cudaEvent_t ev[9];
  for (int i = 0; i < 9; ++i) MGK_CUDA(cudaEventCreate(&ev[i]));
  double acc[6] = {0, 0, 0, 0, 0, 0};
  int rc = MGK_OK;
  for (int r = 0; r < reps && rc == MGK_OK; ++r) {
    cudaEventRecord(ev[0], s);
    for (int k = 0; k < L.n && rc == MGK_OK; ++k) {
      rc = fs_run(L.body[k], s);
      cudaEventRecord(ev[k + 1], s);
    }
    if (rc == MGK_OK && cudaEventSynchronize(ev[L.n]) != cudaSuccess) rc = MGK_CUDA_ERROR;
    for (int k = 0; k < L.n && rc == MGK_OK; ++k) {
      float ms = 0;
      cudaEventElapsedTime(&ms, ev[k], ev[k + 1]);
      acc[slot[k]] += ms;
    }
  }
  for (int i = 0; i < 9; ++i) cudaEventDestroy(ev[i]);
  if (rc != MGK_OK) { cudaGetLastError(); set_error("mgk_fs3d_profile: kernel failure"); return rc; }
  for (int k = 0; k < 6; ++k) ms_out[k] = (float)(acc[k] / reps);
  return MGK_OK;
}

// Autotuner: times one Krylov iteration of each kernel family that can serve
// the plan (register FFTs on the axes that have one; the general passes always)
// on the current state and keeps the faster one.
extern "C" int mgk_fs3d_autotune(mgk_fs3d_t p, int reps, int* chosen, float* best_ms, mgk_stream_t stream) {
  MGK_REQUIRE(p && reps >= 1 && p->has_material, "mgk_fs3d_autotune: bad argument");
  const int f = p->prec == MGK_MIXED ? 1 : 0;
  const bool can_fast = f ? p->line32[0] || p->line32[1] || p->line32[2] : p->line[0] || p->line[1] || p->line[2];
  int best = 0;
  float best_t = 0.0f;
  for (int k = 0; k < (can_fast ? 2 : 1); ++k) {
    p->fast = k;
    if (int rc = fs_raise(p)) return rc;
    float ms[6];
    int st = mgk_fs3d_profile(p, f, reps, ms, stream);
    if (st) return st;
    float t = 0;
    for (float v : ms) t += v;
    if (k == 0 || t < best_t) { best_t = t; best = k; }
  }
  p->fast = best;
  fs_drop_graphs(p);
  if (chosen) *chosen = best;
  if (best_ms) *best_ms = best_t;
  return MGK_OK;
}

extern "C" int mgk_fs3d_set_plane_strain(mgk_fs3d_t p, int on) {
  MGK_REQUIRE(p && (!on || p->ny == 1), "mgk_fs3d_set_plane_strain: the plan must be (nx, 1, ny)");
  p->ff_offset = on ? (double)p->N : 0.0;
  return MGK_OK;
}

extern "C" int mgk_fs3d_set_plane_stress(mgk_fs3d_t p, int on) {
  MGK_REQUIRE(p && (!on || p->ny == 1), "mgk_fs3d_set_plane_stress: the plan must be (nx, 1, ny)");
  p->plane_stress = on ? 1 : 0;
  p->ff_offset = on ? (double)p->N : 0.0;
  return MGK_OK;
}

extern "C" int mgk_fs3d_step(mgk_fs3d_t p, const double* F_bar_in, int drv_i, int drv_j, const double* P_target,
                             const int* P_mask, double E_avg, double nu_avg, double tol_NW, double tol_CG, int max_NW,
                             double tol_macro, int max_iter_macro, double* F_bar_out, mgk_fs_info* info,
                             mgk_stream_t stream) {
  MGK_REQUIRE(p && p->has_material && F_bar_in && F_bar_out, "mgk_fs3d_step: bad argument (material set?)");
  MGK_REQUIRE(max_NW >= 1 && max_iter_macro >= 1, "mgk_fs3d_step: iteration caps must be positive");
  cudaStream_t s = (cudaStream_t)stream;
  double Fb[9], tgt[9] = {0};
  int mask[9] = {0};
  for (int q = 0; q < 9; ++q) {
    Fb[q] = F_bar_in[q];
    if (P_target) tgt[q] = P_target[q];
    if (P_mask) mask[q] = P_mask[q] != 0;
  }
  bool any_mask = false;
  for (int q = 0; q < 9; ++q) any_mask |= mask[q] != 0;
  int upd[3] = {0, 0, 0};
  for (int k = 0; k < 3; ++k) upd[k] = mask[4 * k] && !(k == drv_i && k == drv_j);
  bool have_prev = false;
  double prevF[3] = {0, 0, 0}, prevS[3] = {0, 0, 0};
  p->stat_newton = p->stat_krylov = p->stat_macro = 0;
  double max_err = 0.0;
  int rc = MGK_OK;
  for (int it = 0; it < max_iter_macro; ++it) {
    rc = fs_newton(p, Fb, tol_NW, tol_CG, max_NW, 150, it == 0, s);
    ++p->stat_macro;
    if (rc) break;
    const double* Sm = p->h_sc->sig;
    if (!any_mask) break;
    double err[9] = {0};
    max_err = 0.0;
    for (int q = 0; q < 9; ++q)
      if (mask[q]) { err[q] = tgt[q] - Sm[q]; max_err = std::max(max_err, fabs(err[q])); }
    if (max_err < tol_macro) break;
    const double trerr = err[0] + err[4] + err[8];
    double dF[9];
    for (int q = 0; q < 9; ++q)
      dF[q] = std::min(0.01, std::max(-0.01, (err[q] - ((q % 4 == 0) ? nu_avg * trerr : 0.0)) / E_avg));
    double d_sc[3], Fsc[3], ssc[3];
    for (int k = 0; k < 3; ++k) { d_sc[k] = dF[4 * k]; Fsc[k] = Fb[4 * k]; ssc[k] = Sm[4 * k]; }
    if (have_prev) {
      for (int k = 0; k < 3; ++k) {
        if (!upd[k]) continue;
        const double dh = Fsc[k] - prevF[k];
        const double slope = (ssc[k] - prevS[k]) / dh;
        if (isfinite(slope) && fabs(dh) > 1e-14 && slope > 0.01 * E_avg)
          d_sc[k] = std::min(0.01, std::max(-0.01, err[4 * k] / slope));
      }
    }
    for (int k = 0; k < 3; ++k) { prevF[k] = Fsc[k]; prevS[k] = ssc[k]; }
    have_prev = true;
    for (int k = 0; k < 3; ++k)
      if (upd[k]) Fb[4 * k] += d_sc[k];
    if (it == max_iter_macro - 1) {
      set_error("Outer BC loop did not converge after %d iterations. Final max stress error: %.2e Pa", max_iter_macro,
                max_err);
      rc = MGK_NOT_CONVERGED;
    }
  }
  for (int q = 0; q < 9; ++q) F_bar_out[q] = Fb[q];
  if (info) {
    info->newton_iterations = p->stat_newton;
    info->krylov_iterations = p->stat_krylov;
    info->macro_iterations = p->stat_macro;
    info->status = rc;
    info->max_stress_error = max_err;
    for (int q = 0; q < 9; ++q) info->sig_mean[q] = p->h_sc->sig[q];
  }
  return rc;
}
