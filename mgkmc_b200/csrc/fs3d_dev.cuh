// Shared device code of the finite-strain solver (fs3d.cu: plan, host loops,
// general kernels; fs3d_line.cuh: the matvec kernels on register FFTs).
#pragma once
#include "common.cuh"
#include "fft.cuh"

namespace mgk {

struct FsScalars {
  double rr, pq, alpha, beta, bb;
  double xx, FF, minJe, nan, err;  // err: a bounded wait ran out
  double sig[9];
  double dbar[9];             // F_bar - mean(F)
  double tol2, kmax, kcount;  // device-side CG loop: (tol_CG)^2, iteration cap, iterations run
  double pad;
};

// Whether the device-side Krylov loop of either precision form runs another
// iteration: the residual is finite and above the tolerance, the iteration cap is
// not reached, and no bounded wait gave up (the vectors are stale then).
__device__ __forceinline__ bool fs_go(const FsScalars& S) {
  return isfinite(S.rr) && S.rr > S.tol2 * S.bb && S.kcount < S.kmax && S.err == 0.0;
}

struct FsArgs {
  int nx, ny, nz, nzh, ld;
  int tcx, tcy;  // kz columns per CTA of the general axis passes
  long long N, plane;  // voxels; complex entries of one spectrum plane (nx ny ld)
  double ix, iy, iz;   // 1 / nx, 1 / ny, 1 / nz
  int has_fp, model;   // model 0 SVK, 1 Neo-Hookean
  int plane_stress;    // (nx, 1, ny) plan of a 2D plane-stress solve (lam the plane-stress lambda)
  FftLen fx, fy, fz;
  const double2* rtw[3];  // register-FFT twiddles (x, y, z)
  const double* F;
  const double* Fpi;
  const double* mu;
  const double* lam;
  const double* P;
  const unsigned char* fpf;  // 1 where F_p^-1 is not the identity
  double* X;                 // real increment field (9 planes)
  double* Fout;
  double* Pout;
  double2* spec;                 // 9 planes of half spectra
  double2 *vr, *vp, *vx, *vq;    // Krylov vectors, 3 planes of half spectra each
  double* st;                    // tangent state (kFsState planes)
  double* part;
  unsigned int* counter;
  FsScalars* sc;
};

// Tangent state planes at the current F, with H = Fe^-1 and E = Fe - I:
//   Neo-Hookean: H (9), lambda, mu, c = mu - lambda ln Je   (plane stress: the
//                condensed lambda* and c = mu F33^2)
//   SVK:         E (9), lambda, mu
// What the tangent does with D = d F_p^-1 follows from these alone:
//   Neo-Hookean  R = mu D^T + lambda tr(H D) H + c H D H
//   SVK          R = S D^T + (mu (X + X^T) + lambda tr(X) I) Fe^T,  X = Fe^T D
// and F_p^-1 R is S_ref dF^T + F_p^-1 Y Fe^T of the reference's tangent (Neo-
// Hookean: the terms c C^-1 D^T of S D^T and of Y Fe^T cancel).  24 planes with
// S_ref, C^-1 and a flag stored were half of the matvec's traffic.  SVK keeps
// E, from which the strain (E + E^T + E^T E) / 2 loses no digits.
constexpr int kFsState = 12;

// ------------------------------------------------------- 3x3 helpers ---
template <typename T> __device__ __forceinline__ void mm(const T* A, const T* B, T* C) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) C[3 * i + j] = A[3 * i] * B[j] + A[3 * i + 1] * B[3 + j] + A[3 * i + 2] * B[6 + j];
}
template <typename T> __device__ __forceinline__ void mtm(const T* A, const T* B, T* C) {  // A^T B
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) C[3 * i + j] = A[i] * B[j] + A[3 + i] * B[3 + j] + A[6 + i] * B[6 + j];
}
template <typename T> __device__ __forceinline__ void mmt(const T* A, const T* B, T* C) {  // A B^T
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      C[3 * i + j] = A[3 * i] * B[3 * j] + A[3 * i + 1] * B[3 * j + 1] + A[3 * i + 2] * B[3 * j + 2];
}

// trans2(K4 : trans2(d)) of voxel i from the tangent state: with F_p the
// transpose of the stress increment, without it the increment itself (the two
// branches of the reference's tangent)
template <int MODEL>
__device__ __forceinline__ void fs_kdf(const FsArgs& a, long long i, const double* d, double* out) {
  using T = double;
  const long long N = a.N;
  const T* st = a.st + i;
  T M[9], D[9], R[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) M[q] = st[q * N];
  const T lam = st[9 * N], mu = st[10 * N];
  const bool fp = a.has_fp && a.fpf[i] != 0;
  T Fpi[9];
  if (fp) {
    const T* f = a.Fpi + i;
#pragma unroll
    for (int q = 0; q < 9; ++q) Fpi[q] = f[q * N];
    mm(d, Fpi, D);
  } else {
#pragma unroll
    for (int q = 0; q < 9; ++q) D[q] = d[q];
  }
  if constexpr (MODEL == 1) {
    const T c = st[11 * N];
    T HD[9];
    mm(M, D, HD);
    const T lt = lam * (HD[0] + HD[4] + HD[8]);
    mm(HD, M, R);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int s = 0; s < 3; ++s) R[3 * r + s] = c * R[3 * r + s] + (lt * M[3 * r + s] + mu * D[3 * s + r]);
  } else {
    T S[9], X[9], A[9];
    mtm(M, M, S);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int s = 0; s < 3; ++s) S[3 * r + s] += M[3 * r + s] + M[3 * s + r];  // 2 E_G
    const T le = T(0.5) * lam * (S[0] + S[4] + S[8]);
#pragma unroll
    for (int q = 0; q < 9; ++q) S[q] = mu * S[q] + (q % 4 == 0 ? le : T(0));
    mtm(M, D, X);
#pragma unroll
    for (int q = 0; q < 9; ++q) X[q] += D[q];
    const T lt = lam * (X[0] + X[4] + X[8]);
    mmt(S, D, A);
    T Y[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int s = 0; s < 3; ++s) Y[3 * r + s] = mu * (X[3 * r + s] + X[3 * s + r]) + (r == s ? lt : T(0));
    mmt(Y, M, R);
#pragma unroll
    for (int q = 0; q < 9; ++q) R[q] += Y[q] + A[q];
  }
  if (fp) {
    mm(Fpi, R, out);
  } else if (a.has_fp) {
#pragma unroll
    for (int q = 0; q < 9; ++q) out[q] = R[q];
  } else {
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int s = 0; s < 3; ++s) out[3 * r + s] = R[3 * s + r];
  }
}

// ---------------------------------------------------------- wave vector ---
// u = (kx / nx, ky / ny, kz / nz), signed; G and the inner products leave out
// the mean and the Nyquist planes.
__device__ __forceinline__ int ffq(int k, int n) { return (k < (n + 1) / 2) ? k : k - n; }
__device__ __forceinline__ bool fs_out(int kx, int ky, int kz, int nx, int ny, int nz) {
  return (kx | ky | kz) == 0 || 2 * kx == nx || 2 * ky == ny || 2 * kz == nz;
}

__device__ __forceinline__ double fs_u(int f, double inv_n) { return f * inv_n; }
__device__ __forceinline__ double fs_u2(const FsArgs& a, int kx, int ky, int kz) {
  const double ux = ffq(kx, a.nx) * a.ix, uy = ffq(ky, a.ny) * a.iy, uz = kz * a.iz;
  return ux * ux + uy * uy + uz * uz;
}

// Sum of every CTA's acc in a fixed order by the CTA that arrives last, whose
// thread 0 calls fin(sum).
template <typename Fin>
__device__ __forceinline__ void fs_finish(const FsArgs& a, double acc, double* red, Fin fin) {
  __shared__ int s_last;
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) {
    a.part[blockIdx.x] = acc;
    __threadfence();
    s_last = atomicInc(a.counter, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double s = 0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) s += __ldcg(&a.part[i]);
  s = block_sum(s, red);
  if (threadIdx.x == 0) fin(s);
}

// The end of the forward x pass at (kx, ky, kz), from the transformed X and B
// lines of the three tensor rows: the potential of G:A,
//   v_i = (u . A_i) / (N |u|^2) = (ux X_i + B_i) / (N |u|^2).
// RHS: r = -v, x = 0, |r|^2; otherwise q = v and p.q.  Inner products are those
// of the real fields over N: |u|^2 Re(conj(a) b) per frequency, doubled for the
// frequencies that stand for their conjugates.
//
// In the plane kz = 0 one frequency of each conjugate pair gives both values:
// the transforms leave a rounding error that is no real field's spectrum, the
// matvec cannot see it, and beside the residual of a nearly converged Newton
// step (small against the stress that it is the projection of) it kept CG from
// converging.  Every vector stays exactly symmetric from then on.
template <bool RHS>
__device__ __forceinline__ double fs_contract(const FsArgs& a, int kx, int ky, int kz, const double2* xv,
                                              const double2* bv) {
  const int qx = ffq(kx, a.nx), qy = ffq(ky, a.ny);
  const bool none = fs_out(kx, ky, kz, a.nx, a.ny, a.nz);
  if (kz == 0 && !none && (qy < 0 || (qy == 0 && qx < 0))) return 0.0;
  double2* out = RHS ? a.vr : a.vq;
  const long long at = ((long long)kx * a.ny + ky) * a.ld + kz;
  const long long mirror = ((long long)(kx ? a.nx - kx : 0) * a.ny + (ky ? a.ny - ky : 0)) * a.ld;
  const double u2 = fs_u2(a, kx, ky, kz);
  const double f = none ? 0.0 : (RHS ? -1.0 : 1.0) / ((double)a.N * u2), ux = fs_u(qx, a.ix);
  double s = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double2 v = none ? make_double2(0, 0) : make_double2(f * (ux * xv[i].x + bv[i].x), f * (ux * xv[i].y + bv[i].y));
    out[i * a.plane + at] = v;
    if (kz == 0 && !none) out[i * a.plane + mirror] = make_double2(-v.x, v.y);  // u is odd
    if constexpr (RHS) {
      a.vx[i * a.plane + at] = make_double2(0, 0);
      if (kz == 0 && !none) a.vx[i * a.plane + mirror] = make_double2(0, 0);
      s += v.x * v.x + v.y * v.y;
    } else {
      const double2 p = a.vp[i * a.plane + at];
      s += p.x * v.x + p.y * v.y;
    }
  }
  return 2.0 * s * u2;
}

// scalars after the sums of the forward x pass
template <bool RHS> __device__ __forceinline__ void fs_after_x(const FsArgs& a, double s) {
  FsScalars& S = *a.sc;
  if (RHS) {
    S.rr = s;
    S.bb = s;
    S.beta = 0.0;
    S.kcount = 0.0;
  } else {
    S.pq = s;
    S.alpha = s != 0.0 ? S.rr / s : 0.0;
  }
}

// The start of the inverse x pass: the potential of p = r + beta p (kept) or,
// FINAL, of x.
template <bool FINAL> __device__ __forceinline__ double2 fs_direction(const FsArgs& a, double beta, long long at) {
  if constexpr (FINAL) return a.vx[at];
  double2 r = a.vr[at];
  if (beta != 0.0) {
    const double2 o = a.vp[at];
    r = make_double2(r.x + beta * o.x, r.y + beta * o.y);
  }
  a.vp[at] = r;
  return r;
}

}  // namespace mgk
