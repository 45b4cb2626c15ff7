// Shared device code of the finite-strain solver's mixed form: FP32 matvecs on
// FP32 CG vectors held as 9 real fields.
//
// The FP64 form's vectors are potentials in Fourier space (fs3d.cu), which
// takes half of the time; this form keeps the real fields and every rounding of
// its passes, the FP64 right-hand sides included.  With F_p the tangent as
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
  const void* rtw32[3];  // register-FFT twiddles (x, y, z)
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

}  // namespace fs32
}  // namespace mgk
