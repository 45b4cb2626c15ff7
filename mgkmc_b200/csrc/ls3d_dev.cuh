// Device-side pieces of the 3D small-strain solver shared by its translation
// units: the replica, state and control records, the Green operator, the
// constitutive laws and the convergence decision.
#pragma once
#include <math.h>

#include "common.cuh"
#include "fft.cuh"

namespace mgk {

struct Ls3dRep {
  int nx, ny, nz, nzh, ld, tc;
  int zl_items;      // z-line pairs = nx*ny/2
  int y_items;       // nx * ceil(nzh/tc)
  int x_items;       // ny * ceil(nzh/tc)
  long long N;
  FftLen fx, fy, fz;
  double* mu;
  double* lam;
  double* eps;   // 6 planes
  double* ep;    // 6 planes
  double* epa;   // eps_p yz, xz, xy, zy, zx, yx as given (6 planes) or null
  double2* spec;
  // mixed-precision plans (warp-line kernels only): FP32 copies and tables;
  // the FP32 spectrum reuses `spec`
  float* mu32;
  float* lam32;
  float* eps32;  // 6 planes
  float* ep32;   // 6 planes
  FftLen fx32, fy32, fz32;
  // step twiddles of the register-FFT kernels (x, y, z; null: CTA-wide passes)
  const double2* rtw[3];
  const float2* rtw32[3];
  // per call
  const double* init;
  double* out_eps;
  double* out_sig;
  double eb[9];
  double tol;
  int max_iter;
  int zl_first;
  // constitutive law: 0 linear (elasticity.py:62-67); 1 the secant
  // degradation law with magnitude law_a and rate law_b (FP64 plans)
  int law;
  double law_a, law_b;
  // law 3, Landau: v1, v2, v3, g1, g2, g3, g4, capping (0 none, 1 piecewise,
  // 2 smooth), E_cap, tangent ratio, smooth power
  double lp[11];
};

struct Ls3dState {
  double mu0, lam0, Bc, inv2mu0;
  double ebar[6];
  double abar[3];  // (xy - yx)/2, (xz - zx)/2, (yz - zy)/2 of eps_bar
  double extra_d0, extra_n0;
  int iter, done, status, phase_iter;  // done: 0 active, 1 phase 1 finished, 2 finished
  double diff;
  double means[9];
  double out_eps_mean[9];
  double out_sig_mean[9];
};

struct Ls3dCtl {
  unsigned int n_active, decided, still, bodies;
  int any;
  int error;  // a bounded wait gave up (MGK_TIMEOUT)
};

constexpr double kL3Phase1Tol = 2e-6;  // mixed plans: FP32 iterations down to max(tol, this)
constexpr int kL3Phase1Cap = 64;

// symmetric component c -> (i, j): xx yy zz yz xz xy
static __device__ __constant__ int kSymI[6] = {0, 1, 2, 1, 0, 0};
static __device__ __constant__ int kSymJ[6] = {0, 1, 2, 2, 2, 1};

__device__ __forceinline__ int fftfreq3(int k, int n) { return (k < (n + 1) / 2) ? k : k - n; }

// eps~^ = -Gamma0(n) : tau^ for symmetric tau (3D), n a unit vector.
// t[6] / e[6] in the symmetric order above.
// R = double for the FP64 iterations, float for the FP32 phase of a mixed plan.
template <typename R>
__device__ __forceinline__ void gamma3d_apply_t(const C_t<R>* t, R n0, R n1, R n2, R inv2mu0, R Bc, C_t<R>* e) {
  constexpr int kI[6] = {0, 1, 2, 1, 0, 0}, kJ[6] = {0, 1, 2, 2, 2, 1};
  const R n[3] = {n0, n1, n2};
  // full symmetric tau as 3x3 of complex
  C_t<R> T[3][3];
  T[0][0] = t[0]; T[1][1] = t[1]; T[2][2] = t[2];
  T[1][2] = T[2][1] = t[3];
  T[0][2] = T[2][0] = t[4];
  T[0][1] = T[1][0] = t[5];
  C_t<R> tn[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    tn[i].x = T[i][0].x * n[0] + T[i][1].x * n[1] + T[i][2].x * n[2];
    tn[i].y = T[i][0].y * n[0] + T[i][1].y * n[1] + T[i][2].y * n[2];
  }
  C_t<R> ntn;
  ntn.x = tn[0].x * n[0] + tn[1].x * n[1] + tn[2].x * n[2];
  ntn.y = tn[0].y * n[0] + tn[1].y * n[1] + tn[2].y * n[2];
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const int k = kI[c], h = kJ[c];
    e[c].x = -(inv2mu0 * (n[h] * tn[k].x + n[k] * tn[h].x) - Bc * n[k] * n[h] * ntn.x);
    e[c].y = -(inv2mu0 * (n[h] * tn[k].y + n[k] * tn[h].y) - Bc * n[k] * n[h] * ntn.y);
  }
}
__device__ __forceinline__ void gamma3d_apply(const double2* t, double n0, double n1, double n2, double inv2mu0,
                                              double Bc, double2* e) {
  gamma3d_apply_t<double>(t, n0, n1, n2, inv2mu0, Bc, e);
}

// Secant shear modulus mu (1 - d (1 - exp(-k eq))) (elasticity.py:703-728) at
// the von Mises equivalent strain sqrt(2/3 e':e') of the elastic strain
// (elasticity.py:665-700) given by its symmetric components; each pair of
// shear entries sums to twice the symmetric one.
// 3D Landau small-strain stress (elasticity.py:811-857) of the symmetric
// elastic strain a = (xx, yy, zz, yz, xz, xy), with the strain capping of
// elasticity.py:297-334: deviator scaled by f above the cap E_cap (piecewise)
// or by the tanh profile (smooth), plus 2 (ratio mu) (a - capped) w.
// sigma = (lam I1 + v1/2 I1^2 + v2 I2 + g1/6 I1^3 + g2 I1 I2 + 4/3 g3 I3) I
//       + 2 (mu + v2 I1 + g2/2 I1^2 + g4 I2) e + 4 (v3 + g3 I1) e^2.
__device__ __forceinline__ void landau_sigma3(double mu, double lam, const double* a, const double* __restrict__ lp,
                                              double* sg) {
  const double v1 = lp[0], v2 = lp[1], v3 = lp[2], g1 = lp[3], g2 = lp[4], g3 = lp[5], g4 = lp[6];
  const int cap = (int)lp[7];
  double c[6];
  for (int q = 0; q < 6; ++q) c[q] = a[q];
  double w = 0.0;
  if (cap) {
    const double I1a = a[0] + a[1] + a[2];
    const double m3 = (1.0 / 3.0) * I1a;
    const double d0 = a[0] - m3, d1 = a[1] - m3, d2 = a[2] - m3;
    const double dd = d0 * d0 + d1 * d1 + d2 * d2 + 2.0 * (a[3] * a[3] + a[4] * a[4] + a[5] * a[5]);
    const double Eeq = sqrt(fmax(0.0, (2.0 / 3.0) * dd));
    const double Ecap = lp[8];
    double f = 1.0;
    if (cap == 2) {
      const double pw = lp[10];
      if (Eeq > 1e-12) f = (Ecap / Eeq) * pow(tanh(fmin(100.0, pow(Eeq / Ecap, pw))), 1.0 / pw);
      const double t = tanh(fmin(100.0, pow(Eeq / Ecap, pw)));
      w = t * t;
    } else if (Eeq > Ecap) {
      f = Ecap / Eeq;
      w = 1.0;
    }
    c[0] = d0 * f + m3;
    c[1] = d1 * f + m3;
    c[2] = d2 * f + m3;
    c[3] = a[3] * f;
    c[4] = a[4] * f;
    c[5] = a[5] * f;
  }
  // e^2 of the symmetric tensor [[xx, xy, xz], [xy, yy, yz], [xz, yz, zz]]
  const double xx = c[0], yy = c[1], zz = c[2], yz = c[3], xz = c[4], xy = c[5];
  double e2[6];
  e2[0] = xx * xx + xy * xy + xz * xz;
  e2[1] = xy * xy + yy * yy + yz * yz;
  e2[2] = xz * xz + yz * yz + zz * zz;
  e2[3] = xy * xz + yy * yz + yz * zz;
  e2[4] = xx * xz + xy * yz + xz * zz;
  e2[5] = xx * xy + xy * yy + xz * yz;
  const double I1 = xx + yy + zz;
  const double I2 = e2[0] + e2[1] + e2[2];
  const double I3 = (e2[0] * xx + e2[5] * xy + e2[4] * xz) + (e2[5] * xy + e2[1] * yy + e2[3] * yz) +
                    (e2[4] * xz + e2[3] * yz + e2[2] * zz);
  const double cI = lam * I1 + 0.5 * v1 * (I1 * I1) + v2 * I2 + (1.0 / 6.0) * g1 * (I1 * I1 * I1) + g2 * I1 * I2 +
                    (4.0 / 3.0) * g3 * I3;
  const double ce = 2.0 * (mu + v2 * I1 + 0.5 * g2 * (I1 * I1) + g4 * I2);
  const double ce2 = 4.0 * (v3 + g3 * I1);
  for (int q = 0; q < 6; ++q) sg[q] = (q < 3 ? cI : 0.0) + ce * c[q] + ce2 * e2[q];
  if (cap) {
    const double r = 2.0 * (lp[9] * mu) * w;
    for (int q = 0; q < 6; ++q) sg[q] += r * (a[q] - c[q]);
  }
}

__device__ __forceinline__ double secant_mu3(double m, double xx, double yy, double zz, double yz, double xz,
                                             double xy, double d, double k) {
  const double tr3 = (xx + yy + zz) / 3.0;
  const double a = xx - tr3, b = yy - tr3, c = zz - tr3;
  const double s1 = 2.0 * xy, s2 = 2.0 * xz, s3 = 2.0 * yz;
  const double eq = sqrt((2.0 / 3.0) * (a * a + b * b + c * c + 0.5 * (s1 * s1 + s2 * s2 + s3 * s3)));
  return m * (1.0 - d * (1.0 - exp(-k * eq)));
}

// Partial sums of this z-line item, and (last item of the replica) the
// fixed-order reduction, the convergence decision and the loop condition.
template <bool FINAL>
__device__ void ls3d_decide(const Ls3dRep& R, Ls3dState& S, int r, int item, double d2, double n2,
                            double* partials, unsigned int* rep_counter, Ls3dCtl* ctl,
                            cudaGraphConditionalHandle cond, int use_cond, int guard_cap, double* red,
                            int* s_last_p) {
  int& s_last = *s_last_p;
  const long long N = R.N;
  d2 = block_sum(d2, red);
  n2 = block_sum(n2, red);
  if (threadIdx.x == 0) {
    partials[2 * item] = d2;
    partials[2 * item + 1] = n2;
    __threadfence();
    const unsigned int t = atomicInc(&rep_counter[r], (unsigned int)R.zl_items - 1);
    s_last = (t == (unsigned int)R.zl_items - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double a = 0, b = 0;
  for (int i = threadIdx.x; i < R.zl_items; i += blockDim.x) {
    a += __ldcg(&partials[2 * (R.zl_first + i)]);
    b += __ldcg(&partials[2 * (R.zl_first + i) + 1]);
  }
  a = block_sum(a, red);
  b = block_sum(b, red);
  if (threadIdx.x != 0) return;
  // the control block's words at once, ahead of the chain of atomics below
  const unsigned int n_act = *(volatile unsigned int*)&ctl->n_active, bodies = *(volatile unsigned int*)&ctl->bodies;
  const int error = *(volatile int*)&ctl->error;
  if (S.iter == 0) { a += S.extra_d0; b += S.extra_n0; }
  else b += 2.0 * (double)N * (S.abar[0] * S.abar[0] + S.abar[1] * S.abar[1] + S.abar[2] * S.abar[2]);
  const double diff = sqrt(a) / (sqrt(b) + 1e-20);
  S.diff = diff;
  S.iter += 1;
  S.phase_iter += 1;
  int keep = 0;
  if (!isfinite(diff)) { S.done = 2; S.status = MGK_NONFINITE; }
  else if (FINAL) {
    if (diff < R.tol) { S.done = 2; S.status = MGK_OK; }
    else if (S.iter >= R.max_iter) { S.done = 2; S.status = MGK_NOT_CONVERGED; }
    else keep = 1;
  } else {
    const double tol1 = R.tol > kL3Phase1Tol ? R.tol : kL3Phase1Tol;
    if (S.iter >= R.max_iter) { S.done = 2; S.status = diff < R.tol ? MGK_OK : MGK_NOT_CONVERGED; }
    else if (diff < tol1 || S.phase_iter >= kL3Phase1Cap) S.done = 1;
    else keep = 1;
  }
  if (keep) atomicAdd(&ctl->still, 1u);
  __threadfence();
  const unsigned int dcount = atomicAdd(&ctl->decided, 1u);
  if (dcount == n_act - 1) {
    __threadfence();
    const unsigned int still = atomicExch(&ctl->still, 0u);
    ctl->decided = 0;
    ctl->n_active = still;
    const bool go = still > 0 && bodies <= (unsigned int)guard_cap && error == 0;
    ctl->any = go ? 1 : 0;
    if (use_cond) cudaGraphSetConditional(cond, go ? 1u : 0u);
  }
}

}  // namespace mgk
