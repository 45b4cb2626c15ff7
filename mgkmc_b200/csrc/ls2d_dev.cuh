// Device-side pieces of the 2D small-strain solver shared by its translation
// units: the replica, state and control records, the Anderson mix, the Green
// operator, the constitutive laws and the convergence decision.
#pragma once
#include <math.h>

#include "common.cuh"
#include "fft.cuh"

namespace mgk {

constexpr int kAaMax = 8;  // deepest Anderson history
constexpr int kMaxPairs = 2048;  // row pairs of a replica (sides up to 4096)
struct Ls2dAA;

struct Ls2dRep {
  int nx, ny, nyh, ld, tc;
  int row_items, col_items;
  long long N;
  // constitutive law: 0 linear (elasticity.py:12-18); 1 secant degradation
  // (law_a = d, law_b = k); 2 Rose (law_a = eta, law_b = floor fraction,
  // law_ps = 1 for plane stress); 3 Landau, law_ps = 1 for plane stress (lp: v1, v2, v3,
  // g1, g2, g3, g4, capping 0 none / 1 piecewise / 2 smooth, E_cap, tangent
  // ratio, smooth power)
  int law, law_ps;
  double law_a, law_b;
  double lp[11];
  FftLen fx64, fy64, fx32, fy32;
  // step twiddles of the register-FFT kernels (x, y; null: CTA-wide passes)
  const double2* rtw[2];
  const float2* rtw32[2];
  double* mu;
  double* lam;
  double* eps;   // 3 planes
  double* ep;    // 3 planes
  double* epa;   // 2 planes or null
  float* mu32;   // mixed plans only
  float* lam32;
  float* eps32;
  float* ep32;
  void* spec;    // 3 planes of nx*ld complex (double2, or float2 in FP32 phases)
  // per call
  const double* init;
  double* out_eps;
  double* out_sig;
  double* out_e33;  // Landau plane stress: the out-of-plane strain per voxel (set_e33_out; may be null)
  double eb[4];
  double tol;
  int max_iter;
  int row_first, col_first;  // first work item of this replica in the call's maps
  // Anderson mixing of this call (null: none): state, the ring's dG slots
  // and its x (the mix is applied by the first row pass of each iterate and,
  // when the iteration cap ends the loop, by the output kernel)
  const Ls2dAA* aa;
  const double* aa_dG;
  double* aa_x;
};

struct Ls2dState {
  double mu0, lam0, Bc, inv2mu0;
  double ebar[3];
  double abar;
  double extra_d0, extra_n0;
  int iter;
  int phase_iter;
  int done;    // 0 active, 1 finished the current phase, 2 finished
  int status;
  double diff;
  double means[4];  // warm-start means (xx, xy, yx, yy)
  double out_eps_mean[4];
  double out_sig_mean[4];
};

struct Ls2dCtl {
  unsigned int n_active;  // replicas iterating at the start of the current body
  unsigned int decided;
  unsigned int still;
  unsigned int bodies;    // loop bodies run in the current phase (guard)
  int any;
  int error;              // a bounded wait gave up (MGK_TIMEOUT)
};

struct Ls2dAA {
  int k;          // valid difference columns, in slots 0 .. k-1
  int slot_next;  // ring slot of the next column
  int have_prev;  // a previous (f, g) pair exists
  int nmix;       // columns of the current mix (0: the plain step)
  unsigned int ctr;  // blocks of the update kernel done (self-resetting)
  int pad;
  double A[kAaMax][kAaMax];  // Gram matrix <dF_i, dF_j>
  double gamma[kAaMax];
};

// The Anderson mix x = g - dG gamma of voxel i's three strain planes (g in
// e), written to the plan's strain planes and the ring's x.
__device__ __forceinline__ void aa_mix_voxel(const Ls2dRep& R, long long i, int nmix, const double* gam, double* e) {
  const long long N = R.N, n3 = 3 * N;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double sm = 0.0;
#pragma unroll
    for (int j = 0; j < kAaMax; ++j)
      if (j < nmix) sm += gam[j] * R.aa_dG[(size_t)j * n3 + c * N + i];
    e[c] -= sm;
    R.eps[c * N + i] = e[c];
    R.aa_x[c * N + i] = e[c];
  }
}

__device__ __forceinline__ int aa_load(const Ls2dRep& R, double* gam) {
  const int nmix = R.aa->nmix;
#pragma unroll
  for (int j = 0; j < kAaMax; ++j) gam[j] = j < nmix ? R.aa->gamma[j] : 0.0;
  return nmix;
}

constexpr double kMixedPhase1Tol = 2e-6;
constexpr int kMixedPhase1Cap = 64;

// --------------------------------------------------------------- helpers ---

// eps~^ = -Gamma0(n) : tau^ for symmetric tau (2D), n a unit vector.
template <typename C, typename T>
__device__ __forceinline__ void gamma2d_apply(const C& txx, const C& tyy, const C& txy, T nx, T ny,
                                              T inv2mu0, T Bc, C& exx, C& eyy, C& exy) {
  C tnx = mk<C>(txx.x * nx + txy.x * ny, txx.y * nx + txy.y * ny);
  C tny = mk<C>(txy.x * nx + tyy.x * ny, txy.y * nx + tyy.y * ny);
  C ntn = mk<C>(tnx.x * nx + tny.x * ny, tnx.y * nx + tny.y * ny);
  const T a = T(2) * inv2mu0;
  exx = mk<C>(-(a * nx * tnx.x - Bc * nx * nx * ntn.x), -(a * nx * tnx.y - Bc * nx * nx * ntn.y));
  eyy = mk<C>(-(a * ny * tny.x - Bc * ny * ny * ntn.x), -(a * ny * tny.y - Bc * ny * ny * ntn.y));
  exy = mk<C>(-(inv2mu0 * (ny * tnx.x + nx * tny.x) - Bc * nx * ny * ntn.x),
              -(inv2mu0 * (ny * tnx.y + nx * tny.y) - Bc * nx * ny * ntn.y));
}

__device__ __forceinline__ int fftfreq(int k, int n) { return (k < (n + 1) / 2) ? k : k - n; }

template <typename TS> struct Fields;
template <> struct Fields<double> {
  static __device__ __forceinline__ const double* mu(const Ls2dRep& R) { return R.mu; }
  static __device__ __forceinline__ const double* lam(const Ls2dRep& R) { return R.lam; }
  static __device__ __forceinline__ double* eps(const Ls2dRep& R) { return R.eps; }
  static __device__ __forceinline__ const double* ep(const Ls2dRep& R) { return R.ep; }
  static __device__ __forceinline__ const FftLen& fx(const Ls2dRep& R) { return R.fx64; }
  static __device__ __forceinline__ const FftLen& fy(const Ls2dRep& R) { return R.fy64; }
};
template <> struct Fields<float> {
  static __device__ __forceinline__ const float* mu(const Ls2dRep& R) { return R.mu32; }
  static __device__ __forceinline__ const float* lam(const Ls2dRep& R) { return R.lam32; }
  static __device__ __forceinline__ float* eps(const Ls2dRep& R) { return R.eps32; }
  static __device__ __forceinline__ const float* ep(const Ls2dRep& R) { return R.ep32; }
  static __device__ __forceinline__ const FftLen& fx(const Ls2dRep& R) { return R.fx32; }
  static __device__ __forceinline__ const FftLen& fy(const Ls2dRep& R) { return R.fy32; }
};

// -------------------------------------------------------------- kernels ---

// Secant shear modulus mu (1 - d (1 - exp(-k eps_eq))) (elasticity.py:189-214)
// at the von Mises equivalent strain of the elastic strain (dxx, dyy, sym
// dxy): sqrt(2/3 eps':eps') with the plane-strain eps'_33 = -(dxx + dyy)/3
// (elasticity.py:112-150; the two shear entries sum to 2 dxy).
__device__ __forceinline__ double secant_mu(double m, double dxx, double dyy, double dxy, double d, double k) {
  const double tr3 = (dxx + dyy) / 3.0;
  const double a = dxx - tr3, b = dyy - tr3, c = -(dxx + dyy) / 3.0, sh = 2.0 * dxy;
  const double eq = sqrt((2.0 / 3.0) * (a * a + b * b + c * c + 0.5 * sh * sh));
  return m * (1.0 - d * (1.0 - exp(-k * eq)));
}

// Rose secant model (elasticity.py:868-944) at the elastic strain (dxx, dyy,
// dxy = its [0,1] entry): G = max(mu exp(-eta eq), floor mu), bulk modulus
// K = lam + 2 mu / 3 kept, lam_eff = K - 2 G / 3; plane stress solves
// eps_zz by the reference's five fixed-point steps.  Returns the trace
// (eps_zz included) and sets G and lam_eff.
__device__ __forceinline__ double rose_moduli(double l, double m, double dxx, double dyy, double dxy, double eta,
                                              double floor_f, int pstress, double& G, double& lam_eff) {
  const double K = l + (2.0 / 3.0) * m;
  double ezz = 0.0;
  auto eq_of = [&](double zz) {
    const double tr3 = (dxx + dyy + zz) / 3.0;
    const double a = dxx - tr3, b = dyy - tr3, c = zz - tr3;
    return sqrt((2.0 / 3.0) * (a * a + b * b + c * c + 2.0 * dxy * dxy));
  };
  auto g_of = [&](double eq) { return fmax(m * exp(-eta * eq), floor_f * m); };
  if (pstress) {
    ezz = -l / (l + 2.0 * m) * (dxx + dyy);
    for (int it = 0; it < 5; ++it) {
      const double g = g_of(eq_of(ezz));
      ezz = -((3.0 * K - 2.0 * g) / (3.0 * K + 4.0 * g)) * (dxx + dyy);
    }
  }
  G = g_of(eq_of(ezz));
  lam_eff = K - (2.0 / 3.0) * G;
  return dxx + dyy + ezz;
}

// Landau small-strain stress, plane strain (elasticity.py:487-639 with
// e33 = 0), parameters lp as in Ls2dRep; a12, a21 the two shear entries of
// the elastic strain.  With capping on, every voxel's strain goes through the
// capped form f (a - m) + m, as in the reference.
// Capped components, invariants and coefficients of the Landau law at the
// block-diagonal strain (in-plane a, out-of-plane e33)
// (elasticity.py:527-569).
struct LandauScal {
  double c11, c22, c12, c21, c33, w, I1, I2, cI, ce, ce2;
};

__device__ __forceinline__ LandauScal landau_scal(double mu, double lam, double a11, double a22, double a12,
                                                  double a21, double e33, const double* __restrict__ lp) {
  const double v1 = lp[0], v2 = lp[1], v3 = lp[2], g1 = lp[3], g2 = lp[4], g3 = lp[5], g4 = lp[6];
  const int cap = (int)lp[7];
  LandauScal s;
  s.c11 = a11; s.c22 = a22; s.c12 = a12; s.c21 = a21; s.c33 = e33; s.w = 0.0;
  if (cap) {
    const double m3 = (a11 + a22 + e33) / 3.0;
    const double d11 = a11 - m3, d22 = a22 - m3, d33 = e33 - m3;
    const double Ecap = lp[8];
    const double Eeq = sqrt(fmax(0.0, (2.0 / 3.0) * (d11 * d11 + d22 * d22 + d33 * d33 + 2.0 * a12 * a21)));
    double f = 1.0;
    if (cap == 2) {
      const double pw = lp[10];
      if (Eeq > 1e-12) f = (Ecap / Eeq) * pow(tanh(fmin(100.0, pow(Eeq / Ecap, pw))), 1.0 / pw);
      const double t = tanh(fmin(100.0, pow(Eeq / Ecap, pw)));
      s.w = t * t;
    } else if (Eeq > Ecap) {
      f = Ecap / Eeq;
      s.w = 1.0;
    }
    s.c11 = f * d11 + m3;
    s.c22 = f * d22 + m3;
    s.c12 = f * a12;
    s.c21 = f * a21;
    s.c33 = f * d33 + m3;
  }
  const double c11 = s.c11, c22 = s.c22, c33 = s.c33;
  const double I1 = c11 + c22 + c33;
  const double cross = s.c12 * s.c21;
  const double tr2 = c11 * c11 + c22 * c22 + 2.0 * cross;
  const double I2 = tr2 + c33 * c33;
  const double t_ip = c11 + c22;
  const double I3 = t_ip * (tr2 - (c11 * c22 - cross)) + c33 * c33 * c33;
  s.I1 = I1;
  s.I2 = I2;
  s.cI = lam * I1 + 0.5 * v1 * (I1 * I1) + v2 * I2 + (1.0 / 6.0) * g1 * (I1 * I1 * I1) + g2 * I1 * I2 +
         (4.0 / 3.0) * g3 * I3;
  s.ce = 2.0 * (mu + v2 * I1 + 0.5 * g2 * (I1 * I1) + g4 * I2);
  s.ce2 = 4.0 * (v3 + g3 * I1);
  return s;
}

// The Landau small-strain stress of a 2D voxel (elasticity.py:487-639).
// Plane strain: e33 = 0.  Plane stress (ps): e33 from the reference's Newton
// steps on sigma33 = 0 (:571-616) from the linear guess
// -lam/(lam + 2 mu) tr a, here until the voxel's step is below 1e-14 (at
// most 64 steps); the stress is evaluated at the stepped e33.  The
// reference runs the steps of all voxels together until every step is below
// 1e-9, evaluates each voxel before its last step and warm-starts the next
// call from the stepped field, so across its solver's iterations e33
// converges to the root of sigma33 = 0, which the kernel solves for at
// every evaluation.  With capping the step's derivative leaves out the
// capping factor's dependence on e33 and the steps converge linearly, so a
// single cold solve stopped at 1e-9 would leave ~1e-10 in e33.  e33_out
// (may be null) receives e33.
__device__ __forceinline__ void landau_sigma(double mu, double lam, double a11, double a22, double a12, double a21,
                                             const double* __restrict__ lp, int ps, double& s11, double& s22,
                                             double& s12, double& s21, double* e33_out = nullptr) {
  double e33 = 0.0;
  if (ps) {
    const double v1 = lp[0], v2 = lp[1], g1 = lp[3], g2 = lp[4], g3 = lp[5], g4 = lp[6];
    const double Gt = lp[9] * mu;
    e33 = -lam / (lam + 2.0 * mu) * (a11 + a22);
#pragma unroll 1
    for (int it = 0; it < 64; ++it) {
      const LandauScal t = landau_scal(mu, lam, a11, a22, a12, a21, e33, lp);
      const double c33 = t.c33, I1 = t.I1, I2 = t.I2;
      double s33 = t.cI + t.ce * c33 + t.ce2 * (c33 * c33);
      const double dcI = lam + v1 * I1 + 0.5 * g1 * (I1 * I1) + g2 * I2 + 2.0 * (v2 + g2 * I1) * c33 +
                         4.0 * g3 * (c33 * c33);
      const double dce = 2.0 * (v2 + g2 * I1) + 4.0 * g4 * c33;
      double ds33 = dcI + dce * c33 + t.ce + 4.0 * g3 * (c33 * c33) + 2.0 * t.ce2 * c33;
      if ((int)lp[7]) {
        s33 = s33 + 2.0 * Gt * (e33 - c33) * t.w;
        ds33 = ds33 + 2.0 * Gt * t.w;
      }
      const double delta = -s33 / (ds33 + 1e-12);
      e33 = e33 + delta;
      if (!(fabs(delta) >= 1e-14)) break;  // also leaves on NaN, which the stress then carries
    }
    if (e33_out) *e33_out = e33;
  }
  const LandauScal t = landau_scal(mu, lam, a11, a22, a12, a21, e33, lp);
  const double cross = t.c12 * t.c21;
  const double t_ip = t.c11 + t.c22;
  s11 = t.cI + t.ce * t.c11 + t.ce2 * (t.c11 * t.c11 + cross);
  s22 = t.cI + t.ce * t.c22 + t.ce2 * (t.c22 * t.c22 + cross);
  s12 = t.ce * t.c12 + t.ce2 * (t.c12 * t_ip);
  s21 = t.ce * t.c21 + t.ce2 * (t.c21 * t_ip);
  if ((int)lp[7]) {
    const double r = 2.0 * (lp[9] * mu) * t.w;
    s11 += r * (a11 - t.c11);
    s22 += r * (a22 - t.c22);
    s12 += r * (a12 - t.c12);
    s21 += r * (a21 - t.c21);
  }
}

// stress of the elastic strain (dxx, dyy, dxy) under law LAW; m, l the voxel's
// mu, lambda; LAW 0 is Hooke's law with the reference's operation order
template <int LAW>
__device__ __forceinline__ void law_sigma(double m, double l, double dxx, double dyy, double dxy, double a, double b,
                                          int ps, double& sxx, double& syy, double& sxy,
                                          const double* __restrict__ lp = nullptr) {
  if constexpr (LAW == 3) {
    double syx;
    landau_sigma(m, l, dxx, dyy, dxy, dxy, lp, ps, sxx, syy, sxy, syx);
  } else if constexpr (LAW == 2) {
    double G, le;
    const double tr = rose_moduli(l, m, dxx, dyy, dxy, a, b, ps, G, le);
    sxx = le * tr + 2.0 * G * dxx;
    syy = le * tr + 2.0 * G * dyy;
    sxy = 2.0 * G * dxy;
  } else {
    const double ms = LAW == 1 ? secant_mu(m, dxx, dyy, dxy, a, b) : m;
    const double trd = dxx + dyy;
    sxx = 2 * ms * dxx + l * trd;
    syy = 2 * ms * dyy + l * trd;
    sxy = 2 * ms * dxy;
  }
}

// Convergence decision of replica r once the last of its row pairs' partial sums
// is written (all threads of the CTA call, in whole warps; thread 0 decides): a
// warp tree over every 32 pairs, then one over their results, so that the order of
// the sums does not depend on the CTA's size.  The last replica to decide sets the graph while-node's condition.
// final: this phase's decision is the last one (FP64 iterations).
static __device__ void ls2d_decide(const Ls2dRep& R, Ls2dState& S, const double* partials, Ls2dCtl* ctl,
                                   cudaGraphConditionalHandle cond, int use_cond, int guard_cap, bool final) {
  __shared__ double2 part32[kMaxPairs / 32];
  const double2* p = reinterpret_cast<const double2*>(partials) + R.row_first;
  const int lane = threadIdx.x & 31, n32 = (R.row_items + 31) / 32;
#pragma unroll 2
  for (int g = threadIdx.x >> 5; g < n32; g += blockDim.x >> 5) {
    const int i = 32 * g + lane;
    double2 v = i < R.row_items ? __ldcg(p + i) : make_double2(0.0, 0.0);
    v.x = warp_sum(v.x);
    v.y = warp_sum(v.y);
    if (lane == 0) part32[g] = v;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  double a = 0, b = 0;
  for (int g = lane; g < n32; g += 32) { a += part32[g].x; b += part32[g].y; }
  a = warp_sum(a);
  b = warp_sum(b);
  if (threadIdx.x != 0) return;
  // the control block's words at once, ahead of the chain of atomics below (n_active is
  // stable until every active replica has decided)
  const unsigned int n_act = *(volatile unsigned int*)&ctl->n_active, bodies = *(volatile unsigned int*)&ctl->bodies;
  const int error = *(volatile int*)&ctl->error;
  if (S.iter == 0) { a += S.extra_d0; b += S.extra_n0; }
  else { b += 2.0 * (double)R.N * S.abar * S.abar; }
  const double diff = sqrt(a) / (sqrt(b) + 1e-20);
  S.diff = diff;
  S.iter += 1;
  S.phase_iter += 1;
  int keep = 0;
  if (!isfinite(diff)) { S.done = 2; S.status = MGK_NONFINITE; }
  else if (final) {
    if (diff < R.tol) { S.done = 2; S.status = MGK_OK; }
    else if (S.iter >= R.max_iter) { S.done = 2; S.status = MGK_NOT_CONVERGED; }
    else keep = 1;
  } else {
    const double tol1 = R.tol > kMixedPhase1Tol ? R.tol : kMixedPhase1Tol;
    if (S.iter >= R.max_iter) { S.done = 2; S.status = diff < R.tol ? MGK_OK : MGK_NOT_CONVERGED; }
    else if (diff < tol1 || S.phase_iter >= kMixedPhase1Cap) S.done = 1;
    else keep = 1;
  }
  if (keep) atomicAdd(&ctl->still, 1u);
  __threadfence();
  const unsigned int d = atomicAdd(&ctl->decided, 1u);
  if (d == n_act - 1) {
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
