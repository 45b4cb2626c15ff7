// 2D small-strain Lippmann-Schwinger solver, batched over replicas.
//
// Restates mgkmc/linear_elastic_simulator.py:12-88 (spectral_solver_2d):
//   tau = C:(eps - eps_p) - C0:eps;  eps_new = eps_bar - IFFT(Gamma0 : FFT(tau));
//   diff = ||eps_new - eps|| / (||eps|| + 1e-20); stop when diff < tol.
// with the Green operator of mgkmc/elasticity.py:20-53 evaluated on the fly
// from the wave vector (never materialised).
//
// A plan holds `nrep` independent replicas (grids of any supported size, so a
// batch may be ragged).  A solve call selects a subset of them; every stage
// is one launch per shape among the selected replicas.
//
// HBM layout per replica (SoA planes of N = nx*ny, C order):
//   mu, lam                 Lame fields (plane strain or plane stress lambda)
//   eps[3]                  xx, yy, symmetric xy of the current iterate
//   ep[3]                   xx, yy, symmetric xy of the eigenstrain
//   epa[2] (optional)       eps_p xy and yx when an eigenstrain is given
//   spec[3]                 half spectrum, nx rows of ld = ny/2+1 complex
// Mixed-precision plans also hold FP32 copies of mu, lam, eps and ep.  The
// antisymmetric part of eps is uniform after the first iteration (Gamma0
// returns symmetric tensors), so it is carried as one scalar.
//
// One iteration = two kernels:
//   row kernel  (one CTA per pair of x-rows): C2R along y of the previous
//               spectrum (two real rows packed as one complex line), update
//               eps = eps_bar + eps~, the diff/norm partial sums, then the
//               polarisation tau and the R2C along y of the next iteration;
//   column kernel (one CTA per tile of ky columns): complex FFT along x,
//               eps~^ = -Gamma0_sym(k) : tau^ / N, inverse FFT along x.
// The spectral field crosses HBM once per direction per iteration.  The last
// CTA of each replica to finish a row kernel reduces that replica's partial
// sums in a fixed order (deterministic), decides its convergence on the
// device, and the last replica to decide sets the condition of the CUDA
// graph while-node that holds the loop, so a solve needs no host round trip (new
// selections of several shapes are driven from the host first, see ls2d_host_first).
//
// Precision forms: FP64 (the reference's arithmetic), and mixed: FP32
// storage, FFTs and Gamma0 until the update norm falls below max(tol, 2e-6)
// (phase 1), then FP64 iterations from that field to the requested tol
// (phase 2).  Norms and partial sums are FP64 in both.
//
// Nyquist handling: the reference takes .real of a complex ifft after
// multiplying by Gamma(q) whose sign pattern breaks Hermitian symmetry on
// Nyquist lines; .real of that equals the C2R of the operator averaged over
// q and its mirror, Gamma_sym(q) = (Gamma(q) + Gamma(S q))/2 with S flipping
// the Nyquist components, which is what the column kernel applies.  q uses
// numpy's fftfreq signs (-n/2 on an even axis's Nyquist line): where two axes
// sit on their Nyquist lines at once the average is Gamma(q) itself and the
// signs of the cross terms follow that convention.
#include <math.h>
#include <stddef.h>
#include <stdlib.h>

#include <algorithm>
#include <mutex>
#include <set>
#include <utility>
#include <vector>

#include "common.cuh"
#include "fft.cuh"
#include "ls2d_dev.cuh"
#include "ls2d_line.cuh"

namespace mgk {

const void* twiddles(int n, int prec);

const Ls2Line* ls2_line_a(int n, int kind);
const Ls2Line* ls2_line_b(int n, int kind);
const Ls2Line* ls2_line_c(int n, int kind);
const Ls2Line* ls2_line_d(int n, int kind);
const Ls2Line* ls2_line_e(int n, int kind);
const Ls2Line* ls2_line_f(int n, int kind);
const Ls2Line* ls2_line_g(int n, int kind);
const Ls2Line* ls2_line_h(int n, int kind);
const Ls2Line* ls2_line(int n, int kind) {
  for (auto f : {ls2_line_a, ls2_line_b, ls2_line_c, ls2_line_d, ls2_line_e, ls2_line_f, ls2_line_g, ls2_line_h})
    if (const Ls2Line* k = f(n, kind)) return k;
  return nullptr;
}

// -------------------------------------------------------------- kernels ---

constexpr int kThreads = 256;

// Sums over a replica's CTAs of K <= 8 values per thread, in a fixed order:
// warp trees, the warps, then (in the CTA that arrives last) one warp per
// value over the CTAs' partials.  part: the replica's gridDim.x slots of K;
// ctr: its arrival counter (left at zero).  True in the last CTA only, with
// the sums in res.  A launch for the last step alone took 4 .. 7 us.
template <int K>
__device__ __forceinline__ bool grid_sums(const double* v, double* part, unsigned int* ctr, double* res) {
  __shared__ double w[kThreads / 32][K];
  __shared__ int s_last;
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
    for (int k = 0; k < kThreads / 32; ++k) t += w[k][threadIdx.x];
    part[blockIdx.x * K + threadIdx.x] = t;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicInc(ctr, gridDim.x - 1) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return false;
  __threadfence();
  if (wid < K) {
    double a = 0;
    for (int i = lane; i < (int)gridDim.x; i += 32) a += __ldcg(&part[i * K + wid]);
    a = warp_sum(a);
    if (lane == 0) res[wid] = a;
  }
  __syncthreads();
  return true;
}

// Per-voxel material prep for one replica: mu, lambda from (E, nu) as in
// elasticity.py:3-10 (set_moduli 1), or given directly (set_moduli 2: E holds
// lambda, nu holds mu, as the secant solver takes them), eigenstrain planes
// (and FP32 copies for mixed plans), and the reference medium from the means:
// of E and nu (linear_elastic_simulator.py:22-26), or of lambda and mu (lame_in
// 1: the secant solver, :679-681; lame_in 2: the Rose solver's (mean lambda,
// (mean mu + floor mean mu) / 2), :866-869).
__global__ void __launch_bounds__(kThreads) ls2d_material_kernel(const Ls2dRep* reps, Ls2dState* st, int rep,
                                                                 const double* __restrict__ E,
                                                                 const double* __restrict__ nu,
                                                                 const double* __restrict__ epsp, int plane_mode,
                                                                 int set_moduli, int lame_in, double floor_f,
                                                                 double* partials, unsigned int* ctr) {
  __shared__ double res[2];
  const Ls2dRep& R = reps[rep];
  const long long N = R.N;
  double sm[2] = {0, 0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N;
       i += (long long)gridDim.x * blockDim.x) {
    if (set_moduli) {
      const double e = E[i], v = nu[i];
      const double mu = set_moduli == 2 ? v : e / (2 * (1 + v));
      const double lam = set_moduli == 2 ? e
                         : plane_mode == MGK_PLANE_STRESS ? e * v / (1 - v * v)
                                                          : e * v / ((1 + v) * (1 - 2 * v));
      R.mu[i] = mu;
      R.lam[i] = lam;
      if (R.mu32) { R.mu32[i] = (float)mu; R.lam32[i] = (float)lam; }
      sm[0] += e;
      sm[1] += v;
    }
    double pxx = 0, pxy = 0, pyx = 0, pyy = 0;
    if (epsp) {
      const double4 p = reinterpret_cast<const double4*>(epsp)[i];
      pxx = p.x; pxy = p.y; pyx = p.z; pyy = p.w;
    }
    const double psym = (pxy == pyx) ? pxy : 0.5 * (pxy + pyx);
    R.ep[i] = pxx;
    R.ep[N + i] = pyy;
    R.ep[2 * N + i] = psym;
    if (R.ep32) { R.ep32[i] = (float)pxx; R.ep32[N + i] = (float)pyy; R.ep32[2 * N + i] = (float)psym; }
    if (R.epa) {
      R.epa[i] = pxy;
      R.epa[N + i] = pyx;
    }
  }
  if (!set_moduli || !grid_sums<2>(sm, partials, ctr, res) || threadIdx.x != 0) return;
  const double a = res[0] / (double)N, v = res[1] / (double)N;
  const double mu0 = lame_in == 2 ? 0.5 * (v + floor_f * v) : lame_in ? v : a / (2 * (1 + v));
  const double lam0 = lame_in ? a
                      : plane_mode == MGK_PLANE_STRESS ? a * v / (1 - v * v) : a * v / ((1 + v) * (1 - 2 * v));
  Ls2dState& S = st[rep];
  S.mu0 = mu0;
  S.lam0 = lam0;
  S.Bc = (lam0 + mu0) / (mu0 * (lam0 + 2 * mu0));
  S.inv2mu0 = 1.0 / (2 * mu0);
}

// Warm-start means of the 4 components of each selected replica's init
// field.  grid = (G, nsel).
__global__ void __launch_bounds__(kThreads) ls2d_means_kernel(const Ls2dRep* reps, Ls2dState* st, const int* sel,
                                                              double* partials, unsigned int* ctr) {
  __shared__ double res[4];
  const int r = sel[blockIdx.y];
  const Ls2dRep& R = reps[r];
  if (!R.init) return;
  const long long N = R.N;
  double s[4] = {0, 0, 0, 0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N;
       i += (long long)gridDim.x * blockDim.x) {
    const double4 v = reinterpret_cast<const double4*>(R.init)[i];
    s[0] += v.x; s[1] += v.y; s[2] += v.z; s[3] += v.w;
  }
  if (grid_sums<4>(s, partials + (size_t)blockIdx.y * gridDim.x * 8, ctr + r, res) && threadIdx.x < 4)
    st[r].means[threadIdx.x] = res[threadIdx.x] * (1.0 / (double)N);
}

// Solve start for each selected replica: eps_bar, caps and the initial field
// (linear_elastic_simulator.py:32-41), and the antisymmetric part's
// contribution to the first diff and norm.  fp32: the loop starts with a mixed
// plan's FP32 phase, which needs the FP32 field only.  The replica's arrival
// counter of the row kernel starts at zero whatever the call before it left: a row
// CTA whose copy wait gave up does not arrive.  grid = (G, nsel).
__global__ void __launch_bounds__(kThreads) ls2d_begin_kernel(const Ls2dRep* reps, Ls2dState* st, const int* sel,
                                                              double* partials, unsigned int* ctr,
                                                              unsigned int* arrivals, int fp32) {
  __shared__ double res[2];
  const int r = sel[blockIdx.y];
  const Ls2dRep& R = reps[r];
  Ls2dState& S = st[r];
  const long long N = R.N;
  const double e00 = R.eb[0], e01 = R.eb[1], e10 = R.eb[2], e11 = R.eb[3];
  const double abar = 0.5 * (e01 - e10);
  const double sbar = (e01 == e10) ? e01 : 0.5 * (e01 + e10);
  const double* init = R.init;
  double dn[2] = {0, 0};
  double m00 = 0, m01 = 0, m10 = 0, m11 = 0;
  if (init) { m00 = S.means[0]; m01 = S.means[1]; m10 = S.means[2]; m11 = S.means[3]; }
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N;
       i += (long long)gridDim.x * blockDim.x) {
    double xx, yy, sy;
    if (init) {
      const double4 v = reinterpret_cast<const double4*>(init)[i];
      xx = v.x + (e00 - m00);
      const double xy = v.y + (e01 - m01), yx = v.z + (e10 - m10);
      yy = v.w + (e11 - m11);
      sy = (xy == yx) ? xy : 0.5 * (xy + yx);
      const double a0 = 0.5 * (xy - yx);
      dn[0] += 2 * (abar - a0) * (abar - a0);
      dn[1] += 2 * a0 * a0;
    } else {
      xx = e00; yy = e11; sy = sbar;
    }
    if (!fp32) {
      R.eps[i] = xx;
      R.eps[N + i] = yy;
      R.eps[2 * N + i] = sy;
    }
    if (R.eps32) { R.eps32[i] = (float)xx; R.eps32[N + i] = (float)yy; R.eps32[2 * N + i] = (float)sy; }
  }
  if (init && grid_sums<2>(dn, partials + (size_t)blockIdx.y * gridDim.x * 8, ctr + r, res) && threadIdx.x == 0) {
    S.extra_d0 = res[0];
    S.extra_n0 = res[1];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    S.ebar[0] = e00;
    S.ebar[1] = e11;
    S.ebar[2] = sbar;
    S.abar = abar;
    S.iter = 0;
    S.phase_iter = 0;
    S.done = R.max_iter <= 0 ? 2 : 0;
    S.status = MGK_OK;
    S.diff = 0;
    arrivals[r] = 0;
    if (!init) { S.extra_d0 = 0; S.extra_n0 = 2.0 * (double)N * abar * abar; }
  }
}

// Row kernel.  IN_SPEC: the previous iteration's spectrum is inverted and the
// field updated (with diff/norm and the convergence decision); otherwise the
// field is read as is (first tau of a phase).  FINAL: this phase's decision
// is the last one (FP64 plans, or phase 2 of mixed plans).
template <typename TS, typename TC, bool IN_SPEC, bool FINAL>
__global__ void __launch_bounds__(256) ls2d_row_kernel(const Ls2dRep* __restrict__ reps, Ls2dState* st,
                                                      const int* __restrict__ row_map,
                                                      const int* __restrict__ row_local, double* partials,
                                                      unsigned int* rep_counter, Ls2dCtl* ctl,
                                                      cudaGraphConditionalHandle cond, int use_cond,
                                                      int guard_cap) {
  using C = C_t<TC>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  __shared__ int s_last;
  const int item = blockIdx.x;
  const int r = row_map[item];
  const Ls2dRep& R = reps[r];
  Ls2dState& S = st[r];
  if (IN_SPEC && use_cond && item == 0 && threadIdx.x == 0) {
    // a body with no active replica has no decider: stop here; the body
    // count bounds the loop whatever happens to the deciders
    const unsigned int b = atomicAdd(&ctl->bodies, 1u) + 1u;
    if (ctl->n_active == 0 || b > (unsigned int)guard_cap || *(volatile int*)&ctl->error != 0) {
      ctl->any = 0;
      cudaGraphSetConditional(cond, 0u);
    }
  }
  if (S.done != 0) return;
  const int ny = R.ny, nyh = R.nyh, ld = R.ld, nx = R.nx;
  const long long N = R.N;
  const int x0 = 2 * row_local[item];
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 3 * ny;
  C* spec = reinterpret_cast<C*>(R.spec);
  const double mu0 = S.mu0, lam0 = S.lam0;
  const int law = R.law, law_ps = R.law_ps;
  const double law_a = R.law_a, law_b = R.law_b;
  const double eb0 = S.ebar[0], eb1 = S.ebar[1], eb2 = S.ebar[2];
  TS* eps = Fields<TS>::eps(R);
  const TS* mu = Fields<TS>::mu(R);
  const TS* lam = Fields<TS>::lam(R);
  const TS* ep = Fields<TS>::ep(R);
  const FftLen& fy = Fields<TS>::fy(R);
  double d2 = 0, n2 = 0;
  C* cur = bufA;
  if (IN_SPEC) {
    const int tot = 3 * ny;
    for (int e0 = threadIdx.x; e0 < tot; e0 += 4 * blockDim.x) {
      C av[4], bv[4];
      int kk[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int e = e0 + u * blockDim.x;
        kk[u] = -1;
        if (e < tot) {
          const int c = e / ny, k = e - c * ny;
          const int ks = (2 * k <= ny) ? k : ny - k;
          const C* ra = spec + ((size_t)c * nx + x0) * ld;
          av[u] = ra[ks];
          bv[u] = ra[ld + ks];
          kk[u] = k;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (kk[u] < 0) continue;
        const int e = e0 + u * blockDim.x, k = kk[u];
        C a = av[u], b = bv[u];
        C z;
        if (2 * k <= ny) {
          if (k == 0 || 2 * k == ny) { a.y = 0; b.y = 0; }
          z = mk<C>(a.x - b.y, a.y + b.x);
        } else {
          z = mk<C>(a.x + b.y, b.x - a.y);
        }
        bufA[e] = z;  // e = c * ny + k
      }
    }
    __syncthreads();
    cur = fft_any<+1>(bufA, bufB, 3, ny, fy);
  }
  C* out = (IN_SPEC && cur == bufA) ? bufB : bufA;
  double gam[kAaMax];
  const int nmix = (!IN_SPEC && sizeof(TS) == 8 && R.aa) ? aa_load(R, gam) : 0;
  // with Anderson mixing the image's tau is never used (the next tau is the
  // mixed iterate's): the pass stops at the image and its update norm
  const bool img_only = IN_SPEC && sizeof(TS) == 8 && law != 0 && R.aa != nullptr;
  for (int y = threadIdx.x; y < ny; y += blockDim.x) {
    TC tr[2][3];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long i = (long long)(x0 + h) * ny + y;
      double e[3];
      const double o0 = (double)eps[i], o1 = (double)eps[N + i], o2 = (double)eps[2 * N + i];
      const double m = (double)mu[i], l = (double)lam[i];
      const double p0 = (double)ep[i], p1 = (double)ep[N + i], p2 = (double)ep[2 * N + i];
      if (IN_SPEC) {
        const C z0 = cur[y], z1 = cur[ny + y], z2 = cur[2 * ny + y];
        e[0] = eb0 + (double)(h == 0 ? z0.x : z0.y);
        e[1] = eb1 + (double)(h == 0 ? z1.x : z1.y);
        e[2] = eb2 + (double)(h == 0 ? z2.x : z2.y);
        const double q0 = e[0] - o0, q1 = e[1] - o1, q2 = e[2] - o2;
        d2 += q0 * q0 + q1 * q1 + 2.0 * q2 * q2;
        n2 += o0 * o0 + o1 * o1 + 2.0 * o2 * o2;
        eps[i] = (TS)e[0];
        eps[N + i] = (TS)e[1];
        eps[2 * N + i] = (TS)e[2];
      } else {
        e[0] = o0; e[1] = o1; e[2] = o2;
        if (!IN_SPEC && sizeof(TS) == 8 && R.aa) aa_mix_voxel(R, i, nmix, gam, e);  // the mixed iterate
      }
      if (img_only) continue;
      const double dxx = e[0] - p0, dyy = e[1] - p1, dxy = e[2] - p2;
      const double tre = e[0] + e[1];
      double s0, s1, s2;  // nonlinear laws only in FP64 kernels (their plans are FP64)
      if (sizeof(TS) == 8 && law == 1) law_sigma<1>(m, l, dxx, dyy, dxy, law_a, law_b, law_ps, s0, s1, s2);
      else if (sizeof(TS) == 8 && law == 2) law_sigma<2>(m, l, dxx, dyy, dxy, law_a, law_b, law_ps, s0, s1, s2);
      else if (sizeof(TS) == 8 && law == 3) law_sigma<3>(m, l, dxx, dyy, dxy, 0.0, 0.0, law_ps, s0, s1, s2, R.lp);
      else law_sigma<0>(m, l, dxx, dyy, dxy, 0.0, 0.0, 0, s0, s1, s2);
      tr[h][0] = (TC)(s0 - (2 * mu0 * e[0] + lam0 * tre));
      tr[h][1] = (TC)(s1 - (2 * mu0 * e[1] + lam0 * tre));
      tr[h][2] = (TC)(s2 - 2 * mu0 * e[2]);
    }
    if (img_only) continue;
#pragma unroll
    for (int c = 0; c < 3; ++c) out[c * ny + y] = mk<C>(tr[0][c], tr[1][c]);
  }
  if (!img_only) {
    __syncthreads();
    C* scratch = (out == bufA) ? bufB : bufA;
    C* Z = fft_any<-1>(out, scratch, 3, ny, fy);
    for (int e = threadIdx.x; e < 3 * nyh; e += blockDim.x) {
      const int c = e / nyh, k = e - c * nyh;
      const C z = Z[c * ny + k];
      const C w = Z[c * ny + (k == 0 ? 0 : ny - k)];
      C* ra = spec + ((size_t)c * nx + x0) * ld;
      ra[k] = mk<C>(TC(0.5) * (z.x + w.x), TC(0.5) * (z.y - w.y));
      ra[ld + k] = mk<C>(TC(0.5) * (z.y + w.y), TC(-0.5) * (z.x - w.x));
    }
  }
  if (!IN_SPEC) return;
  // partial sums -> fixed slot; the replica's last CTA reduces and decides
  d2 = block_sum(d2, red);
  n2 = block_sum(n2, red);
  if (threadIdx.x == 0) {
    partials[2 * item] = d2;
    partials[2 * item + 1] = n2;
    __threadfence();
    const unsigned int t = atomicInc(&rep_counter[r], (unsigned int)R.row_items - 1);  // self-resetting
    s_last = (t == (unsigned int)R.row_items - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  ls2d_decide(R, S, partials, ctl, cond, use_cond, guard_cap, FINAL);
}

// Column kernel: FFT along x, Gamma0_sym, inverse FFT along x, for a tile of
// tc consecutive ky columns and all three components.
template <typename TS, typename TC>
__global__ void __launch_bounds__(256) ls2d_col_kernel(const Ls2dRep* __restrict__ reps,
                                                      const Ls2dState* __restrict__ st,
                                                      const int* __restrict__ col_map,
                                                      const int* __restrict__ col_local) {
  using C = C_t<TC>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int item = blockIdx.x;
  const int r = col_map[item];
  const Ls2dRep& R = reps[r];
  const Ls2dState& S = st[r];
  if (S.done != 0) return;
  const int nx = R.nx, ny = R.ny, nyh = R.nyh, ld = R.ld, tc = R.tc;
  const int ky0 = col_local[item] * tc;
  const int tcw = min(tc, nyh - ky0);
  const FftLen& fx = Fields<TS>::fx(R);
  C* bufA = reinterpret_cast<C*>(smem_raw);
  C* bufB = bufA + 3 * tc * nx;
  C* spec = reinterpret_cast<C*>(R.spec);
  const int tot = 3 * tcw * nx;
  for (int e0 = threadIdx.x; e0 < tot; e0 += 4 * blockDim.x) {
    C v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * blockDim.x;
      if (e < tot) {
        const int c = e / (tcw * nx);
        const int rem = e - c * tcw * nx;
        const int x = rem / tcw, t = rem - x * tcw;
        v[u] = spec[((size_t)c * nx + x) * ld + ky0 + t];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * blockDim.x;
      if (e < tot) {
        const int c = e / (tcw * nx);
        const int rem = e - c * tcw * nx;
        const int x = rem / tcw, t = rem - x * tcw;
        bufA[(c * tc + t) * nx + x] = v[u];
      }
    }
  }
  __syncthreads();
  // lines (c * tc + t); only t < tcw are meaningful, all 3*tc are transformed
  C* F = fft_any<-1>(bufA, bufB, 3 * tc, nx, fx);
  const TC inv2mu0 = (TC)S.inv2mu0, Bc = (TC)S.Bc;
  const TC sc = (TC)(1.0 / ((double)nx * (double)ny));
  for (int e = threadIdx.x; e < tcw * nx; e += blockDim.x) {
    const int t = e / nx, kx = e - t * nx;
    const int ky = ky0 + t;
    C* pxx = &F[(0 * tc + t) * nx + kx];
    C* pyy = &F[(1 * tc + t) * nx + kx];
    C* pxy = &F[(2 * tc + t) * nx + kx];
    if (kx == 0 && ky == 0) {
      *pxx = mk<C>(TC(0), TC(0)); *pyy = *pxx; *pxy = *pxx;
      continue;
    }
    // fftfreq signs matter where several axes sit on their Nyquist line
    const double ux = (double)fftfreq(kx, nx) / nx, uy = (double)fftfreq(ky, ny) / ny;
    const double inv = 1.0 / sqrt(ux * ux + uy * uy);
    const TC nxv = (TC)(ux * inv), nyv = (TC)(uy * inv);
    const C txx = *pxx, tyy = *pyy, txy = *pxy;
    C exx, eyy, exy;
    gamma2d_apply(txx, tyy, txy, nxv, nyv, inv2mu0, Bc, exx, eyy, exy);
    const bool nqx = (nx & 1) == 0 && 2 * kx == nx, nqy = (ny & 1) == 0 && 2 * ky == ny;
    if (nqx || nqy) {
      C fxx, fyy, fxy;
      gamma2d_apply(txx, tyy, txy, nqx ? -nxv : nxv, nqy ? -nyv : nyv, inv2mu0, Bc, fxx, fyy, fxy);
      exx = mk<C>(TC(0.5) * (exx.x + fxx.x), TC(0.5) * (exx.y + fxx.y));
      eyy = mk<C>(TC(0.5) * (eyy.x + fyy.x), TC(0.5) * (eyy.y + fyy.y));
      exy = mk<C>(TC(0.5) * (exy.x + fxy.x), TC(0.5) * (exy.y + fxy.y));
    }
    *pxx = mk<C>(exx.x * sc, exx.y * sc);
    *pyy = mk<C>(eyy.x * sc, eyy.y * sc);
    *pxy = mk<C>(exy.x * sc, exy.y * sc);
  }
  __syncthreads();
  C* G = (F == bufA) ? bufB : bufA;
  C* Rz = fft_any<+1>(F, G, 3 * tc, nx, fx);
  for (int e = threadIdx.x; e < tot; e += blockDim.x) {
    const int c = e / (tcw * nx);
    const int rem = e - c * tcw * nx;
    const int x = rem / tcw, t = rem - x * tcw;
    spec[((size_t)c * nx + x) * ld + ky0 + t] = Rz[(c * tc + t) * nx + x];
  }
}

// Mixed plans with CTA-wide replicas, between the phases: their FP64 field
// from the FP32 one (the register-FFT row pass promotes its own).  grid = (G,
// replicas).
__global__ void ls2d_promote_kernel(const Ls2dRep* reps, const int* sel) {
  const int r = sel[blockIdx.y];
  const Ls2dRep& R = reps[r];
  const long long n3 = 3 * R.N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n3;
       i += (long long)gridDim.x * blockDim.x)
    R.eps[i] = (double)R.eps32[i];
}

// Replicas that finished phase 1 re-enter for phase 2; resets the control block.
// One warp.
__global__ void ls2d_phase2_kernel(Ls2dState* st, const int* sel, int nsel, Ls2dCtl* ctl) {
  unsigned int n = 0;
  for (int q = threadIdx.x; q < nsel; q += 32) {
    Ls2dState& S = st[sel[q]];
    if (S.done == 1) { S.done = 0; S.phase_iter = 0; ++n; }
  }
  n = __reduce_add_sync(0xffffffffu, n);
  if (threadIdx.x != 0) return;
  ctl->n_active = n;
  ctl->decided = 0;
  ctl->still = 0;
  ctl->bodies = 0;
  ctl->any = n > 0;
}

// Outputs in the reference layout: eps, sig (nx,ny,2,2) and the means of
// their components (linear_elastic_simulator.py:83-88).
// grid = (G, nsel).
template <int LAW = 0>  // 1: the secant law, 2: the Rose law, 3: the Landau law
__global__ void __launch_bounds__(kThreads) ls2d_output_kernel(const Ls2dRep* reps, Ls2dState* st, const int* sel,
                                                               double* partials, unsigned int* ctr) {
  __shared__ double res[8];
  const int r = sel[blockIdx.y];
  const Ls2dRep& R = reps[r];
  Ls2dState& S = st[r];
  const long long N = R.N;
  const double abar = S.abar;
  double* eps_out = R.out_eps;
  double* sig_out = R.out_sig;
  const int law_ps = R.law_ps;
  const double law_a = R.law_a, law_b = R.law_b;
  const bool capped_mix = R.aa && S.done == 2 && S.status == MGK_NOT_CONVERGED;
  double gam[kAaMax];
  const int nmix = capped_mix ? aa_load(R, gam) : 0;
  double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N;
       i += (long long)gridDim.x * blockDim.x) {
    double ev[3] = {R.eps[i], R.eps[N + i], R.eps[2 * N + i]};
    if (capped_mix) aa_mix_voxel(R, i, nmix, gam, ev);  // the loop ended at the cap: the last mixed iterate
    const double sxy = ev[2];
    const double exx = ev[0], eyy = ev[1];
    const double exy = abar == 0 ? sxy : sxy + abar;
    const double eyx = abar == 0 ? sxy : sxy - abar;
    double pxx = R.ep[i], pyy = R.ep[N + i], pxy, pyx;
    if (R.epa) { pxy = R.epa[i]; pyx = R.epa[N + i]; }
    else { pxy = R.ep[2 * N + i]; pyx = pxy; }
    const double lam = R.lam[i];
    const double dxx = exx - pxx, dxy = exy - pxy, dyx = eyx - pyx, dyy = eyy - pyy;
    double mu = R.mu[i];
    double sxx, syy, sxy2, syx2;
    if constexpr (LAW == 3) {
      landau_sigma(mu, lam, dxx, dyy, dxy, dyx, R.lp, law_ps, sxx, syy, sxy2, syx2, R.out_e33 ? R.out_e33 + i : nullptr);
    } else if constexpr (LAW == 2) {
      // Rose: sigma_yx is a copy of sigma_xy, from the [0,1] strain entry
      law_sigma<2>(mu, lam, dxx, dyy, dxy, law_a, law_b, law_ps, sxx, syy, sxy2);
      syx2 = sxy2;
    } else {
      if constexpr (LAW == 1) mu = secant_mu(mu, dxx, dyy, 0.5 * (dxy + dyx), law_a, law_b);
      const double tr = dxx + dyy;
      sxx = 2 * mu * dxx + lam * tr;
      syy = 2 * mu * dyy + lam * tr;
      sxy2 = 2 * mu * dxy;
      syx2 = 2 * mu * dyx;
    }
    if (eps_out) reinterpret_cast<double4*>(eps_out)[i] = make_double4(exx, exy, eyx, eyy);
    if (sig_out) reinterpret_cast<double4*>(sig_out)[i] = make_double4(sxx, sxy2, syx2, syy);
    s[0] += exx; s[1] += exy; s[2] += eyx; s[3] += eyy;
    s[4] += sxx; s[5] += sxy2; s[6] += syx2; s[7] += syy;
  }
  if (grid_sums<8>(s, partials + (size_t)blockIdx.y * gridDim.x * 8, ctr + r, res) && threadIdx.x < 8)
    (threadIdx.x < 4 ? S.out_eps_mean : S.out_sig_mean)[threadIdx.x & 3] = res[threadIdx.x] * (1.0 / (double)N);
}

// Anderson mixing over fields of n doubles (linear_elastic_simulator.py:
// 1185-1209), kept as differences: hist holds 2 m + 2 vectors of n doubles,
// dF columns 0..m-1, dG columns 0..m-1, then f_prev and g_prev.  One pass
// forms f = g - x, writes column `slot` (dF = f - f_prev, dG = g - g_prev)
// when a previous pair exists, stores f and g as the previous pair, and
// accumulates <dF_j, dF_slot> and <dF_j, f> for the ncols valid columns.
constexpr int kAaBlocks = 296;

__global__ void __launch_bounds__(256) aa_update_kernel(long long n, const double* __restrict__ x,
                                                        const double* __restrict__ g, double* __restrict__ hist,
                                                        int m, int slot, int have_prev, int ncols,
                                                        double* __restrict__ partials) {
  __shared__ double red[32];
  double* dF = hist;
  double* dG = hist + (size_t)m * n;
  double* fp = hist + 2 * (size_t)m * n;
  double* gp = fp + n;
  double an[kAaMax], ar[kAaMax];
#pragma unroll
  for (int j = 0; j < kAaMax; ++j) { an[j] = 0.0; ar[j] = 0.0; }
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double gi = g[i], fi = gi - x[i];
    double df = 0.0;
    if (have_prev) {
      df = fi - fp[i];
      dF[(size_t)slot * n + i] = df;
      dG[(size_t)slot * n + i] = gi - gp[i];
    }
    fp[i] = fi;
    gp[i] = gi;
#pragma unroll
    for (int j = 0; j < kAaMax; ++j)
      if (j < ncols) {
        const double c = (j == slot && have_prev) ? df : dF[(size_t)j * n + i];
        an[j] += c * df;
        ar[j] += c * fi;
      }
  }
#pragma unroll
  for (int j = 0; j < kAaMax; ++j)
    if (j < ncols) {
      const double a = block_sum(an[j], red);
      const double b = block_sum(ar[j], red);
      if (threadIdx.x == 0) {
        partials[(size_t)blockIdx.x * 2 * kAaMax + j] = a;
        partials[(size_t)blockIdx.x * 2 * kAaMax + kAaMax + j] = b;
      }
    }
}

// sums the per-block partials: out[j] = <dF_j, dF_slot>, out[kAaMax + j] = <dF_j, f>
__global__ void aa_sum_kernel(const double* __restrict__ partials, int nb, int ncols, double* __restrict__ out) {
  __shared__ double red[32];
  for (int q = 0; q < 2 * kAaMax; ++q) {
    if ((q % kAaMax) >= ncols) continue;
    double a = 0.0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) a += partials[(size_t)b * 2 * kAaMax + q];
    a = block_sum(a, red);
    if (threadIdx.x == 0) out[q] = a;
  }
}

struct AaCoef { double v[kAaMax]; };

// x = g - sum_j gamma_j dG_j
__global__ void aa_mix_kernel(long long n, const double* __restrict__ g, const double* __restrict__ hist, int m,
                              int ncols, AaCoef gam, double* __restrict__ x) {
  const double* dG = hist + (size_t)m * n;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < kAaMax; ++j)
      if (j < ncols) s += gam.v[j] * dG[(size_t)j * n + i];
    x[i] = g[i] - s;
  }
}


// ------------------------------------- Anderson mixing inside the LS loop ---
// Type-II Anderson mixing of one replica's fixed-point iterates, run in the
// loop body between the row kernel that forms the image g = G(x) (with the
// update norm and the convergence decision) and the first row pass of the
// next iterate (linear_elastic_simulator.py:1185-1209): residual f = g - x;
// differences dF, dG of consecutive (f, g) pairs, at most m of them;
// gamma = argmin |dF gamma - f|; x = g - dG gamma.  When the coefficients are
// not finite the step is the plain one (x = g) and the history restarts from
// the last pair, as the reference's fallback does.  Fields are the replica's
// symmetric strain planes (xx, yy, xy); inner products weight the xy plane
// by 2, as the reference's sums over the four tensor entries do.  The
// differences sit in a ring of m slots; the least-squares solution does not
// depend on the order of the columns.

// Mixing follows every iteration except the converged or non-finite one:
// the reference leaves its loop with the image g there, and with the last
// mixed iterate when the iteration cap ends the loop.
__device__ __forceinline__ bool aa_skip(const Ls2dState& S) {
  return S.done != 0 && S.status != MGK_NOT_CONVERGED;
}

// Ring buffer of one plan (n3 = 3 N doubles each): x, f_prev, g_prev, then
// dF slots 0 .. m-1 and dG slots 0 .. m-1.
__global__ void ls2d_aa_init_kernel(const Ls2dRep* reps, const int* sel, double* buf, Ls2dAA* aa) {
  const Ls2dRep& R = reps[sel[0]];
  const long long n3 = 3 * R.N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n3; i += (long long)gridDim.x * blockDim.x)
    buf[i] = R.eps[i];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    aa->k = 0;
    aa->slot_next = 0;
    aa->have_prev = 0;
    aa->nmix = 0;
    aa->ctr = 0;
  }
}

// Sum over the warp, the same value in every lane (reduced to lane 0, then
// broadcast: a butterfly would round differently per lane).
__device__ __forceinline__ double warp_allsum(double v) {
  return __shfl_sync(0xffffffffu, warp_sum(v), 0);
}

// Least squares of the mix, one warp (lanes = matrix rows): gamma = sum
// over eigenpairs (lambda_i, v_i) of the k x k Gram matrix with lambda_i
// above 1e-14 lambda_max of (v_i . b / lambda_i) v_i, the minimum-norm
// solution with the small singular values of dF cut off.  Eigenpairs by
// cyclic Jacobi rotations (Golub & Van Loan, Matrix Computations, 8.5), each
// rotation's row and column updates spread over the lanes.  sa, sv: k x k
// shared scratch; b in sb.  Writes gamma and nmix (0 for the plain step,
// and the history restarts from the last pair when the coefficients are
// not finite).
// Fast path of the same least squares (one thread): when the Gram matrix
// is comfortably conditioned no eigenvalue falls under the cut-off, so the
// truncated eigen solution is A^-1 b, solved here by Cholesky.  The test:
// lambda_min >= 1 / tr(A^-1) = 1 / ||L^-1||_F^2 and lambda_max <= tr(A);
// when 1 / ||L^-1||_F^2 > 1e-12 tr(A) every eigenvalue is above
// 1e-14 lambda_max with margin for the rounding of the estimate.  Returns
// false (nothing written) when the factorisation fails or the test does not
// hold: the eigen path decides then.
__device__ bool aa_lstsq_cholesky(Ls2dAA* aa, int k, const double* sb) {
  double Lm[kAaMax][kAaMax];
  double tr = 0.0;
  for (int i = 0; i < k; ++i) tr += aa->A[i][i];
  for (int j = 0; j < k; ++j) {
    double d = aa->A[j][j];
    for (int q = 0; q < j; ++q) d -= Lm[j][q] * Lm[j][q];
    if (!(d > 0.0)) return false;
    const double ljj = sqrt(d);
    Lm[j][j] = ljj;
    for (int i = j + 1; i < k; ++i) {
      double v = aa->A[i][j];
      for (int q = 0; q < j; ++q) v -= Lm[i][q] * Lm[j][q];
      Lm[i][j] = v / ljj;
    }
  }
  // ||L^-1||_F^2, column by column of L^-1 (forward substitution on e_c)
  double fro = 0.0;
  for (int c = 0; c < k; ++c) {
    double z[kAaMax];
    for (int i = 0; i < k; ++i) {
      double v = i == c ? 1.0 : 0.0;
      for (int q = c; q < i; ++q) v -= Lm[i][q] * z[q];
      z[i] = i < c ? 0.0 : v / Lm[i][i];
      if (i >= c) fro += z[i] * z[i];
    }
  }
  if (!(isfinite(fro) && 1.0 / fro > 1e-12 * tr)) return false;
  double y[kAaMax], g[kAaMax];
  for (int i = 0; i < k; ++i) {
    double v = sb[i];
    for (int q = 0; q < i; ++q) v -= Lm[i][q] * y[q];
    y[i] = v / Lm[i][i];
  }
  for (int i = k - 1; i >= 0; --i) {
    double v = y[i];
    for (int q = i + 1; q < k; ++q) v -= Lm[q][i] * g[q];
    g[i] = v / Lm[i][i];
  }
  for (int i = 0; i < k; ++i)
    if (!isfinite(g[i])) return false;
  for (int i = 0; i < k; ++i) aa->gamma[i] = g[i];
  aa->nmix = k;
  return true;
}

__device__ void aa_lstsq_warp(Ls2dAA* aa, int k, double (*sa)[kAaMax], double (*sv)[kAaMax], const double* sb) {
  const int l = threadIdx.x;  // lane, < 32
  for (int e = l; e < k * k; e += 32) {
    const int i = e / k, j = e - (e / k) * k;
    sa[i][j] = aa->A[i][j];
    sv[i][j] = i == j ? 1.0 : 0.0;
  }
  __syncwarp();
  double fro = 0.0;
  for (int e = l; e < k * k; e += 32) {
    const int i = e / k, j = e - (e / k) * k;
    fro += sa[i][j] * sa[i][j];
  }
  fro = warp_allsum(fro);
  for (int sweep = 0; sweep < 40; ++sweep) {
    double off = 0.0;
    for (int e = l; e < k * k; e += 32) {
      const int i = e / k, j = e - (e / k) * k;
      if (j > i) off += sa[i][j] * sa[i][j];
    }
    off = warp_allsum(off);
    if (!(off > 1e-30 * fro)) break;  // also leaves on NaN (uniform: every lane has the same sums)
    for (int p = 0; p < k; ++p)
      for (int q = p + 1; q < k; ++q) {
        const double apq = sa[p][q], app = sa[p][p], aqq = sa[q][q];
        __syncwarp();
        if (fabs(apq) <= 1e-18 * sqrt(fabs(app * aqq))) {  // negligible: no rotation
          if (l == 0) { sa[p][q] = 0.0; sa[q][p] = 0.0; }
          __syncwarp();
          continue;
        }
        const double th = (aqq - app) / (2.0 * apq);
        const double t = (th >= 0.0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
        const double c = 1.0 / sqrt(t * t + 1.0), sn = t * c;
        double x0 = 0.0, x1 = 0.0;
        if (l < k) { x0 = sa[l][p]; x1 = sa[l][q]; }
        __syncwarp();
        if (l < k) { sa[l][p] = c * x0 - sn * x1; sa[l][q] = sn * x0 + c * x1; }
        __syncwarp();
        if (l < k) { x0 = sa[p][l]; x1 = sa[q][l]; }
        __syncwarp();
        if (l < k) {
          sa[p][l] = c * x0 - sn * x1;
          sa[q][l] = sn * x0 + c * x1;
          const double v0 = sv[l][p], v1 = sv[l][q];
          sv[l][p] = c * v0 - sn * v1;
          sv[l][q] = sn * v0 + c * v1;
        }
        __syncwarp();
      }
  }
  double lmax = 0.0;
  for (int i = 0; i < k; ++i) lmax = fmax(lmax, sa[i][i]);
  // gamma_j (lane j) = sum_i [lambda_i kept] v_ji (v_i . b) / lambda_i
  double g = 0.0;
  bool ok = isfinite(lmax);
  if (ok && lmax > 0.0 && l < k) {
    for (int i = 0; i < k; ++i) {
      const double li = sa[i][i];
      if (!(li > 1e-14 * lmax)) continue;
      double vb = 0.0;
      for (int j = 0; j < k; ++j) vb += sv[j][i] * sb[j];
      g += sv[l][i] * (vb / li);
    }
  }
  ok = __all_sync(0xffffffffu, ok && (l >= k || isfinite(g)));
  if (!ok) {  // the plain step; the history restarts from the last pair
    if (l == 0) {
      aa->k = 0;
      aa->slot_next = 0;
      aa->nmix = 0;
    }
    return;
  }
  if (l < k) aa->gamma[l] = g;
  if (l == 0) aa->nmix = k;
}

// f = g - x; with a previous pair, the new column dF = f - f_prev and
// dG = g - g_prev goes to slot slot_next; (f, g) become the previous pair.
// Per-block partial sums of <dF_j, dF_new> and <dF_j, f> over the columns
// valid after this update; the last block to finish sums them, updates the
// Gram matrix and solves the least-squares problem of the mix.
constexpr int kAaThreads = 256, kAaWarps = kAaThreads / 32;
// K: the history depth m, compile-time so that only m accumulator pairs
// live in registers
template <int K>
__global__ void __launch_bounds__(kAaThreads) ls2d_aa_update_kernel(const Ls2dRep* reps, const Ls2dState* st,
                                                                    const int* sel, double* buf, Ls2dAA* aa, int m,
                                                                    double* part) {
  __shared__ double wred[kAaWarps][2 * kAaMax];
  __shared__ double lred[kAaThreads / (2 * kAaMax)][2 * kAaMax];
  __shared__ double sums[2 * kAaMax];
  __shared__ double sa[kAaMax][kAaMax], sv[kAaMax][kAaMax];
  __shared__ int s_last;
  const int r = sel[0];
  const Ls2dRep& R = reps[r];
  if (aa_skip(st[r])) return;
  const long long N = R.N, n3 = 3 * N;
  const int have_prev = aa->have_prev;
  const int slot = have_prev ? aa->slot_next : -1;
  const int ncols = have_prev ? min(aa->k + 1, m) : aa->k;
  const double* x = buf;
  double* fp = buf + n3;
  double* gp = buf + 2 * n3;
  double* dF = buf + 3 * n3;
  double* dG = dF + (size_t)m * n3;
  double an[K], ar[K];
#pragma unroll
  for (int j = 0; j < K; ++j) { an[j] = 0.0; ar[j] = 0.0; }
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n3; i += (long long)gridDim.x * blockDim.x) {
    const double w = i >= 2 * N ? 2.0 : 1.0;
    const double gi = R.eps[i], fi = gi - x[i];
    double df = 0.0;
    if (have_prev) {
      df = fi - fp[i];
      dF[(size_t)slot * n3 + i] = df;
      dG[(size_t)slot * n3 + i] = gi - gp[i];
    }
    fp[i] = fi;
    gp[i] = gi;
#pragma unroll
    for (int j = 0; j < K; ++j)
      if (j < ncols) {
        const double c = w * (j == slot ? df : dF[(size_t)j * n3 + i]);
        an[j] += c * df;
        ar[j] += c * fi;
      }
  }
  // block partials in a fixed order: warp trees, then the warps in order
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < K; ++j)
    if (j < ncols) {
      const double a = warp_sum(an[j]), b = warp_sum(ar[j]);
      if (lane == 0) { wred[wid][j] = a; wred[wid][kAaMax + j] = b; }
    }
  __syncthreads();
  constexpr int Q = 2 * kAaMax;
  if (threadIdx.x < Q && threadIdx.x % kAaMax < ncols) {
    double t = 0.0;
    for (int w = 0; w < kAaWarps; ++w) t += wred[w][threadIdx.x];
    part[(size_t)blockIdx.x * Q + threadIdx.x] = t;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int t = atomicInc(&aa->ctr, gridDim.x - 1);  // self-resetting
    s_last = t == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // the last block: sums over the blocks (value q = thread % Q, blocks in
  // strides of the thread's group, then the groups in order)
  const int nb = gridDim.x;
  {
    const int q = threadIdx.x % Q, g0 = threadIdx.x / Q;
    double a = 0.0;
    if (q % kAaMax < ncols)
      for (int b = g0; b < nb; b += kAaThreads / Q) a += __ldcg(&part[(size_t)b * Q + q]);
    lred[g0][q] = a;
  }
  __syncthreads();
  if (threadIdx.x < Q) {
    double t = 0.0;
    for (int g = 0; g < kAaThreads / Q; ++g) t += lred[g][threadIdx.x];
    sums[threadIdx.x] = t;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  if (threadIdx.x == 0) {
    if (have_prev) {
      for (int j = 0; j < ncols; ++j) {
        aa->A[slot][j] = sums[j];
        aa->A[j][slot] = sums[j];
      }
      aa->k = ncols;
      aa->slot_next = (slot + 1) % m;
    }
    aa->have_prev = 1;
    aa->nmix = 0;
  }
  __syncwarp();
  if (ncols == 0) return;
  int fast = 0;
  if (threadIdx.x == 0) fast = aa_lstsq_cholesky(aa, ncols, sums + kAaMax) ? 1 : 0;
  if (__shfl_sync(0xffffffffu, fast, 0)) return;
  aa_lstsq_warp(aa, ncols, sa, sv, sums + kAaMax);
}


}  // namespace mgk

// ================================================================== plan ===
using namespace mgk;

namespace {

constexpr int kPerVoxelBlocks = 256;  // G: CTAs per replica for per-voxel kernels

int grid_blocks(long long maxN) {
  long long b = (maxN + kThreads - 1) / kThreads;
  if (b > kPerVoxelBlocks) b = kPerVoxelBlocks;
  if (b < 1) b = 1;
  return (int)b;
}

// columns per CTA: largest power of two <= 8 whose double-buffered tile fits
// `cap` bytes (keeps several CTAs resident per SM)
int pick_tc(int nx, size_t csz, size_t cap) {
  int tc = 8;
  while (tc > 1 && 2 * 3 * (size_t)tc * nx * csz > cap) tc >>= 1;
  return tc;
}

}  // namespace

// One launch group of a solve: the selected replicas of one shape on the
// register-FFT kernels, or every other replica on the CTA-wide passes (ky
// null), which find their replica in work maps.
struct Grp2 {
  const Ls2Line *kx = nullptr, *ky = nullptr, *kx32 = nullptr, *ky32 = nullptr;
  const int* sel = nullptr;  // the group's slice of the selection (device)
  int n = 0;                 // replicas
  int nx = 0, nyh = 0;
  int wr = 0, wc = 0, wc32 = 0;  // narrow or wide forms
  const int *row_map = nullptr, *row_local = nullptr, *col_map = nullptr, *col_local = nullptr;
  int rows = 0, cols = 0;    // CTA-wide: items over its replicas
  int lead = 0;              // counts the loop bodies
  Ls2dCtl* ctl = nullptr;    // its loop's control block
};

struct Loop2 {
  const Ls2dRep* reps = nullptr;
  Ls2dState* st = nullptr;
  double* part = nullptr;
  unsigned int* ctr = nullptr;
  Ls2dCtl* ctl = nullptr;                     // one for the graph's loop, or one per group (host_loop)
  size_t rs = 0, cs = 0, rs32 = 0, cs32 = 0;  // shared memory of the CTA-wide passes
  const int* sel = nullptr;
  int nsel = 0, G = 0, law = 0;
  // Anderson mixing (FP64 loop of a one-replica selection; aa_m = 0: none)
  int aa_m = 0, aa_nb = 0;
  double* aa_buf = nullptr;
  Ls2dAA* aa = nullptr;
  double* aa_part = nullptr;
  std::vector<Grp2> grp;
};

struct mgk_ls2d_plan {
  int nrep = 0;
  int plane_mode = 0, prec = 0;
  long long maxN = 0;
  size_t row_smem = 0, col_smem = 0;      // CTA-wide FP64 iteration kernels
  size_t row_smem32 = 0, col_smem32 = 0;  // and FP32
  // Kernel family: 256/512/1024 asks for the register-FFT kernels, 0 for the
  // CTA-wide passes where every side is one of the lengths 64 .. 1024 of
  // warp_fft_len (fast_nat: its smallest family); a plan with other sides has
  // family 0 only, which then means each replica's natural kernels.
  int fast = 0, fast_nat = 0;
  std::vector<int> order;                 // the last selection in launch order
  std::vector<char> line_ok;              // replicas whose sides both have a register-FFT kernel
  int law = 0;                            // 1: secant degradation law, 2: Rose law
  double law_a = 0, law_b = 0;            // the law's parameters (set_secant, set_rose)
  int law_ps = 0;
  std::vector<Ls2dRep> reps;      // host copy (static part)
  std::vector<char> has_material;
  Ls2dRep* h_reps = nullptr;      // pinned staging of the table
  int* h_maps = nullptr;          // pinned staging: row_map, row_local, col_map, col_local, sel
  Ls2dCtl* h_ctl = nullptr;       // 2 nctl: staging, and the host-driven loop's copies
  int nctl = 0;                   // control blocks: the plan's distinct shapes, and one
  Ls2dState* h_state = nullptr;
  cudaEvent_t staged = nullptr;   // last upload from the staging buffers
  bool staged_pending = false;
  Ls2dRep* d_reps = nullptr;
  Ls2dState* d_st = nullptr;
  Ls2dCtl* d_ctl = nullptr;
  int* d_maps = nullptr;
  unsigned int* d_repctr = nullptr;
  double* d_part = nullptr;
  double* d_mat_part = nullptr;   // partials of the material kernel, each replica's from mat_off
  std::vector<size_t> mat_off;
  size_t part_doubles = 0;
  int total_row_items = 0, total_col_items = 0;
  unsigned int* d_voxctr = nullptr;  // arrival counters of the per-voxel kernels, per replica
  std::vector<void*> allocations;
  // spectra of all replicas, one slab
  void* spec_slab = nullptr;
  size_t spec_bytes = 0;
  // instantiated loop graphs by the selection's shapes and widths (its
  // signature): a serving loop selects varying numbers of replicas
  struct GraphEntry {
    std::vector<int> sig;
    int cap;
    cudaGraph_t g;
    cudaGraphExec_t x;
  };
  std::vector<GraphEntry> gcache;
  int graph_mode = 1;  // 0: host-driven loop
  std::vector<std::pair<std::vector<int>, int>> sights;  // uses of selections of several shapes without a graph
  Loop2 last;          // the last call's launches (the timing hook repeats its stages)
  // Anderson mixing inside the loop (one replica per solve): depth, ring
  // buffer of (3 + 2 m) strain fields, state and per-block partial sums
  int aa_m = 0;
  double* aa_buf = nullptr;
  size_t aa_doubles = 0;
  Ls2dAA* d_aa = nullptr;
  double* aa_part = nullptr;
  int aa_nb = 0;
};

static int plan_alloc(mgk_ls2d_t p, void** ptr, size_t bytes) {
  if (cudaMalloc(ptr, bytes) != cudaSuccess) {
    cudaGetLastError();
    set_error("mgk_ls2d: cudaMalloc of %zu bytes failed", bytes);
    return MGK_OOM;
  }
  p->allocations.push_back(*ptr);
  return MGK_OK;
}

static void ls2d_drop_graphs(mgk_ls2d_t p) {
  for (auto& e : p->gcache) {
    cudaGraphExecDestroy(e.x);
    cudaGraphDestroy(e.g);
  }
  p->gcache.clear();
}

// whether a replica runs on the register-FFT kernels under the plan's family
static bool ls2d_on_line(mgk_ls2d_t p, int r) { return p->line_ok[r] && (p->fast != 0 || p->fast_nat == 0); }

template <typename TS, typename TC>
static int ls2d_set_attrs(size_t row_smem, size_t col_smem) {
  MGK_CUDA(raise_smem((const void*)ls2d_row_kernel<TS, TC, true, true>, (int)row_smem));
  MGK_CUDA(raise_smem((const void*)ls2d_row_kernel<TS, TC, false, true>, (int)row_smem));
  MGK_CUDA(raise_smem((const void*)ls2d_row_kernel<TS, TC, true, false>, (int)row_smem));
  MGK_CUDA(raise_smem((const void*)ls2d_row_kernel<TS, TC, false, false>, (int)row_smem));
  MGK_CUDA(raise_smem((const void*)ls2d_col_kernel<TS, TC>, (int)col_smem));
  return MGK_OK;
}

extern "C" int mgk_ls2d_destroy(mgk_ls2d_t p) {
  if (!p) return MGK_OK;
  ls2d_drop_graphs(p);
  if (p->staged) cudaEventDestroy(p->staged);
  for (void* a : p->allocations) cudaFree(a);
  if (p->aa_buf) cudaFree(p->aa_buf);
  if (p->d_aa) cudaFree(p->d_aa);
  if (p->aa_part) cudaFree(p->aa_part);
  if (p->h_reps) cudaFreeHost(p->h_reps);
  if (p->h_maps) cudaFreeHost(p->h_maps);
  if (p->h_ctl) cudaFreeHost(p->h_ctl);
  if (p->h_state) cudaFreeHost(p->h_state);
  delete p;
  return MGK_OK;
}

extern "C" int mgk_ls2d_create_batch(int nrep, const int* nxs, const int* nys, int plane_mode, int precision,
                                     mgk_ls2d_t* out) {
  MGK_REQUIRE(out != nullptr, "mgk_ls2d_create_batch: null output handle");
  *out = nullptr;
  MGK_REQUIRE(nrep >= 1 && nrep <= 65535 && nxs && nys, "mgk_ls2d_create_batch: bad replica count");
  MGK_REQUIRE(plane_mode == MGK_PLANE_STRAIN || plane_mode == MGK_PLANE_STRESS,
              "mgk_ls2d_create: plane_mode must be 0 (strain) or 1 (stress)");
  MGK_REQUIRE(precision == MGK_FP64 || precision == MGK_MIXED, "mgk_ls2d_create: bad precision");
  for (int r = 0; r < nrep; ++r) {
    FftLen f;
    MGK_REQUIRE(fft_schedule(nxs[r], &f) && fft_schedule(nys[r], &f) && nxs[r] % 2 == 0,
                "mgk_ls2d_create: grid %dx%d unsupported (each side 2^a 3^b up to 4096, nx even)", nxs[r],
                nys[r]);
    MGK_REQUIRE(2 * 3 * (size_t)nys[r] * sizeof(double2) <= 220 * 1024 &&
                    2 * 3 * (size_t)pick_tc(nxs[r], sizeof(double2), 64 * 1024) * nxs[r] * sizeof(double2) <=
                        220 * 1024,
                "mgk_ls2d_create: grid too large for the shared-memory FFT");
  }
  mgk_ls2d_t p = new mgk_ls2d_plan();
  p->nrep = nrep;
  p->plane_mode = plane_mode;
  p->prec = precision;
  const bool mixed = precision == MGK_MIXED;
  const size_t c64 = sizeof(double2);
  auto fail = [&](int s) { mgk_ls2d_destroy(p); return s; };
  p->reps.resize(nrep);
  p->has_material.assign(nrep, 0);
  const char* env = getenv("MGK_FAST");
  const bool no_line = env && env[0] == '0';
  {
    bool fast = true;
    int side = 0;
    for (int r = 0; r < nrep; ++r) {
      fast = fast && warp_fft_len(nxs[r]) && warp_fft_len(nys[r]);
      side = std::max(side, std::max(nxs[r], nys[r]));
    }
    p->fast_nat = fast ? (side > 512 ? 1024 : side > 256 ? 512 : 256) : 0;
    p->fast = no_line ? 0 : p->fast_nat;
  }
  p->line_ok.assign(nrep, 0);
  std::vector<size_t> spec_off(nrep, 0);
  size_t row_smem = 0, col_smem = 0, row_smem32 = 0, col_smem32 = 0;
  for (int r = 0; r < nrep; ++r) {
    const int nx = nxs[r], ny = nys[r];
    Ls2dRep& R = p->reps[r];
    memset(&R, 0, sizeof(R));
    p->line_ok[r] = !no_line && ls2_line(nx, kLs2Fp64) && ls2_line(ny, kLs2Fp64);
    R.nx = nx; R.ny = ny; R.nyh = ny / 2 + 1;
    R.ld = p->line_ok[r] ? ls2_ld(ny) : R.nyh;  // register-FFT tiles read rows of 64 aligned bytes
    R.N = (long long)nx * ny;
    R.tc = pick_tc(nx, c64, 64 * 1024);
    R.row_items = nx / 2;
    R.col_items = (R.nyh + R.tc - 1) / R.tc;
    fft_schedule(nx, &R.fx64);
    fft_schedule(ny, &R.fy64);
    R.fx32 = R.fx64;
    R.fy32 = R.fy64;
    R.fx64.tw = twiddles(nx, MGK_FP64);
    R.fy64.tw = twiddles(ny, MGK_FP64);
    if (!R.fx64.tw || !R.fy64.tw) return fail(MGK_OOM);
    if (mixed) {
      R.fx32.tw = twiddles(nx, 1 /* float table */);
      R.fy32.tw = twiddles(ny, 1 /* float table */);
      if (!R.fx32.tw || !R.fy32.tw) return fail(MGK_OOM);
    }
    if (p->line_ok[r]) {
      const int n[2] = {nx, ny};
      for (int q = 0; q < 2; ++q) {
        R.rtw[q] = reinterpret_cast<const double2*>(twiddles_reg(n[q], MGK_FP64));
        if (mixed) R.rtw32[q] = reinterpret_cast<const float2*>(twiddles_reg(n[q], MGK_MIXED));
        if (!R.rtw[q] || (mixed && !R.rtw32[q])) return fail(MGK_OOM);
      }
    }
    row_smem = std::max(row_smem, 2 * 3 * (size_t)ny * c64);
    col_smem = std::max(col_smem, 2 * 3 * (size_t)R.tc * nx * c64);
    row_smem32 = row_smem / 2;
    col_smem32 = col_smem / 2;
    p->maxN = std::max(p->maxN, R.N);
    p->total_row_items += R.row_items;
    p->total_col_items += R.col_items;
    void* f = nullptr;
    int st = plan_alloc(p, &f, sizeof(double) * R.N * 10);
    if (st) return fail(st);
    double* d = reinterpret_cast<double*>(f);
    R.mu = d; R.lam = d + R.N; R.eps = d + 2 * R.N; R.ep = d + 5 * R.N; R.epa = nullptr;
    // spectra of all replicas sit in one slab (assigned after the loop)
    spec_off[r] = p->spec_bytes;
    p->spec_bytes += (3 * (size_t)nx * R.ld * c64 + 255) / 256 * 256;
    if (mixed) {
      void* g = nullptr;
      st = plan_alloc(p, &g, sizeof(float) * R.N * 8);
      if (st) return fail(st);
      float* fl = reinterpret_cast<float*>(g);
      R.mu32 = fl; R.lam32 = fl + R.N; R.eps32 = fl + 2 * R.N; R.ep32 = fl + 5 * R.N;
    }
  }
  {
    void* slab = nullptr;
    int st = plan_alloc(p, &slab, p->spec_bytes);
    if (st) return fail(st);
    p->spec_slab = slab;
    for (int r = 0; r < nrep; ++r) p->reps[r].spec = reinterpret_cast<char*>(slab) + spec_off[r];
  }
  p->row_smem = row_smem;
  p->col_smem = col_smem;
  p->row_smem32 = row_smem32;
  p->col_smem32 = col_smem32;
  int st = MGK_OK;
  const int G = grid_blocks(p->maxN);
  p->part_doubles = std::max((size_t)2 * p->total_row_items, (size_t)nrep * G * 8);
  void* v = nullptr;
  if ((st = plan_alloc(p, &v, sizeof(double) * p->part_doubles))) return fail(st);
  p->d_part = reinterpret_cast<double*>(v);
  // two sums per CTA: replicas may be set on different streams, so each has its own
  size_t mat = 0;
  for (int r = 0; r < nrep; ++r) {
    p->mat_off.push_back(mat);
    mat += 2 * (size_t)grid_blocks(p->reps[r].N);
  }
  if ((st = plan_alloc(p, &v, sizeof(double) * mat))) return fail(st);
  p->d_mat_part = reinterpret_cast<double*>(v);
  if ((st = plan_alloc(p, &v, sizeof(Ls2dRep) * nrep))) return fail(st);
  p->d_reps = reinterpret_cast<Ls2dRep*>(v);
  if ((st = plan_alloc(p, &v, sizeof(Ls2dState) * nrep))) return fail(st);
  p->d_st = reinterpret_cast<Ls2dState*>(v);
  {
    std::set<std::pair<int, int>> shapes;
    for (int r = 0; r < nrep; ++r) shapes.insert({nxs[r], nys[r]});
    p->nctl = (int)shapes.size() + 1;
  }
  if ((st = plan_alloc(p, &v, sizeof(Ls2dCtl) * p->nctl))) return fail(st);
  p->d_ctl = reinterpret_cast<Ls2dCtl*>(v);
  const size_t nmaps = 2 * (size_t)p->total_row_items + 2 * (size_t)p->total_col_items + nrep;
  if ((st = plan_alloc(p, &v, sizeof(int) * nmaps))) return fail(st);
  p->d_maps = reinterpret_cast<int*>(v);
  if ((st = plan_alloc(p, &v, sizeof(unsigned int) * 2 * nrep))) return fail(st);
  p->d_repctr = reinterpret_cast<unsigned int*>(v);
  p->d_voxctr = p->d_repctr + nrep;
  if (cudaMemset(p->d_repctr, 0, sizeof(unsigned int) * 2 * nrep) != cudaSuccess ||
      cudaMemset(p->d_st, 0, sizeof(Ls2dState) * nrep) != cudaSuccess ||
      cudaMemset(p->d_ctl, 0, sizeof(Ls2dCtl) * p->nctl) != cudaSuccess)
    return fail(MGK_CUDA_ERROR);
  if (cudaMallocHost(&p->h_reps, sizeof(Ls2dRep) * nrep) != cudaSuccess ||
      cudaMallocHost(&p->h_maps, sizeof(int) * nmaps) != cudaSuccess ||
      cudaMallocHost(&p->h_ctl, sizeof(Ls2dCtl) * 2 * p->nctl) != cudaSuccess ||
      cudaMallocHost(&p->h_state, sizeof(Ls2dState) * nrep) != cudaSuccess)
    return fail(MGK_OOM);
  if (cudaEventCreateWithFlags(&p->staged, cudaEventDisableTiming) != cudaSuccess) return fail(MGK_CUDA_ERROR);
  memcpy(p->h_reps, p->reps.data(), sizeof(Ls2dRep) * nrep);
  if (cudaMemcpy(p->d_reps, p->h_reps, sizeof(Ls2dRep) * nrep, cudaMemcpyHostToDevice) != cudaSuccess)
    return fail(MGK_CUDA_ERROR);
  *out = p;
  return MGK_OK;
}

extern "C" int mgk_ls2d_create(int nx, int ny, int plane_mode, int precision, mgk_ls2d_t* out) {
  return mgk_ls2d_create_batch(1, &nx, &ny, plane_mode, precision, out);
}

// wait until the previous upload from the pinned staging buffers has run
static int staging_wait(mgk_ls2d_t p) {
  if (p->staged_pending) {
    MGK_CUDA(cudaEventSynchronize(p->staged));
    p->staged_pending = false;
  }
  return MGK_OK;
}

static int ls2d_set_fields(mgk_ls2d_t p, int rep, const double* E, const double* nu, const double* epsp,
                           int set_moduli, cudaStream_t s) {
  Ls2dRep& R = p->reps[rep];
  const bool want_epa = epsp != nullptr;
  if (want_epa != (R.epa != nullptr)) {
    R.epa = want_epa ? R.mu + 8 * R.N : nullptr;
    int st = staging_wait(p);
    if (st) return st;
    p->h_reps[rep] = R;
    MGK_CUDA(cudaMemcpyAsync(&p->d_reps[rep], &p->h_reps[rep], sizeof(Ls2dRep), cudaMemcpyHostToDevice, s));
    MGK_CUDA(cudaEventRecord(p->staged, s));
    p->staged_pending = true;
  }
  const int grid = grid_blocks(R.N);
  ls2d_material_kernel<<<grid, kThreads, 0, s>>>(p->d_reps, p->d_st, rep, E, nu, epsp, p->plane_mode, set_moduli,
                                                 set_moduli == 2 ? (p->law == 2 ? 2 : 1) : 0, p->law_b,
                                                 p->d_mat_part + p->mat_off[rep], p->d_voxctr + rep);
  MGK_CUDA(cudaGetLastError());
  return MGK_OK;
}

extern "C" int mgk_ls2d_set_material_rep(mgk_ls2d_t p, int rep, const double* E, const double* nu,
                                         const double* epsp, mgk_stream_t stream) {
  MGK_REQUIRE(p && E && nu, "mgk_ls2d_set_material: null argument");
  MGK_REQUIRE(rep >= 0 && rep < p->nrep, "mgk_ls2d_set_material: replica %d out of range", rep);
  int st = ls2d_set_fields(p, rep, E, nu, epsp, 1, (cudaStream_t)stream);
  if (st == MGK_OK) p->has_material[rep] = 1;
  return st;
}

extern "C" int mgk_ls2d_set_material(mgk_ls2d_t p, const double* E, const double* nu, const double* epsp,
                                     mgk_stream_t stream) {
  return mgk_ls2d_set_material_rep(p, 0, E, nu, epsp, stream);
}

extern "C" int mgk_ls2d_set_lame_rep(mgk_ls2d_t p, int rep, const double* lam, const double* mu,
                                     const double* epsp, mgk_stream_t stream) {
  MGK_REQUIRE(p && lam && mu, "mgk_ls2d_set_lame: null argument");
  MGK_REQUIRE(rep >= 0 && rep < p->nrep, "mgk_ls2d_set_lame: replica %d out of range", rep);
  int st = ls2d_set_fields(p, rep, lam, mu, epsp, 2, (cudaStream_t)stream);
  if (st == MGK_OK) p->has_material[rep] = 1;
  return st;
}

// switches every replica of the plan to law (a, b, ps); cached loop graphs
// hold the previous law's row kernel and are dropped
static int ls2d_set_law(mgk_ls2d_t p, int law, double a, double b, int ps, const double* lp = nullptr) {
  for (auto& R : p->reps) {
    R.law = law; R.law_a = a; R.law_b = b; R.law_ps = ps;
    for (int q = 0; q < 11; ++q) R.lp[q] = lp ? lp[q] : 0.0;
  }
  p->law_a = a; p->law_b = b; p->law_ps = ps;
  if (law != p->law) {
    ls2d_drop_graphs(p);
    p->law = law;
  }
  return MGK_OK;
}

extern "C" int mgk_ls2d_set_secant(mgk_ls2d_t p, double d, double k) {
  MGK_REQUIRE(p, "mgk_ls2d_set_secant: null plan");
  MGK_REQUIRE(d >= 0.0 && d <= 1.0 && k >= 0.0 && isfinite(k), "mgk_ls2d_set_secant: need 0 <= d <= 1, k >= 0");
  MGK_REQUIRE(d == 0.0 || p->prec == MGK_FP64, "mgk_ls2d_set_secant: the secant law runs in FP64 plans only");
  return ls2d_set_law(p, d != 0.0 ? 1 : 0, d, k, 0);
}

extern "C" int mgk_ls2d_set_rose(mgk_ls2d_t p, double eta, double floor_fraction, int plane_stress) {
  MGK_REQUIRE(p, "mgk_ls2d_set_rose: null plan");
  MGK_REQUIRE(eta >= 0.0 && isfinite(eta) && floor_fraction >= 0.0 && floor_fraction <= 1.0,
              "mgk_ls2d_set_rose: need eta >= 0, 0 <= floor_fraction <= 1");
  MGK_REQUIRE(p->prec == MGK_FP64, "mgk_ls2d_set_rose: the Rose law runs in FP64 plans only");
  return ls2d_set_law(p, 2, eta, floor_fraction, plane_stress ? 1 : 0);
}

extern "C" int mgk_ls2d_set_landau(mgk_ls2d_t p, const double* v, int capping, double e_cap, double tangent_ratio,
                                   double smooth_power, int plane_stress) {
  MGK_REQUIRE(p && v, "mgk_ls2d_set_landau: null argument");
  MGK_REQUIRE(p->prec == MGK_FP64, "mgk_ls2d_set_landau: the Landau law runs in FP64 plans only");
  MGK_REQUIRE(capping >= 0 && capping <= 2, "mgk_ls2d_set_landau: capping must be 0, 1 or 2");
  MGK_REQUIRE(!capping || (e_cap > 0.0 && isfinite(e_cap) && isfinite(tangent_ratio) &&
                           (capping != 2 || (smooth_power > 0.0 && isfinite(smooth_power)))),
              "mgk_ls2d_set_landau: need e_cap > 0 (and smooth_power > 0 for smooth capping)");
  double lp[11];
  for (int q = 0; q < 7; ++q) {
    MGK_REQUIRE(isfinite(v[q]), "mgk_ls2d_set_landau: non-finite coefficient");
    lp[q] = v[q];
  }
  lp[7] = capping; lp[8] = e_cap; lp[9] = tangent_ratio; lp[10] = smooth_power;
  return ls2d_set_law(p, 3, 0.0, 0.0, plane_stress ? 1 : 0, lp);
}

extern "C" int mgk_ls2d_set_e33_out(mgk_ls2d_t p, int rep, double* e33) {
  MGK_REQUIRE(p && rep >= 0 && rep < p->nrep, "mgk_ls2d_set_e33_out: bad argument");
  p->reps[rep].out_e33 = e33;
  return MGK_OK;
}

extern "C" int mgk_ls2d_set_anderson(mgk_ls2d_t p, int m) {
  MGK_REQUIRE(p, "mgk_ls2d_set_anderson: null plan");
  MGK_REQUIRE(m >= 0 && m <= kAaMax, "mgk_ls2d_set_anderson: depth must be 0..%d", kAaMax);
  MGK_REQUIRE(m == 0 || p->prec == MGK_FP64, "mgk_ls2d_set_anderson: Anderson mixing runs in FP64 plans only");
  if (m == p->aa_m) return MGK_OK;
  int rc = staging_wait(p);
  if (rc) return rc;
  ls2d_drop_graphs(p);  // loop graphs hold the ring's address: rebuild them
  if (m > 0) {
    const size_t need = (size_t)(3 + 2 * m) * 3 * (size_t)p->maxN;
    if (need > p->aa_doubles) {
      MGK_CUDA(cudaDeviceSynchronize());  // the old ring may be in use by queued work
      if (p->aa_buf) cudaFree(p->aa_buf);
      p->aa_buf = nullptr;
      p->aa_doubles = 0;
      if (cudaMalloc((void**)&p->aa_buf, need * sizeof(double)) != cudaSuccess) {
        cudaGetLastError();
        p->aa_buf = nullptr;
        p->aa_m = 0;
        set_error("mgk_ls2d_set_anderson: cudaMalloc of %zu bytes failed", need * sizeof(double));
        return MGK_OOM;
      }
      p->aa_doubles = need;
    }
    if (!p->d_aa) {
      int dev = 0, sms = 148;
      if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      p->aa_nb = std::max(1, std::min(8 * sms, ceil_div(3 * p->maxN, kAaThreads)));
      // zeroed (the legacy stream waited for): the timing hooks run first passes before
      // any solve has set the mix
      if (cudaMalloc((void**)&p->d_aa, sizeof(Ls2dAA)) != cudaSuccess ||
          cudaMemset(p->d_aa, 0, sizeof(Ls2dAA)) != cudaSuccess || cudaStreamSynchronize(0) != cudaSuccess ||
          cudaMalloc((void**)&p->aa_part, sizeof(double) * 2 * kAaMax * p->aa_nb) != cudaSuccess) {
        cudaGetLastError();
        set_error("mgk_ls2d_set_anderson: cudaMalloc failed");
        p->aa_m = 0;
        return MGK_OOM;
      }
    }
  }
  p->aa_m = m;
  return MGK_OK;
}

extern "C" int mgk_ls2d_set_eigenstrain_rep(mgk_ls2d_t p, int rep, const double* epsp, mgk_stream_t stream) {
  MGK_REQUIRE(p && rep >= 0 && rep < p->nrep && p->has_material[rep],
              "mgk_ls2d_set_eigenstrain: replica has no material");
  return ls2d_set_fields(p, rep, nullptr, nullptr, epsp, 0, (cudaStream_t)stream);
}

extern "C" int mgk_ls2d_set_eigenstrain(mgk_ls2d_t p, const double* epsp, mgk_stream_t stream) {
  return mgk_ls2d_set_eigenstrain_rep(p, 0, epsp, stream);
}

// ------------------------------------------------------------- the loop ---

struct Launch2 {
  const void* fn;
  dim3 grid, block;
  size_t smem;
};

// Row stages of a group: 0 an iteration's, 1 the first of a phase (or of a
// mixed iterate), 2 the first after the FP32 phase; -1 the column stage.
enum { kCol = -1, kRow = 0, kFirst = 1, kPromote = 2 };

// Calls f(launch, args) with a stage's launch and arguments; final: as
// ls2d_decide's.
template <typename F>
static cudaError_t with_stage2(Loop2& a, Grp2& g, int stage, bool f32, int final, cudaGraphConditionalHandle h, int use,
                               int cap, F f) {
  if (g.ky) {
    const Ls2Line *kx = f32 ? g.kx32 : g.kx, *ky = f32 ? g.ky32 : g.ky;
    if (stage == kCol) {
      const int w = f32 ? g.wc32 : g.wc;
      void* x[] = {&a.reps, &a.st, &g.sel};
      return f(Launch2{kx->col[w], dim3(g.n * ceil_div(g.nyh, kx->cols[w])), dim3(kx->c_threads[w]),
                       (size_t)kx->c_bytes[w]}, x);
    }
    const int w = g.wr;
    void* x[] = {&a.reps, &a.st, &g.sel, &a.part, &a.ctr, &g.ctl, &h, &use, &cap, &g.lead, &stage, &final};
    return f(Launch2{ky->row[f32 ? 0 : a.law][w], dim3(g.n * ceil_div(g.nx / 2, ky->pairs[w])),
                     dim3(ky->r_threads[w]), (size_t)ky->r_bytes[w]}, x);
  }
  if (stage == kCol) {
    void* x[] = {&a.reps, &a.st, &g.col_map, &g.col_local};
    return f(Launch2{f32 ? (const void*)ls2d_col_kernel<float, float> : (const void*)ls2d_col_kernel<double, double>,
                     dim3(g.cols), dim3(kThreads), f32 ? a.cs32 : a.cs}, x);
  }
  const void* fn = f32 ? (stage == kRow ? (final ? (const void*)ls2d_row_kernel<float, float, true, true>
                                                 : (const void*)ls2d_row_kernel<float, float, true, false>)
                                        : (const void*)ls2d_row_kernel<float, float, false, false>)
                       : (stage == kRow ? (const void*)ls2d_row_kernel<double, double, true, true>
                                        : (const void*)ls2d_row_kernel<double, double, false, true>);
  void* x[] = {&a.reps, &a.st, &g.row_map, &g.row_local, &a.part, &a.ctr, &g.ctl, &h, &use, &cap};
  return f(Launch2{fn, dim3(g.rows), dim3(kThreads), f32 ? a.rs32 : a.rs}, x);
}

static int launch2(Loop2& a, Grp2& g, int stage, bool f32, int final, cudaStream_t s) {
  MGK_CUDA(with_stage2(a, g, stage, f32, final, 0, 0, 0, [&](const Launch2& L, void** args) {
    return cudaLaunchKernel(L.fn, L.grid, L.block, args, L.smem, s);
  }));
  return MGK_OK;
}
static int launch2(Loop2& a, int stage, bool f32, int final, cudaStream_t s) {
  for (Grp2& g : a.grp)
    if (int rc = launch2(a, g, stage, f32, final, s)) return rc;
  return MGK_OK;
}

// the history kernel of depth m (1..kAaMax)
static void* aa_update_fn(int m) {
  switch (m) {
    case 1: return (void*)ls2d_aa_update_kernel<1>;
    case 2: return (void*)ls2d_aa_update_kernel<2>;
    case 3: return (void*)ls2d_aa_update_kernel<3>;
    case 4: return (void*)ls2d_aa_update_kernel<4>;
    case 5: return (void*)ls2d_aa_update_kernel<5>;
    case 6: return (void*)ls2d_aa_update_kernel<6>;
    case 7: return (void*)ls2d_aa_update_kernel<7>;
    default: return (void*)ls2d_aa_update_kernel<8>;
  }
}

static int launch_body(Loop2& a, Grp2& g, bool f32, cudaStream_t s) {
  int rc = launch2(a, g, kCol, f32, !f32, s);
  if (rc == MGK_OK) rc = launch2(a, g, kRow, f32, !f32, s);
  if (rc == MGK_OK && !f32 && a.aa_m > 0) {
    void* args[] = {&a.reps, &a.st, &a.sel, &a.aa_buf, &a.aa, &a.aa_m, &a.aa_part};
    MGK_CUDA(cudaLaunchKernel(aa_update_fn(a.aa_m), dim3(a.aa_nb), dim3(kAaThreads), args, 0, s));
    rc = launch2(a, g, kFirst, false, 1, s);  // the mix and tau of the mixed iterate
  }
  return rc;
}

static cudaError_t add_node2(cudaGraph_t g, cudaGraphNode_t* node, const cudaGraphNode_t* dep, size_t ndep,
                             const Launch2& L, void** args) {
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
static int add_while(cudaGraph_t g, cudaGraphNode_t* node, const cudaGraphNode_t* dep, size_t ndep, Loop2& a, bool f32,
                     int cap) {
  cudaGraphConditionalHandle h;
  MGK_CUDA(cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault));
  // cudaGraphNodeParams has no default constructor in C++: zeroed storage
  alignas(cudaGraphNodeParams) unsigned char raw[sizeof(cudaGraphNodeParams)];
  memset(raw, 0, sizeof(raw));
  cudaGraphNodeParams& cp = *reinterpret_cast<cudaGraphNodeParams*>(raw);
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  MGK_CUDA(cudaGraphAddNode(node, g, dep, ndep, &cp));
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  for (Grp2& gr : a.grp) {
    cudaGraphNode_t prev, next;
    MGK_CUDA(with_stage2(a, gr, kCol, f32, !f32, h, 1, cap, [&](const Launch2& L, void** args) {
      return add_node2(body, &prev, nullptr, 0, L, args);
    }));
    MGK_CUDA(with_stage2(a, gr, kRow, f32, !f32, h, 1, cap, [&](const Launch2& L, void** args) {
      return add_node2(body, &next, &prev, 1, L, args);
    }));
    if (f32 || a.aa_m == 0) continue;
    // Anderson history and least squares, then the mix and tau of the mixed
    // iterate in the first row pass (one replica, one group)
    cudaGraphNode_t hist, first;
    void* ah[] = {&a.reps, &a.st, &a.sel, &a.aa_buf, &a.aa, &a.aa_m, &a.aa_part};
    MGK_CUDA(add_node2(body, &hist, &next, 1, {aa_update_fn(a.aa_m), dim3(a.aa_nb), dim3(kAaThreads), 0}, ah));
    MGK_CUDA(with_stage2(a, gr, kFirst, false, 1, 0, 0, 0, [&](const Launch2& L, void** args) {
      return add_node2(body, &first, &hist, 1, L, args);
    }));
  }
  return MGK_OK;
}

// Graph of a selection: mixed plans run [phase-1 while, phase-2 set-up, first
// FP64 row pass] before the final while node.
static int build_graph(mgk_ls2d_t p, Loop2& a, int cap, cudaGraph_t* gout, cudaGraphExec_t* xout) {
  cudaGraph_t g = nullptr;
  MGK_CUDA(cudaGraphCreate(&g, 0));
  auto build = [&]() -> int {
    cudaGraphNode_t last;
    if (p->prec != MGK_MIXED) return add_while(g, &last, nullptr, 0, a, false, cap);
    cudaGraphNode_t w1, ph2;
    int rc = add_while(g, &w1, nullptr, 0, a, true, cap);
    if (rc) return rc;
    if (!a.grp[0].ky) {  // the CTA-wide replicas' FP64 field
      cudaGraphNode_t prom;
      void* ap[] = {&a.reps, &a.sel};
      MGK_CUDA(add_node2(g, &prom, &w1, 1, {(const void*)ls2d_promote_kernel, dim3(a.G, a.grp[0].n), dim3(kThreads), 0},
                         ap));
      w1 = prom;
    }
    void* ap2[] = {&a.st, &a.sel, &a.nsel, &a.ctl};
    MGK_CUDA(add_node2(g, &ph2, &w1, 1, {(const void*)ls2d_phase2_kernel, dim3(1), dim3(32), 0}, ap2));
    std::vector<cudaGraphNode_t> row0(a.grp.size());
    for (size_t i = 0; i < a.grp.size(); ++i)
      MGK_CUDA(with_stage2(a, a.grp[i], kPromote, false, 1, 0, 0, 0, [&](const Launch2& L, void** args) {
        return add_node2(g, &row0[i], &ph2, 1, L, args);
      }));
    return add_while(g, &last, row0.data(), row0.size(), a, false, cap);
  };
  int rc = build();
  cudaGraphExec_t x = nullptr;
  if (rc == MGK_OK && cudaGraphInstantiate(&x, g, 0) != cudaSuccess) rc = MGK_CUDA_ERROR;
  if (rc != MGK_OK) {
    cudaGraphDestroy(g);
    cudaGetLastError();
    return rc;
  }
  *gout = g;
  *xout = x;
  return MGK_OK;
}

// The loop driven from the host, from the first tau on; the caller's stream has
// drained when it returns.  Each group runs on a stream of its own (as far as there
// are side streams) with its own control block and phase.  The host launches kBodies iterations per group (body by
// body, the groups in turn) before it looks at the control blocks: a body too many is
// two launches that return at once.
static int host_loop(mgk_ls2d_t p, Loop2& a, int max_iter, cudaStream_t s) {
  constexpr int kBodies = 4;
  const bool mixed = p->prec == MGK_MIXED;
  const size_t G = a.grp.size();
  struct Run {
    cudaStream_t s;
    bool f32;
    int left;  // bodies of this phase yet to launch
  };
  std::vector<Run> run(G);
  int priority = 0;
  MGK_CUDA(cudaStreamGetPriority(s, &priority));
  const SideStreams side(G - 1, priority);
  auto loop = [&]() -> int {
    // the fork's event joins later: a wait means the record before it
    if (side.size()) MGK_CUDA(cudaEventRecord(side[0].done, s));
    for (size_t i = 0; i < side.size(); ++i) MGK_CUDA(cudaStreamWaitEvent(side[i].s, side[0].done, 0));
    for (size_t i = 0; i < G; ++i) {
      run[i] = {i > 0 && i <= side.size() ? side[i - 1].s : s, mixed, max_iter};
      if (int e = launch2(a, a.grp[i], kFirst, mixed, !mixed, run[i].s)) return e;
    }
    for (size_t open = G; open > 0;) {
      for (int b = 0; b < kBodies; ++b)
        for (size_t i = 0; i < G; ++i)
          if (run[i].left > 0) {
            if (int e = launch_body(a, a.grp[i], run[i].f32, run[i].s)) return e;
            --run[i].left;
          }
      for (size_t i = 0; i < side.size(); ++i) {
        MGK_CUDA(cudaEventRecord(side[i].done, side[i].s));
        MGK_CUDA(cudaStreamWaitEvent(s, side[i].done, 0));
      }
      Ls2dCtl* c = p->h_ctl + p->nctl;
      MGK_CUDA(cudaMemcpyAsync(c, a.ctl, sizeof(Ls2dCtl) * G, cudaMemcpyDeviceToHost, s));
      MGK_CUDA(cudaStreamSynchronize(s));
      open = 0;
      for (size_t i = 0; i < G; ++i) {
        if (c[i].error) {
          set_error("mgk_ls2d_solve: a bulk copy wait gave up (device timeout)");
          return MGK_TIMEOUT;
        }
        if (!c[i].any) run[i].left = 0;
        if (run[i].left == 0 && run[i].f32) {  // the FP32 phase is over: on to the FP64 iterations
          Grp2& g = a.grp[i];
          run[i].f32 = false;
          run[i].left = max_iter;
          if (!g.ky) ls2d_promote_kernel<<<dim3(a.G, g.n), kThreads, 0, run[i].s>>>(a.reps, g.sel);
          ls2d_phase2_kernel<<<1, 32, 0, run[i].s>>>(a.st, g.sel, g.n, g.ctl);
          MGK_CUDA(cudaGetLastError());
          if (int e = launch2(a, g, kPromote, false, 1, run[i].s)) return e;
        }
        open += run[i].left > 0;
      }
    }
    return MGK_OK;
  };
  const int rc = loop();
  if (rc)
    for (size_t i = 0; i < side.size(); ++i) cudaStreamSynchronize(side[i].s);
  return rc;
}

// Switches the plan's kernel family (see mgk_ls2d_plan::fast).
static int ls2d_set_variant(mgk_ls2d_t p, int v) {
  MGK_REQUIRE(v == 0 || (p->fast_nat && v >= p->fast_nat && (v == 256 || v == 512 || v == 1024)),
              "mgk_ls2d: kernel family %d cannot serve this plan", v);
  p->fast = v;
  ls2d_drop_graphs(p);
  return MGK_OK;
}

static int profile_setup(mgk_ls2d_t p, int nsel, const int* sel, const double* eps_bar, cudaStream_t s);

// Mean time of an iteration as the loop's body runs it, the groups side by side:
// a graph of `reps` bodies, each waiting for the whole one before it.
static int time_iterations(mgk_ls2d_t p, bool f32, int reps, float* ms, cudaStream_t s) {
  Loop2& a = p->last;
  int rc = launch2(a, kFirst, f32, 1, s);
  if (rc) return rc;
  cudaGraph_t g = nullptr;
  cudaGraphExec_t x = nullptr;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  auto run = [&]() -> int {
    MGK_CUDA(cudaGraphCreate(&g, 0));
    std::vector<cudaGraphNode_t> prev, rows;
    for (int r = 0; r < reps; ++r) {
      rows.clear();
      for (Grp2& gr : a.grp) {
        cudaGraphNode_t col, row;
        MGK_CUDA(with_stage2(a, gr, kCol, f32, 1, 0, 0, 0, [&](const Launch2& L, void** args) {
          return add_node2(g, &col, prev.data(), prev.size(), L, args);
        }));
        MGK_CUDA(with_stage2(a, gr, kRow, f32, 1, 0, 0, 0, [&](const Launch2& L, void** args) {
          return add_node2(g, &row, &col, 1, L, args);
        }));
        rows.push_back(row);
      }
      prev = rows;
    }
    MGK_CUDA(cudaGraphInstantiate(&x, g, 0));
    for (int i = 0; i < 2; ++i) MGK_CUDA(cudaEventCreate(&ev[i]));
    MGK_CUDA(cudaGraphLaunch(x, s));  // warm-up
    MGK_CUDA(cudaEventRecord(ev[0], s));
    MGK_CUDA(cudaGraphLaunch(x, s));
    MGK_CUDA(cudaEventRecord(ev[1], s));
    MGK_CUDA(cudaEventSynchronize(ev[1]));
    MGK_CUDA(cudaEventElapsedTime(ms, ev[0], ev[1]));
    *ms /= reps;
    return MGK_OK;
  };
  rc = run();
  for (int i = 0; i < 2; ++i)
    if (ev[i]) cudaEventDestroy(ev[i]);
  if (x) cudaGraphExecDestroy(x);
  if (g) cudaGraphDestroy(g);
  return rc;
}

extern "C" int mgk_ls2d_set_family(mgk_ls2d_t p, int family) {
  MGK_REQUIRE(p, "mgk_ls2d_set_family: null plan");
  MGK_CUDA(cudaDeviceSynchronize());  // no loop graph of this plan in flight
  return ls2d_set_variant(p, family);
}

extern "C" int mgk_ls2d_autotune(mgk_ls2d_t p, int nsel, const int* sel, const double* eps_bar, int reps,
                                 int* chosen, float* best_ms, mgk_stream_t stream) {
  MGK_REQUIRE(p && eps_bar && nsel >= 1 && reps >= 1, "mgk_ls2d_autotune: bad argument");
  // families 256/512/1024 share their kernels: the natural one stands for them
  int cands[2];
  int nc = 0;
  if (p->fast_nat) cands[nc++] = p->fast_nat;
  cands[nc++] = 0;
  int best = p->fast;
  float best_t = 0.0f;
  for (int k = 0; k < nc; ++k) {
    int st = ls2d_set_variant(p, cands[k]);
    if (st) return st;
    float t64 = 0, t32 = 0;
    st = profile_setup(p, nsel, sel, eps_bar, (cudaStream_t)stream);
    if (st == MGK_OK) st = time_iterations(p, false, reps, &t64, (cudaStream_t)stream);
    if (st == MGK_OK && p->prec == MGK_MIXED) {
      st = profile_setup(p, nsel, sel, eps_bar, (cudaStream_t)stream);
      if (st == MGK_OK) st = time_iterations(p, true, reps, &t32, (cudaStream_t)stream);
    }
    if (st) return st;
    const float t = t64 + t32;
    if (k == 0 || t < best_t) { best_t = t; best = cands[k]; }
  }
  int st = ls2d_set_variant(p, best);
  if (st) return st;
  if (chosen) *chosen = best;
  if (best_ms) *best_ms = best_t;
  return MGK_OK;
}

// Copies the replicas' states to the host (one synchronisation of the
// stream) and fills infos for the selection.
static int ls2d_collect(mgk_ls2d_t p, int nsel, const int* selv, mgk_ls_info* infos, cudaStream_t s) {
  MGK_CUDA(cudaMemcpyAsync(p->h_state, p->d_st, sizeof(Ls2dState) * p->nrep, cudaMemcpyDeviceToHost, s));
  Ls2dCtl hc;
  MGK_CUDA(cudaMemcpyAsync(&hc, p->d_ctl, sizeof(Ls2dCtl), cudaMemcpyDeviceToHost, s));
  MGK_CUDA(cudaStreamSynchronize(s));
  if (hc.error) {
    set_error("mgk_ls2d_solve: a bulk copy wait gave up (device timeout)");
    return MGK_TIMEOUT;
  }
  int worst = MGK_OK;
  for (int q = 0; q < nsel; ++q) {
    const Ls2dState& S = p->h_state[selv[q]];
    infos[q].iterations = S.iter;
    infos[q].status = S.status;
    infos[q].final_diff = S.diff;
    for (int k = 0; k < 4; ++k) { infos[q].eps_mean[k] = S.out_eps_mean[k]; infos[q].sig_mean[k] = S.out_sig_mean[k]; }
    if (S.status == MGK_NONFINITE) worst = MGK_NONFINITE;
  }
  if (worst == MGK_NONFINITE) {
    set_error("mgk_ls2d_solve: non-finite residual");
    return MGK_NONFINITE;
  }
  return MGK_OK;
}

extern "C" int mgk_ls2d_collect(mgk_ls2d_t p, int nsel, const int* sel, mgk_ls_info* infos, mgk_stream_t stream) {
  MGK_REQUIRE(p && sel && infos && nsel >= 1 && nsel <= p->nrep, "mgk_ls2d_collect: bad argument");
  for (int q = 0; q < nsel; ++q)
    MGK_REQUIRE(sel[q] >= 0 && sel[q] < p->nrep, "mgk_ls2d_collect: replica %d out of range", sel[q]);
  return ls2d_collect(p, nsel, sel, infos, (cudaStream_t)stream);
}

// The selection by launch groups (the CTA-wide replicas first, then each
// shape), its order and the loop's signature.  A group takes the wide forms
// when these give at least two CTAs per SM.  The shared-memory limits are raised
// here and not in the constructor: of five sides' 50 kernels (4 laws, 2 widths) a
// solve launches 10, and the first one named of a translation unit loads it (created
// after a plan of other sides, one 64^2 grid 18 -> 3 ms, five sides 40 -> 5 ms).
static int ls2d_group(mgk_ls2d_t p, const std::vector<int>& selv, Loop2& a, std::vector<int>& sig) {
  const int nsel = (int)selv.size();
  constexpr int kFill = 296;
  a = Loop2();
  a.reps = p->d_reps; a.st = p->d_st; a.part = p->d_part; a.ctr = p->d_repctr; a.ctl = p->d_ctl;
  a.rs = p->row_smem; a.cs = p->col_smem; a.rs32 = p->row_smem32; a.cs32 = p->col_smem32;
  a.sel = p->d_maps; a.nsel = nsel; a.G = grid_blocks(p->maxN); a.law = p->law;
  p->order.clear();
  Grp2 c;
  for (int r : selv)
    if (!ls2d_on_line(p, r)) {
      p->order.push_back(r);
      ++c.n;
      c.rows += p->reps[r].row_items;
      c.cols += p->reps[r].col_items;
    }
  c.row_map = p->d_maps + nsel;
  c.row_local = c.row_map + c.rows;
  c.col_map = c.row_local + c.rows;
  c.col_local = c.col_map + c.cols;
  if (c.n) {
    int rc = ls2d_set_attrs<double, double>(a.rs, a.cs);
    if (rc == MGK_OK && p->prec == MGK_MIXED) rc = ls2d_set_attrs<float, float>(a.rs32, a.cs32);
    if (rc) return rc;
  }
  sig = {p->law, p->aa_m, nsel, c.n, c.rows, c.cols};
  c.sel = p->d_maps;
  if (c.n) a.grp.push_back(c);
  std::vector<char> placed(p->nrep, 0);
  for (int q = 0; q < nsel; ++q) {
    const Ls2dRep& R = p->reps[selv[q]];
    if (placed[selv[q]] || !ls2d_on_line(p, selv[q])) continue;
    Grp2 g;
    g.kx = ls2_line(R.nx, kLs2Fp64);
    g.ky = ls2_line(R.ny, kLs2Fp64);
    if (p->prec == MGK_MIXED) {
      // the FP32 roundings of the kernels that the plan's family stands for
      const int kind = p->fast ? kLs2Fp32 : kLs2Fp32Wide;
      g.kx32 = ls2_line(R.nx, kind);
      g.ky32 = ls2_line(R.ny, kind);
    }
    g.nx = R.nx;
    g.nyh = R.nyh;
    g.sel = p->d_maps + p->order.size();
    for (int w = q; w < nsel; ++w) {
      const int r = selv[w];
      if (placed[r] || !ls2d_on_line(p, r) || p->reps[r].nx != R.nx || p->reps[r].ny != R.ny) continue;
      placed[r] = 1;
      p->order.push_back(r);
      ++g.n;
    }
    g.wr = (long long)g.n * ceil_div(g.nx / 2, g.ky->pairs[1]) >= kFill;
    g.wc = (long long)g.n * ceil_div(g.nyh, g.kx->cols[1]) >= kFill;
    if (g.kx32) g.wc32 = (long long)g.n * ceil_div(g.nyh, g.kx32->cols[1]) >= kFill;
    MGK_CUDA(raise_smem(g.ky->row[p->law][g.wr], g.ky->r_bytes[g.wr]));
    MGK_CUDA(raise_smem(g.kx->col[g.wc], g.kx->c_bytes[g.wc]));
    if (g.kx32) {
      MGK_CUDA(raise_smem(g.ky32->row[0][g.wr], g.ky32->r_bytes[g.wr]));
      MGK_CUDA(raise_smem(g.kx32->col[g.wc32], g.kx32->c_bytes[g.wc32]));
    }
    sig.insert(sig.end(), {R.nx, R.ny, g.n});
    a.grp.push_back(g);
  }
  a.grp[0].lead = 1;
  for (Grp2& g : a.grp) g.ctl = a.ctl;
  return MGK_OK;
}

// Whether a selection of several shapes whose caller waits for it is driven from the
// host: at its first kHostUses uses.  Its graph takes 360 us to instantiate with five
// shapes (135 with one, 55 for every further branch of a body; mixed plans have two
// bodies), most of a warm-started solve, and an ensemble's selections change from
// round to round; a host-driven solve of 3 .. 5 shapes takes 20 us less to 80 us more.
// First solve of a fresh plan of the five sides 128 .. 512, warm: 815 -> 466 us (660
// with the one pair of kernels for all shapes that the register passes replaced).
static bool ls2d_host_first(mgk_ls2d_t p, const std::vector<int>& sig) {
  constexpr int kHostUses = 4;
  constexpr size_t kSights = 64;
  for (auto& e : p->sights)
    if (e.first == sig) return e.second < kHostUses && ++e.second <= kHostUses;
  if (p->sights.size() >= kSights) p->sights.erase(p->sights.begin());
  p->sights.push_back({sig, 1});
  return true;
}

extern "C" int mgk_ls2d_solve_batch(mgk_ls2d_t p, int nsel, const int* sel, const double* eps_bar,
                                    const double* const* eps_init, double* const* eps_out, double* const* sig_out,
                                    int max_iter, double tol, mgk_ls_info* infos, mgk_stream_t stream) {
  MGK_REQUIRE(p && eps_bar && nsel >= 1 && nsel <= p->nrep, "mgk_ls2d_solve_batch: bad argument");
  MGK_REQUIRE(max_iter >= 0 && max_iter <= 1000000, "mgk_ls2d_solve: max_iter out of range");
  MGK_REQUIRE(p->aa_m == 0 || nsel == 1, "mgk_ls2d_solve_batch: Anderson mixing solves one replica per call");
  MGK_REQUIRE(p->aa_m == 0 || p->law != 0, "mgk_ls2d_solve_batch: Anderson mixing runs with a nonlinear law");
  cudaStream_t s = (cudaStream_t)stream;
  std::vector<int> selv(nsel);
  std::vector<char> seen(p->nrep, 0);
  for (int q = 0; q < nsel; ++q) {
    const int r = sel ? sel[q] : q;
    MGK_REQUIRE(r >= 0 && r < p->nrep && !seen[r], "mgk_ls2d_solve_batch: bad or repeated replica index");
    MGK_REQUIRE(p->has_material[r], "mgk_ls2d_solve: replica %d has no material (call set_material)", r);
    // the Rose law reads the [0,1] strain entry; the symmetric storage carries it
    // when macro strain and eigenstrain are symmetric (the eigenstrain is the
    // caller's to keep symmetric)
    MGK_REQUIRE(p->law < 2 || eps_bar[4 * q + 1] == eps_bar[4 * q + 2],
                "mgk_ls2d_solve: the Rose and Landau laws need a symmetric macro strain");
    seen[r] = 1;
    selv[q] = r;
  }
  int rc = staging_wait(p);
  if (rc) return rc;
  Loop2& a = p->last;
  std::vector<int> sig;
  if ((rc = ls2d_group(p, selv, a, sig))) return rc;
  // per-call records, the selection and the CTA-wide group's maps
  const Grp2& cg = a.grp[0];
  int* row_map = p->h_maps + nsel;
  int* row_local = row_map + cg.rows;
  int* col_map = row_local + cg.rows;
  int* col_local = col_map + cg.cols;
  std::vector<int> at(p->nrep, 0);
  for (int q = 0; q < nsel; ++q) at[selv[q]] = q;
  int first = 0, k = 0, ri = 0, ci = 0;
  for (const Grp2& g : a.grp)
    for (int e = 0; e < g.n; ++e, ++k) {
      const int r = p->order[k], q = at[r];
      Ls2dRep& H = p->h_reps[r];
      H = p->reps[r];
      H.init = eps_init ? eps_init[q] : nullptr;
      H.out_eps = eps_out ? eps_out[q] : nullptr;
      H.out_sig = sig_out ? sig_out[q] : nullptr;
      for (int c = 0; c < 4; ++c) H.eb[c] = eps_bar[4 * q + c];
      H.tol = tol;
      H.max_iter = max_iter;
      H.aa = p->aa_m > 0 ? p->d_aa : nullptr;
      H.aa_x = p->aa_m > 0 ? p->aa_buf : nullptr;
      H.aa_dG = p->aa_m > 0 ? p->aa_buf + (size_t)(3 + p->aa_m) * 3 * (size_t)H.N : nullptr;
      H.row_first = first;
      first += H.row_items;
      p->h_maps[k] = r;
      if (g.ky) continue;
      for (int i = 0; i < H.row_items; ++i) { row_map[ri] = r; row_local[ri] = i; ++ri; }
      for (int i = 0; i < H.col_items; ++i) { col_map[ci] = r; col_local[ci] = i; ++ci; }
    }
  const int n_active = max_iter > 0 ? nsel : 0;
  const char* env = getenv("MGK_NO_GRAPH_WHILE");
  if (env && env[0] == '1') p->graph_mode = 0;
  const bool hosted = p->graph_mode == 0 || (infos && a.grp.size() > 1 && ls2d_host_first(p, sig));
  const size_t nc = hosted ? a.grp.size() : 1;
  for (size_t i = 0; i < nc; ++i) {
    const int n = n_active == 0 ? 0 : hosted ? a.grp[i].n : nsel;
    p->h_ctl[i] = Ls2dCtl{(unsigned int)n, 0u, 0u, 0u, n > 0, 0};
    if (hosted) a.grp[i].ctl = a.ctl + i;
  }
  const size_t nm = nsel + 2 * (size_t)(ri + ci);
  MGK_CUDA(cudaMemcpyAsync(p->d_maps, p->h_maps, sizeof(int) * nm, cudaMemcpyHostToDevice, s));
  MGK_CUDA(cudaMemcpyAsync(p->d_reps, p->h_reps, sizeof(Ls2dRep) * p->nrep, cudaMemcpyHostToDevice, s));
  MGK_CUDA(cudaMemcpyAsync(p->d_ctl, p->h_ctl, sizeof(Ls2dCtl) * nc, cudaMemcpyHostToDevice, s));
  MGK_CUDA(cudaEventRecord(p->staged, s));
  p->staged_pending = true;

  const int* d_sel = a.sel;
  const int G = a.G;
  const bool mixed = p->prec == MGK_MIXED;
  bool any_init = false;
  for (int q = 0; q < nsel && eps_init; ++q) any_init |= eps_init[q] != nullptr;
  if (any_init)
    ls2d_means_kernel<<<dim3(G, nsel), kThreads, 0, s>>>(p->d_reps, p->d_st, d_sel, p->d_part, p->d_voxctr);
  ls2d_begin_kernel<<<dim3(G, nsel), kThreads, 0, s>>>(p->d_reps, p->d_st, d_sel, p->d_part, p->d_voxctr,
                                                       p->d_repctr, mixed && n_active > 0);
  MGK_CUDA(cudaGetLastError());
  if (n_active > 0) {
    if (p->aa_m > 0) {
      a.aa_m = p->aa_m;
      a.aa_nb = p->aa_nb;
      a.aa_buf = p->aa_buf;
      a.aa = p->d_aa;
      a.aa_part = p->aa_part;
      ls2d_aa_init_kernel<<<p->aa_nb, kThreads, 0, s>>>(p->d_reps, d_sel, p->aa_buf, p->d_aa);
      MGK_CUDA(cudaGetLastError());
    }
    cudaGraphExec_t exec = nullptr;
    if (!hosted) {
      const int cap = (max_iter + 2 > 1000 ? max_iter + 2 : 1000);
      for (auto& e : p->gcache)
        if (e.cap >= cap && e.sig == sig) exec = e.x;
      if (!exec) {
        cudaGraph_t g;
        if (build_graph(p, a, cap, &g, &exec) == MGK_OK) {
          constexpr size_t kMaxGraphs = 48;
          if (p->gcache.size() >= kMaxGraphs) {
            cudaGraphExecDestroy(p->gcache.front().x);
            cudaGraphDestroy(p->gcache.front().g);
            p->gcache.erase(p->gcache.begin());
          }
          p->gcache.push_back({sig, cap, g, exec});
        } else {
          exec = nullptr;
          p->graph_mode = 0;
        }
      }
    }
    if (exec) {
      if ((rc = launch2(a, kFirst, mixed, !mixed, s))) return rc;
      MGK_CUDA(cudaGraphLaunch(exec, s));
    } else {
      if (!hosted && a.grp.size() > 1) {  // no graph after all: the groups' own control blocks
        for (size_t i = 0; i < a.grp.size(); ++i) {
          p->h_ctl[p->nctl + i] = Ls2dCtl{(unsigned int)a.grp[i].n, 0u, 0u, 0u, 1, 0};
          a.grp[i].ctl = a.ctl + i;
        }
        MGK_CUDA(cudaMemcpyAsync(p->d_ctl, p->h_ctl + p->nctl, sizeof(Ls2dCtl) * a.grp.size(), cudaMemcpyHostToDevice, s));
      }
      if ((rc = host_loop(p, a, max_iter, s))) return rc;
    }
  }
  auto out = p->law == 1   ? ls2d_output_kernel<1>
             : p->law == 2 ? ls2d_output_kernel<2>
             : p->law == 3 ? ls2d_output_kernel<3>
                           : ls2d_output_kernel<0>;
  out<<<dim3(G, nsel), kThreads, 0, s>>>(p->d_reps, p->d_st, d_sel, p->d_part, p->d_voxctr);
  MGK_CUDA(cudaGetLastError());
  if (infos) return ls2d_collect(p, nsel, selv.data(), infos, s);
  return MGK_OK;
}

extern "C" int mgk_ls2d_solve(mgk_ls2d_t p, const double* eps_bar, const double* eps_init, double* eps_out,
                              double* sig_out, int max_iter, double tol, mgk_ls_info* info, mgk_stream_t stream) {
  MGK_REQUIRE(p && eps_bar, "mgk_ls2d_solve: null argument");
  int r0 = 0;
  return mgk_ls2d_solve_batch(p, 1, &r0, eps_bar, &eps_init, &eps_out, &sig_out, max_iter, tol, info, stream);
}

extern "C" int mgk_ls2d_leave_arrivals(mgk_ls2d_t p, int rep, int count, mgk_stream_t stream) {
  MGK_REQUIRE(p && rep >= 0 && rep < p->nrep && count >= 0 && count < p->reps[rep].row_items && count < 256,
              "mgk_ls2d_leave_arrivals: bad argument");
  MGK_CUDA(cudaMemsetAsync(p->d_repctr + rep, count, 1, (cudaStream_t)stream));  // the low byte; the others are zero
  return MGK_OK;
}

// ----------------------------------------------------------- profiling ---

// times the stages of the plan's last selection
static int profile_stages(mgk_ls2d_t p, bool f32, float* row_ms, float* col_ms, int reps, cudaStream_t s) {
  Loop2& a = p->last;
  int rc = launch2(a, kFirst, f32, 1, s);
  if (rc) return rc;
  cudaEvent_t ev[3];
  for (int i = 0; i < 3; ++i) MGK_CUDA(cudaEventCreate(&ev[i]));
  float tr = 0, tc = 0;
  for (int r = 0; r < reps && rc == MGK_OK; ++r) {
    cudaEventRecord(ev[0], s);
    rc = launch2(a, kCol, f32, 1, s);
    cudaEventRecord(ev[1], s);
    if (rc == MGK_OK) rc = launch2(a, kRow, f32, 1, s);
    cudaEventRecord(ev[2], s);
    if (cudaEventSynchronize(ev[2]) != cudaSuccess) { rc = MGK_CUDA_ERROR; break; }
    float x = 0, y = 0;
    cudaEventElapsedTime(&x, ev[0], ev[1]);
    cudaEventElapsedTime(&y, ev[1], ev[2]);
    tc += x;
    tr += y;
  }
  for (int i = 0; i < 3; ++i) cudaEventDestroy(ev[i]);
  MGK_CUDA(cudaGetLastError());
  if (rc != MGK_OK) { set_error("mgk_ls2d_profile: kernel failure"); return rc; }
  *row_ms = tr / reps;
  *col_ms = tc / reps;
  return MGK_OK;
}

static int profile_setup(mgk_ls2d_t p, int nsel, const int* sel, const double* eps_bar, cudaStream_t s) {
  // set up the selection with a zero-iteration solve, then time iterations
  // with tolerance 0 and an unreachable cap so every replica stays active
  std::vector<const double*> init(nsel, nullptr);
  std::vector<double*> outs(nsel, nullptr);
  int rc = mgk_ls2d_solve_batch(p, nsel, sel, eps_bar, init.data(), outs.data(), outs.data(), 0, 0.0, nullptr,
                                (mgk_stream_t)s);
  if (rc) return rc;
  rc = staging_wait(p);
  if (rc) return rc;
  for (int q = 0; q < nsel; ++q) {
    Ls2dRep& H = p->h_reps[sel ? sel[q] : q];
    H.max_iter = 1 << 30;
    H.tol = 0.0;
  }
  MGK_CUDA(cudaMemcpyAsync(p->d_reps, p->h_reps, sizeof(Ls2dRep) * p->nrep, cudaMemcpyHostToDevice, s));
  for (int q = 0; q < nsel; ++q) {
    const int r = sel ? sel[q] : q;
    MGK_CUDA(cudaMemsetAsync(reinterpret_cast<char*>(&p->d_st[r]) + offsetof(Ls2dState, done), 0, sizeof(int), s));
  }
  p->h_ctl->n_active = nsel;
  p->h_ctl->decided = 0;
  p->h_ctl->still = 0;
  p->h_ctl->bodies = 0;
  MGK_CUDA(cudaMemcpyAsync(p->d_ctl, p->h_ctl, sizeof(Ls2dCtl), cudaMemcpyHostToDevice, s));
  MGK_CUDA(cudaStreamSynchronize(s));
  return MGK_OK;
}

extern "C" int mgk_ls2d_profile_batch(mgk_ls2d_t p, int nsel, const int* sel, const double* eps_bar, int fp32,
                                      int reps, float* row_ms, float* col_ms, mgk_stream_t stream) {
  MGK_REQUIRE(p && eps_bar && row_ms && col_ms && reps > 0, "mgk_ls2d_profile: bad argument");
  MGK_REQUIRE(!fp32 || p->prec == MGK_MIXED, "mgk_ls2d_profile: FP32 kernels need a mixed-precision plan");
  cudaStream_t s = (cudaStream_t)stream;
  int rc = profile_setup(p, nsel, sel, eps_bar, s);
  if (rc) return rc;
  return profile_stages(p, fp32 != 0, row_ms, col_ms, reps, s);
}

extern "C" int mgk_ls2d_profile(mgk_ls2d_t p, const double* eps_bar, int reps, float* row_ms, float* col_ms,
                                mgk_stream_t stream) {
  int r0 = 0;
  return mgk_ls2d_profile_batch(p, 1, &r0, eps_bar, 0, reps, row_ms, col_ms, stream);
}

// ------------------------------------------------- one-voxel eigenstrain ---

namespace mgk {
// Copy voxel (x, y) = d_xy[0..1] of the caller's eigenstrain field (after a
// flip) into the plan's planes; a negative x means no event happened.
__global__ void ls2d_sync_voxel_kernel(const Ls2dRep* reps, int rep, const double* __restrict__ epsp,
                                       const long long* __restrict__ d_xy) {
  const long long x = d_xy[0], y = d_xy[1];
  const Ls2dRep& R = reps[rep];
  if (x < 0 || y < 0 || x >= R.nx || y >= R.ny) return;
  const long long N = R.N, i = x * R.ny + y;
  const double4 p = reinterpret_cast<const double4*>(epsp)[i];
  const double psym = (p.y == p.z) ? p.y : 0.5 * (p.y + p.z);
  R.ep[i] = p.x;
  R.ep[N + i] = p.w;
  R.ep[2 * N + i] = psym;
  if (R.ep32) { R.ep32[i] = (float)p.x; R.ep32[N + i] = (float)p.w; R.ep32[2 * N + i] = (float)psym; }
  if (R.epa) { R.epa[i] = p.y; R.epa[N + i] = p.z; }
}
}  // namespace mgk

extern "C" int mgk_ls2d_sync_voxel(mgk_ls2d_t p, int rep, const double* eps_plastic, const int64_t* d_xy,
                                   mgk_stream_t stream) {
  MGK_REQUIRE(p && eps_plastic && d_xy && rep >= 0 && rep < p->nrep && p->has_material[rep],
              "mgk_ls2d_sync_voxel: bad argument");
  MGK_REQUIRE(p->reps[rep].epa != nullptr, "mgk_ls2d_sync_voxel: set the material with an eigenstrain field first");
  ls2d_sync_voxel_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(p->d_reps, rep, eps_plastic, (const long long*)d_xy);
  MGK_CUDA(cudaGetLastError());
  return MGK_OK;
}

// ============================================================ no-alloc ===
// Allocation-free 2D LS solve.  Some callers cannot call cudaMalloc: a host
// application or framework whose caching allocator already reserves the
// device memory, a serving process with a fixed memory budget that must not
// allocate after start-up, or code that must avoid the device-wide
// synchronisation cudaFree performs.  For them every buffer the solve needs
// beyond its inputs and outputs lives in one file-scope device array, sized
// for grids up to MGK_NOALLOC_MAX_SIDE per side; each GPU that loads this
// library holds it (about 7 MB) until the process exits.
namespace {
constexpr long long kNaMaxN = (long long)MGK_NOALLOC_MAX_SIDE * MGK_NOALLOC_MAX_SIDE;
constexpr size_t kNaPlanes = 10 * (size_t)kNaMaxN;                                          // 10 real planes
constexpr size_t kNaSpec = 3 * (size_t)MGK_NOALLOC_MAX_SIDE * (MGK_NOALLOC_MAX_SIDE / 2 + 1) * 2;  // complex
constexpr size_t kNaTw = 2 * (size_t)MGK_NOALLOC_MAX_SIDE * 2;                               // two tables
constexpr size_t kNaPart = 8 * 2048;                                                         // partial sums
constexpr size_t kNaMisc = 1024;                    // plan record, state, control, work maps
constexpr size_t kNaDoubles = kNaPlanes + kNaSpec + kNaTw + kNaPart + kNaMisc;
// byte offsets inside the misc region
constexpr size_t kNaRep = 0, kNaState = 1024, kNaCtl = 2048, kNaCtr = 2112, kNaMaps = 2176;
constexpr int kNaMapInts = 128 + 128 + 256 + 256 + 1;
static_assert(kNaMaps + 4 * kNaMapInts <= kNaMisc * sizeof(double), "no-alloc misc region");
}  // namespace

// Device-side storage.  In host code this name is only a stand-in for the
// device address, which cudaGetSymbolAddress resolves per device.
static __device__ __align__(256) double g_ls2d_noalloc_scratch[kNaDoubles];

namespace mgk {

// Writes the plan record and the work maps, clears the state, the control
// block and the arrival counter, and fills the twiddle tables (sincospi):
// everything a call must start from.
__global__ void ls2d_noalloc_setup_kernel(Ls2dRep rep, Ls2dRep* dst, Ls2dState* st, Ls2dCtl* ctl,
                                          unsigned int* repctr, int* maps, int rows, int cols, int n_active,
                                          double2* twx, int nx, double2* twy, int ny) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int stride = gridDim.x * blockDim.x;
  int* row_map = maps;
  int* row_local = row_map + rows;
  int* col_map = row_local + rows;
  int* col_local = col_map + cols;
  int* sel = col_local + cols;
  for (int i = t; i < rows; i += stride) { row_map[i] = 0; row_local[i] = i; }
  for (int i = t; i < cols; i += stride) { col_map[i] = 0; col_local[i] = i; }
  for (int m = t; m < nx; m += stride) {
    double s, c;
    sincospi(2.0 * m / nx, &s, &c);
    twx[m] = make_double2(c, -s);
  }
  for (int m = t; m < ny; m += stride) {
    double s, c;
    sincospi(2.0 * m / ny, &s, &c);
    twy[m] = make_double2(c, -s);
  }
  if (t == 0) {
    *dst = rep;
    sel[0] = 0;
    repctr[0] = 0;
    repctr[1] = 0;
    Ls2dState z;
    memset(&z, 0, sizeof(z));
    *st = z;
    ctl->n_active = (unsigned int)n_active;
    ctl->decided = 0;
    ctl->still = 0;
    ctl->bodies = 0;
    ctl->any = n_active > 0;
  }
}

}  // namespace mgk

static std::mutex g_noalloc_mu;
static void* g_noalloc_addr[128];  // resolved scratch address per device

// First call on a device: resolve the device address of the scratch array
// (this loads the module if it is not loaded yet).  Later calls reuse it.
static int noalloc_scratch(double** out) {
  int dev = -1;
  MGK_CUDA(cudaGetDevice(&dev));
  MGK_REQUIRE(dev >= 0 && dev < 128, "mgk_ls2d_solve_noalloc: device index %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_ls2d_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) {
      set_error("mgk_ls2d_solve_noalloc: cudaGetSymbolAddress failed on device %d: %s", dev, cudaGetErrorString(e));
      return MGK_CUDA_ERROR;
    }
    g_noalloc_addr[dev] = p;
  }
  *out = reinterpret_cast<double*>(g_noalloc_addr[dev]);
  return MGK_OK;
}

extern "C" int mgk_ls2d_solve_noalloc(int nx, int ny, int plane_mode, const double* E, const double* nu,
                                      const double* eps_plastic, const double* eps_bar, const double* eps_init,
                                      double* eps_out, double* sig_out, int max_iter, double tol,
                                      mgk_ls_info* info, mgk_stream_t stream) {
  MGK_REQUIRE(nx >= 2 && ny >= 1 && nx <= MGK_NOALLOC_MAX_SIDE && ny <= MGK_NOALLOC_MAX_SIDE,
              "mgk_ls2d_solve_noalloc: grid %dx%d exceeds the maximum of %dx%d for the allocation-free entry "
              "point (use mgk_ls2d_create/mgk_ls2d_solve)", nx, ny, MGK_NOALLOC_MAX_SIDE, MGK_NOALLOC_MAX_SIDE);
  FftLen fx, fy;
  MGK_REQUIRE(fft_schedule(nx, &fx) && fft_schedule(ny, &fy) && nx % 2 == 0,
              "mgk_ls2d_solve_noalloc: grid %dx%d unsupported (each side 2^a 3^b, nx even)", nx, ny);
  MGK_REQUIRE(plane_mode == MGK_PLANE_STRAIN || plane_mode == MGK_PLANE_STRESS,
              "mgk_ls2d_solve_noalloc: plane_mode must be 0 (strain) or 1 (stress)");
  MGK_REQUIRE(E && nu && eps_bar && eps_out && sig_out, "mgk_ls2d_solve_noalloc: null argument");
  MGK_REQUIRE(max_iter >= 0 && max_iter <= 1000000, "mgk_ls2d_solve_noalloc: max_iter out of range");
  double* base = nullptr;
  int st = noalloc_scratch(&base);
  if (st != MGK_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;

  const long long N = (long long)nx * ny;
  const int nyh = ny / 2 + 1;
  const int tc = pick_tc(nx, sizeof(double2), 64 * 1024);
  const int rows = nx / 2, cols = (nyh + tc - 1) / tc;
  const size_t row_smem = 2 * 3 * (size_t)ny * sizeof(double2);
  const size_t col_smem = 2 * 3 * (size_t)tc * nx * sizeof(double2);
  st = ls2d_set_attrs<double, double>(row_smem, col_smem);
  if (st != MGK_OK) return st;

  // carve the scratch array (offsets in doubles, each region 256-byte aligned)
  double* planes = base;
  double2* spec = reinterpret_cast<double2*>(base + kNaPlanes);
  double2* twx = reinterpret_cast<double2*>(base + kNaPlanes + kNaSpec);
  double2* twy = twx + MGK_NOALLOC_MAX_SIDE;
  double* part = base + kNaPlanes + kNaSpec + kNaTw;
  char* misc = reinterpret_cast<char*>(base + kNaPlanes + kNaSpec + kNaTw + kNaPart);
  Ls2dRep* d_rep = reinterpret_cast<Ls2dRep*>(misc + kNaRep);
  Ls2dState* d_st = reinterpret_cast<Ls2dState*>(misc + kNaState);
  Ls2dCtl* d_ctl = reinterpret_cast<Ls2dCtl*>(misc + kNaCtl);
  unsigned int* d_ctr = reinterpret_cast<unsigned int*>(misc + kNaCtr);
  unsigned int* d_vox = d_ctr + 1;  // arrival counter of the per-voxel kernels
  int* d_maps = reinterpret_cast<int*>(misc + kNaMaps);
  static_assert(sizeof(Ls2dRep) <= 1024 && sizeof(Ls2dState) <= 1024 && sizeof(Ls2dCtl) <= 64,
                "no-alloc record sizes");
  const int* d_row_map = d_maps;
  const int* d_row_local = d_row_map + rows;
  const int* d_col_map = d_row_local + rows;
  const int* d_col_local = d_col_map + cols;
  const int* d_sel = d_col_local + cols;

  fx.tw = twx;
  fy.tw = twy;
  Ls2dRep R;
  memset(&R, 0, sizeof(R));
  R.nx = nx; R.ny = ny; R.nyh = nyh; R.ld = nyh; R.tc = tc;
  R.row_items = rows; R.col_items = cols;
  R.N = N; R.fx64 = fx; R.fy64 = fy; R.fx32 = fx; R.fy32 = fy;
  R.mu = planes; R.lam = planes + N; R.eps = planes + 2 * N; R.ep = planes + 5 * N;
  R.epa = eps_plastic ? planes + 8 * N : nullptr;
  R.spec = spec;
  R.init = eps_init; R.out_eps = eps_out; R.out_sig = sig_out;
  for (int k = 0; k < 4; ++k) R.eb[k] = eps_bar[k];
  R.tol = tol; R.max_iter = max_iter; R.row_first = 0; R.col_first = 0;

  ls2d_noalloc_setup_kernel<<<4, 256, 0, s>>>(R, d_rep, d_st, d_ctl, d_ctr, d_maps, rows, cols,
                                              max_iter > 0 ? 1 : 0, twx, nx, twy, ny);
  MGK_CUDA(cudaGetLastError());
  const int G = grid_blocks(N);
  ls2d_material_kernel<<<G, kThreads, 0, s>>>(d_rep, d_st, 0, E, nu, eps_plastic, plane_mode, 1, 0, 0.0, part, d_vox);
  MGK_CUDA(cudaGetLastError());
  if (eps_init) ls2d_means_kernel<<<dim3(G, 1), kThreads, 0, s>>>(d_rep, d_st, d_sel, part, d_vox);
  ls2d_begin_kernel<<<dim3(G, 1), kThreads, 0, s>>>(d_rep, d_st, d_sel, part, d_vox, d_ctr, 0);
  MGK_CUDA(cudaGetLastError());
  if (max_iter > 0) {
    ls2d_row_kernel<double, double, false, true><<<rows, kThreads, row_smem, s>>>(
        d_rep, d_st, d_row_map, d_row_local, part, d_ctr, d_ctl, 0, 0, 0);
    MGK_CUDA(cudaGetLastError());
    // host-driven loop in chunks of 4 iterations; finished replicas skip
    // their work on the device, and the host polls the activity flag
    int it = 0;
    while (it < max_iter) {
      const int chunk = max_iter - it < 4 ? max_iter - it : 4;
      for (int c = 0; c < chunk; ++c) {
        ls2d_col_kernel<double, double><<<cols, kThreads, col_smem, s>>>(d_rep, d_st, d_col_map, d_col_local);
        ls2d_row_kernel<double, double, true, true><<<rows, kThreads, row_smem, s>>>(
            d_rep, d_st, d_row_map, d_row_local, part, d_ctr, d_ctl, 0, 0, 0);
        MGK_CUDA(cudaGetLastError());
      }
      it += chunk;
      Ls2dCtl hc;
      MGK_CUDA(cudaMemcpyAsync(&hc, d_ctl, sizeof(Ls2dCtl), cudaMemcpyDeviceToHost, s));
      MGK_CUDA(cudaStreamSynchronize(s));
      if (!hc.any) break;
    }
  }
  ls2d_output_kernel<0><<<dim3(G, 1), kThreads, 0, s>>>(d_rep, d_st, d_sel, part, d_vox);
  MGK_CUDA(cudaGetLastError());
  Ls2dState h;
  MGK_CUDA(cudaMemcpyAsync(&h, d_st, sizeof(Ls2dState), cudaMemcpyDeviceToHost, s));
  MGK_CUDA(cudaStreamSynchronize(s));
  if (info) {
    info->iterations = h.iter;
    info->status = h.status;
    info->final_diff = h.diff;
    for (int q = 0; q < 4; ++q) { info->eps_mean[q] = h.out_eps_mean[q]; info->sig_mean[q] = h.out_sig_mean[q]; }
  }
  if (h.status == MGK_NONFINITE) {
    set_error("mgk_ls2d_solve_noalloc: non-finite residual at iteration %d", h.iter);
    return MGK_NONFINITE;
  }
  return MGK_OK;
}

extern "C" int64_t mgk_aa_work_bytes(int64_t n) {
  (void)n;
  return (int64_t)sizeof(double) * kAaBlocks * 2 * kAaMax;
}

extern "C" int mgk_aa_update(int64_t n, const double* x, const double* g, double* hist, int m, int slot,
                             int have_prev, int ncols, double* dots, void* work, mgk_stream_t stream) {
  MGK_REQUIRE(n > 0 && x && g && hist && work && dots, "mgk_aa_update: bad argument");
  MGK_REQUIRE(m >= 1 && m <= kAaMax && ncols >= 0 && ncols <= m && slot >= 0 && slot < m &&
                  (!have_prev || slot < ncols),
              "mgk_aa_update: need 1 <= m <= %d, 0 <= ncols <= m, slot < m (and < ncols with a previous pair)",
              kAaMax);
  cudaStream_t s = (cudaStream_t)stream;
  const int nb = (int)std::min<long long>(kAaBlocks, (n + 255) / 256);
  double* part = reinterpret_cast<double*>(work);
  aa_update_kernel<<<nb, 256, 0, s>>>(n, x, g, hist, m, slot, have_prev, ncols, part);
  MGK_CUDA(cudaGetLastError());
  if (ncols > 0) {
    aa_sum_kernel<<<1, 256, 0, s>>>(part, nb, ncols, dots);
    MGK_CUDA(cudaGetLastError());
  }
  return MGK_OK;
}

extern "C" int mgk_aa_mix(int64_t n, const double* g, const double* hist, int m, int ncols, const double* gamma,
                          double* x, mgk_stream_t stream) {
  MGK_REQUIRE(n > 0 && g && hist && x && (ncols == 0 || gamma), "mgk_aa_mix: bad argument");
  MGK_REQUIRE(m >= 1 && m <= kAaMax && ncols >= 0 && ncols <= m, "mgk_aa_mix: need 1 <= m <= %d, ncols <= m",
              kAaMax);
  AaCoef c;
  for (int j = 0; j < kAaMax; ++j) {
    c.v[j] = j < ncols ? gamma[j] : 0.0;
    MGK_REQUIRE(isfinite(c.v[j]), "mgk_aa_mix: non-finite coefficient");
  }
  const int nb = (int)std::min<long long>(4 * kAaBlocks, (n + 255) / 256);
  aa_mix_kernel<<<nb, 256, 0, (cudaStream_t)stream>>>(n, g, hist, m, ncols, c, x);
  MGK_CUDA(cudaGetLastError());
  return MGK_OK;
}
