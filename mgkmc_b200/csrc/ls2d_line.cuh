// 2D small-strain iteration kernels on register FFTs (fft_reg.cuh), one
// instantiation per line length; lengths without one take the CTA-wide passes
// of ls2d.cu.
//
//   row kernel     CTA of P pairs of x-rows x 3 components x T threads: C2R
//                  along y of the previous spectrum, eps update with the
//                  diff/norm partials and the convergence decision, tau, R2C
//                  along y;
//   column kernel  CTA of W ky columns x 3 components x T threads: FFT along
//                  x, Gamma0, inverse FFT along x.
//
// A large selection is bound by HBM (136 and 48 bytes per voxel in FP64), a
// small one by the chain of one CTA: loads, two transforms, the law.  So each
// kernel comes in two widths: P pairs or W columns per CTA for a selection
// that fills the GPU twice over, one pair or column (the sector waste is served
// by L2) below that, which spreads a 64^2 grid over 32 CTAs instead of 8.
// CUDA events around each launch, the warp-line kernels before and these: FP64,
// 256^2 x 32: row 94.6 and 70.2 us (285 MB: 0.62 of the measured copy rate), column
// 60.5 and 44 us (0.35); 1024^2 x 1: 67 and 45 us, 43 and 40 us.  FP32, 256^2 x 32: row
// 49.9 and 51 us, column 38 and 30.6 us; 1024^2 x 1: 50.7 and 36 us, 33 and 24 us.
// 432x324, 162x243 and 288x216 together, whose sides had no warp-line kernel: an
// iteration took 101 us in the CTA-wide passes and takes 45 us.
#pragma once
#include "fft_reg.cuh"
#include "ls2d_dev.cuh"
#include "tma.cuh"

namespace mgk {

// ------------------------------------------------------------ geometry ---
constexpr int ls2_round32(int n) { return (n + 31) / 32 * 32; }
// Threads per line: the schedule's, or half of them in the wide form of FP32 lines of
// three steps of at most 8 points, whose butterflies then fill a thread's registers
// (256^2 x 32: row 55.0 -> 51.5 us, column 34.6 -> 31.1; 512^2 x 8: 61.1 -> 59.5, 39.4 ->
// 31.7; the kernels before the register passes: 49.8 and 38.0, 78 and 61).  One small
// grid wants the warps (256^2 x 1: row 15.7, at half 16.6), radix 9 the registers (162^2
// x 64: row 48.8, at half 57.3).
constexpr int ls2_t(int n, int csz, bool wide) {
  const RegSched q = reg_sched(n, csz);
  return wide && csz == 8 && q.ns == 3 && q.r[0] <= 8 && q.r[1] <= 8 && q.r[2] <= 8 ? q.t / 2 : q.t;
}
// row pairs per CTA of the wide kernel: about 100 transform threads in FP64
// (the same in FP32: a replica's items do not depend on the phase)
constexpr int ls2_pairs(int n) { return reg_sched64(n).t <= 9 ? 4 : reg_sched64(n).t <= 18 ? 2 : 1; }
// threads: those of the transforms, and enough for equal rounds of the voxel
// stage of at most 128 (256 for the longer lines) voxel pairs
constexpr int ls2_r_threads(int n, int p, int tl) {
  const int fft = 3 * tl * p, vox = p * ls2_round32(n), cap = n <= 256 ? 128 : 256;
  const int rounds = (vox + cap - 1) / cap, per = (vox + rounds - 1) / rounds;
  return ls2_round32(fft > per ? fft : per);
}
// columns per CTA: rows of 64 bytes in the wide kernel where the CTA stays
// below 432 threads, of 32 or 16 otherwise; 16 in the narrow one.  Lines of at most
// 32 points have the wide form only: their narrow CTA is a single warp, whose
// one-round loops the compiler contracts differently.
constexpr int ls2_cols(int n, int csz, bool wide) {
  const int t = ls2_t(n, csz, wide), one = 16 / csz;
  return wide || n <= 32 ? (t * one <= 36 ? 4 * one : t * one <= 72 ? 2 * one : csz == 16 ? 2 : one) : one;
}
constexpr int ls2_c_threads(int w, int tl) { return ls2_round32(3 * w * tl); }
// row pitch of the half spectra
constexpr int ls2_ld(int n) { return (n / 2 + 1 + 3) / 4 * 4; }
// exchange buffers; they first hold the pairs' spectrum rows as copied
constexpr int ls2_r_bytes(int n, int p, int csz) {
  const int a = p * 3 * reg_slots(n, csz), b = p * 6 * ls2_ld(n);
  return (a > b ? a : b) * csz;
}
constexpr int ls2_c_bytes(int n, int w, int csz) { return 3 * w * reg_slots(n, csz) * csz; }
// Resident CTAs asked of the register allocator: as many as 128 registers per thread
// allow in FP64, 80 in FP32, rounded down.  Where that leaves registers over, the
// compiler takes them: blocks of 192 threads get two CTAs and up to 168 registers
// (the FP64 column pass: 158 at 256 points, 160 at 1024, 12 warps per SM).
constexpr int ls2_minb(int threads, int csz) {
  const int b = 65536 / (threads * (csz == 16 ? 128 : 80));
  return b < 1 ? 1 : b > 16 ? 16 : b;
}

template <typename T> struct Twid;
template <> struct Twid<double> {
  static __device__ __forceinline__ const double2* get(const Ls2dRep& R, int axis) { return R.rtw[axis]; }
};
template <> struct Twid<float> {
  static __device__ __forceinline__ const float2* get(const Ls2dRep& R, int axis) { return R.rtw32[axis]; }
};

// eps~^ = -Gamma0(n) : tau^ of one real part in FP32, with the contractions of
// the FP32 passes written out (see fmul32)
__device__ __forceinline__ void gamma2d_f32(float txx, float tyy, float txy, float nx, float ny, float inv2mu0,
                                            float Bc, float& exx, float& eyy, float& exy) {
  const float tnx = __fmaf_rn(txx, nx, __fmul_rn(txy, ny)), tny = __fmaf_rn(tyy, ny, __fmul_rn(txy, nx));
  const float ntn = __fmaf_rn(tnx, nx, __fmul_rn(tny, ny)), a = 2.0f * inv2mu0;
  const float bx = __fmul_rn(Bc, nx), by = __fmul_rn(Bc, ny);
  exx = -__fmaf_rn(__fmul_rn(a, nx), tnx, -__fmul_rn(__fmul_rn(bx, nx), ntn));
  eyy = -__fmaf_rn(__fmul_rn(a, ny), tny, -__fmul_rn(__fmul_rn(by, ny), ntn));
  exy = -__fmaf_rn(inv2mu0, __fmaf_rn(ny, tnx, __fmul_rn(nx, tny)), -__fmul_rn(__fmul_rn(bx, ny), ntn));
}

// ask `bytes` at p into L2 when both suit the bulk prefetch (16-byte pieces)
__device__ __forceinline__ void l2_prefetch2(const void* p, uint32_t bytes) {
  if (((reinterpret_cast<uintptr_t>(p) | bytes) & 15) == 0)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// The launch covers the replicas sel[0 ..) of one shape, their items in
// order.  first: 0 inverts the previous spectrum and updates the field; 1 reads
// the field as is (first tau of a phase, or of a mixed iterate); 2 does so
// from the FP32 field of a mixed plan, which becomes the FP64 one.  final: see
// ls2d_decide.  lead: this launch counts the loop bodies.
template <typename T, int NY, int P, int TL, int LAW, int ALT>
__global__ void __launch_bounds__(ls2_r_threads(NY, P, TL), ls2_minb(ls2_r_threads(NY, P, TL), 2 * (int)sizeof(T)))
    ls2_row_reg(const Ls2dRep* __restrict__ reps, Ls2dState* st, const int* __restrict__ sel, double* partials,
                unsigned int* rep_counter, Ls2dCtl* ctl, cudaGraphConditionalHandle cond, int use_cond, int guard_cap,
                int lead, int first, int final) {
  using C = C_t<T>;
  constexpr int TH = ls2_r_threads(NY, P, TL), SL = reg_slots(NY, sizeof(C));
  constexpr int NYH = NY / 2 + 1;
  // A pair's sums behind the update norm do not depend on P: its voxel pairs, padded
  // to whole warps, are folded warp by warp (K = 1), or after the K rounds in which the
  // CTA of either form takes them up alike; where there is one form, after the loop.
  constexpr bool ONE = ls2_pairs(NY) == 1 && ls2_t(NY, sizeof(C), false) == ls2_t(NY, sizeof(C), true);
  constexpr int NYP = ls2_round32(NY), T1 = ls2_r_threads(NY, 1, ls2_t(NY, sizeof(C), false));
  constexpr int T2 = ls2_r_threads(NY, ls2_pairs(NY), ls2_t(NY, sizeof(C), true));
  constexpr int K = T1 == T2 && NYP % T1 == 0 ? NYP / T1 : 1;
  constexpr int NCH = ONE || K > 1 ? TH / 32 : NYP / 32;  // parts of a pair's sum
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double chunk[2][P * NCH];
  __shared__ int s_last;
  __shared__ __align__(8) uint64_t bar;
  const int per = (reps[sel[0]].nx / 2 + P - 1) / P;
  const int r = sel[blockIdx.x / per], loc = blockIdx.x % per;
  const Ls2dRep& R = reps[r];
  Ls2dState& S = st[r];
  if (first == 0 && use_cond && lead && blockIdx.x == 0 && threadIdx.x == 0) {
    // a body with no active replica has no decider: stop here; the body
    // count bounds the loop whatever happens to the deciders
    const unsigned int b = atomicAdd(&ctl->bodies, 1u) + 1u;
    if (ctl->n_active == 0 || b > (unsigned int)guard_cap || *(volatile int*)&ctl->error != 0) {
      ctl->any = 0;
      cudaGraphSetConditional(cond, 0u);
    }
  }
  const long long N = R.N;
  const int ld = R.ld, nx = R.nx;
  const int p0 = loc * P, np = min(P, nx / 2 - p0);
  if (S.done != 0) {
    // a replica that ended in the FP32 phase still becomes FP64 for the outputs
    if (sizeof(T) == 8 && first == 2)
      for (int c = 0; c < 3; ++c)
        for (int e = threadIdx.x; e < 2 * np * NY; e += TH)
          R.eps[c * N + 2LL * p0 * NY + e] = (double)R.eps32[c * N + 2LL * p0 * NY + e];
    return;
  }
  T* eps = Fields<T>::eps(R);
  const T *mu = Fields<T>::mu(R), *lam = Fields<T>::lam(R), *ep = Fields<T>::ep(R);
  C* spec = reinterpret_cast<C*>(R.spec);
  C* lines = reinterpret_cast<C*>(smem_raw);
  if (first == 0 && threadIdx.x == 0) {
    // the pairs' half-spectrum rows, contiguous per component
    const uint32_t bytes = 2u * np * ld * sizeof(C);
    mbar_init(&bar, 1);
    fence_mbar_init();
    mbar_arrive_expect_tx(&bar, 3u * bytes);
#pragma unroll
    for (int q = 0; q < 3; ++q)
      bulk_g2s(lines + q * 2 * P * ld, spec + ((long long)q * nx + 2 * p0) * ld, bytes, &bar);
  }
  if (threadIdx.x >= 16 && threadIdx.x < 24) {
    const int q = threadIdx.x - 16;
    const T* f = q < 3 ? eps + q * N : q == 3 ? mu : q == 4 ? lam : ep + (q - 5) * N;
    l2_prefetch2(f + 2LL * p0 * NY, (uint32_t)(2 * np * NY * sizeof(T)));
  }
  const C* tw = Twid<T>::get(R, 1);
  const int line = threadIdx.x / TL, t = threadIdx.x % TL;  // line = 3 pair + component
  const int pr = line / 3, c = line - 3 * pr;
  const bool act = line < 3 * P && pr < np;
  C* buf = lines + (line < 3 * P ? line : 0) * SL;
  auto at = [&](int s) -> C& { return buf[s]; };
  auto put = [&](int i, C v) { buf[reg_slot<NY, C>(i)] = v; };
  auto sync = [] {
    if constexpr (32 % TL == 0) __syncwarp();
    else __syncthreads();
  };
  if (first == 0) {
    __syncthreads();  // the barrier is initialised
    if (!__syncthreads_and(mbar_wait(&bar, 0) ? 1 : 0)) {
      if (threadIdx.x == 0) { ctl->error = 1; ctl->any = 0; }
      return;
    }
    const C* sa = lines + (c * P + pr) * 2 * ld;
    auto load = [&](int k) -> C {
      const int ks = 2 * k <= NY ? k : NY - k;
      C a = sa[ks], b = sa[ld + ks];
      if (k == 0 || 2 * k == NY) { a.y = 0; b.y = 0; }
      return 2 * k <= NY ? mk<C>(a.x - b.y, a.y + b.x) : mk<C>(a.x + b.y, b.x - a.y);
    };
    reg_line<NY, +1, ALT, C, TL>(t, act, tw, load, at, put, sync, [] { __syncthreads(); });
  }
  __syncthreads();
  const double mu0 = S.mu0, lam0 = S.lam0;
  const int law_ps = R.law_ps;
  const double law_a = R.law_a, law_b = R.law_b;
  const double eb0 = S.ebar[0], eb1 = S.ebar[1], eb2 = S.ebar[2];
  // Anderson mixing (nonlinear laws): a first pass applies the mix; the image's
  // tau is never used (the next tau is the mixed iterate's), so an image pass
  // stops at the update norm
  double gam[kAaMax];
  int nmix = 0;
  if constexpr (LAW != 0)
    if (first != 0 && R.aa) nmix = aa_load(R, gam);
  const bool img_only = LAW != 0 && first == 0 && R.aa != nullptr;
  double d2 = 0, n2 = 0;
  // the warp's 32 sums of each kind: the low lanes fold d2, the high ones n2
  auto fold = [&](int part) {
    const bool low = (threadIdx.x & 16) == 0;
    double v = (low ? d2 : n2) + __shfl_xor_sync(0xffffffffu, low ? n2 : d2, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o, 16);
    if ((threadIdx.x & 15) == 0) chunk[low ? 0 : 1][part] = v;
    d2 = n2 = 0;
  };
#pragma unroll 1
  for (int e = threadIdx.x; e < np * NYP; e += TH) {
    const int q = e / NYP, y = e - q * NYP;
    if (NY == NYP || y < NY) {
      C* vx = lines + q * 3 * SL + reg_slot<NY, C>(y);
      // every input of the two voxels before the first store
      double o[2][3], m[2], l[2], pl[2][3];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const long long i = (2LL * (p0 + q) + h) * NY + y;
#pragma unroll
        for (int k = 0; k < 3; ++k)
          o[h][k] = sizeof(T) == 8 && first == 2 ? (double)R.eps32[k * N + i] : (double)eps[k * N + i];
        m[h] = (double)mu[i];
        l[h] = (double)lam[i];
#pragma unroll
        for (int k = 0; k < 3; ++k) pl[h][k] = (double)ep[k * N + i];
      }
      T tr[2][3];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const long long i = (2LL * (p0 + q) + h) * NY + y;
        double ev[3];
        if (first == 0) {
          const C z0 = vx[0], z1 = vx[SL], z2 = vx[2 * SL];
          ev[0] = eb0 + (double)(h == 0 ? z0.x : z0.y);
          ev[1] = eb1 + (double)(h == 0 ? z1.x : z1.y);
          ev[2] = eb2 + (double)(h == 0 ? z2.x : z2.y);
          const double q0 = ev[0] - o[h][0], q1 = ev[1] - o[h][1], q2 = ev[2] - o[h][2];
          d2 += q0 * q0 + q1 * q1 + 2.0 * q2 * q2;
          n2 += o[h][0] * o[h][0] + o[h][1] * o[h][1] + 2.0 * o[h][2] * o[h][2];
#pragma unroll
          for (int k = 0; k < 3; ++k) eps[k * N + i] = (T)ev[k];
        } else {
#pragma unroll
          for (int k = 0; k < 3; ++k) ev[k] = o[h][k];
          if constexpr (LAW != 0)
            if (R.aa) aa_mix_voxel(R, i, nmix, gam, ev);  // the mixed iterate
          if (sizeof(T) == 8 && first == 2)
#pragma unroll
            for (int k = 0; k < 3; ++k) eps[k * N + i] = (T)ev[k];
        }
        if (img_only) continue;
        const double tre = ev[0] + ev[1];
        double s0, s1, s2;  // LAW 0 linear; 1 secant, 2 Rose, 3 Landau (FP64 plans)
        law_sigma<LAW>(m[h], l[h], ev[0] - pl[h][0], ev[1] - pl[h][1], ev[2] - pl[h][2], law_a, law_b, law_ps, s0, s1,
                       s2, R.lp);
        tr[h][0] = (T)(s0 - (2 * mu0 * ev[0] + lam0 * tre));
        tr[h][1] = (T)(s1 - (2 * mu0 * ev[1] + lam0 * tre));
        tr[h][2] = (T)(s2 - 2 * mu0 * ev[2]);
      }
      if (!img_only)
#pragma unroll
        for (int k = 0; k < 3; ++k) vx[k * SL] = mk<C>(tr[0][k], tr[1][k]);
    }
    if constexpr (!ONE)
      if (first == 0 && (K == 1 || y >= NYP - TH)) fold(K == 1 ? e >> 5 : q * NCH + (threadIdx.x >> 5));
  }
  if constexpr (ONE)
    if (first == 0) fold(threadIdx.x >> 5);
  if (!img_only) {
    __syncthreads();
    reg_line<NY, -1, ALT, C, TL>(t, act, tw, [&](int i) -> C { return buf[reg_slot<NY, C>(i)]; }, at, put, sync, sync);
    sync();
    if (act) {
      C* ra = spec + ((long long)c * nx + 2 * (p0 + pr)) * ld;
      for (int k = t; k < NYH; k += TL) {
        const C z = buf[reg_slot<NY, C>(k)];
        const C w = buf[reg_slot<NY, C>(k == 0 ? 0 : NY - k)];
        ra[k] = mk<C>(T(0.5) * (z.x + w.x), T(0.5) * (z.y - w.y));
        ra[ld + k] = mk<C>(T(0.5) * (z.y + w.y), T(-0.5) * (z.x - w.x));
      }
    }
  }
  if (first != 0) return;
  __syncthreads();
  for (int q = threadIdx.x >> 5; q < np; q += TH / 32) {
    const int lane = threadIdx.x & 31;
    const double a = warp_sum(lane < NCH ? chunk[0][q * NCH + lane] : 0.0);
    const double b = warp_sum(lane < NCH ? chunk[1][q * NCH + lane] : 0.0);
    if (lane == 0) {
      reinterpret_cast<double2*>(partials)[R.row_first + p0 + q] = make_double2(a, b);
      __threadfence();
    }
  }
  if constexpr (P > 1) __syncthreads();
  if (threadIdx.x == 0) s_last = atomicInc(&rep_counter[r], (unsigned int)per - 1) == (unsigned int)per - 1;  // self-resetting
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  ls2d_decide(R, S, partials, ctl, cond, use_cond, guard_cap, final != 0);
}

// Thread = (component, t, column), the column fastest: a warp's loads cover
// whole rows of the tile, and the exchange is stored column-fastest too.
template <typename T, int NX, int W, int TL, int ALT>
__global__ void __launch_bounds__(ls2_c_threads(W, TL), ls2_minb(ls2_c_threads(W, TL), 2 * (int)sizeof(T)))
    ls2_col_reg(const Ls2dRep* __restrict__ reps, const Ls2dState* __restrict__ st, const int* __restrict__ sel) {
  using C = C_t<T>;
  constexpr int SL = reg_slots(NX, sizeof(C)), TH = ls2_c_threads(W, TL);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nyh = reps[sel[0]].nyh, per = (nyh + W - 1) / W;
  const int r = sel[blockIdx.x / per], k0 = blockIdx.x % per * W;
  const Ls2dRep& R = reps[r];
  const Ls2dState& S = st[r];
  if (S.done != 0) return;
  const int ny = R.ny, ld = R.ld, tcw = min(W, nyh - k0);
  const int col = threadIdx.x % W, t = threadIdx.x / W % TL, c = threadIdx.x / (W * TL);
  const bool act = c < 3 && col < tcw;
  C* g = reinterpret_cast<C*>(R.spec) + (long long)min(c, 2) * NX * ld + k0 + (col < tcw ? col : 0);
  C* lines = reinterpret_cast<C*>(smem_raw);
  C* buf = lines + min(c, 2) * (SL * W) + col;
  const C* tw = Twid<T>::get(R, 0);
  auto at = [&](int s) -> C& { return buf[s * W]; };
  auto put = [&](int i, C v) { buf[reg_slot<NX, C>(i) * W] = v; };
  auto sync = [] {
    if constexpr (32 % (TL * W) == 0) __syncwarp();
    else __syncthreads();
  };
  reg_line<NX, -1, ALT, C, TL>(t, act, tw, [&](int i) -> C { return g[i * ld]; }, at, put, sync, [] {});
  __syncthreads();
  // Gamma0 in the precision of the pass.
  const T scale = (T)(1.0 / ((double)NX * (double)ny));
  const T a0 = (T)S.inv2mu0, b0 = (T)S.Bc;
#pragma unroll 1
  for (int e = threadIdx.x; e < W * NX; e += TH) {
    const int w = e % W, kx = e / W, ky = k0 + w;
    if (w >= tcw) continue;
    C* p = lines + reg_slot<NX, C>(kx) * W + w;
    const C txx = p[0], tyy = p[SL * W], txy = p[2 * SL * W];
    const bool nqx = (NX & 1) == 0 && 2 * kx == NX, nqy = (ny & 1) == 0 && 2 * ky == ny;
    const bool nq = nqx || nqy;
    C exx, eyy, exy;
    if constexpr (sizeof(T) == 8) {
      // with u the wave vector, n = u/|u| only enters squared, so one division
      // by |u|^2 replaces the square root
      const T ux = (T)fftfreq(kx, NX) / (T)NX, uy = (T)fftfreq(ky, ny) / (T)ny;
      const T uu = ux * ux + uy * uy;
      const T i2 = uu > T(0) ? T(1) / uu : T(0);  // the mean stays zero
      const T f = (nq ? T(0.5) : T(1)) * scale * i2;
      gamma2d_apply(txx, tyy, txy, ux, uy, a0 * f, b0 * f * i2, exx, eyy, exy);
      if (nq) {
        C fxx, fyy, fxy;
        gamma2d_apply(txx, tyy, txy, nqx ? -ux : ux, nqy ? -uy : uy, a0 * f, b0 * f * i2, fxx, fyy, fxy);
        exx = cadd(exx, fxx);
        eyy = cadd(eyy, fyy);
        exy = cadd(exy, fxy);
      }
    } else {
      // the roundings of the FP32 passes (see reg_sched32): the direction from
      // double in the CTA-wide ones
      T nxv, nyv;
      if constexpr (ALT) {
        const double ux = (double)fftfreq(kx, NX) / NX, uy = (double)fftfreq(ky, ny) / ny;
        const double inv = 1.0 / sqrt(ux * ux + uy * uy);
        nxv = (T)(ux * inv);
        nyv = (T)(uy * inv);
      } else {
        const T ux = (T)fftfreq(kx, NX) / (T)NX, uy = (T)fftfreq(ky, ny) / (T)ny;
        const T inv = T(1) / sqrtf(__fmaf_rn(ux, ux, __fmul_rn(uy, uy)));
        nxv = ux * inv;
        nyv = uy * inv;
      }
      gamma2d_f32(txx.x, tyy.x, txy.x, nxv, nyv, a0, b0, exx.x, eyy.x, exy.x);
      gamma2d_f32(txx.y, tyy.y, txy.y, nxv, nyv, a0, b0, exx.y, eyy.y, exy.y);
      if (nq) {
        C fxx, fyy, fxy;
        const T mx = nqx ? -nxv : nxv, my = nqy ? -nyv : nyv;
        gamma2d_f32(txx.x, tyy.x, txy.x, mx, my, a0, b0, fxx.x, fyy.x, fxy.x);
        gamma2d_f32(txx.y, tyy.y, txy.y, mx, my, a0, b0, fxx.y, fyy.y, fxy.y);
        exx = mk<C>(T(0.5) * (exx.x + fxx.x), T(0.5) * (exx.y + fxx.y));
        eyy = mk<C>(T(0.5) * (eyy.x + fyy.x), T(0.5) * (eyy.y + fyy.y));
        exy = mk<C>(T(0.5) * (exy.x + fxy.x), T(0.5) * (exy.y + fxy.y));
      }
      const bool mean = kx == 0 && ky == 0;
      exx = mean ? mk<C>(T(0), T(0)) : mk<C>(exx.x * scale, exx.y * scale);
      eyy = mean ? mk<C>(T(0), T(0)) : mk<C>(eyy.x * scale, eyy.y * scale);
      exy = mean ? mk<C>(T(0), T(0)) : mk<C>(exy.x * scale, exy.y * scale);
    }
    p[0] = exx;
    p[SL * W] = eyy;
    p[2 * SL * W] = exy;
  }
  __syncthreads();
  reg_line<NX, +1, ALT, C, TL>(t, act, tw, [&](int i) -> C { return buf[reg_slot<NX, C>(i) * W]; }, at,
                      [&](int i, C v) { g[i * ld] = v; }, sync, sync);
}

// ------------------------------------------------------------- kernels ---
// The kernels of one line length with their launch shapes; index 0 the narrow
// form, 1 the wide one (the same where they coincide).  Kinds: FP64; FP32 with
// the roundings of the former warp-line kernels (the lengths of warp_fft_len)
// or of the CTA-wide passes (every length).
enum { kLs2Fp64 = 0, kLs2Fp32 = 1, kLs2Fp32Wide = 2 };
struct Ls2Line {
  const void* row[4][2];  // by law; FP32: linear only
  const void* col[2];
  int pairs[2], r_threads[2], r_bytes[2];
  int cols[2], c_threads[2], c_bytes[2];
};
const Ls2Line* ls2_line(int n, int kind);  // null: no instantiation

template <typename T, int N, int ALT> static const Ls2Line* ls2_make() {
  constexpr int cs = 2 * (int)sizeof(T);
  static const Ls2Line L = [] {
    constexpr int P = ls2_pairs(N), W0 = ls2_cols(N, cs, false), W1 = ls2_cols(N, cs, true);
    constexpr int T0 = ls2_t(N, cs, false), T1 = ls2_t(N, cs, true);
    Ls2Line k{};
    k.row[0][0] = (const void*)ls2_row_reg<T, N, 1, T0, 0, ALT>;
    k.row[0][1] = (const void*)ls2_row_reg<T, N, P, T1, 0, ALT>;
    if constexpr (sizeof(T) == 8) {
      k.row[1][0] = (const void*)ls2_row_reg<T, N, 1, T0, 1, 0>;
      k.row[1][1] = (const void*)ls2_row_reg<T, N, P, T1, 1, 0>;
      k.row[2][0] = (const void*)ls2_row_reg<T, N, 1, T0, 2, 0>;
      k.row[2][1] = (const void*)ls2_row_reg<T, N, P, T1, 2, 0>;
      k.row[3][0] = (const void*)ls2_row_reg<T, N, 1, T0, 3, 0>;
      k.row[3][1] = (const void*)ls2_row_reg<T, N, P, T1, 3, 0>;
    }
    k.col[0] = (const void*)ls2_col_reg<T, N, W0, T0, ALT>;
    k.col[1] = (const void*)ls2_col_reg<T, N, W1, T1, ALT>;
    const int p[2] = {1, P}, w[2] = {W0, W1}, t[2] = {T0, T1};
    for (int i = 0; i < 2; ++i) {
      k.pairs[i] = p[i];
      k.r_threads[i] = ls2_r_threads(N, p[i], t[i]);
      k.r_bytes[i] = ls2_r_bytes(N, p[i], cs);
      k.cols[i] = w[i];
      k.c_threads[i] = ls2_c_threads(w[i], t[i]);
      k.c_bytes[i] = ls2_c_bytes(N, w[i], cs);
    }
    return k;
  }();
  return &L;
}

template <int N> static const Ls2Line* ls2_pick(int kind) {
  if (kind == kLs2Fp64) return ls2_make<double, N, 0>();
  if constexpr (warp_fft_len(N)) {
    if (kind == kLs2Fp32) return ls2_make<float, N, 0>();
  }
  return kind == kLs2Fp32Wide ? ls2_make<float, N, 1>() : nullptr;
}

}  // namespace mgk
