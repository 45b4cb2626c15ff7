// 3D small-strain iteration kernels on register FFTs (fft_reg.cuh), one
// instantiation per line length; lengths without one take the CTA-wide passes
// of ls3d.cu.
//
//   z-line   CTA of ls3_zp pairs of z-lines x 6 components x T threads: C2R
//            along z of the previous spectrum, eps update with the diff/norm
//            partials and the convergence decision, tau, R2C along z;
//   y pass   CTA of 3 components x tile of kz columns x T threads;
//   x pass   the same with all 6 components: forward, Gamma0, inverse.
//
// What bounds them: each pass moves its spectrum once in each direction
// (6 x 16 bytes per frequency), the z-line kernel also 20 fields of 8 bytes per
// voxel, so HBM; the former passes through padded shared memory (radix 8 and 4
// steps, two shared-memory accesses per point and step, strided twiddles) ran
// at 60 % of the L1 rate and 0.25 .. 0.4 of HBM with 12 .. 15 warps per SM.  Here
// a point crosses shared memory once per transform (twice more around Gamma0),
// a thread has 8 .. 16 independent loads in flight, the spectrum rows of the
// z-lines come by bulk copies, and their fields are asked into L2 while the
// spectrum is inverted.  FP64 at 128^3, before and now: z-lines 197 and 130 us
// (540 MB: 0.63 of the measured copy rate), x pass 113 and 70 us, y pass 71 and
// 42 us (204 MB each: 0.45 and 0.74).
#pragma once
#include "fft_reg.cuh"
#include "ls3d_dev.cuh"
#include "tma.cuh"

namespace mgk {

// ------------------------------------------------------------ geometry ---
constexpr int round32(int n) { return (n + 31) / 32 * 32; }
// Line pairs per z-line CTA, and its threads: those of the transforms, and
// enough for the voxel stage to run in one round of at most 192 voxel pairs or
// two equal ones (at 128 points 96 threads would take three rounds).
constexpr int ls3_zp(int n) { return reg_sched64(n).t <= 9 ? 2 : 1; }
constexpr int ls3_z_threads(int n, int csz) {
  const int fft = 6 * reg_sched(n, csz).t * ls3_zp(n), vox = ls3_zp(n) * n, rounds = (vox + 191) / 192;
  const int per = (vox + rounds - 1) / rounds;
  return round32(fft > per ? fft : per);
}
// row pitch of the half spectra (see mgk_ls3d_create_batch)
constexpr int ls3_ld(int n) { return (n / 2 + 1 + 3) / 4 * 4; }
// kz columns per tile: rows of 64 bytes (whole 32-byte sectors, spectra rows
// start on 64-byte boundaries), fewer where a CTA would pass 432 threads.  The
// x pass spends its time in the load-store pipe (58 % of its rate at 128^3,
// half of it the exchanges and Gamma0): tiles of 2 columns (79 us) and a third
// resident CTA at 96 registers (77 us) were slower than this (70 us).
constexpr int ls3_tile(int n, int csz) {
  return csz == 8 ? 8 : 6 * 4 * reg_sched64(n).t <= 432 ? 4 : 2;
}
constexpr int ls3_ax_threads(int n, int csz, int nc) { return round32(nc * ls3_tile(n, csz) * reg_sched(n, csz).t); }
// exchange buffers; they first hold the pairs' spectrum rows as copied
constexpr int ls3_z_bytes(int n, int csz) {
  const int a = ls3_zp(n) * 6 * reg_slots(n, csz), b = ls3_zp(n) * 12 * ls3_ld(n);
  return (a > b ? a : b) * csz;
}
constexpr int ls3_ax_bytes(int n, int csz, int nc) { return nc * ls3_tile(n, csz) * reg_slots(n, csz) * csz; }
// resident CTAs asked of the register allocator: as many as 128 registers per thread
// allow in FP64, 80 in FP32, rounded down (blocks of 192 threads, as the x pass at 128
// points, get two and up to 168 registers: 162)
constexpr int ls3_minb(int threads, int csz) {
  const int b = 65536 / (threads * (csz == 16 ? 128 : 80));
  return b < 1 ? 1 : b;
}

template <typename T> struct L3F;
template <> struct L3F<double> {
  static __device__ __forceinline__ double* eps(const Ls3dRep& R) { return R.eps; }
  static __device__ __forceinline__ const double* ep(const Ls3dRep& R) { return R.ep; }
  static __device__ __forceinline__ const double* mu(const Ls3dRep& R) { return R.mu; }
  static __device__ __forceinline__ const double* lam(const Ls3dRep& R) { return R.lam; }
  static __device__ __forceinline__ double2* spec(const Ls3dRep& R) { return R.spec; }
  static __device__ __forceinline__ const double2* tw(const Ls3dRep& R, int axis) { return R.rtw[axis]; }
};
template <> struct L3F<float> {
  static __device__ __forceinline__ float* eps(const Ls3dRep& R) { return R.eps32; }
  static __device__ __forceinline__ const float* ep(const Ls3dRep& R) { return R.ep32; }
  static __device__ __forceinline__ const float* mu(const Ls3dRep& R) { return R.mu32; }
  static __device__ __forceinline__ const float* lam(const Ls3dRep& R) { return R.lam32; }
  static __device__ __forceinline__ float2* spec(const Ls3dRep& R) { return reinterpret_cast<float2*>(R.spec); }
  static __device__ __forceinline__ const float2* tw(const Ls3dRep& R, int axis) { return R.rtw32[axis]; }
};

// ask `bytes` (a multiple of 16) at a 16-byte aligned address into L2
__device__ __forceinline__ void l2_prefetch(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// ------------------------------------------------------------- z-lines ---
// The launch covers the replicas sel[0 ..) of one shape, their items in
// order.  first: the field is read as is (first tau of a phase); otherwise the
// previous spectrum is inverted and the field updated.  lead: this launch
// counts the loop bodies.
template <typename T, int NZ, bool FINAL, int LAW>
__global__ void __launch_bounds__(ls3_z_threads(NZ, 2 * (int)sizeof(T)),
                                  ls3_minb(ls3_z_threads(NZ, 2 * (int)sizeof(T)), 2 * (int)sizeof(T)))
    ls3_zline_reg(const Ls3dRep* __restrict__ reps, Ls3dState* st, const int* __restrict__ sel, double* partials,
                  unsigned int* rep_counter, Ls3dCtl* ctl, cudaGraphConditionalHandle cond, int use_cond,
                  int guard_cap, int lead, int first) {
  using C = C_t<T>;
  constexpr int TL = reg_sched(NZ, sizeof(C)).t, P = ls3_zp(NZ), TH = ls3_z_threads(NZ, sizeof(C)), SL = reg_slots(NZ, sizeof(C));
  constexpr int NZH = NZ / 2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  __shared__ int s_last;
  __shared__ __align__(8) uint64_t bar;
  const int per = reps[sel[0]].zl_items;
  const int r = sel[blockIdx.x / per], loc = blockIdx.x % per;
  const Ls3dRep& R = reps[r];
  Ls3dState& S = st[r];
  if (!first && use_cond && lead && blockIdx.x == 0 && threadIdx.x == 0) {
    // a body with no active replica has no decider: stop here; the body
    // count bounds the loop whatever happens to the deciders
    const unsigned int b = atomicAdd(&ctl->bodies, 1u) + 1u;
    if (ctl->n_active == 0 || b > (unsigned int)guard_cap || *(volatile int*)&ctl->error != 0) {
      ctl->any = 0;
      cudaGraphSetConditional(cond, 0u);
    }
  }
  if (S.done != 0) return;
  const long long N = R.N;
  const int ld = R.ld;
  const long long plane = (long long)R.nx * R.ny * ld;
  const long long p0 = (long long)loc * P;  // first pair
  const int np = (int)min((long long)P, (long long)R.nx * R.ny / 2 - p0);
  T* eps = L3F<T>::eps(R);
  const T *mu = L3F<T>::mu(R), *lam = L3F<T>::lam(R), *ep = L3F<T>::ep(R);
  C* lines = reinterpret_cast<C*>(smem_raw);
  if (!first && threadIdx.x == 0) {
    // the pairs' half-spectrum rows, contiguous per component
    const uint32_t bytes = 2u * np * ld * sizeof(C);
    mbar_init(&bar, 1);
    fence_mbar_init();
    mbar_arrive_expect_tx(&bar, 6u * bytes);
#pragma unroll
    for (int q = 0; q < 6; ++q)
      bulk_g2s(lines + q * 2 * P * ld, L3F<T>::spec(R) + q * plane + 2 * p0 * ld, bytes, &bar);
  }
  if (threadIdx.x >= 32 && threadIdx.x < 46) {
    const int q = threadIdx.x - 32;
    const T* f = q < 6 ? eps + q * N : q == 6 ? mu : q == 7 ? lam : ep + (q - 8) * N;
    l2_prefetch(f + 2 * p0 * NZ, (uint32_t)(2 * np * NZ * sizeof(T)));
  }
  const C* tw = L3F<T>::tw(R, 2);
  const int line = threadIdx.x / TL, t = threadIdx.x % TL;  // line = 6 pair + component
  const int pr = line / 6, c = line - 6 * pr;
  const bool act = line < 6 * P && pr < np;
  C* buf = lines + (line < 6 * P ? line : 0) * SL;
  C* ra = L3F<T>::spec(R) + c * plane + 2 * (p0 + pr) * ld;  // the pair's two rows: ra, ra + ld
  auto at = [&](int s) -> C& { return buf[s]; };
  auto put = [&](int i, C v) { buf[reg_slot<NZ, C>(i)] = v; };
  auto sync = [] {
    if constexpr (32 % TL == 0) __syncwarp();
    else __syncthreads();
  };
  if (!first) {
    __syncthreads();  // the barrier is initialised
    if (!__syncthreads_and(mbar_wait(&bar, 0) ? 1 : 0)) {
      if (threadIdx.x == 0) { ctl->error = 1; ctl->any = 0; }
      return;
    }
    const C* sa = lines + (c * P + pr) * 2 * ld;
    auto load = [&](int k) -> C {
      const int ks = 2 * k <= NZ ? k : NZ - k;
      C a = sa[ks], b = sa[ld + ks];
      if (k == 0 || 2 * k == NZ) { a.y = 0; b.y = 0; }
      return 2 * k <= NZ ? mk<C>(a.x - b.y, a.y + b.x) : mk<C>(a.x + b.y, b.x - a.y);
    };
    reg_line<NZ, +1, 0, C>(t, act, tw, load, at, put, sync, [] { __syncthreads(); });
  }
  __syncthreads();
  const double mu0 = S.mu0, lam0 = S.lam0;
  double d2 = 0, n2 = 0;
#pragma unroll 1
  for (int e = threadIdx.x; e < np * NZ; e += TH) {
    const int q = e / NZ, z = e - q * NZ;
    C* vx = lines + q * 6 * SL + reg_slot<NZ, C>(z);
    // every input of the two voxels before the first store
    T o[2][6], m[2], l[2], pl[2][6];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long i = (2 * (p0 + q) + h) * NZ + z;
#pragma unroll
      for (int k = 0; k < 6; ++k) o[h][k] = eps[k * N + i];
      m[h] = mu[i];
      l[h] = lam[i];
#pragma unroll
      for (int k = 0; k < 6; ++k) pl[h][k] = ep[k * N + i];
    }
    T tr[2][6];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long i = (2 * (p0 + q) + h) * NZ + z;
      double ev[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const double ov = (double)o[h][k];
        if (!first) {
          const C zz = vx[k * SL];
          const double nw = S.ebar[k] + (double)(h == 0 ? zz.x : zz.y);
          const double dd = nw - ov, w = k < 3 ? 1.0 : 2.0;
          d2 += w * dd * dd;
          n2 += w * ov * ov;
          eps[k * N + i] = (T)nw;
          ev[k] = nw;
        } else {
          ev[k] = ov;
        }
      }
      double mm = (double)m[h];
      const double ll = (double)l[h];
      double d[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) d[k] = ev[k] - (double)pl[h][k];
      if constexpr (LAW == 1) mm = secant_mu3(mm, d[0], d[1], d[2], d[3], d[4], d[5], R.law_a, R.law_b);
      const double trd = d[0] + d[1] + d[2], tre = ev[0] + ev[1] + ev[2];
      if constexpr (LAW == 3) {
        double sg[6];
        landau_sigma3(mm, ll, d, R.lp, sg);
#pragma unroll
        for (int k = 0; k < 6; ++k) tr[h][k] = (T)(sg[k] - (2 * mu0 * ev[k] + (k < 3 ? lam0 * tre : 0.0)));
      } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) tr[h][k] = (T)((2 * mm * d[k] + ll * trd) - (2 * mu0 * ev[k] + lam0 * tre));
#pragma unroll
        for (int k = 3; k < 6; ++k) tr[h][k] = (T)(2 * mm * d[k] - 2 * mu0 * ev[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) vx[k * SL] = mk<C>(tr[0][k], tr[1][k]);
  }
  __syncthreads();
  reg_line<NZ, -1, 0, C>(t, act, tw, [&](int i) -> C { return buf[reg_slot<NZ, C>(i)]; }, at, put, sync, sync);
  sync();
  if (act) {
    for (int k = t; k < NZH; k += TL) {
      const C z = buf[reg_slot<NZ, C>(k)];
      const C w = buf[reg_slot<NZ, C>(k == 0 ? 0 : NZ - k)];
      ra[k] = mk<C>(T(0.5) * (z.x + w.x), T(0.5) * (z.y - w.y));
      ra[ld + k] = mk<C>(T(0.5) * (z.y + w.y), T(-0.5) * (z.x - w.x));
    }
  }
  if (first) return;
  ls3d_decide<FINAL>(R, S, r, R.zl_first + loc, d2, n2, partials, rep_counter, ctl, cond, use_cond, guard_cap, red, &s_last);
}

// ---------------------------------------------------------- axis passes ---
// AXIS 1: FFT of sign SIGN along y; AXIS 0: FFT along x, Gamma0, inverse.
// Item of a replica: the other in-plane index o and a tile of kz columns;
// grid = items * (6 / NC), the component group fastest.  Thread = (component, t, column),
// the column fastest, so that a warp's loads cover whole 64-byte rows; the
// exchange is stored column-fastest too.
template <typename T, int NL, int AXIS, int SIGN>
__global__ void __launch_bounds__(ls3_ax_threads(NL, 2 * (int)sizeof(T), AXIS ? 3 : 6),
                                  ls3_minb(ls3_ax_threads(NL, 2 * (int)sizeof(T), AXIS ? 3 : 6), 2 * (int)sizeof(T)))
    ls3_axis_reg(const Ls3dRep* __restrict__ reps, const Ls3dState* __restrict__ st, const int* __restrict__ sel) {
  using C = C_t<T>;
  constexpr int NC = AXIS ? 3 : 6, TL = reg_sched(NL, sizeof(C)).t, W = ls3_tile(NL, sizeof(C)), SL = reg_slots(NL, sizeof(C));
  constexpr int TH = ls3_ax_threads(NL, sizeof(C), NC);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int c0 = (blockIdx.x % (6 / NC)) * NC;
  int item = blockIdx.x / (6 / NC);
  const int ntile = (reps[sel[0]].nzh + W - 1) / W;
  const int per = (AXIS ? reps[sel[0]].nx : reps[sel[0]].ny) * ntile;
  const int r = sel[item / per];
  item %= per;
  const Ls3dRep& R = reps[r];
  const Ls3dState& S = st[r];
  if (S.done != 0) return;
  const int nx = R.nx, ny = R.ny, nz = R.nz, nzh = R.nzh, ld = R.ld;
  const int o = item / ntile, k0 = (item - o * ntile) * W;
  const int tcw = min(W, nzh - k0);
  const long long plane = (long long)nx * ny * ld;
  const long long js = AXIS ? ld : (long long)ny * ld;
  const int col = threadIdx.x % W, t = threadIdx.x / W % TL, c = threadIdx.x / (W * TL);
  const bool act = c < NC && col < tcw;
  C* g = L3F<T>::spec(R) + (c0 + min(c, NC - 1)) * plane + (AXIS ? (long long)o * ny : (long long)o) * ld + k0 +
         (col < tcw ? col : 0);
  C* lines = reinterpret_cast<C*>(smem_raw);
  C* buf = lines + min(c, NC - 1) * (SL * W) + col;
  const C* tw = L3F<T>::tw(R, AXIS);
  auto at = [&](int s) -> C& { return buf[s * W]; };
  auto sync = [] {
    if constexpr (32 % (TL * W) == 0) __syncwarp();
    else __syncthreads();
  };
  auto load = [&](int i) -> C { return g[i * js]; };
  if constexpr (AXIS) {
    reg_line<NL, SIGN, 0, C>(t, act, tw, load, at, [&](int i, C v) { g[i * js] = v; }, sync, [] {});
  } else {
    auto put = [&](int i, C v) { buf[reg_slot<NL, C>(i) * W] = v; };

    reg_line<NL, -1, 0, C>(t, act, tw, load, at, put, sync, [] {});
    __syncthreads();
    // Gamma0 in the precision of the pass: FP64 iterations in double, the
    // FP32 phase of a mixed plan in float
    const T scale = T(1.0 / (double)R.N);
    const T a0 = (T)S.inv2mu0, b0 = (T)S.Bc;
    const T uy = (T)fftfreq3(o, ny) / (T)ny;
    const bool nqy = (ny & 1) == 0 && 2 * o == ny;
#pragma unroll 1
    for (int e = threadIdx.x; e < W * NL; e += TH) {
      const int w = e % W, kx = e / W, kz = k0 + w;
      if (w >= tcw) continue;
      C* p = lines + reg_slot<NL, C>(kx) * W + w;
      C tv[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) tv[k] = p[k * (SL * W)];
      const T ux = (T)fftfreq3(kx, nx) / (T)nx, uz = (T)fftfreq3(kz, nz) / (T)nz;
      const T uu = ux * ux + uy * uy + uz * uz;
      const bool nqx = (nx & 1) == 0 && 2 * kx == nx, nqz = (nz & 1) == 0 && 2 * kz == nz;
      const bool nq = nqx || nqy || nqz;
      C ev[6];
      if constexpr (sizeof(T) == 8) {
        // with u the wave vector, n = u/|u| only enters squared, so one
        // division by |u|^2 replaces the square root
        const T i2 = uu > T(0) ? T(1) / uu : T(0);  // the mean stays zero
        const T f = (nq ? T(0.5) : T(1)) * scale * i2;
        gamma3d_apply_t<T>(tv, ux, uy, uz, a0 * f, b0 * f * i2, ev);
        if (nq) {
          C fv[6];
          gamma3d_apply_t<T>(tv, nqx ? -ux : ux, nqy ? -uy : uy, nqz ? -uz : uz, a0 * f, b0 * f * i2, fv);
#pragma unroll
          for (int k = 0; k < 6; ++k) ev[k] = cadd(ev[k], fv[k]);
        }
      } else {
        // the roundings of the FP32 passes (see reg_sched32)
        const T inv = T(1) / sqrt(uu), n0 = ux * inv, n1 = uy * inv, n2 = uz * inv;
        gamma3d_apply_t<T>(tv, n0, n1, n2, a0, b0, ev);
        if (nq) {
          C fv[6];
          gamma3d_apply_t<T>(tv, nqx ? -n0 : n0, nqy ? -n1 : n1, nqz ? -n2 : n2, a0, b0, fv);
#pragma unroll
          for (int k = 0; k < 6; ++k) ev[k] = mk<C>(T(0.5) * (ev[k].x + fv[k].x), T(0.5) * (ev[k].y + fv[k].y));
        }
        const bool mean = kx == 0 && o == 0 && kz == 0;
#pragma unroll
        for (int k = 0; k < 6; ++k)
          ev[k] = mean ? mk<C>(T(0), T(0)) : mk<C>(ev[k].x * scale, ev[k].y * scale);
      }
#pragma unroll
      for (int k = 0; k < 6; ++k) p[k * (SL * W)] = ev[k];
    }
    __syncthreads();
    reg_line<NL, +1, 0, C>(t, act, tw, [&](int i) -> C { return buf[reg_slot<NL, C>(i) * W]; }, at,
                        [&](int i, C v) { g[i * js] = v; }, sync, sync);
  }
}

// ------------------------------------------------------------- kernels ---
// The kernels of one line length in one precision, with their launch shapes
// (FP32: the mixed form's, sides 64, 96 and 128).
struct Ls3Line {
  const void* zline[4];  // by law (2 unused)
  const void* y[2];      // forward, inverse
  const void* x;
  int zp, z_threads, tile, y_threads, x_threads;
  int z_bytes, y_bytes, x_bytes;
};
const Ls3Line* ls3_line(int n, int prec);  // null: no instantiation

template <typename T, int N, bool FINAL> static const Ls3Line* ls3_make() {
  constexpr int cs = 2 * (int)sizeof(T);
  static const Ls3Line L = [] {
    Ls3Line k{};
    k.zline[0] = (const void*)ls3_zline_reg<T, N, FINAL, 0>;
    if constexpr (sizeof(T) == 8) {
      k.zline[1] = (const void*)ls3_zline_reg<T, N, FINAL, 1>;
      k.zline[3] = (const void*)ls3_zline_reg<T, N, FINAL, 3>;
    }
    k.y[0] = (const void*)ls3_axis_reg<T, N, 1, -1>;
    k.y[1] = (const void*)ls3_axis_reg<T, N, 1, 1>;
    k.x = (const void*)ls3_axis_reg<T, N, 0, 0>;
    k.zp = ls3_zp(N);
    k.z_threads = ls3_z_threads(N, cs);
    k.tile = ls3_tile(N, cs);
    k.y_threads = ls3_ax_threads(N, cs, 3);
    k.x_threads = ls3_ax_threads(N, cs, 6);
    k.z_bytes = ls3_z_bytes(N, cs);
    k.y_bytes = ls3_ax_bytes(N, cs, 3);
    k.x_bytes = ls3_ax_bytes(N, cs, 6);
    return k;
  }();
  return &L;
}

}  // namespace mgk
