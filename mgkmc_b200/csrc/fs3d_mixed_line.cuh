// The mixed form's FP32 matvec passes on register FFTs (fft_reg.cuh), one
// instantiation per line length, with the roundings of the passes they replace:
// the radices of fft.cuh, and ALT, the product that a complex multiplication
// rounds (0 the warp-line kernels that served sides 64, 96 and 128 only, 1 the
// CTA-wide passes of other grids, which remain for lengths without a register
// FFT).  Sums keep their order.
//
//   z forward  CTA of a pair of z-lines x 9 components x T threads: p = r + beta
//              p, A = K:p per voxel into shared memory, R2C;
//   y          CTA of one tensor row (3 components) x tile of kz columns;
//   x          all 9 components x tile: forward, G, inverse;
//   z inverse  CTA of one pair: C2R, q, the p.q partial.
//
// What bounds them: HBM, 45 + 2 x 18 + 18 + 27 floats per voxel.  The former
// passes crossed shared memory about twice per radix pass and wrote A to memory
// between K:p and the z transform.  At 128^3, before and now (CUDA events around
// each launch): K:p with z forward 202 and 133 us, y 56 and 37, x 88 and 61, y
// inverse 53 and 33, z inverse 66 and 54.  72^3, from CTA-wide passes: 301 and
// 129 us an iteration.
#pragma once
#include "fft_reg.cuh"
#include "fs3d_mixed_dev.cuh"
#include "tma.cuh"

namespace mgk {
namespace fs32 {

constexpr int up32(int n) { return (n + 31) / 32 * 32; }
constexpr int ml_t(int n) { return reg_sched32(n).t; }
constexpr int ml_ld(int n) { return (n / 2 + 1 + 3) / 4 * 4; }  // row pitch of the half spectra
// one pair of lines per z CTA: with two, 64^3 took 13.9 instead of 12.7 ms a load
// step, 96^3 45 instead of 39
constexpr int ml_zf_threads(int n) { return up32(9 * ml_t(n)); }
// z inverse: the threads (and with them the order of the sums) of the passes
// that it replaces.  The nine lines have to fit: 256 points, 32 threads a line, have
// no instantiation, and an axis of that length takes the CTA-wide passes (the FP64
// form has one)
constexpr int ml_zi_threads(int alt) { return alt ? 256 : 96; }
// columns per tile: 64-byte rows in y, 32-byte rows in x, less on lines of many
// threads
constexpr int ml_yw(int n) { return ml_t(n) <= 9 ? 8 : ml_t(n) <= 18 ? 4 : 2; }
constexpr int ml_xw(int n) { return ml_t(n) <= 14 ? 4 : 2; }
constexpr int ml_y_threads(int n) { return up32(3 * ml_yw(n) * ml_t(n)); }
constexpr int ml_x_threads(int n) { return up32(9 * ml_xw(n) * ml_t(n)); }
constexpr int ml_zf_bytes(int n) { return 9 * reg_slots(n, 8) * 8; }
constexpr int ml_zi_bytes(int n) {
  const int a = 9 * reg_slots(n, 8), b = 18 * ml_ld(n);
  return (a > b ? a : b) * 8;
}
constexpr int ml_y_bytes(int n) { return 3 * ml_yw(n) * reg_slots(n, 8) * 8; }
constexpr int ml_x_bytes(int n) { return 9 * ml_xw(n) * reg_slots(n, 8) * 8; }
constexpr int ml_minb(int threads, int regs = 80) { return 65536 / (threads * regs) < 1 ? 1 : 65536 / (threads * regs); }
// x pass: a third CTA of 288 threads where no step has more than 16 points per
// thread (128 points: 65 -> 60 us; 96 points, radix 24: 39.0 and 39.5 us)
constexpr int ml_x_regs(int n) { return reg_sched32(n).r[0] > 16 || reg_sched32(n).r[1] > 16 ? 80 : 72; }

template <int NZ, int ALT>
__global__ void __launch_bounds__(ml_zf_threads(NZ), ml_minb(ml_zf_threads(NZ))) ml_zfwd(Fs32Args a) {
  using C = float2;
  constexpr int TL = ml_t(NZ), TH = ml_zf_threads(NZ), SL = reg_slots(NZ, 8), NZH = NZ / 2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const long long N = a.N, plane = (long long)a.nx * a.ny * a.ld;
  const long long l0 = 2LL * blockIdx.x;  // first line
  C* lines = reinterpret_cast<C*>(smem_raw);
  const double beta = a.sc->beta;
  // one voxel per thread and round, the two lines of a pair interleaved
#pragma unroll 1
  for (int e = threadIdx.x; e < 2 * NZ; e += TH) {
    const int h = e & 1, z = e >> 1;
    const long long i = (l0 + h) * NZ + z;
    float* vx = reinterpret_cast<float*>(lines + reg_slot<NZ, C>(z)) + h;
    float d[9], out[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const double rv = (double)a.r32[k * N + i];
      d[k] = beta == 0.0 ? (float)rv : (float)(rv + beta * (double)a.p32[k * N + i]);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) a.p32[k * N + i] = d[k];
    kdf_state<float>(a, i, d, out);
#pragma unroll
    for (int k = 0; k < 9; ++k) vx[k * 2 * SL] = out[k];
  }
  __syncthreads();
  const int c = min(threadIdx.x / TL, 8), t = threadIdx.x % TL;
  const bool act = threadIdx.x < 9 * TL;
  C* buf = lines + c * SL;
  auto at = [&](int s) -> C& { return buf[s]; };
  auto sync = [] {
    if constexpr (32 % TL == 0) __syncwarp();
    else __syncthreads();
  };
  reg_line<NZ, -1, ALT, C>(t, act, reinterpret_cast<const C*>(a.rtw32[2]),
                           [&](int i) -> C { return buf[reg_slot<NZ, C>(i)]; }, at,
                           [&](int i, C v) { buf[reg_slot<NZ, C>(i)] = v; }, sync, sync);
  sync();
  if (act) {
    C* ra = reinterpret_cast<C*>(a.spec) + c * plane + l0 * a.ld;
    for (int k = t; k < NZH; k += TL) {
      const C z = buf[reg_slot<NZ, C>(k)];
      const C w = buf[reg_slot<NZ, C>(k == 0 ? 0 : NZ - k)];
      ra[k] = mk<C>(0.5f * (z.x + w.x), 0.5f * (z.y - w.y));
      ra[a.ld + k] = mk<C>(0.5f * (z.y + w.y), -0.5f * (z.x - w.x));
    }
  }
}

template <int NZ, int ALT> __global__ void __launch_bounds__(ml_zi_threads(ALT)) ml_zinv(Fs32Args a) {
  using C = float2;
  constexpr int TL = ml_t(NZ), TH = ml_zi_threads(ALT), SL = reg_slots(NZ, 8), ld = ml_ld(NZ);
  static_assert(9 * TL <= TH, "lines");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  __shared__ __align__(8) uint64_t bar;
  const long long N = a.N, plane = (long long)a.nx * a.ny * ld;
  const long long l0 = 2LL * blockIdx.x;
  C* lines = reinterpret_cast<C*>(smem_raw);
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    mbar_arrive_expect_tx(&bar, 18u * ld * sizeof(C));
#pragma unroll
    for (int q = 0; q < 9; ++q)
      bulk_g2s(lines + q * 2 * ld, reinterpret_cast<const C*>(a.spec) + q * plane + l0 * ld, 2u * ld * sizeof(C), &bar);
  }
  const int c = min(threadIdx.x / TL, 8), t = threadIdx.x % TL;
  const bool act = threadIdx.x < 9 * TL;
  C* buf = lines + c * SL;
  const C* sa = lines + c * 2 * ld;
  auto at = [&](int s) -> C& { return buf[s]; };
  auto sync = [] {
    if constexpr (32 % TL == 0) __syncwarp();
    else __syncthreads();
  };
  __syncthreads();  // the barrier is initialised
  if (!__syncthreads_and(mbar_wait(&bar, 0) ? 1 : 0)) {
    if (threadIdx.x == 0) { a.sc->err = 1.0; a.part[blockIdx.x] = 0.0; }
    return;
  }
  auto load = [&](int k) -> C {
    const int ks = 2 * k <= NZ ? k : NZ - k;
    C x = sa[ks], y = sa[ld + ks];
    if (k == 0 || 2 * k == NZ) { x.y = 0; y.y = 0; }
    return 2 * k <= NZ ? mk<C>(x.x - y.y, x.y + y.x) : mk<C>(x.x + y.y, y.x - x.y);
  };
  reg_line<NZ, +1, ALT, C>(t, act, reinterpret_cast<const C*>(a.rtw32[2]), load, at,
                           [&](int i, C v) { buf[reg_slot<NZ, C>(i)] = v; }, sync, [] { __syncthreads(); });
  __syncthreads();
  double acc = 0;
  if constexpr (ALT == 0) {
#pragma unroll 1
    for (int z = threadIdx.x; z < NZ; z += TH) {
      const C* vx = lines + reg_slot<NZ, C>(z);
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const C v = vx[k * SL];
        const long long i = k * N + l0 * NZ + z;
        a.q32[i] = v.x;
        acc += (double)a.p32[i] * (double)v.x;
        a.q32[i + NZ] = v.y;
        acc += (double)a.p32[i + NZ] * (double)v.y;
      }
    }
  } else {
    for (int e = threadIdx.x; e < 9 * NZ; e += TH) {
      const int k = e / NZ, z = e - k * NZ;
      const C v = lines[k * SL + reg_slot<NZ, C>(z)];
      const long long i = k * N + l0 * NZ + z;
      a.q32[i] = v.x;
      acc += (double)a.p32[i] * (double)v.x;
      a.q32[i + NZ] = v.y;
      acc += (double)a.p32[i + NZ] * (double)v.y;
    }
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) a.part[blockIdx.x] = acc;
}

// y pass of one tensor row; grid = nx * ntile * 3, the row fastest
template <int NL, int SIGN, int ALT>
__global__ void __launch_bounds__(ml_y_threads(NL), ml_minb(ml_y_threads(NL))) ml_ypass(Fs32Args a) {
  using C = float2;
  constexpr int TL = ml_t(NL), W = ml_yw(NL), SL = reg_slots(NL, 8);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int row = blockIdx.x % 3, item = blockIdx.x / 3;
  const int ld = a.ld, ntile = (a.nzh + W - 1) / W;
  const int o = item / ntile, k0 = (item - o * ntile) * W;
  const int tcw = min(W, a.nzh - k0);
  const long long plane = (long long)a.nx * NL * ld;
  const int col = threadIdx.x % W, t = threadIdx.x / W % TL, c = min(threadIdx.x / (W * TL), 2);
  const bool act = threadIdx.x < 3 * W * TL && col < tcw;
  C* g = reinterpret_cast<C*>(a.spec) + (3 * row + c) * plane + (long long)o * NL * ld + k0 + (col < tcw ? col : 0);
  C* buf = reinterpret_cast<C*>(smem_raw) + c * (SL * W) + col;
  auto at = [&](int s) -> C& { return buf[s * W]; };
  auto sync = [] {
    if constexpr (32 % (TL * W) == 0) __syncwarp();
    else __syncthreads();
  };
  reg_line<NL, SIGN, ALT, C>(t, act, reinterpret_cast<const C*>(a.rtw32[1]), [&](int i) -> C { return g[(long long)i * ld]; },
                             at, [&](int i, C v) { g[(long long)i * ld] = v; }, sync, [] {});
}

// x pass with G; grid = ny * ntile
template <int NL, int ALT>
__global__ void __launch_bounds__(ml_x_threads(NL), ml_minb(ml_x_threads(NL), ml_x_regs(NL))) ml_xpass(Fs32Args a) {
  using C = float2;
  constexpr int TL = ml_t(NL), W = ml_xw(NL), SL = reg_slots(NL, 8), TH = ml_x_threads(NL);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ld = a.ld, ny = a.ny, nz = a.nz, ntile = (a.nzh + W - 1) / W;
  const int ky = blockIdx.x / ntile, k0 = (blockIdx.x - ky * ntile) * W;
  const int tcw = min(W, a.nzh - k0);
  const long long js = (long long)ny * ld, plane = js * NL;
  const int col = threadIdx.x % W, t = threadIdx.x / W % TL, c = min(threadIdx.x / (W * TL), 8);
  const bool act = threadIdx.x < 9 * W * TL && col < tcw;
  C* g = reinterpret_cast<C*>(a.spec) + c * plane + (long long)ky * ld + k0 + (col < tcw ? col : 0);
  C* lines = reinterpret_cast<C*>(smem_raw);
  C* buf = lines + c * (SL * W) + col;
  const C* tw = reinterpret_cast<const C*>(a.rtw32[0]);
  auto at = [&](int s) -> C& { return buf[s * W]; };
  auto sync = [] {
    if constexpr (32 % (TL * W) == 0) __syncwarp();
    else __syncthreads();
  };
  reg_line<NL, -1, ALT, C>(t, act, tw, [&](int i) -> C { return g[i * js]; }, at,
                           [&](int i, C v) { buf[reg_slot<NL, C>(i) * W] = v; }, sync, [] {});
  __syncthreads();
  const float scale = (float)(1.0 / (double)a.N);
  const double uy = (double)ffq(ky, ny) / ny;
  const bool nqy = (ny & 1) == 0 && 2 * ky == ny;
#pragma unroll 1
  for (int e = threadIdx.x; e < W * NL; e += TH) {
    const int w = e % W, kx = e / W, kz = k0 + w;
    if (w >= tcw) continue;
    C* p = lines + reg_slot<NL, C>(kx) * W + w;
    const bool nqx = (NL & 1) == 0 && 2 * kx == NL, nqz = (nz & 1) == 0 && 2 * kz == nz;
    if ((kx == 0 && ky == 0 && kz == 0) || nqx || nqy || nqz) {
#pragma unroll
      for (int k = 0; k < 9; ++k) p[k * (SL * W)] = mk<C>(0.0f, 0.0f);
      continue;
    }
    const double ux = (double)ffq(kx, NL) / NL, uz = (double)ffq(kz, nz) / nz;
    const double inv = 1.0 / sqrt(ux * ux + uy * uy + uz * uz);
    const float n[3] = {(float)(ux * inv), (float)(uy * inv), (float)(uz * inv)};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      float vx = 0, vy = 0;
#pragma unroll
      for (int l = 0; l < 3; ++l) {
        const C A = p[(3 * i + l) * (SL * W)];
        vx += A.x * n[l];
        vy += A.y * n[l];
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) p[(3 * i + j) * (SL * W)] = mk<C>(vx * n[j] * scale, vy * n[j] * scale);
    }
  }
  __syncthreads();
  reg_line<NL, +1, ALT, C>(t, act, tw, [&](int i) -> C { return buf[reg_slot<NL, C>(i) * W]; }, at,
                           [&](int i, C v) { g[i * js] = v; }, sync, sync);
}

// The kernels of one line length, with their launch shapes.
struct MixedLine {
  const void *zfwd, *zinv, *y[2], *x;
  int zf_threads, zi_threads, yw, xw, y_threads, x_threads;
  int zf_bytes, zi_bytes, y_bytes, x_bytes;
};
const MixedLine* mixed_line(int n, int alt);  // null: no instantiation

template <int N, int ALT> static const MixedLine* mixed_make() {
  static const MixedLine L = [] {
    MixedLine k{};
    k.zfwd = (const void*)ml_zfwd<N, ALT>;
    k.zinv = (const void*)ml_zinv<N, ALT>;
    k.y[0] = (const void*)ml_ypass<N, -1, ALT>;
    k.y[1] = (const void*)ml_ypass<N, 1, ALT>;
    k.x = (const void*)ml_xpass<N, ALT>;
    k.zf_threads = ml_zf_threads(N);
    k.zi_threads = ml_zi_threads(ALT);
    k.yw = ml_yw(N);
    k.xw = ml_xw(N);
    k.y_threads = ml_y_threads(N);
    k.x_threads = ml_x_threads(N);
    k.zf_bytes = ml_zf_bytes(N);
    k.zi_bytes = ml_zi_bytes(N);
    k.y_bytes = ml_y_bytes(N);
    k.x_bytes = ml_x_bytes(N);
    return k;
  }();
  return &L;
}

}  // namespace fs32
}  // namespace mgk
