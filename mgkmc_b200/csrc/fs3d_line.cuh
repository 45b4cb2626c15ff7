// Finite-strain matvec kernels on register FFTs (fft_reg.cuh), one
// instantiation per line length; axes of other lengths take the general
// kernels of fs3d.cu.
//
//   z-line   CTA of a pair of z-lines x 9 components x T threads: C2R of
//            the increment's spectrum, K:p per voxel, R2C of the product; the
//            real fields exist in shared memory only;
//   y pass   CTA of one tensor row (3 components) x tile of kz columns;
//   x pass   CTA of three rows (2 lines each) x tile of kz columns.
//
// See fs3d.cu for what the lines of a row are.
#pragma once
#include "fft_reg.cuh"
#include "fs3d_dev.cuh"
#include "tma.cuh"

namespace mgk {

// ------------------------------------------------------------ geometry ---
constexpr int fs_round32(int n) { return (n + 31) / 32 * 32; }
// row pitch of the half spectra: rows start on 64-byte boundaries
__host__ __device__ constexpr int fs_ld(int n) { return (n / 2 + 1 + 3) / 4 * 4; }
constexpr int fs_z_threads(int n) { return fs_round32(9 * reg_sched64(n).t); }
// kz columns per tile: whole 32-byte sectors per row, within 432 threads for
// the six lines of the x pass
constexpr int fs_tile(int n) { return reg_sched64(n).t <= 18 ? 4 : 2; }
constexpr int fs_ax_threads(int n, int nc) { return fs_round32(nc * fs_tile(n) * reg_sched64(n).t); }
// exchange buffers; they first hold the pairs' spectrum rows as copied
constexpr int fs_z_bytes(int n) {
  const int a = 9 * reg_slots(n, 16), b = 18 * fs_ld(n);
  return (a > b ? a : b) * 16;
}
constexpr int fs_ax_bytes(int n, int nc) { return nc * fs_tile(n) * reg_slots(n, 16) * 16; }
// resident CTAs asked of the register allocator: as many as 128 registers per thread
// allow, rounded down (the compiler takes what is left over), in the x passes 112 (a third CTA of 192 threads at 128 points, 118 registers without
// being asked: 80 and 98 us -> 73 and 80 us; in the y passes the spills cost more:
// 57 and 63 us -> 96 and 82 us)
constexpr int fs_minb(int threads, int regs = 128) {
  const int b = 65536 / (threads * regs);
  return b < 1 ? 1 : b;
}

// ------------------------------------------------------------- z-lines ---
// MODE 0: the matvec's (inverse, K:p, forward); 1: forward of K:dbar; 2:
// forward of P; 3: inverse of the increment into the real field X.
template <int NZ, int MODE, int MODEL>
__global__ void __launch_bounds__(fs_z_threads(NZ),
                                  fs_minb(fs_z_threads(NZ)))
    fs_zline_reg(FsArgs a) {
  using C = double2;
  constexpr int TL = reg_sched64(NZ).t, TH = fs_z_threads(NZ), SL = reg_slots(NZ, sizeof(C));
  constexpr int NZH = NZ / 2 + 1, ld = fs_ld(NZ);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar;
  const long long N = a.N, plane = a.plane;
  const long long l0 = 2LL * blockIdx.x;  // first line
  C* lines = reinterpret_cast<C*>(smem_raw);
  C* spec = reinterpret_cast<C*>(a.spec);
  if constexpr (MODE == 0 || MODE == 3) {
    if (threadIdx.x == 0) {
      // the pair's half-spectrum rows, contiguous per component
      const uint32_t bytes = 2u * ld * sizeof(C);
      mbar_init(&bar, 1);
      fence_mbar_init();
      mbar_arrive_expect_tx(&bar, 9u * bytes);
#pragma unroll
      for (int q = 0; q < 9; ++q) bulk_g2s(lines + q * 2 * ld, spec + q * plane + l0 * ld, bytes, &bar);
    }
  }
  if constexpr (MODE == 0) {
    // the voxels' tangent state into L2 meanwhile (rows that start on 16 bytes)
    if (threadIdx.x >= 32 && threadIdx.x < 32 + (MODEL == 1 ? 12 : 11)) {
      const double* f = reinterpret_cast<const double*>(a.st) + (threadIdx.x - 32) * N + l0 * NZ;
      const uint32_t bytes = 2u * NZ * sizeof(double);
      if (((reinterpret_cast<uintptr_t>(f) | bytes) & 15) == 0)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(f), "r"(bytes) : "memory");
    }
  }
  const C* tw = reinterpret_cast<const C*>(a.rtw[2]);
  const int c = min(threadIdx.x / TL, 8), t = threadIdx.x % TL;
  const bool act = threadIdx.x < 9 * TL;
  const bool third = c % 3 == 2;  // its spectrum is uz times the potential's
  C* buf = lines + c * SL;
  C* ra = spec + c * plane + l0 * ld;  // the pair's two rows: ra, ra + ld
  auto at = [&](int s) -> C& { return buf[s]; };
  auto put = [&](int i, C v) { buf[reg_slot<NZ, C>(i)] = v; };
  auto sync = [] {
    if constexpr (32 % TL == 0) __syncwarp();
    else __syncthreads();
  };
  if constexpr (MODE == 0 || MODE == 3) {
    __syncthreads();  // the barrier is initialised
    if (!__syncthreads_and(mbar_wait(&bar, 0) ? 1 : 0)) {
      if (threadIdx.x == 0) a.sc->err = 1.0;
      return;
    }
    const C* sa = lines + c * 2 * ld;
    auto load = [&](int k) -> C {
      const int ks = 2 * k <= NZ ? k : NZ - k;
      C x = sa[ks], y = sa[ld + ks];
      if (k == 0 || 2 * k == NZ) { x.y = 0; y.y = 0; }
      C z = 2 * k <= NZ ? mk<C>(x.x - y.y, x.y + y.x) : mk<C>(x.x + y.y, y.x - x.y);
      if (third) {
        const double u = ks * (1.0 / NZ);
        z.x *= u;
        z.y *= u;
      }
      return z;
    };
    reg_line<NZ, +1, 0, C>(t, act, tw, load, at, put, sync, [] { __syncthreads(); });
    __syncthreads();
  }
  if constexpr (MODE == 3) {
    for (int e = threadIdx.x; e < 9 * NZ; e += TH) {
      const int k = e / NZ, z = e - k * NZ;
      const C v = lines[k * SL + reg_slot<NZ, C>(z)];
      double* X = a.X + k * N + l0 * NZ + z;
      X[0] = v.x;
      X[NZ] = v.y;
    }
    return;
  }
  // one voxel per thread and round, the two lines of a pair interleaved
  // (8-byte words of consecutive lanes in consecutive banks)
#pragma unroll 1
  for (int e = threadIdx.x; e < 2 * NZ; e += TH) {
    const int h = e & 1, z = e >> 1;
    const long long i = (l0 + h) * NZ + z;
    double* vx = reinterpret_cast<double*>(lines + reg_slot<NZ, C>(z)) + h;
    double d[9], out[9];
    if constexpr (MODE == 2) {
#pragma unroll
      for (int k = 0; k < 9; ++k) out[k] = a.P[k * N + i];
    } else {
#pragma unroll
      for (int k = 0; k < 9; ++k) d[k] = MODE == 0 ? vx[k * 2 * SL] : a.sc->dbar[k];
      fs_kdf<MODEL>(a, i, d, out);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) vx[k * 2 * SL] = out[k];
  }
  __syncthreads();
  reg_line<NZ, -1, 0, C>(t, act, tw, [&](int i) -> C { return buf[reg_slot<NZ, C>(i)]; }, at, put, sync, sync);
  sync();
  if (act) {
    for (int k = t; k < NZH; k += TL) {
      const C z = buf[reg_slot<NZ, C>(k)];
      const C w = buf[reg_slot<NZ, C>(k == 0 ? 0 : NZ - k)];
      const double f = third ? 0.5 * (k * (1.0 / NZ)) : 0.5;
      ra[k] = mk<C>(f * (z.x + w.x), f * (z.y - w.y));
      ra[ld + k] = mk<C>(f * (z.y + w.y), -f * (z.x - w.x));
    }
  }
}

// ---------------------------------------------------------- axis passes ---
// Thread = (line, t, column), the column fastest, so that a warp's loads cover
// whole rows; the exchange is stored column-fastest too.

// y pass of one tensor row; grid = nx * ntile * 3, the row fastest.  SIGN -1:
// A_x, A_y, uz A_z -> X, B = uy A_y + uz A_z (planes 3 row, 3 row + 1); SIGN +1:
// X, the potential -> the row's increments along x and y, and the potential
// for the z pass.
template <int NL, int SIGN>
__global__ void __launch_bounds__(fs_ax_threads(NL, 3),
                                  fs_minb(fs_ax_threads(NL, 3)))
    fs_yline_reg(FsArgs a) {
  using C = double2;
  constexpr int TL = reg_sched(NL, sizeof(C)).t, W = fs_tile(NL), SL = reg_slots(NL, sizeof(C));
  constexpr int TH = fs_ax_threads(NL, 3);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int row = blockIdx.x % 3, item = blockIdx.x / 3;
  const int ld = a.ld, ntile = (a.nzh + W - 1) / W;
  const int o = item / ntile, k0 = (item - o * ntile) * W;
  const int tcw = min(W, a.nzh - k0);
  const int col = threadIdx.x % W, t = threadIdx.x / W % TL, c = min(threadIdx.x / (W * TL), 2);
  const bool act = threadIdx.x < 3 * W * TL && col < tcw;
  const long long base = (long long)o * NL * ld + k0;
  C* g = reinterpret_cast<C*>(a.spec) + 3 * row * a.plane + base + (col < tcw ? col : 0);
  C* out = g + c * a.plane;
  C* lines = reinterpret_cast<C*>(smem_raw);
  C* buf = lines + c * (SL * W) + col;
  const C* tw = reinterpret_cast<const C*>(a.rtw[1]);
  auto at = [&](int s) -> C& { return buf[s * W]; };
  auto sync = [] {
    if constexpr (32 % (TL * W) == 0) __syncwarp();
    else __syncthreads();
  };
  if constexpr (SIGN > 0) {
    // the row's second and third line both come from its second plane, which
    // the second one replaces: every load before the first store
    const C* in = g + (c == 0 ? 0 : a.plane);
    auto load = [&](int i) -> C {
      C v = in[(long long)i * ld];
      if (c == 1) {
        const double u = ffq(i, NL) * (1.0 / NL);
        v.x *= u;
        v.y *= u;
      }
      return v;
    };
    reg_line<NL, +1, 0, C>(t, act, tw, load, at, [&](int i, C v) { out[(long long)i * ld] = v; }, sync,
                           [] { __syncthreads(); });
  } else {
    auto store = [&](int i, C v) {
      if (c == 0) out[(long long)i * ld] = v;
      else buf[reg_slot<NL, C>(i) * W] = v;
    };
    reg_line<NL, -1, 0, C>(t, act, tw, [&](int i) -> C { return out[(long long)i * ld]; }, at, store, sync, [] {});
    __syncthreads();
    C* gb = reinterpret_cast<C*>(a.spec) + (3 * row + 1) * a.plane + base;
    for (int e = threadIdx.x; e < W * NL; e += TH) {
      const int w = e % W, ky = e / W;
      if (w >= tcw) continue;
      const C* p = lines + SL * W + reg_slot<NL, C>(ky) * W + w;
      const C y = p[0], z = p[SL * W];
      const double u = ffq(ky, NL) * (1.0 / NL);
      gb[(long long)ky * ld + w] = mk<C>(u * y.x + z.x, u * y.y + z.y);
    }
  }
}

// Forward x pass with G's contraction; grid = ny * ntile.  RHS: see
// fs_contract().
template <int NL, bool RHS>
__global__ void __launch_bounds__(fs_ax_threads(NL, 6),
                                  fs_minb(fs_ax_threads(NL, 6), 112))
    fs_xfwd_reg(FsArgs a) {
  using C = double2;
  constexpr int TL = reg_sched(NL, sizeof(C)).t, W = fs_tile(NL), SL = reg_slots(NL, sizeof(C));
  constexpr int TH = fs_ax_threads(NL, 6);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  const int ld = a.ld, ntile = (a.nzh + W - 1) / W;
  const int o = blockIdx.x / ntile, k0 = (blockIdx.x - o * ntile) * W;
  const int tcw = min(W, a.nzh - k0);
  const long long js = (long long)a.ny * ld;
  const int col = threadIdx.x % W, t = threadIdx.x / W % TL, c = min(threadIdx.x / (W * TL), 5);
  const bool act = threadIdx.x < 6 * W * TL && col < tcw;
  const C* g = reinterpret_cast<const C*>(a.spec) + (3 * (c >> 1) + (c & 1)) * a.plane + (long long)o * ld + k0 +
               (col < tcw ? col : 0);
  C* lines = reinterpret_cast<C*>(smem_raw);
  C* buf = lines + c * (SL * W) + col;
  const C* tw = reinterpret_cast<const C*>(a.rtw[0]);
  auto at = [&](int s) -> C& { return buf[s * W]; };
  auto sync = [] {
    if constexpr (32 % (TL * W) == 0) __syncwarp();
    else __syncthreads();
  };
  reg_line<NL, -1, 0, C>(t, act, tw, [&](int i) -> C { return g[i * js]; }, at,
                         [&](int i, C v) { buf[reg_slot<NL, C>(i) * W] = v; }, sync, [] {});
  __syncthreads();
  double s = 0;
#pragma unroll 1
  for (int e = threadIdx.x; e < W * NL; e += TH) {
    const int w = e % W, kx = e / W;
    if (w >= tcw) continue;
    const C* p = lines + reg_slot<NL, C>(kx) * W + w;
    C xv[3], bv[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) { xv[i] = p[2 * i * (SL * W)]; bv[i] = p[(2 * i + 1) * (SL * W)]; }
    s += fs_contract<RHS>(a, kx, o, k0 + w, xv, bv);
  }
  fs_finish(a, s, red, [&](double v) { fs_after_x<RHS>(a, v); });
}

// Inverse x pass: the direction's potential v and its lines X = ux v and v.
template <int NL, bool FINAL>
__global__ void __launch_bounds__(fs_ax_threads(NL, 6),
                                  fs_minb(fs_ax_threads(NL, 6), 112))
    fs_xinv_reg(FsArgs a) {
  using C = double2;
  constexpr int TL = reg_sched(NL, sizeof(C)).t, W = fs_tile(NL), SL = reg_slots(NL, sizeof(C));
  constexpr int TH = fs_ax_threads(NL, 6);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ld = a.ld, ntile = (a.nzh + W - 1) / W;
  const int o = blockIdx.x / ntile, k0 = (blockIdx.x - o * ntile) * W;
  const int tcw = min(W, a.nzh - k0);
  const long long js = (long long)a.ny * ld, base = (long long)o * ld + k0;
  C* lines = reinterpret_cast<C*>(smem_raw);
  const double beta = a.sc->beta;
#pragma unroll 2
  for (int e = threadIdx.x; e < W * NL; e += TH) {
    const int w = e % W, kx = e / W;
    if (w >= tcw) continue;
    C* p = lines + reg_slot<NL, C>(kx) * W + w;
    const double u = ffq(kx, NL) * (1.0 / NL);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const C v = fs_direction<FINAL>(a, beta, i * a.plane + kx * js + base + w);
      p[2 * i * (SL * W)] = mk<C>(u * v.x, u * v.y);
      p[(2 * i + 1) * (SL * W)] = v;
    }
  }
  __syncthreads();
  const int col = threadIdx.x % W, t = threadIdx.x / W % TL, c = min(threadIdx.x / (W * TL), 5);
  const bool act = threadIdx.x < 6 * W * TL && col < tcw;
  C* g = reinterpret_cast<C*>(a.spec) + (3 * (c >> 1) + (c & 1)) * a.plane + base + (col < tcw ? col : 0);
  C* buf = lines + c * (SL * W) + col;
  const C* tw = reinterpret_cast<const C*>(a.rtw[0]);
  auto at = [&](int s) -> C& { return buf[s * W]; };
  auto sync = [] {
    if constexpr (32 % (TL * W) == 0) __syncwarp();
    else __syncthreads();
  };
  reg_line<NL, +1, 0, C>(t, act, tw, [&](int i) -> C { return buf[reg_slot<NL, C>(i) * W]; }, at,
                         [&](int i, C v) { g[i * js] = v; }, sync, sync);
}

// ------------------------------------------------------------- kernels ---
// The kernels of one line length, with their launch shapes.
struct FsLine {
  const void* z[2][4];  // [model][mode]
  const void* y[2];     // forward, inverse
  const void* xf[2];    // matvec, right-hand side
  const void* xi[2];    // direction, final
  int z_threads, tile, y_threads, x_threads;
  int z_bytes, y_bytes, x_bytes;
};
const FsLine* fs_line(int n);  // null: no instantiation

template <int N> static const FsLine* fs_make() {
  static const FsLine L = [] {
    FsLine k{};
    k.z[0][0] = (const void*)fs_zline_reg<N, 0, 0>;
    k.z[1][0] = (const void*)fs_zline_reg<N, 0, 1>;
    k.z[0][1] = (const void*)fs_zline_reg<N, 1, 0>;
    k.z[1][1] = (const void*)fs_zline_reg<N, 1, 1>;
    k.z[0][2] = k.z[1][2] = (const void*)fs_zline_reg<N, 2, 0>;
    k.z[0][3] = k.z[1][3] = (const void*)fs_zline_reg<N, 3, 0>;
    k.y[0] = (const void*)fs_yline_reg<N, -1>;
    k.y[1] = (const void*)fs_yline_reg<N, 1>;
    k.xf[0] = (const void*)fs_xfwd_reg<N, false>;
    k.xf[1] = (const void*)fs_xfwd_reg<N, true>;
    k.xi[0] = (const void*)fs_xinv_reg<N, false>;
    k.xi[1] = (const void*)fs_xinv_reg<N, true>;
    k.z_threads = fs_z_threads(N);
    k.tile = fs_tile(N);
    k.y_threads = fs_ax_threads(N, 3);
    k.x_threads = fs_ax_threads(N, 6);
    k.z_bytes = fs_z_bytes(N);
    k.y_bytes = fs_ax_bytes(N, 3);
    k.x_bytes = fs_ax_bytes(N, 6);
    return k;
  }();
  return &L;
}

}  // namespace mgk
