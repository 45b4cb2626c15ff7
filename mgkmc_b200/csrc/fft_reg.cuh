// Register FFTs of compile-time lengths N = 2^a 3^b (24 <= N <= 1024).
//
// A line of N points is transformed by T threads in two or three Stockham
// steps of composite radices (up to 24): a thread loads a step's points into
// registers straight from where they are (global memory for the first step of
// a pass), transforms them there and exchanges through shared memory only
// between steps.  The shared-memory passes of radix 3, 2, 4 and 8 that this
// replaces touch shared memory about twice per pass and load a strided twiddle
// per point; here a two-step line crosses shared memory once and its twiddles
// lie in the order in which the threads read them.
//
// Step s has radix R_s and stride NS_s = R_0 .. R_{s-1}; butterfly j reads
// a[j + r N/R_s], multiplies by W_{NS_s R_s}^{r (j mod NS_s)}, and writes
// a'[(j - j mod NS_s) R_s + j mod NS_s + r NS_s]: natural order in and out.
// The last step writes the indices that it read, so its results may replace
// its inputs in place.
#pragma once
#include "common.cuh"
#include "fft.cuh"

namespace mgk {

// Radices and threads per line.
//
// FP64: two steps wherever both radices stay at or below 16 (more points per
// thread would leave too few warps per SM), three above; the smallest radix
// first, so that the threads of the first step are those that the transposed
// exchange feeds without bank conflicts.
//
// FP32: the passes of make_sched() (fft.cuh: radix 3 first, then 8, 4, 2), two
// of them fused into one step where the registers allow (9 = 3 x 3, 24 = 3 x 8,
// 16 = 4 x 4, ...), with the same twiddles, so that every rounding is that of
// the shared-memory passes.  The FP32 phase of a mixed solve decides when the
// FP64 iterations start, and its rounding noise moves their update norms by
// some 0.2 %: with other roundings 3 % of the 256^2 problems took one more
// iteration.  rb: second radix of a fused step (1: none).
struct RegSched {
  int ns, r[3], t, rb[3];
};
constexpr RegSched reg_sched64(int n) {
  switch (n) {
    case 24: return {2, {4, 6, 1}, 6};
    case 27: return {2, {3, 9, 1}, 9};
    case 32: return {2, {4, 8, 1}, 8};
    case 36: return {2, {6, 6, 1}, 6};
    case 48: return {2, {6, 8, 1}, 8};
    case 54: return {2, {6, 9, 1}, 9};
    case 64: return {2, {8, 8, 1}, 8};
    case 72: return {2, {8, 9, 1}, 9};
    case 81: return {2, {9, 9, 1}, 9};
    case 96: return {2, {8, 12, 1}, 12};
    case 108: return {2, {9, 12, 1}, 12};
    case 128: return {2, {8, 16, 1}, 8};
    case 144: return {2, {12, 12, 1}, 12};
    case 162: return {3, {3, 6, 9}, 18};
    case 192: return {2, {12, 16, 1}, 16};
    case 216: return {3, {6, 6, 6}, 36};
    case 243: return {3, {3, 9, 9}, 27};
    case 256: return {2, {16, 16, 1}, 16};
    case 288: return {3, {6, 6, 8}, 36};
    case 324: return {3, {6, 6, 9}, 36};
    case 384: return {3, {6, 8, 8}, 48};
    case 432: return {3, {6, 8, 9}, 54};
    case 486: return {3, {6, 9, 9}, 54};
    case 512: return {3, {8, 8, 8}, 64};
    case 576: return {3, {8, 8, 9}, 64};
    case 648: return {3, {8, 9, 9}, 72};
    case 729: return {3, {9, 9, 9}, 81};
    case 768: return {3, {8, 8, 12}, 64};
    case 864: return {3, {8, 9, 12}, 72};
    case 972: return {3, {9, 9, 12}, 81};
    case 1024: return {3, {8, 8, 16}, 64};
    default: return {0, {1, 1, 1}, 1};
  }
}
constexpr RegSched reg_sched32(int n) {
  switch (n) {
    case 24: return {2, {3, 8, 1}, 8, {1, 1, 1}};
    case 27: return {2, {9, 3, 1}, 9, {3, 1, 1}};
    case 32: return {2, {8, 4, 1}, 8, {1, 1, 1}};
    case 36: return {2, {9, 4, 1}, 9, {3, 1, 1}};
    case 48: return {2, {12, 4, 1}, 6, {4, 1, 1}};
    case 54: return {2, {9, 6, 1}, 9, {3, 2, 1}};
    case 64: return {2, {8, 8, 1}, 8, {1, 1, 1}};
    case 72: return {2, {9, 8, 1}, 9, {3, 1, 1}};
    case 81: return {2, {9, 9, 1}, 9, {3, 3, 1}};
    case 96: return {2, {24, 4, 1}, 8, {8, 1, 1}};
    case 108: return {2, {9, 12, 1}, 12, {3, 4, 1}};
    case 128: return {2, {8, 16, 1}, 8, {1, 4, 1}};
    case 144: return {2, {9, 16, 1}, 16, {3, 4, 1}};
    case 162: return {3, {9, 9, 2}, 18, {3, 3, 1}};
    case 192: return {2, {24, 8, 1}, 8, {8, 1, 1}};
    case 216: return {2, {9, 24, 1}, 24, {3, 8, 1}};
    case 243: return {3, {9, 9, 3}, 27, {3, 3, 1}};
    case 256: return {3, {8, 8, 4}, 32, {1, 1, 1}};
    case 288: return {3, {9, 8, 4}, 36, {3, 1, 1}};
    case 324: return {3, {9, 9, 4}, 36, {3, 3, 1}};
    case 384: return {2, {24, 16, 1}, 24, {8, 4, 1}};
    case 432: return {3, {9, 12, 4}, 48, {3, 4, 1}};
    case 486: return {3, {9, 9, 6}, 54, {3, 3, 2}};
    case 512: return {3, {8, 8, 8}, 64, {1, 1, 1}};
    case 576: return {3, {9, 8, 8}, 72, {3, 1, 1}};
    case 648: return {3, {9, 9, 8}, 81, {3, 3, 1}};
    case 729: return {3, {9, 9, 9}, 81, {3, 3, 3}};
    case 768: return {3, {24, 8, 4}, 48, {8, 1, 1}};
    case 864: return {3, {9, 24, 4}, 72, {3, 8, 1}};
    case 972: return {3, {9, 9, 12}, 108, {3, 3, 4}};
    case 1024: return {3, {8, 8, 16}, 64, {1, 1, 4}};
    default: return {0, {1, 1, 1}, 1, {1, 1, 1}};
  }
}
// csz: bytes of a complex number (16: FP64, 8: FP32)
constexpr RegSched reg_sched(int n, int csz) { return csz == 16 ? reg_sched64(n) : reg_sched32(n); }
constexpr bool reg_len(int n) { return reg_sched64(n).ns != 0; }

// padding of the first exchange: one slot after every R_0 points when R_0 is
// even (the transposed writes then hit distinct 16-byte banks)
constexpr int reg_p0(int n, int csz) { return reg_sched(n, csz).r[0] + (reg_sched(n, csz).r[0] % 2 == 0 ? 1 : 0); }
// slots of one line's exchange buffer
constexpr int reg_slots(int n, int csz) { return n / reg_sched(n, csz).r[0] * reg_p0(n, csz); }
// slot of point i (the layout of the first exchange, of a pass's input held
// in shared memory and of its in-place result)
template <int N, typename C> __device__ __forceinline__ int reg_slot(int i) {
  constexpr int R0 = reg_sched(N, sizeof(C)).r[0], P0 = reg_p0(N, sizeof(C));
  return R0 == P0 ? i : i + i / R0;
}

// Table of pass twiddles: every pass after the first (a fused step is two
// passes) in order, entry [r - 1][k] = W_{NS R}^{r k}, k < NS; host-built.
const void* twiddles_reg(int n, int prec);

// ------------------------------------------------------- small DFTs ---
template <int SIGN, typename C> __device__ __forceinline__ void rdft3(C& a, C& b, C& c) {
  using R = decltype(C::x);
  const R s3 = R(0.86602540378443864676372317075294);
  const C s = cadd(b, c), d = csub(b, c);
  const C m = mk<C>(a.x - R(0.5) * s.x, a.y - R(0.5) * s.y);
  const C t = cmul_i<SIGN>(mk<C>(s3 * d.x, s3 * d.y));
  a = cadd(a, s);
  b = cadd(m, t);
  c = csub(m, t);
}
template <int SIGN, typename C> __device__ __forceinline__ void rdft4(C& a, C& b, C& c, C& d) {
  const C a0 = cadd(a, c), a1 = csub(a, c), a2 = cadd(b, d), a3 = cmul_i<SIGN>(csub(b, d));
  a = cadd(a0, a2);
  c = csub(a0, a2);
  b = cadd(a1, a3);
  d = csub(a1, a3);
}
// times exp(SIGN 2 pi i m / n) given (cos, sin) of 2 pi m / n
template <int SIGN, typename C>
__device__ __forceinline__ C crot(C a, decltype(C::x) c, decltype(C::x) s) {
  return SIGN < 0 ? mk<C>(a.x * c + a.y * s, a.y * c - a.x * s) : mk<C>(a.x * c - a.y * s, a.y * c + a.x * s);
}
// times exp(SIGN 2 pi i / 8) and its cube
template <int SIGN, typename C> __device__ __forceinline__ C crot8(C a) {
  using R = decltype(C::x);
  const R h = R(0.70710678118654752440084436210485);
  return SIGN < 0 ? mk<C>(h * (a.x + a.y), h * (a.y - a.x)) : mk<C>(h * (a.x - a.y), h * (a.x + a.y));
}
template <int SIGN, typename C> __device__ __forceinline__ C crot83(C a) {
  using R = decltype(C::x);
  const R h = R(0.70710678118654752440084436210485);
  return SIGN < 0 ? mk<C>(h * (a.y - a.x), -h * (a.x + a.y)) : mk<C>(-h * (a.x + a.y), h * (a.x - a.y));
}

template <int R, int SIGN, typename C> __device__ __forceinline__ void rdft(C* v) {
  using F = decltype(C::x);
  if constexpr (R == 2) {
    dft2<SIGN>(v);
  } else if constexpr (R == 3) {
    rdft3<SIGN>(v[0], v[1], v[2]);
  } else if constexpr (R == 4) {
    rdft4<SIGN>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 6) {
    // 2 x 3 by the prime-factor map: n = 3 n1 + 2 n2, k = 3 k1 + 4 k2 (mod 6)
    C x[2][3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const C p = v[(2 * b) % 6], q = v[(3 + 2 * b) % 6];
      x[0][b] = cadd(p, q);
      x[1][b] = csub(p, q);
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      rdft3<SIGN>(x[a][0], x[a][1], x[a][2]);
#pragma unroll
      for (int b = 0; b < 3; ++b) v[(3 * a + 4 * b) % 6] = x[a][b];
    }
  } else if constexpr (R == 8) {
    rdft4<SIGN>(v[0], v[2], v[4], v[6]);
    rdft4<SIGN>(v[1], v[3], v[5], v[7]);
    const C e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    const C o1 = crot8<SIGN>(v[3]), o2 = cmul_i<SIGN>(v[5]), o3 = crot83<SIGN>(v[7]);
    v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1); v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2); v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3); v[7] = csub(e3, o3);
  } else if constexpr (R == 9) {
    // 3 x 3: x[3 a + b] -> X[k1 + 3 k2]
    const F c1 = F(0.76604444311897803520239265055542), s1 = F(0.64278760968653932632264340990726);
    const F c2 = F(0.17364817766693034885171662676931), s2 = F(0.98480775301220805936674302458952);
    const F c4 = F(-0.93969262078590838405410927732473), s4 = F(0.34202014332566873304409961468226);
#pragma unroll
    for (int b = 0; b < 3; ++b) rdft3<SIGN>(v[b], v[3 + b], v[6 + b]);
    // v[3 k1 + b] times W9^{b k1}
    v[4] = crot<SIGN>(v[4], c1, s1);
    v[5] = crot<SIGN>(v[5], c2, s2);
    v[7] = crot<SIGN>(v[7], c2, s2);
    v[8] = crot<SIGN>(v[8], c4, s4);
#pragma unroll
    for (int a = 0; a < 3; ++a) rdft3<SIGN>(v[3 * a], v[3 * a + 1], v[3 * a + 2]);
    // v[3 k1 + k2] -> X[k1 + 3 k2]
    C t;
    t = v[1]; v[1] = v[3]; v[3] = t;
    t = v[2]; v[2] = v[6]; v[6] = t;
    t = v[5]; v[5] = v[7]; v[7] = t;
  } else if constexpr (R == 12) {
    // 4 x 3 by the prime-factor map: n = 3 n1 + 4 n2, k = 9 k1 + 4 k2 (mod 12)
    C x[3][4];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
#pragma unroll
      for (int a = 0; a < 4; ++a) x[b][a] = v[(3 * a + 4 * b) % 12];
      rdft4<SIGN>(x[b][0], x[b][1], x[b][2], x[b][3]);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      rdft3<SIGN>(x[0][a], x[1][a], x[2][a]);
#pragma unroll
      for (int b = 0; b < 3; ++b) v[(9 * a + 4 * b) % 12] = x[b][a];
    }
  } else {
    static_assert(R == 16, "radix");
    // 4 x 4: x[4 a + b] -> X[k1 + 4 k2]
    const F c1 = F(0.92387953251128675612818318939679), s1 = F(0.38268343236508977172845998403040);
#pragma unroll
    for (int b = 0; b < 4; ++b) rdft4<SIGN>(v[b], v[4 + b], v[8 + b], v[12 + b]);
    // v[4 k1 + b] times W16^{b k1}
    v[5] = crot<SIGN>(v[5], c1, s1);
    v[6] = crot8<SIGN>(v[6]);
    v[7] = crot<SIGN>(v[7], s1, c1);
    v[9] = crot8<SIGN>(v[9]);
    v[10] = cmul_i<SIGN>(v[10]);
    v[11] = crot83<SIGN>(v[11]);
    v[13] = crot<SIGN>(v[13], s1, c1);
    v[14] = crot83<SIGN>(v[14]);
    v[15] = crot<SIGN>(v[15], -c1, -s1);
#pragma unroll
    for (int a = 0; a < 4; ++a) rdft4<SIGN>(v[4 * a], v[4 * a + 1], v[4 * a + 2], v[4 * a + 3]);
    // v[4 k1 + k2] -> X[k1 + 4 k2]
    C t;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = a + 1; b < 4; ++b) { t = v[4 * a + b]; v[4 * a + b] = v[4 * b + a]; v[4 * b + a] = t; }
  }
}

// The FP32 passes' arithmetic with its contractions written out: the compiler
// is free to round either product of a complex multiplication first, and chose
// differently from kernel to kernel (40 % of the values of a 256-point line
// changed in the last bit).  ALT: which product of the imaginary part the
// forward transforms round, 0 as the former warp-line kernels did, 1 as the
// CTA-wide passes do.
template <int SIGN, int ALT> __device__ __forceinline__ float2 fmul32(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)),
                     SIGN < 0 && ALT ? __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x))
                                     : __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y)));
}
template <int SIGN> __device__ __forceinline__ void fdft3(float2* v) {
  const float s3 = 0.86602540378443864676372317075294f;
  const float2 s = cadd(v[1], v[2]), d = csub(v[1], v[2]);
  const float2 m = make_float2(__fmaf_rn(-0.5f, s.x, v[0].x), __fmaf_rn(-0.5f, s.y, v[0].y));
  const float2 i = cmul_i<SIGN>(d);  // the products s3 d enter the sums unrounded
  v[0] = cadd(v[0], s);
  v[1] = make_float2(__fmaf_rn(s3, i.x, m.x), __fmaf_rn(s3, i.y, m.y));
  v[2] = make_float2(__fmaf_rn(-s3, i.x, m.x), __fmaf_rn(-s3, i.y, m.y));
}
template <int SIGN> __device__ __forceinline__ void fdft8(float2* v) {
  const float h = 0.70710678118654752440084436210485f;
  dft4<SIGN>(v[0], v[2], v[4], v[6]);
  dft4<SIGN>(v[1], v[3], v[5], v[7]);
  const float2 s1 = make_float2(v[3].x - SIGN * v[3].y, v[3].y + SIGN * v[3].x), o2 = cmul_i<SIGN>(v[5]);
  const float2 s3 = make_float2(-(v[7].x + SIGN * v[7].y), SIGN * v[7].x - v[7].y);
  const float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
  v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
  v[2] = cadd(e2, o2); v[6] = csub(e2, o2);
  v[1] = make_float2(__fmaf_rn(h, s1.x, e1.x), __fmaf_rn(h, s1.y, e1.y));
  v[5] = make_float2(__fmaf_rn(-h, s1.x, e1.x), __fmaf_rn(-h, s1.y, e1.y));
  v[3] = make_float2(__fmaf_rn(h, s3.x, e3.x), __fmaf_rn(h, s3.y, e3.y));
  v[7] = make_float2(__fmaf_rn(-h, s3.x, e3.x), __fmaf_rn(-h, s3.y, e3.y));
}

// one FP32 pass of a step: twiddles at w (null: none) and DFT
template <int R, int SIGN, int ALT>
__device__ __forceinline__ void pass_bfly(float2* v, const float2* __restrict__ w, int ns) {
  if (w) {
#pragma unroll
    for (int r = 1; r < R; ++r) {
      float2 x = __ldg(w + (r - 1) * ns);
      if (SIGN > 0) x.y = -x.y;
      v[r] = fmul32<SIGN, ALT>(v[r], x);
    }
  }
  if constexpr (R == 2) dft2<SIGN>(v);
  else if constexpr (R == 3) fdft3<SIGN>(v);
  else if constexpr (R == 4) dft4<SIGN>(v[0], v[1], v[2], v[3]);
  else fdft8<SIGN>(v);
}

// One step of butterfly j.  FP32, fused step R = Ra Rb: point q = r' + Rb r;
// pass a over r for each r' (stride NS), then pass b over r' (stride NS Ra) for
// each r, whose twiddle index is j mod NS + r NS; output s of r is r + Ra s.
template <int N, int S, int SIGN, int ALT, typename C>
__device__ __forceinline__ void reg_bfly(C* v, int j, const C* __restrict__ tw) {
  constexpr RegSched Q = reg_sched(N, sizeof(C));
  constexpr int R = Q.r[S], NS = S == 0 ? 1 : S == 1 ? Q.r[0] : Q.r[0] * Q.r[1];
  constexpr int OFF = NS - 1;  // the passes before this step have NS - 1 entries, less the first pass's
  const int k = S == 0 ? 0 : S == Q.ns - 1 ? j : j % NS;  // the last step has j < NS
  if constexpr (sizeof(C) == 16) {
    if constexpr (S > 0) {
      const C* w0 = tw + (OFF - (Q.r[0] - 1)) + k;
#pragma unroll
      for (int r = 1; r < R; ++r) {
        C w = __ldg(w0 + (r - 1) * NS);
        if (SIGN > 0) w.y = -w.y;
        v[r] = cmul(v[r], w);
      }
    }
    rdft<R, SIGN>(v);
  } else {
    constexpr int Rb = Q.rb[S], Ra = R / Rb, A0 = Q.r[0] / Q.rb[0];  // A0: radix of the first pass
    if constexpr (Rb == 1) {
      pass_bfly<R, SIGN, ALT>(v, S > 0 ? tw + (OFF - (A0 - 1)) + k : nullptr, NS);
    } else {
      C x[Ra][Rb];
#pragma unroll
      for (int b = 0; b < Rb; ++b) {
        C y[Ra];
#pragma unroll
        for (int r = 0; r < Ra; ++r) y[r] = v[b + Rb * r];
        pass_bfly<Ra, SIGN, ALT>(y, S > 0 ? tw + (OFF - (A0 - 1)) + k : nullptr, NS);
#pragma unroll
        for (int r = 0; r < Ra; ++r) x[r][b] = y[r];
      }
#pragma unroll
      for (int r = 0; r < Ra; ++r) {
        pass_bfly<Rb, SIGN, ALT>(x[r], tw + (NS * Ra - 1 - (A0 - 1)) + k + r * NS, NS * Ra);
#pragma unroll
        for (int s = 0; s < Rb; ++s) v[r + Ra * s] = x[r][s];
      }
    }
  }
}

// The transform of one line by its T threads (t in [0, T); TT: other than the
// schedule's, which changes no rounding).
//   load(i)      the input point i (any source)
//   at(slot)     reference to the line's exchange slot
//   store(i, v)  the result point i; it may write at(reg_slot(i)) in place
//   sync()       synchronises the threads that share the line
// Threads with act == false take part in the synchronisations only.
//   pre()        called once by every thread between its loads and the first
//                exchange: inputs that lie in exchange buffers have been read
//                by the threads it synchronises
template <int N, int SIGN, int ALT, typename C, int TT = 0, typename Load, typename At, typename Store, typename Sync,
          typename Pre>
__device__ __forceinline__ void reg_line(int t, bool act, const C* __restrict__ tw, Load load, At at, Store store,
                                         Sync sync, Pre pre) {
  constexpr RegSched Q = reg_sched(N, sizeof(C));
  constexpr int R0 = Q.r[0], T = TT ? TT : Q.t, P0 = reg_p0(N, sizeof(C));
  {
    constexpr int NB = N / R0, U = (NB + T - 1) / T;
    C v[U][R0];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = t + T * u;
      if (act && (NB % T == 0 || j < NB)) {
#pragma unroll
        for (int r = 0; r < R0; ++r) v[u][r] = load(j + r * NB);
      }
    }
    pre();
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = t + T * u;
      if (act && (NB % T == 0 || j < NB)) {
        reg_bfly<N, 0, SIGN, ALT>(v[u], j, tw);
#pragma unroll
        for (int r = 0; r < R0; ++r) at(j * P0 + r) = v[u][r];
      }
    }
  }
  sync();
  constexpr int R1 = Q.r[1], NB1 = N / R1, U1 = (NB1 + T - 1) / T;
  if constexpr (Q.ns == 2) {
#pragma unroll
    for (int u = 0; u < U1; ++u) {
      const int j = t + T * u;
      if (act && (NB1 % T == 0 || j < NB1)) {
        C v[R1];
#pragma unroll
        for (int r = 0; r < R1; ++r) v[r] = at(j + r * P0);  // NB1 = R0
        reg_bfly<N, 1, SIGN, ALT>(v, j, tw);
#pragma unroll
        for (int r = 0; r < R1; ++r) store(j + r * NB1, v[r]);
      }
    }
  } else {
    constexpr int R2 = Q.r[2], NB2 = N / R2, U2 = (NB2 + T - 1) / T;
    {
      C v[U1][R1];
#pragma unroll
      for (int u = 0; u < U1; ++u) {
        const int j = t + T * u;
        if (act && (NB1 % T == 0 || j < NB1)) {
          const int s0 = reg_slot<N, C>(j);
#pragma unroll
          for (int r = 0; r < R1; ++r) v[u][r] = at(s0 + r * (NB1 / R0) * P0);  // NB1 is a multiple of R0
          reg_bfly<N, 1, SIGN, ALT>(v[u], j, tw);
        }
      }
      sync();
#pragma unroll
      for (int u = 0; u < U1; ++u) {
        const int j = t + T * u;
        if (act && (NB1 % T == 0 || j < NB1)) {
          const int k = j % R0;
          const int s0 = reg_slot<N, C>((j - k) * R1) + k;  // rows of R0 points: k stays inside one
#pragma unroll
          for (int r = 0; r < R1; ++r) at(s0 + r * P0) = v[u][r];
        }
      }
    }
    sync();
#pragma unroll
    for (int u = 0; u < U2; ++u) {
      const int j = t + T * u;
      if (act && (NB2 % T == 0 || j < NB2)) {
        C v[R2];
        const int s0 = reg_slot<N, C>(j);
#pragma unroll
        for (int r = 0; r < R2; ++r) v[r] = at(s0 + r * (NB2 / R0) * P0);
        reg_bfly<N, 2, SIGN, ALT>(v, j, tw);
#pragma unroll
        for (int r = 0; r < R2; ++r) store(j + r * NB2, v[r]);
      }
    }
  }
}

}  // namespace mgk
