// Library-wide runtime pieces: error text, status names, FFT schedules and
// the per-device twiddle-table cache.
#include <stdarg.h>

#include <map>
#include <tuple>
#include <mutex>
#include <vector>
#include <cmath>

#include "common.cuh"
#include "fft.cuh"
#include "fft_reg.cuh"

namespace mgk {

static thread_local char g_err[2048] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

cudaError_t raise_smem(const void* fn, size_t bytes) {
  // naming a kernel loads it, and the first of a translation unit loads that (5 .. 15
  // ms); up to 46 KB (48 less what kernels declare themselves) none needs it
  if (bytes <= 46 * 1024) return cudaSuccess;
  static std::mutex m;
  static std::map<std::pair<int, const void*>, size_t> set;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> g(m);
  size_t& cur = set[{dev, fn}];
  if (bytes <= cur) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) cur = bytes;
  return e;
}

namespace {
struct SidePool {
  std::mutex m;
  struct Kind {
    size_t made = 0;
    std::vector<SideStream> free;
  };
  std::map<std::pair<int, int>, Kind> kinds;  // by device and priority
};
// never destroyed: it may be needed while the process ends
SidePool& side_pool() {
  static SidePool* p = new SidePool();
  return *p;
}
}  // namespace

SideStreams::SideStreams(size_t want, int prio) : priority(prio) {
  if (want == 0 || cudaGetDevice(&device) != cudaSuccess) return;
  SidePool& P = side_pool();
  std::lock_guard<std::mutex> g(P.m);
  SidePool::Kind& k = P.kinds[{device, priority}];
  while (v.size() < want) {
    if (k.free.empty()) {
      SideStream n{};
      if (k.made == kSideStreams || cudaStreamCreateWithPriority(&n.s, cudaStreamNonBlocking, priority) != cudaSuccess) break;
      if (cudaEventCreateWithFlags(&n.done, cudaEventDisableTiming) != cudaSuccess) {
        cudaStreamDestroy(n.s);
        break;
      }
      ++k.made;
      k.free.push_back(n);
    }
    v.push_back(k.free.back());
    k.free.pop_back();
  }
}

SideStreams::~SideStreams() {
  if (v.empty()) return;
  SidePool& P = side_pool();
  std::lock_guard<std::mutex> g(P.m);
  SidePool::Kind& k = P.kinds[{device, priority}];
  k.free.insert(k.free.end(), v.begin(), v.end());
}

bool fft_schedule(int n, FftLen* f) {
  if (n < 1 || n > 4096) return false;
  int m = n, a = 0, b = 0;
  while (m % 3 == 0) { m /= 3; ++b; }
  while (m % 2 == 0) { m /= 2; ++a; }
  if (m != 1) return false;
  int np = 0;
  for (int i = 0; i < b; ++i) f->radix[np++] = 3;
  int p8 = a / 3, rem = a % 3;
  if (rem == 1 && p8 >= 1) { p8 -= 1; rem = 4; }  // 2^(3k+1) = 8^(k-1) * 4 * 4
  for (int i = 0; i < p8; ++i) f->radix[np++] = 8;
  if (rem == 4) { f->radix[np++] = 4; f->radix[np++] = 4; }
  else if (rem == 2) f->radix[np++] = 4;
  else if (rem == 1) f->radix[np++] = 2;
  if (np > 8) return false;
  f->n = n;
  f->npass = np;
  f->tw = nullptr;
  return true;
}

// A device copy of the table h, complete on return: a copy from pageable memory
// may still be on its way when cudaMemcpy returns, and the streams that will read
// the table need not wait for the legacy one.
template <typename C> static void* upload(const std::vector<C>& h) {
  void* d = nullptr;
  if (cudaMalloc(&d, h.size() * sizeof(C)) != cudaSuccess) return nullptr;
  if (cudaMemcpy(d, h.data(), h.size() * sizeof(C), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaStreamSynchronize(0) != cudaSuccess) {
    cudaFree(d);
    return nullptr;
  }
  return d;
}

template <typename C> static void* upload_twiddles(int n) {
  std::vector<C> h(n);
  for (int m = 0; m < n; ++m) {
    const long double ang = -2.0L * 3.14159265358979323846264338327950288L * (long double)m / (long double)n;
    h[m].x = (decltype(C::x))cosl(ang);
    h[m].y = (decltype(C::x))sinl(ang);
  }
  return upload(h);
}

// Twiddle tables W_n^m = exp(-2 pi i m / n), one per (device, n, precision);
// they live until process exit (a few tens of KB in total).
const void* twiddles(int n, int prec) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, int>, void*> cache;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  auto key = std::make_tuple(dev, n, prec);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  void* d = prec == MGK_FP64 ? upload_twiddles<double2>(n) : upload_twiddles<float2>(n);
  if (!d) return nullptr;
  cache[key] = d;
  return d;
}

// Twiddles of the register FFT of length n: for each pass after the first
// (the steps' radices in FP64; make_sched's passes in FP32, the angle as m / n
// there, so that the floats are those of twiddles()) the entries W_{NS R}^{r k}
// at [r - 1][k], k < NS; one table per (device, n, precision), kept until
// process exit.
template <typename C> static void fill_reg(int n, std::vector<C>& h) {
  const RegSched q = reg_sched(n, sizeof(C));
  std::vector<int> pass;
  for (int s = 0; s < q.ns; ++s) {
    const int rb = sizeof(C) == 16 ? 1 : q.rb[s];
    pass.push_back(q.r[s] / rb);
    if (rb > 1) pass.push_back(rb);
  }
  int ns = pass[0];
  for (size_t p = 1; p < pass.size(); ++p) {
    for (int r = 1; r < pass[p]; ++r)
      for (int k = 0; k < ns; ++k) {
        const int m = r * k * (n / (ns * pass[p]));
        const long double ang = -2.0L * 3.14159265358979323846264338327950288L * (long double)m / (long double)n;
        C c;
        c.x = (decltype(C::x))cosl(ang);
        c.y = (decltype(C::x))sinl(ang);
        h.push_back(c);
      }
    ns *= pass[p];
  }
}

const void* twiddles_reg(int n, int prec) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, int>, void*> cache;
  int dev = 0;
  if (!reg_len(n) || cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  void*& d = cache[std::make_tuple(dev, n, prec)];
  if (!d) {
    if (prec == MGK_FP64) {
      std::vector<double2> h;
      fill_reg(n, h);
      d = upload(h);
    } else {
      std::vector<float2> h;
      fill_reg(n, h);
      d = upload(h);
    }
  }
  return d;
}

}  // namespace mgk

extern "C" {

int mgk_version(void) { return 100; }

const char* mgk_status_string(int s) {
  switch (s) {
    case MGK_OK: return "ok";
    case MGK_NOT_CONVERGED: return "not converged";
    case MGK_NONFINITE: return "non-finite value";
    case MGK_BAD_ARG: return "bad argument";
    case MGK_OOM: return "out of device memory";
    case MGK_TIMEOUT: return "timeout";
    case MGK_CUDA_ERROR: return "CUDA error";
    default: return "unknown status";
  }
}

const char* mgk_last_error(void) { return mgk::g_err; }

int mgk_fft_supported(int n) {
  mgk::FftLen f;
  return mgk::fft_schedule(n, &f) ? 1 : 0;
}

}  // extern "C"
