// Device twiddle tables: exp(-2 pi i m / N) for every compiled length N,
// followed by the w^(4m) copy used by the radix-8/16 stages (tw_len(N)
// entries per length), computed on the host in FP64 and rounded to float.
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include <cuda_fp16.h>

#include "host.cuh"
#include "tcgen05.cuh"

namespace cx {

static __device__ float2 g_twiddles[kTwTotal];
static __device__ float2 g_unit_twiddles[kTwTotal];

// Of the floats on either side of c and of s (cos and sin of an angle), the
// pair with the least m^2 + p^2 / 2, where its modulus is 1 + 5e-9 + m and its
// angle is off by p.  Rounded to nearest, the few factors of a short block and
// the rounded constants of the radix-8 and radix-16 butterflies are below unit
// modulus on average: a 1024-point transform came out 5.2e-8 too small, all
// points alike, and the four of a round trip added up to half of its error.
// With these tables every planned length (pair_fft.cuh) is within 2.5e-8 of
// its mean gain 1, and the rest of the error stays as it was (1.13e-7 at 1024,
// with the mean 1.25e-7 -> 1.12e-7; the 5e-9 make up for the constants).
static float2 unit_rounded(double c, double s) {
  auto other = [](double v) {
    const float r = (float)v;
    return (double)r == v ? r : std::nextafterf(r, (double)r < v ? 2.f : -2.f);
  };
  const float cs[2] = {(float)c, other(c)}, sn[2] = {(float)s, other(s)};
  float2 best = make_float2(cs[0], sn[0]);
  double least = 1.0;
  for (float a : cs)
    for (float b : sn) {
      const double m = std::hypot((double)a, (double)b) - 1.0 - 5e-9, p = a * s - b * c;
      const double e = m * m + 0.5 * p * p;
      if (e < least) {
        least = e;
        best = make_float2(a, b);
      }
    }
  return best;
}

// DFT matrices of lengths 32 and 40 (see tc_dft_mats), 16-byte aligned
constexpr int kTcLens[] = {32, 40};
constexpr uint32_t kTcMatTotal = tc_dft_mat_bytes(32) + tc_dft_mat_bytes(40);
static __device__ uint4 g_tc_mats[kTcMatTotal / 16];
static const uint8_t* g_tc_addr[64] = {nullptr};
static __device__ int g_tc_timeouts;
static int* g_tc_timeouts_addr[64] = {nullptr};

int* tc_timeout_counter() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  return g_tc_timeouts_addr[dev];
}

// row j = output (re | im), column k = input (re | im) of the length-R DFT
// exp(-2 pi i n k / R), as tc_fft_build_b lays it out on the device
static void build_tc_mat(int R, uint8_t* dst) {
  const int K = 2 * R;
  const double pi = 3.141592653589793238462643383279502884;
  for (int j = 0; j < K; ++j)
    for (int k = 0; k < K; ++k) {
      const int n = k % R, kk = j % R, pin = k / R, pout = j / R;
      const double a = -2.0 * pi * (double)((n * kk) % R) / (double)R;
      const float v = (float)(pin == pout ? std::cos(a) : (pin == 0 ? std::sin(a) : -std::sin(a)));
      const __half h = __float2half_rn(v);
      const __half l = __float2half_rn(v - __half2float(h));
      std::memcpy(dst + tc::off_kmajor(K, j, k), &h, 2);
      std::memcpy(dst + K * K * 2 + tc::off_kmajor(K, j, k), &l, 2);
    }
}

const uint8_t* tc_dft_mats(int R) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !g_tc_addr[dev]) return nullptr;
  uint32_t off = 0;
  for (int L : kTcLens) {
    if (L == R) return g_tc_addr[dev] + off;
    off += tc_dft_mat_bytes(L);
  }
  return nullptr;
}

cx_status ensure_twiddles(const float2** table, bool unit) {
  static std::mutex mu;
  static const float2 *addr[64] = {nullptr}, *unit_addr[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    set_error("no current CUDA device");
    return CX_ERR_CUDA;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (addr[dev]) {
    if (table) *table = unit ? unit_addr[dev] : addr[dev];
    return CX_OK;
  }
  static std::vector<float2> host, unit_host;
  if (host.empty()) {
    host.resize(kTwTotal);
    unit_host.resize(kTwTotal);
    const double pi = 3.141592653589793238462643383279502884;
    for (int i = 0; i < kNumSizes; ++i) {
      const int N = kSizes[i];
      float2* t = host.data() + tw_offset(N);
      for (int m = 0; m < tw_len(N); ++m) {
        const long e = m < N ? m : (4L * (m - N)) % N;
        // exact symmetric reduction keeps the argument small: angle = 2 pi e / N
        const double a = 2.0 * pi * (double)e / (double)N;
        t[m] = make_float2((float)std::cos(a), (float)(-std::sin(a)));
        // (multiples of a quarter turn stay as they are: no other factor is exact)
        unit_host[tw_offset(N) + m] = 4 * e % N == 0 ? t[m] : unit_rounded(std::cos(a), -std::sin(a));
      }
    }
  }
  static std::vector<uint8_t> mats;
  if (mats.empty()) {
    mats.resize(kTcMatTotal);
    uint32_t off = 0;
    for (int L : kTcLens) {
      build_tc_mat(L, mats.data() + off);
      off += tc_dft_mat_bytes(L);
    }
  }
  // synchronous copies: visible to every stream once this returns; a first
  // call inside a stream capture is refused by the runtime (call cx_init first)
  CX_CUDA_TRY(cudaMemcpyToSymbol(g_twiddles, host.data(), sizeof(float2) * kTwTotal));
  CX_CUDA_TRY(cudaMemcpyToSymbol(g_unit_twiddles, unit_host.data(), sizeof(float2) * kTwTotal));
  CX_CUDA_TRY(cudaMemcpyToSymbol(g_tc_mats, mats.data(), kTcMatTotal));
  void* q = nullptr;
  CX_CUDA_TRY(cudaGetSymbolAddress(&q, g_tc_mats));
  g_tc_addr[dev] = static_cast<const uint8_t*>(q);
  void* c = nullptr;
  CX_CUDA_TRY(cudaGetSymbolAddress(&c, g_tc_timeouts));
  g_tc_timeouts_addr[dev] = static_cast<int*>(c);
  void *p = nullptr, *u = nullptr;
  CX_CUDA_TRY(cudaGetSymbolAddress(&p, g_twiddles));
  CX_CUDA_TRY(cudaGetSymbolAddress(&u, g_unit_twiddles));
  unit_addr[dev] = static_cast<const float2*>(u);
  addr[dev] = static_cast<const float2*>(p);
  if (table) *table = unit ? unit_addr[dev] : addr[dev];
  return CX_OK;
}

}  // namespace cx

extern "C" cx_status cx_init(void) { return cx::ensure_twiddles(nullptr); }

extern "C" cx_status cx_tc_timeouts(int32_t* count, int32_t reset) {
  if (!count) {
    cx::set_error("null count pointer");
    return CX_ERR_INVALID;
  }
  cx_status s = cx::ensure_twiddles(nullptr);
  if (s != CX_OK) return s;
  int v = 0;
  CX_CUDA_TRY(cudaMemcpyFromSymbol(&v, cx::g_tc_timeouts, sizeof(int)));
  *count = v;
  if (reset) {
    const int zero = 0;
    CX_CUDA_TRY(cudaMemcpyToSymbol(cx::g_tc_timeouts, &zero, sizeof(int)));
  }
  return CX_OK;
}
