// Plane-wise convolution (conv.cuh) on pairs: the sample and the kernel of a
// plane are the two vectors of a pair, in the row and in the column pass.
//
// T holds the row spectra as (zc, NC, ldY): column k of a plane is contiguous
// over the rows y, each element one float4 (sample re, kernel re, sample im,
// kernel im) as the engine's registers hold it.  The row pass writes it 32
// bytes at a time (two rows of one column, whole sectors), the column pass
// reads it contiguously, and neither packs or unpacks anything.
#pragma once

#include "conv.cuh"
#include "pair_fft.cuh"

namespace cx {

// first-stage inputs r >= R_1 / 2: zero when the vector lives on [0, N / 2)
template <int N>
constexpr unsigned pair_lower_mask() {
  unsigned m = 0u;
  for (int r = PairPlan<N>::R1 / 2; r < PairPlan<N>::R1; ++r) m |= 1u << r;
  return m;
}

// --------------------------------------------------------------------------
// rows: r2c of row y of the sample and of the kernel, two rows per CTA
// --------------------------------------------------------------------------
// Z = FFT_M(x[2n] + i x[2n+1]) stays in the buffer, then per k <= M / 2
//   E = (Z[k] + conj Z[M-k]) / 2, O = (Z[k] - conj Z[M-k]) / (2i),
//   X[k] = E + W^k O,  X[M-k] = conj(E - W^k O),  W = exp(-2 pi i / Q).
template <int M>
struct ConvPairRows {
  using F = PairFFT<M, 1>;
  static constexpr int L = F::L;
  static constexpr int ROWS = 2;  // teams: two adjacent rows y, so that a column's two elements fill a sector
  static constexpr int THREADS = ROWS * L;
  static constexpr int TWB = (F::TW * (int)sizeof(float2) + 15) & ~15;
  static constexpr size_t SMEM = TWB + sizeof(float4) * (size_t)ROWS * F::ELEMS;
  static constexpr int WARPS = (THREADS + 31) / 32;
  // 20 warps per SM: the pass waits on loads and barriers.  16 -> 20: 1243 -> 1114 us at M = 1536 (64 planes; two
  // CTAs -> three), 794 -> 752 at 1280, 449 -> 443 at 1024; one-warp CTAs only lose registers (256: 28 -> 30)
  static constexpr int MINB = WARPS == 1 ? 16 : (20 / WARPS > 0 ? 20 / WARPS : 1);
};

template <int M>
__global__ void __launch_bounds__(ConvPairRows<M>::THREADS, ConvPairRows<M>::MINB) k_conv_rows_pair(ConvArgs a) {
  using C = ConvPairRows<M>;
  using F = typename C::F;
  constexpr int ROWS = C::ROWS, NB = M / F::RL;
  constexpr int OFF_Q = tw_offset(2 * M);
  static_assert(OFF_Q >= 0, "row length Q = 2 M has no twiddle table");
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  float4* s0 = reinterpret_cast<float4*>(smem + C::TWB);
  F::load_tables(tw, a.twg, threadIdx.x, blockDim.x);
  const float2* wq = a.twg + OFF_Q;  // exp(-2 pi i k / Q)
  const int team = threadIdx.x / C::L, t = threadIdx.x % C::L;
  float4* s = s0 + (size_t)team * F::ELEMS;
  auto sync = [] { __syncthreads(); };
  float4* T = reinterpret_cast<float4*>(a.T);
  const int groups = a.ldY / ROWS;  // row groups of a plane
  const long total = (long)a.zc * groups;
  for (long item = blockIdx.x; item < total; item += gridDim.x) {
    const int zl = (int)(item / groups), y0 = (int)(item % groups) * ROWS, y = y0 + team;
    const float* xa = a.a + ((size_t)(a.z0 + zl) * a.h + y) * a.w;
    const float* xb = a.b + (size_t)(a.z0 + zl) * a.b_plane + (size_t)y * a.kw;
    const int wa = y < a.h ? a.w : 0, wb = y < a.kh ? a.kw : 0;  // a missing row is a row of zeros
    // even width on an 8-byte boundary: one float2 load per input pair
    const bool pa = (a.w % 2) == 0 && (reinterpret_cast<uintptr_t>(a.a) & 7u) == 0;
    const bool pb = (a.kw % 2) == 0 && (a.b_plane % 2) == 0 && (reinterpret_cast<uintptr_t>(a.b) & 7u) == 0;
    const bool both = pa && pb;
    auto load2 = [&](int n) -> c2 {
      const int x = 2 * n;
      return ppack(ld2z(xa + x, x < wa), ld2z(xb + x, x < wb));
    };
    auto load1 = [&](int n) -> c2 {
      const int x = 2 * n;
      return ppack(make_float2(x < wa ? xa[x] : 0.f, x + 1 < wa ? xa[x + 1] : 0.f),
                   make_float2(x < wb ? xb[x] : 0.f, x + 1 < wb ? xb[x + 1] : 0.f));
    };
    __syncthreads();  // the previous rows have been read
    // z[n] = 0 for n >= M / 2 (Q >= 2 max(w, kw))
    if (both)
      F::template first<false, pair_lower_mask<M>()>(s, tw, t, load2);
    else
      F::template first<false, pair_lower_mask<M>()>(s, tw, t, load1);
    F::template inner<false>(s, tw, t, sync);
    F::template last_in_place<false>(s, t);
    __syncthreads();
    float4* dst = T + (size_t)zl * a.NC * a.ldY + y0;
    // lanes of the two rows side by side: 32 bytes of one column
    for (int e = threadIdx.x; e < (M / 2 + 1) * ROWS; e += C::THREADS) {
      const int k = e / ROWS, row = e % ROWS, km = M - k;
      float4* b = s0 + (size_t)row * F::ELEMS;
      const c2 zk = sload(F::last_ptr(b, k % NB) + k / NB);
      const int kz = k == 0 ? 0 : km;
      c2 zm = sload(F::last_ptr(b, kz % NB) + kz / NB);
      zm.im = f2neg(zm.im);
      const c2 E = pscale(padd(zk, zm), 0.5f), d = psub(zk, zm);
      const c2 O = {__fmul2_rn(d.im, f2dup(0.5f)), __fmul2_rn(d.re, f2dup(-0.5f))};
      const c2 wo = pmulw<false>(O, wq[k]);
      sstore(dst + (size_t)k * a.ldY + row, padd(E, wo));
      if (km != k) {
        c2 x = psub(E, wo);
        x.im = f2neg(x.im);
        sstore(dst + (size_t)km * a.ldY + row, x);
      }
    }
  }
}

// --------------------------------------------------------------------------
// columns: FFT_P of a spectrum column of the sample and of the kernel, the
// product of the two summed over the planes in shared memory
// --------------------------------------------------------------------------
// Work units (column, plane) split in equal contiguous ranges over the
// resident CTAs (no last wave); a range's sums go to St when it leaves a column.
// With at least as many columns as CTAs a column belongs to two CTAs at most,
// and 0 + a + b is the same in both orders.  With fewer (images of up to about
// a thousand pixels) more CTAs share one, and the order in which they finish
// would decide the rounding: each then stores its sum to a slab of its own,
// and k_conv_sum adds a column's slabs to St in order.
// The first stage's twiddles stay in registers: 6 KB less shared memory let a
// third CTA per SM in at 3072 (64 planes: 1347 -> 1284 us; 4096: 2404 -> 2271;
// 512 to 2560: within 3 %).
template <int P>
struct ConvPairCols {
  using F = PairFFT<P, 1>;
  static constexpr int L = F::L;
  static constexpr int THREADS = L;
  static constexpr int TWB = ((F::TW - F::T2) * (int)sizeof(float2) + 15) & ~15;
  static constexpr size_t ACC_OFF = TWB + sizeof(float4) * (size_t)F::ELEMS;
  static constexpr size_t SMEM = ACC_OFF + sizeof(float2) * (size_t)P;
  static constexpr int WARPS = (THREADS + 31) / 32;
  // up to 20 warps per SM, as far as their shared memory goes
  static constexpr int FIT = (int)(227 * 1024 / (SMEM + 1024));
  static constexpr int MINB = 20 / WARPS < 1 || FIT < 1 ? 1 : (20 / WARPS < FIT ? 20 / WARPS : FIT);
  static constexpr int CTAS = 148 * MINB;
  static_assert(SMEM <= 227 * 1024, "convolution column does not fit one CTA");
};

// the range that holds unit u of `units` in `ctas` ranges
__device__ __forceinline__ long conv_owner(long u, long units, long ctas) { return ((u + 1) * ctas - 1) / units; }

// SLAB: a.slabs > 1 (in a kernel of its own: the other one has no registers to spare, 1907 -> 1951 us at 128 x 1024^2)
template <int P, bool SLAB>
__global__ void __launch_bounds__(ConvPairCols<P>::THREADS, ConvPairCols<P>::MINB) k_conv_cols_pair(ConvArgs a) {
  using C = ConvPairCols<P>;
  using F = typename C::F;
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  float4* s = reinterpret_cast<float4*>(smem + C::TWB);
  float2* acc = reinterpret_cast<float2*>(smem + C::ACC_OFF);
  F::template load_tables<F::T2>(tw, a.twg, threadIdx.x, blockDim.x);
  tw -= F::T2;
  const int t = threadIdx.x;
  const typename F::Powers w1 = F::first_powers(a.twg, t);
  auto sync = [] { __syncthreads(); };
  const float4* T = reinterpret_cast<const float4*>(a.T);
  const long units = (long)a.NC * a.zc;
  const long u0 = units * blockIdx.x / gridDim.x, u1 = units * (blockIdx.x + 1) / gridDim.x;
  bool fresh = true;  // no plane of this column summed yet
  for (long u = u0; u < u1; ++u) {
    const int kc = (int)(u / a.zc), zl = (int)(u % a.zc);
    const float4* src = T + ((size_t)zl * a.NC + kc) * a.ldY;
    auto load = [&](int n) -> c2 {
      const float4 v = ld4z(src + n, n < a.ldY);
      return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
    };
    const bool leave = u + 1 == u1 || zl + 1 == a.zc;
    float2* col = (SLAB ? a.part : a.St) + (size_t)kc * a.P;
    // this CTA's number among those of the column
    if (SLAB && leave) col += (blockIdx.x - conv_owner((long)kc * a.zc, units, gridDim.x)) * a.NC * a.P;
    // acc[k] belongs to one lane: no barrier between its updates
    auto out = [&](int k, c2 v) {
      float2 p = cmul(make_float2(v.re.x, v.im.x), make_float2(v.re.y, v.im.y));
      if (!fresh) p = cadd(acc[k], p);
      if (!leave)
        acc[k] = p;
      else if (SLAB)
        col[k] = p;
      else
        atomicAdd(col + k, p);
    };
    __syncthreads();  // the previous column has been read
    // rows >= HB are zero and P >= 2 HB
    F::template first<false, pair_lower_mask<P>()>(s, w1, t, load);
    F::template inner<false>(s, tw, t, sync);
    F::template last<false>(s, t, out);
    fresh = leave;
  }
}

// St[kc][k] (+)= the slabs of column kc, one thread per element (the whole sum
// of 64 planes of 256^2 with its 6 MB of slabs: 84 -> 88 us, of 48 x 768^2 454 ->
// 461; with the slabs added in the final pass's loader 110 and 492).
static __global__ void k_conv_sum(ConvArgs a, int ctas) {
  const long units = (long)a.NC * a.zc, n = (long)a.NC * a.P;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
    const long u = e / a.P * a.zc;
    const int count = (int)(conv_owner(u + a.zc - 1, units, ctas) - conv_owner(u, units, ctas)) + 1;
    float2 v = a.fresh ? make_float2(0.f, 0.f) : a.St[e];
#pragma unroll 8
    for (int s = 0; s < count; ++s) v = cadd(v, a.part[s * n + e]);
    a.St[e] = v;
  }
}

// lengths with both passes on pairs
inline bool conv_on_pairs(int m, int p) { return m <= 2048 && p <= 4096 && pair_length(m) && pair_length(p); }

}  // namespace cx
