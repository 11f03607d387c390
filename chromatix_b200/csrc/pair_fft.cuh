// In-place FFT engine for PAIRS of complex64 vectors, on packed FP32 pairs.
//
// sm_100a issues one FADD2 / FMUL2 / FFMA2 for two independent FP32 lanes
// (add/mul/fma.rn.f32x2): the FP32 pipe does the same 128 lane-operations per
// clock and SM as with scalar instructions, in half the issue slots (measured:
// 63 packed against 51-62 pairs of scalar operations per clock and SM, and 31
// against 25 with two integer operations beside each).  The transforms here
// were bound by issue (45 of 86 instructions per point were FP32), so each
// lane works on the same elements of two vectors (two adjacent columns, two
// rows) at once: c2 holds their real parts in one packed pair and their
// imaginary parts in the other, and addressing, control, barriers and twiddle
// arithmetic are shared by both vectors.
//
// Decimation in frequency, in place: N = R_1 R_2 ... R_S.  Stage 1 takes
// elements j + r N/R_1 (j < M = N/R_1), and every later stage works inside
// blocks of its predecessor's length, on the positions that it reads.  A
// lane's butterfly writes only what it has read, so one barrier per exchange
// suffices, and the butterflies of a lane need not be held at the same time.
// The last stage's outputs come in digit-reversed position but are handed to
// the caller with their frequency k = b + r N/R_S (b = butterfly number):
// consecutive lanes get consecutive k.  The round trip (transform -> pointwise
// product -> inverse) then runs the stages backwards from those positions:
// the last forward and first inverse stage share one pass over shared memory.
//
// Shared memory: element (position p, pair c of VP) as one float4 at
// ((q1 (M + 1) + p mod M) VP + c), q1 = p / M.  M is even for every compiled
// length, so lanes that step through q1 (stages after the first) or through j
// (stage 1) hit distinct 16-byte banks.
#pragma once

#include "host.cuh"

namespace cx {

struct c2 {
  float2 re, im;  // real / imaginary parts of the two vectors
};

__device__ __forceinline__ float2 f2neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 f2dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ c2 padd(c2 a, c2 b) { return {__fadd2_rn(a.re, b.re), __fadd2_rn(a.im, b.im)}; }
__device__ __forceinline__ c2 psub(c2 a, c2 b) { return {__fadd2_rn(a.re, f2neg(b.re)), __fadd2_rn(a.im, f2neg(b.im))}; }
// a + (-i) b (forward) / a + i b (inverse), and with the other sign
template <bool INV>
__device__ __forceinline__ c2 padd_mi(c2 a, c2 b) {
  return INV ? c2{__fadd2_rn(a.re, f2neg(b.im)), __fadd2_rn(a.im, b.re)}
             : c2{__fadd2_rn(a.re, b.im), __fadd2_rn(a.im, f2neg(b.re))};
}
template <bool INV>
__device__ __forceinline__ c2 psub_mi(c2 a, c2 b) {
  return padd_mi<!INV>(a, b);
}
// both vectors times one complex factor w (conjugated when CONJ)
template <bool CONJ>
__device__ __forceinline__ c2 pmulw(c2 a, float2 w) {
  const float2 wr = f2dup(w.x), wi = f2dup(CONJ ? -w.y : w.y);
  return {__ffma2_rn(a.im, f2neg(wi), __fmul2_rn(a.re, wr)), __ffma2_rn(a.im, wr, __fmul2_rn(a.re, wi))};
}
// each vector times its own complex factor (h as a pair)
__device__ __forceinline__ c2 pmul(c2 a, c2 h) {
  return {__ffma2_rn(a.im, f2neg(h.im), __fmul2_rn(a.re, h.re)), __ffma2_rn(a.im, h.re, __fmul2_rn(a.re, h.im))};
}
__device__ __forceinline__ c2 pscale(c2 a, float s) {
  return {__fmul2_rn(a.re, f2dup(s)), __fmul2_rn(a.im, f2dup(s))};
}
__device__ __forceinline__ c2 pzero() { return {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }
__device__ __forceinline__ c2 ppack(float2 a, float2 b) { return {make_float2(a.x, b.x), make_float2(a.y, b.y)}; }
__device__ __forceinline__ c2 ppack(float4 v) { return {make_float2(v.x, v.z), make_float2(v.y, v.w)}; }
__device__ __forceinline__ float4 punpack(c2 a) { return make_float4(a.re.x, a.im.x, a.re.y, a.im.y); }
__device__ __forceinline__ float2 pfirst(c2 a) { return make_float2(a.re.x, a.im.x); }
__device__ __forceinline__ float2 psecond(c2 a) { return make_float2(a.re.y, a.im.y); }
__device__ __forceinline__ c2 sload(const float4* s) {
  const float4 v = *s;
  return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ void sstore(float4* s, c2 a) { *s = make_float4(a.re.x, a.re.y, a.im.x, a.im.y); }

// Predicated global loads, zero where !ok.  As one instruction each (not a
// branch around a load and its use) all loads of a stage are issued before the
// first is waited for.  volatile: they stay behind barriers and grid waits.
__device__ __forceinline__ float4 ld4z(const void* p, bool ok) {
  float4 v;
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.u32 q, %5, 0;\n mov.f32 %0, 0f00000000;\n mov.f32 %1, 0f00000000;\n"
      " mov.f32 %2, 0f00000000;\n mov.f32 %3, 0f00000000;\n @q ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];\n}"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(p), "r"((unsigned)ok));
  return v;
}
__device__ __forceinline__ float2 ld2z(const void* p, bool ok) {
  float2 v;
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.u32 q, %3, 0;\n mov.f32 %0, 0f00000000;\n mov.f32 %1, 0f00000000;\n"
      " @q ld.global.v2.f32 {%0, %1}, [%2];\n}"
      : "=f"(v.x), "=f"(v.y)
      : "l"(p), "r"((unsigned)ok));
  return v;
}

// ---------------------------------------------------------------------------
// small DFTs of c2 (natural order in and out)
// ---------------------------------------------------------------------------
template <int R, bool INV>
struct PDFT;

template <bool INV>
__device__ __forceinline__ void pdft4(c2& x0, c2& x1, c2& x2, c2& x3) {
  const c2 t0 = padd(x0, x2), t1 = psub(x0, x2), t2 = padd(x1, x3), t3 = psub(x1, x3);
  x0 = padd(t0, t2);
  x2 = psub(t0, t2);
  x1 = padd_mi<INV>(t1, t3);
  x3 = psub_mi<INV>(t1, t3);
}

template <bool INV>
struct PDFT<2, INV> {
  __device__ __forceinline__ static void run(c2* v) {
    const c2 t = v[0];
    v[0] = padd(t, v[1]);
    v[1] = psub(t, v[1]);
  }
};

template <bool INV>
struct PDFT<4, INV> {
  __device__ __forceinline__ static void run(c2* v) { pdft4<INV>(v[0], v[1], v[2], v[3]); }
};

// odd prime radices by symmetric pairs: y_k = x0 + sum_m (x_m + x_{R-m}) cos -/+ i sum_m (x_m - x_{R-m}) sin
template <int R, bool INV>
struct PDFTOdd {
  __device__ __forceinline__ static void run(c2* v) {
    constexpr int H = (R - 1) / 2;
    c2 sp[H + 1], dm[H + 1];
#pragma unroll
    for (int m = 1; m <= H; ++m) {
      sp[m] = padd(v[m], v[R - m]);
      dm[m] = psub(v[m], v[R - m]);
    }
    const c2 x0 = v[0];
#pragma unroll
    for (int m = 1; m <= H; ++m) v[0] = padd(v[0], sp[m]);
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      c2 re = x0, im;
#pragma unroll
      for (int m = 1; m <= H; ++m) {
        const int idx = (k * m) % R;
        const int ii = idx <= H ? idx : R - idx;
        const float c = OddConst<R>::c(ii);
        const float s = (idx <= H ? 1.f : -1.f) * OddConst<R>::s(ii);
        re = {__ffma2_rn(sp[m].re, f2dup(c), re.re), __ffma2_rn(sp[m].im, f2dup(c), re.im)};
        if (m == 1)
          im = {__fmul2_rn(dm[m].re, f2dup(s)), __fmul2_rn(dm[m].im, f2dup(s))};
        else
          im = {__ffma2_rn(dm[m].re, f2dup(s), im.re), __ffma2_rn(dm[m].im, f2dup(s), im.im)};
      }
      v[k] = padd_mi<INV>(re, im);
      v[R - k] = psub_mi<INV>(re, im);
    }
  }
};
template <bool INV>
struct PDFT<3, INV> : PDFTOdd<3, INV> {};
template <bool INV>
struct PDFT<5, INV> : PDFTOdd<5, INV> {};
template <bool INV>
struct PDFT<7, INV> : PDFTOdd<7, INV> {};

template <bool INV>
struct PDFT<8, INV> {
  __device__ __forceinline__ static void run(c2* v) {
    pdft4<INV>(v[0], v[2], v[4], v[6]);  // even inputs -> a_k in v[0], v[2], v[4], v[6]
    pdft4<INV>(v[1], v[3], v[5], v[7]);  // odd inputs -> b_k in v[1], v[3], v[5], v[7]
    // w8 = h (1 - i), w8^3 = -h (1 + i); products by FMA: a sum scaled by h would round once more at full size
    const float h = 0.70710678118654752440f;
    const c2 w1 = pmulw<INV>(v[3], make_float2(h, -h)), w3 = pmulw<INV>(v[7], make_float2(-h, -h));
    const c2 a0 = v[0], a1 = v[2], a2 = v[4], a3 = v[6], b0 = v[1], b2 = v[5];
    v[0] = padd(a0, b0);
    v[4] = psub(a0, b0);
    v[1] = padd(a1, w1);
    v[5] = psub(a1, w1);
    v[2] = padd_mi<INV>(a2, b2);
    v[6] = psub_mi<INV>(a2, b2);
    v[3] = padd(a3, w3);
    v[7] = psub(a3, w3);
  }
};

template <bool INV>
struct PDFT<16, INV> {
  __device__ __forceinline__ static void run(c2* v) {
    const float c1 = 0.92387953251128675613f;  // cos(pi/8)
    const float s1 = 0.38268343236508977173f;  // sin(pi/8)
    const float h = 0.70710678118654752440f;
#pragma unroll
    for (int r1 = 0; r1 < 4; ++r1) pdft4<INV>(v[r1], v[r1 + 4], v[r1 + 8], v[r1 + 12]);
    // v[r1 + 4 k2] *= w16^(r1 k2), w16 = (c1, -s1) forward
    v[5] = pmulw<INV>(v[5], make_float2(c1, -s1));
    v[13] = pmulw<INV>(v[13], make_float2(s1, -c1));
    v[7] = pmulw<INV>(v[7], make_float2(s1, -c1));
    v[15] = pmulw<INV>(v[15], make_float2(-c1, s1));
    // w16^2 = h (1 - i), w16^6 = -h (1 + i)
    v[9] = pmulw<INV>(v[9], make_float2(h, -h));
    v[6] = pmulw<INV>(v[6], make_float2(h, -h));
    v[14] = pmulw<INV>(v[14], make_float2(-h, -h));
    v[11] = pmulw<INV>(v[11], make_float2(-h, -h));
    // r1 = 2, k2 = 2: w16^4 = -i, folded into the second step's butterflies
    c2 y[16];
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
      const c2 a0 = v[4 * k2], a1 = v[4 * k2 + 1], a2 = v[4 * k2 + 2], a3 = v[4 * k2 + 3];
      const c2 t0 = k2 == 2 ? padd_mi<INV>(a0, a2) : padd(a0, a2);
      const c2 t1 = k2 == 2 ? psub_mi<INV>(a0, a2) : psub(a0, a2);
      const c2 t2 = padd(a1, a3), t3 = psub(a1, a3);
      y[k2] = padd(t0, t2);
      y[k2 + 8] = psub(t0, t2);
      y[k2 + 4] = padd_mi<INV>(t1, t3);
      y[k2 + 12] = psub_mi<INV>(t1, t3);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = y[i];
  }
};

// coprime factors A B without twiddles (Good 1958): input n = (B n1 + A n2) mod AB,
// output k with k mod A = k1 and k mod B = k2
template <int A, int B, bool INV>
struct PDFTGood {
  __host__ __device__ static constexpr int crt(int k1, int k2) {
    for (int k = 0; k < A * B; ++k)
      if (k % A == k1 && k % B == k2) return k;
    return 0;
  }
  __device__ __forceinline__ static void run(c2* v) {
    c2 y[A * B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      c2 t[A];
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) t[n1] = v[(B * n1 + A * n2) % (A * B)];
      PDFT<A, INV>::run(t);
#pragma unroll
      for (int k1 = 0; k1 < A; ++k1) y[k1 * B + n2] = t[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      PDFT<B, INV>::run(y + k1 * B);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[crt(k1, k2)] = y[k1 * B + k2];
    }
  }
};
template <bool INV>
struct PDFT<6, INV> : PDFTGood<2, 3, INV> {};
template <bool INV>
struct PDFT<10, INV> : PDFTGood<2, 5, INV> {};
template <bool INV>
struct PDFT<12, INV> : PDFTGood<4, 3, INV> {};
template <bool INV>
struct PDFT<14, INV> : PDFTGood<2, 7, INV> {};

// v[r] *= w^r, r < R, from the table's w, w^2, w^4 and w^8 (`tw` at w's entry,
// BLOCK entries between the powers): every other power is a product of at most
// two of them and w^3 or w^12, formed once for both vectors in scalar FP32.
// (Broadcast tables and packed products need no moves but twice the FP32
// lanes: the row passes of 64 1024^2 fields went from 78 to 81 and from 174 to
// 176 us.  With w and w^4 only, the error against FP64 was a tenth larger.)
__host__ __device__ constexpr int ptw_powers(int R) { return R > 8 ? 4 : (R > 4 ? 3 : (R > 2 ? 2 : 1)); }
// (cmul with the contraction written out: every kernel forms the same bits)
__device__ __forceinline__ float2 cmul_rn(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
template <int R, bool CONJ, int BLOCK>
__device__ __forceinline__ void ptwiddle(c2* v, const float2* tw) {
  const float2 w1 = tw[0];
  v[1] = pmulw<CONJ>(v[1], w1);
  if constexpr (R > 2) {
    const float2 w2 = tw[BLOCK];
    v[2] = pmulw<CONJ>(v[2], w2);
    if constexpr (R > 3) {
      const float2 w3 = cmul_rn(w2, w1);
      v[3] = pmulw<CONJ>(v[3], w3);
      if constexpr (R > 4) {
        const float2 w4 = tw[2 * BLOCK];
        float2 wq = w4;  // w^(4 q)
#pragma unroll
        for (int q = 1; 4 * q < R; ++q) {
          if (q == 2) wq = tw[3 * BLOCK];
          if (q == 3) wq = cmul_rn(wq, w4);
          v[4 * q] = pmulw<CONJ>(v[4 * q], wq);
          if (4 * q + 1 < R) v[4 * q + 1] = pmulw<CONJ>(v[4 * q + 1], cmul_rn(wq, w1));
          if (4 * q + 2 < R) v[4 * q + 2] = pmulw<CONJ>(v[4 * q + 2], cmul_rn(wq, w2));
          if (4 * q + 3 < R) v[4 * q + 3] = pmulw<CONJ>(v[4 * q + 3], cmul_rn(wq, w3));
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// plans
// ---------------------------------------------------------------------------
// Lengths with a pair plan: N, lanes L per pair, radices in stage order (1:
// no stage).  The first radix is a power of two; L divides N / R_1 (a
// lane's first stage is one butterfly: every global load of a tile is in
// flight before the first is used).  16 points per lane from 640 up and 8 at
// 224 .. 512 (below 224, two stages of up to 16).  Below 128 points a pass is
// bound by its launch: those lengths keep the scalar engine.
// (8192: only the propagation passes.)
#define CX_PAIR_PLANS_4096(X)                                                                         \
  X(128, 8, 16, 8, 1, 1) X(160, 10, 16, 10, 1, 1) X(192, 12, 16, 12, 1, 1) X(224, 28, 8, 4, 7, 1)   \
  X(256, 16, 16, 16, 1, 1) X(320, 40, 8, 8, 5, 1) X(384, 48, 8, 8, 6, 1) X(448, 56, 8, 8, 7, 1)     \
  X(512, 64, 8, 8, 8, 1) X(640, 40, 16, 8, 5, 1) X(768, 48, 16, 8, 6, 1) X(896, 56, 16, 8, 7, 1)      \
  X(1024, 64, 16, 8, 8, 1) X(1280, 80, 16, 8, 10, 1) X(1536, 96, 16, 16, 6, 1)                        \
  X(1792, 112, 16, 16, 7, 1) X(2048, 128, 16, 16, 8, 1) X(2560, 160, 16, 16, 10, 1)                   \
  X(3072, 192, 16, 16, 12, 1) X(3584, 224, 16, 16, 14, 1) X(4096, 256, 16, 16, 16, 1)
#define CX_PAIR_PLANS(X) CX_PAIR_PLANS_4096(X) X(8192, 512, 16, 8, 8, 8)

template <int N, bool LONE = false>
struct PairPlan : PairPlan<N, false> {};
template <int N>
struct PairPlan<N, false> {
  static constexpr int L = 0, R1 = 0, R2 = 0, R3 = 0, R4 = 0;
};
#define CX_PAIR_PLAN_(N_, L_, A_, B_, C_, D_)                                          \
  template <>                                                                          \
  struct PairPlan<N_, false> {                                                         \
    static constexpr int L = L_, R1 = A_, R2 = B_, R3 = C_, R4 = D_;                   \
    static_assert(A_ * B_ * C_ * D_ == N_ && N_ / A_ % L_ == 0 && N_ / A_ % 2 == 0, ""); \
  };
CX_PAIR_PLANS(CX_PAIR_PLAN_)
#undef CX_PAIR_PLAN_

// LONE: plans for passes over one plane, where a pass is a single wave and
// its time the length of one lane's work: 8 points per lane where the plans
// above have 16, at the price of a fourth stage from 1024 up.
#define CX_PAIR_LONE_PLANS(X)                                                                           \
  X(640, 80, 8, 8, 10, 1) X(768, 96, 8, 8, 12, 1) X(896, 112, 8, 8, 14, 1) X(1024, 128, 8, 8, 4, 4)     \
  X(1280, 160, 8, 8, 5, 4) X(1536, 192, 8, 8, 6, 4) X(1792, 224, 8, 8, 7, 4) X(2048, 256, 8, 8, 8, 4)   \
  X(2560, 320, 8, 8, 10, 4) X(3072, 384, 8, 8, 12, 4) X(3584, 448, 8, 8, 14, 4) X(4096, 512, 8, 8, 16, 4)
#define CX_PAIR_PLAN_(N_, L_, A_, B_, C_, D_)                                          \
  template <>                                                                          \
  struct PairPlan<N_, true> {                                                          \
    static constexpr int L = L_, R1 = A_, R2 = B_, R3 = C_, R4 = D_;                   \
    static_assert(A_ * B_ * C_ * D_ == N_ && N_ / A_ % L_ == 0 && N_ / A_ % 2 == 0, ""); \
  };
CX_PAIR_LONE_PLANS(CX_PAIR_PLAN_)
#undef CX_PAIR_PLAN_

template <int N>
constexpr bool pair_planned() {
  return PairPlan<N>::L > 0;
}
// run-time counterpart of pair_planned
inline bool pair_length(int n) {
  switch (n) {
#define CX_CASE_(N_, L_, A_, B_, C_, D_) case N_:
    CX_PAIR_PLANS(CX_CASE_)
#undef CX_CASE_
    return true;
  }
  return false;
}

// One transform length on VP interleaved pairs per buffer.  `t` is the lane
// inside the pair (0 .. L-1); `s` points at the pair's element 0 (its index c
// is already added); `tw` at the twiddle tables in shared memory (TW float2).
template <int N, int VP = 1, bool LONE = false>
struct PairFFT {
  using P = PairPlan<N, LONE>;
  static constexpr int L = P::L, R1 = P::R1, R2 = P::R2, R3 = P::R3, R4 = P::R4;
  static constexpr int S = R3 == 1 ? 2 : (R4 == 1 ? 3 : 4);
  static constexpr int M = N / R1, M2 = M / R2, M3 = M2 / R3;  // block lengths
  static constexpr int RL = S == 2 ? R2 : (S == 3 ? R3 : R4);  // last radix
  static constexpr int PITCH = M + 1;
  static constexpr int ELEMS = R1 * PITCH * VP;  // float4 per buffer
  // twiddles, each as blocks of its 1st, 2nd, 4th and 8th powers (as many as the radix needs): stage 1 w_N^j
  // (j < M), stage 2 w_M^j (j < M2), stage 3 of four w_M2^j (j < M3); the last stage has none
  static constexpr int T2 = ptw_powers(R1) * M, T3 = T2 + (S > 2 ? ptw_powers(R2) * M2 : 0);
  static constexpr int TW = T3 + (S > 3 ? ptw_powers(R3) * M3 : 0);

  // fill the tables from the length's table w_N^m (m < N) in global memory; FROM = T2: all but the first stage's
  // (a kernel that keeps its lanes' first-stage powers in registers passes `tw` - T2 from there on)
  template <int FROM = 0>
  __device__ static void load_tables(float2* tw, const float2* __restrict__ twg, int tid, int nthreads) {
    const float2* g = twg + tw_offset(N);
    for (int i = FROM + tid; i < TW; i += nthreads) {
      const int base = i < T2 ? 0 : (i < T3 ? T2 : T3), block = i < T2 ? M : (i < T3 ? M2 : M3);
      const int step = i < T2 ? 1 : (i < T3 ? R1 : R1 * R2);
      const int j = (i - base) % block, pw = (i - base) / block;
      tw[i - FROM] = g[((j * step) << pw) % N];
    }
  }

  template <int NB, class F>
  __device__ __forceinline__ static void each(int t, F f) {
#pragma unroll
    for (int it = 0; it < (NB + L - 1) / L; ++it) {
      const int b = t + it * L;
      if (NB % L == 0 || b < NB) f(b);
    }
  }
  // stage 1 of a forward chain: v[r] = load(j + r M); ZM: r whose inputs are zero
  template <bool INV, unsigned ZM = 0u, class Load>
  __device__ __forceinline__ static void first(float4* s, const float2* tw, int t, Load& load) {
    each<M>(t, [&](int j) {
      c2 v[R1];
#pragma unroll
      for (int r = 0; r < R1; ++r) v[r] = ((ZM >> r) & 1u) ? pzero() : load(j + r * M);
      PDFT<R1, INV>::run(v);
      ptwiddle<R1, INV, M>(v, tw + j);
#pragma unroll
      for (int q = 0; q < R1; ++q) sstore(s + (q * PITCH + j) * VP, v[q]);
    });
  }
  // A lane's first butterfly is always its t-th: its powers can stay in
  // registers over all of a kernel's transforms, 8 registers for a quarter of
  // the first stage's shared-memory reads and the largest table.
  struct Powers {
    float2 w[ptw_powers(R1)];
  };
  __device__ __forceinline__ static Powers first_powers(const float2* __restrict__ twg, int t) {
    Powers p;
#pragma unroll
    for (int i = 0; i < ptw_powers(R1); ++i) p.w[i] = twg[tw_offset(N) + ((t << i) % N)];
    return p;
  }
  template <bool INV, unsigned ZM = 0u, class Load>
  __device__ __forceinline__ static void first(float4* s, const Powers& w, int t, Load& load) {
    static_assert(M == L, "one first-stage butterfly per lane");
    c2 v[R1];
#pragma unroll
    for (int r = 0; r < R1; ++r) v[r] = ((ZM >> r) & 1u) ? pzero() : load(t + r * M);
    PDFT<R1, INV>::run(v);
    ptwiddle<R1, INV, 1>(v, w.w);
#pragma unroll
    for (int q = 0; q < R1; ++q) sstore(s + (q * PITCH + t) * VP, v[q]);
  }
  // the inner stages (2 of three; 2 and 3 of four)
  template <bool INV, bool BACK>
  __device__ __forceinline__ static void mid2(float4* s, const float2* tw, int t) {
    each<N / R2>(t, [&](int b) {
      const int q = b % R1, j = b / R1;
      float4* p = s + (q * PITCH + j) * VP;
      c2 v[R2];
#pragma unroll
      for (int r = 0; r < R2; ++r) v[r] = sload(p + r * M2 * VP);
      if constexpr (BACK) ptwiddle<R2, INV, M2>(v, tw + T2 + j);
      PDFT<R2, INV>::run(v);
      if constexpr (!BACK) ptwiddle<R2, INV, M2>(v, tw + T2 + j);
#pragma unroll
      for (int r = 0; r < R2; ++r) sstore(p + r * M2 * VP, v[r]);
    });
  }
  template <bool INV, bool BACK>
  __device__ __forceinline__ static void mid3(float4* s, const float2* tw, int t) {
    each<N / R3>(t, [&](int b) {
      const int q = b % R1, j = (b / R1) % M3, q2 = b / (R1 * M3);
      float4* p = s + (q * PITCH + q2 * M2 + j) * VP;
      c2 v[R3];
#pragma unroll
      for (int r = 0; r < R3; ++r) v[r] = sload(p + r * M3 * VP);
      if constexpr (BACK) ptwiddle<R3, INV, M3>(v, tw + T3 + j);
      PDFT<R3, INV>::run(v);
      if constexpr (!BACK) ptwiddle<R3, INV, M3>(v, tw + T3 + j);
#pragma unroll
      for (int r = 0; r < R3; ++r) sstore(p + r * M3 * VP, v[r]);
    });
  }
  // address of butterfly b of the last stage (frequencies b + r N / RL)
  __device__ __forceinline__ static float4* last_ptr(float4* s, int b) {
    const int q = b % R1, rest = b / R1;
    if constexpr (S == 2) return s + (q * PITCH) * VP;
    if constexpr (S == 3) return s + (q * PITCH + rest * R3) * VP;
    const int q2 = rest % R2, q3 = rest / R2;
    return s + (q * PITCH + q2 * M2 + q3 * R4) * VP;
  }
  // stages 2 .. S-1 of the forward chain, with a barrier after each stage
  template <bool INV, class Sync>
  __device__ __forceinline__ static void inner(float4* s, const float2* tw, int t, Sync& sync) {
    sync();
    if constexpr (S >= 3) {
      mid2<INV, false>(s, tw, t);
      sync();
    }
    if constexpr (S >= 4) {
      mid3<INV, false>(s, tw, t);
      sync();
    }
  }

  // last stage: out(k, v) for every k (unnormalised)
  template <bool INV, class Out>
  __device__ __forceinline__ static void last(float4* s, int t, Out& out) {
    each<N / RL>(t, [&](int b) {
      const float4* p = last_ptr(s, b);
      c2 v[RL];
#pragma unroll
      for (int r = 0; r < RL; ++r) v[r] = sload(p + r * VP);
      PDFT<RL, INV>::run(v);
#pragma unroll
      for (int r = 0; r < RL; ++r) out(b + r * (N / RL), v[r]);
    });
  }

  // transform: out(k, v) for every k (unnormalised); the caller separates
  // successive uses of the buffer by a barrier (`sync` first thing on entry)
  template <bool INV, unsigned ZM = 0u, class Load, class Out, class Sync>
  __device__ __forceinline__ static void transform(float4* s, const float2* tw, int t, Load& load, Out& out, Sync& sync) {
    first<INV, ZM>(s, tw, t, load);
    inner<INV>(s, tw, t, sync);
    last<INV>(s, t, out);
  }

  // last stage with the outputs left in the buffer: frequency k = b + r N / RL at last_ptr(b) + r VP
  template <bool INV>
  __device__ __forceinline__ static void last_in_place(float4* s, int t) {
    each<N / RL>(t, [&](int b) {
      float4* p = last_ptr(s, b);
      c2 v[RL];
#pragma unroll
      for (int r = 0; r < RL; ++r) v[r] = sload(p + r * VP);
      PDFT<RL, INV>::run(v);
#pragma unroll
      for (int r = 0; r < RL; ++r) sstore(p + r * VP, v[r]);
    });
  }

  // centre of a round trip over butterflies [b0, b1): last stage, v <- f(b, r, v) at frequency b + r N / RL,
  // first stage back, in place.  Rolled: the body is emitted once.
  template <bool INV, class G>
  __device__ __forceinline__ static void centre(float4* s, int t, G& f, int b0 = 0, int b1 = N / RL) {
#pragma unroll 1
    for (int b = b0 + t; b < b1; b += L) {
      float4* p = last_ptr(s, b);
      c2 v[RL];
#pragma unroll
      for (int r = 0; r < RL; ++r) v[r] = sload(p + r * VP);
      PDFT<RL, INV>::run(v);
#pragma unroll
      for (int r = 0; r < RL; ++r) v[r] = f(b, r, v[r]);
      PDFT<RL, !INV>::run(v);
#pragma unroll
      for (int r = 0; r < RL; ++r) sstore(p + r * VP, v[r]);
    }
  }
  // the second half of a round trip on loaded values, v[r] = load(b + r N / RL): with back() a whole transform
  // in the operation order of a round trip's way back
  template <bool INV, class Load>
  __device__ __forceinline__ static void enter(float4* s, int t, Load& load) {
    each<N / RL>(t, [&](int b) {
      float4* p = last_ptr(s, b);
      c2 v[RL];
#pragma unroll
      for (int r = 0; r < RL; ++r) v[r] = load(b + r * (N / RL));
      PDFT<RL, INV>::run(v);
#pragma unroll
      for (int r = 0; r < RL; ++r) sstore(p + r * VP, v[r]);
    });
  }
  // the way back from the centre: out(n, v), natural order, unnormalised
  template <bool INV, class Out, class Sync>
  __device__ __forceinline__ static void back(float4* s, const float2* tw, int t, Out& out, Sync& sync) {
    sync();
    if constexpr (S >= 4) {
      mid3<INV, true>(s, tw, t);
      sync();
    }
    if constexpr (S >= 3) {
      mid2<INV, true>(s, tw, t);
      sync();
    }
    back_last<INV>(s, tw, t, out);
  }
  template <bool INV, class Out>
  __device__ __forceinline__ static void back_last(float4* s, const float2* tw, int t, Out& out) {
    each<M>(t, [&](int j) {
      c2 v[R1];
#pragma unroll
      for (int r = 0; r < R1; ++r) v[r] = sload(s + (r * PITCH + j) * VP);
      ptwiddle<R1, INV, M>(v, tw + j);
      PDFT<R1, INV>::run(v);
#pragma unroll
      for (int r = 0; r < R1; ++r) out(j + r * M, v[r]);
    });
  }
};

// Row kernels on pairs of rows: one buffer per pair, TEAMS pairs per CTA.
// Pairs of whole warps synchronise on a named barrier of their own; pairs that
// do not tile warps run in lockstep on the CTA's barrier (every team of the
// CTA then runs the same number of transforms).
template <int N, int TARGET = 128, int LANES = 512>
struct PairRows {
  using F = PairFFT<N, 1>;
  static constexpr int L = F::L;
  static constexpr bool OWN = L % 32 == 0;  // own barrier per pair
  static constexpr int T0 = TARGET / L > 0 ? TARGET / L : 1;
  static constexpr int T1 = OWN && T0 > 15 ? 15 : T0;
  static constexpr int teams() {
    int t = T1;
    while (!OWN && (t * L) % 32 != 0) ++t;
    return t;
  }
  static constexpr int TEAMS = teams();
  static constexpr int THREADS = TEAMS * L;
  static constexpr int TWB = (F::TW * (int)sizeof(float2) + 15) & ~15;
  static constexpr size_t SMEM = TWB + sizeof(float4) * (size_t)TEAMS * F::ELEMS;
  // LANES resident lanes per SM set the register budget: at 512, 128 registers hold a radix-16 stage of a pair (64
  // for the values, the rest addresses and twiddles); at 640, 96 just do
  static constexpr int MINB = LANES / THREADS > 0 ? LANES / THREADS : 1;
  __device__ __forceinline__ static void sync(int team) {
    if constexpr (OWN) {
      asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(L) : "memory");
    } else {
      __syncthreads();
    }
  }
};

// Column kernels: VP adjacent column pairs per CTA, the pair index fastest
// over the lanes, so that lanes read and write 16 VP contiguous bytes of a row
// straight from and to global memory (no staging through shared memory).
template <int N, int VPMAX = 4>
struct PairCols {
  static constexpr int L = PairPlan<N>::L;
  static constexpr size_t bytes(int vp) {
    return (size_t)PairPlan<N>::R1 * (N / PairPlan<N>::R1 + 1) * vp * sizeof(float4);
  }
  // two CTAs per SM where four pairs fit that way, else fewer pairs; 1024 threads at most
  static constexpr int vp() {
    int v = VPMAX;
    while (v > 1 && (v * L > 512 || bytes(v) > 100 * 1024)) v /= 2;
    return v;
  }
  static constexpr int VP = vp();
  using F = PairFFT<N, VP>;
  static constexpr int V = 2 * VP;
  static constexpr int THREADS = VP * L;
  static constexpr int TWB = (F::TW * (int)sizeof(float2) + 15) & ~15;
  static constexpr size_t SMEM = TWB + sizeof(float4) * (size_t)F::ELEMS;
  static constexpr int MINB = 512 / THREADS > 0 ? 512 / THREADS : 1;
};

}  // namespace cx
