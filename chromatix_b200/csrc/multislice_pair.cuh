// Row passes of the multislice loop (multislice.cuh) on row pairs, for every
// length with a pair plan (pair_fft.cuh).
//
// One padded plane is N / 2 row pairs: a pass of 1024^2 is 512 teams of 128
// lanes, about fourteen warps per SM, so it is bound by latency.  The slice's dn
// and absorption rows are inputs of the call, not of the previous pass: they
// are copied to shared memory and turned into the transmittance there before
// the pass waits for its predecessor (programmatic launch), so that part of
// the pass runs beside the end of the previous one.  The inverse transform,
// the product at the row's pixels and the forward transform share one pass
// over shared memory (PairFFT::centre).
#pragma once

#include "multislice.cuh"
#include "pair_fft.cuh"

namespace cx {

// One row pair per CTA.  Shared memory: twiddles | transform buffer | per row
// of the pair the transmittance (re, im) [MS_FLUOR: and the source (re, im)]
// [MS_BWD: and the recorded field] | mbarrier.
template <int NX, int MODE>
struct MsPairCfg {
  using F = PairFFT<NX, 1, true>;
  static constexpr int L = F::L;
  static constexpr int THREADS = L;
  static constexpr bool PF = MODE == MS_FWD || MODE == MS_BWD || MODE == MS_FLUOR;
  static constexpr int MAPS = MODE == MS_FWD ? 2 : 4;  // floats per pixel and row (MS_FLUOR: 3 copied, 4 kept)
  static constexpr int TWB = (F::TW * (int)sizeof(float2) + 15) & ~15;
  static constexpr size_t PF_OFF = TWB + sizeof(float4) * (size_t)F::ELEMS;
  static constexpr size_t BAR_OFF = PF_OFF + (PF ? sizeof(float) * 2 * (size_t)MAPS * NX : 0);
  static constexpr size_t SMEM = BAR_OFF + 16;
  static constexpr int WARPS = (THREADS + 31) / 32;
  static constexpr int MINB = SMEM > 113 * 1024 ? 1 : (16 / WARPS > 0 ? 16 / WARPS : 1);
  static constexpr int POLLS = 1 << 20;
  static_assert(SMEM <= 227 * 1024, "row pair does not fit one CTA");
};

template <int NX, int MODE>
__global__ void __launch_bounds__(MsPairCfg<NX, MODE>::THREADS, MsPairCfg<NX, MODE>::MINB) k_ms_rows_pair(MsArgs a) {
  using C = MsPairCfg<NX, MODE>;
  using F = typename C::F;
  constexpr int NB = NX / F::RL;
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  float4* s = reinterpret_cast<float4*>(smem + C::TWB);
  float* pf = reinterpret_cast<float*>(smem + C::PF_OFF);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + C::BAR_OFF);
  const int t = threadIdx.x;
  auto sync = [] { __syncthreads(); };
  pdl_trigger();
  // rows y, y + 1 of the padded grid (MS_FINAL: of its cropped part)
  const int r0 = MODE == MS_FINAL ? a.pad_y : 0, nrows = MODE == MS_FINAL ? a.ny : a.py;
  const int y = r0 + 2 * blockIdx.x;
  const bool two = 2 * (int)blockIdx.x + 1 < nrows;
  const int yd = y - a.pad_y;
  const bool in0 = yd >= 0 && yd < a.ny, in1 = two && yd + 1 >= 0 && yd + 1 < a.ny;
  F::load_tables(tw, a.twg, t, C::THREADS);
  const size_t off0 = (size_t)a.slice * a.ny * a.nx + (size_t)(in0 ? yd : 0) * a.nx;
  const size_t off1 = (size_t)a.slice * a.ny * a.nx + (size_t)(in1 ? yd + 1 : 0) * a.nx;
  // per row j: [dn -> t.re][ab -> t.im] ([fl -> source re][source im]) or ([recorded field])
  float* p0 = pf;
  float* p1 = pf + (size_t)C::MAPS * NX;
  if constexpr (C::PF) {
    if (t == 0) bulk_mbar_init(bar);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    __syncthreads();
    const float* m1 = MODE == MS_FLUOR ? a.fl : a.ab;
    bool bulk = a.nx % 4 == 0 && ((reinterpret_cast<size_t>(a.dn) | reinterpret_cast<size_t>(m1)) & 15) == 0;
    if constexpr (MODE == MS_FLUOR) bulk = bulk && (reinterpret_cast<size_t>(a.ph) & 15) == 0;
    if constexpr (MODE == MS_BWD) bulk = bulk && a.px % 2 == 0 && (reinterpret_cast<size_t>(a.rec_u) & 15) == 0;
    if (bulk && (in0 || in1)) {
      if (t == 0) {
        // read once per pass: evict first (the field state and the propagator stay in L2)
        const uint64_t pol = l2_evict_first();
        const unsigned rb = (unsigned)a.nx * 4u, ub = (unsigned)a.px * 8u;
        const unsigned per = MODE == MS_FWD ? 2 * rb : (MODE == MS_FLUOR ? 3 * rb : 2 * rb + ub);
        bulk_expect(bar, per * ((in0 ? 1u : 0u) + (in1 ? 1u : 0u)));
        auto row = [&](float* p, size_t off, int yy) {
          bulk_copy_g2s_hint(p, a.dn + off, rb, bar, pol);
          bulk_copy_g2s_hint(p + NX, m1 + off, rb, bar, pol);
          if constexpr (MODE == MS_FLUOR) bulk_copy_g2s_hint(p + 2 * NX, a.ph + off, rb, bar, pol);
          if constexpr (MODE == MS_BWD) bulk_copy_g2s_hint(p + 2 * NX, a.rec_u + (size_t)yy * a.px, ub, bar, pol);
        };
        if (in0) row(p0, off0, y);
        if (in1) row(p1, off1, y + 1);
      }
      // past the (generous) poll limit the rows are read from global memory instead
      bulk = bulk_wait(bar, 0, C::POLLS);
    }
    // transmittance (and source) of the rows, in place of what they are made of
#pragma unroll 1
    for (int i = t; i < 2 * a.nx; i += C::THREADS) {
      const int j = i >= a.nx, x = i - (j ? a.nx : 0);
      if (!(j ? in1 : in0)) continue;
      float* p = j ? p1 : p0;
      const size_t off = (j ? off1 : off0) + x;
      const float dnv = bulk ? p[x] : a.dn[off];
      const float abv = bulk ? p[NX + x] : m1[off];
      if constexpr (MODE == MS_FLUOR) {
        float sp, cp;
        sincosf(bulk ? p[2 * NX + x] : a.ph[off], &sp, &cp);
        const float2 tr = ms_transmittance(a, dnv, 0.f);
        p[x] = tr.x;
        p[NX + x] = tr.y;
        p[2 * NX + x] = abv * cp;
        p[3 * NX + x] = abv * sp;
      } else {
        const float2 tr = ms_transmittance(a, dnv, abv);
        p[x] = tr.x;
        p[NX + x] = tr.y;
      }
    }
    if constexpr (MODE == MS_BWD) {
      if (!bulk)
        for (int i = t; i < 2 * a.px; i += C::THREADS) {
          const int j = i >= a.px, x = i - (j ? a.px : 0);
          if (j ? in1 : in0)
            reinterpret_cast<float2*>((j ? p1 : p0) + 2 * NX)[x] = a.rec_u[(size_t)(y + j) * a.px + x];
        }
    }
  }
  __syncthreads();
  pdl_wait();
  float2* row = a.buf + (size_t)y * a.px;
  const size_t up = two ? (size_t)a.px : 0;
  if constexpr (MODE == MS_LOAD) {
    const int ys = y - a.oy;
    const bool s0 = ys >= 0 && ys < a.sy, s1 = two && ys + 1 >= 0 && ys + 1 < a.sy;
    const float2* srow = a.src + (ptrdiff_t)ys * a.sx;
    float2* rrow = a.rec + (size_t)y * a.px;
    auto load = [&](int n) -> c2 {
      const int xs = n - a.ox;
      const bool xin = xs >= 0 && xs < a.sx;
      const float2 z = make_float2(0.f, 0.f);
      const c2 v = ppack(xin && s0 ? cscale(srow[xs], a.load_scale) : z, xin && s1 ? cscale(srow[a.sx + xs], a.load_scale) : z);
      if (a.record) {
        rrow[n] = pfirst(v);
        if (two) rrow[a.px + n] = psecond(v);
      }
      return v;
    };
    auto out = [&](int k, c2 v) {
      row[k] = pfirst(v);
      if (two) row[up + k] = psecond(v);
    };
    // in the operation order of MS_FWD's forward transform: a segment recomputed from its record gives the same bits
    F::template enter<false>(s, t, load);
    F::template back<false>(s, tw, t, out, sync);
  } else {
    auto load = [&](int n) -> c2 { return ppack(ld2z(row + n, true), ld2z(row + up + n, true)); };
    F::template first<true>(s, tw, t, load);
    F::template inner<true>(s, tw, t, sync);
    if constexpr (MODE == MS_FINAL) {
      float2* drow = a.dst + (size_t)yd * a.nx;
      auto out = [&](int k, c2 v) {
        const int xd = k - a.pad_x;
        if (xd >= 0 && xd < a.nx) {
          drow[xd] = pfirst(v);
          if (two) drow[a.nx + xd] = psecond(v);
        }
      };
      F::template last<true>(s, t, out);
    } else {
      const uint64_t pol = l2_evict_first();  // records are read back once, by the adjoint
      float2* rrow = a.record ? a.rec + (size_t)y * a.px : nullptr;
      auto f = [&](int b, int r, c2 v) -> c2 {
        const int n = b + r * NB, xd = n - a.pad_x;
        const bool xin = (unsigned)xd < (unsigned)a.nx;
        const bool h0 = xin && in0, h1 = xin && in1;
        const int xi = xin ? xd : 0;
        if constexpr (MODE == MS_BWD) {
          // w = g conj(u): dL/d dn = k dz Im w, dL/d abs = -k dz Re w (k dz as a sum of two floats: the products
          // round as from FP64)
          const float2* u0 = reinterpret_cast<const float2*>(p0 + 2 * NX);
          const float2* u1 = reinterpret_cast<const float2*>(p1 + 2 * NX);
          auto grad = [&](float2 g, float2 u, size_t gi) {
            const float wr = g.x * u.x + g.y * u.y, wi = g.y * u.x - g.x * u.y;
            a.gdn[gi] = fmaf(a.kdz_f, wi, a.kdz_lo * wi);
            a.gab[gi] = -fmaf(a.kdz_f, wr, a.kdz_lo * wr);
          };
          if (h0) grad(pfirst(v), u0[n], (size_t)yd * a.nx + xi);
          if (h1) grad(psecond(v), u1[n], (size_t)(yd + 1) * a.nx + xi);
        }
        c2 tr = ppack(h0 ? make_float2(p0[xi], p0[NX + xi]) : make_float2(1.f, 0.f),
                      h1 ? make_float2(p1[xi], p1[NX + xi]) : make_float2(1.f, 0.f));
        if constexpr (MODE == MS_BWD) tr.im = f2neg(tr.im);
        v = pmul(v, tr);
        if constexpr (MODE == MS_FLUOR) {
          if (h0) v.re.x += p0[2 * NX + xi], v.im.x += p0[3 * NX + xi];
          if (h1) v.re.y += p1[2 * NX + xi], v.im.y += p1[3 * NX + xi];
        }
        if constexpr (MODE == MS_FWD) {
          if (rrow) {
            st_hint(rrow + n, pfirst(v), pol);
            if (two) st_hint(rrow + a.px + n, psecond(v), pol);
          }
        }
        return v;
      };
      F::template centre<true>(s, t, f);
      auto out = [&](int k, c2 v) {
        row[k] = pfirst(v);
        if (two) row[up + k] = psecond(v);
      };
      F::template back<false>(s, tw, t, out, sync);
    }
  }
}

}  // namespace cx
