// lw_rt64.cuh -- FP64 McICA radiative transfer, thread = g-point.
//
// Replaces rtrnmc (physics/Radiation/RRTMG/radlw_main.F90, RLM:3420-3785) and
// the output mapping of rrtmg_lw_run (RLM:1228-1304) in FP64; the spectral
// heating rates (hlwb) and the FP32 path run lw_rt.cuh.  A CTA of five warps
// owns one column, a thread one of its 140 g-points: it walks the layers down
// and then up in the reference's order, four at a time, so the four layers'
// optical depths and table records are in flight together and the recurrence
// behind them is one FMA per layer and sweep.
//
// Bound: FP64 issue and the table gathers.  Against a column per warp with the
// layers across the lanes (both sweeps as affine scans: a composition, five
// shuffle steps and a replay per g-point, lw_rt.cuh), a layer's terms cost two
// evaluations but no scan, a column spreads over five warps, and a layer count
// of 64 leaves no lane idle.  16,384 x 127: 5.02 ms as scans, 4.26 here;
// 5,003 x 127: 2.06 -> 1.35 ms; 1,024 x 64: 493 -> 174 us; 32 x 64: 569 -> 47 us.
// The way down leaves {transmittance, upward source} in place of {tau, frac}
// (recomputing both on the way up: 6.06 ms); with exp_tbl and tfn_tbl in shared
// memory, three columns per CTA: 5.83 ms; four CTAs per SM at 96 registers:
// 5.93 ms.
#pragma once

#include "fp64_util.cuh"
#include "lw_gas.cuh"

namespace lw {

constexpr int kRt64Threads = 160, kRt64Warps = kRt64Threads / 32;

// tau and frac of this path, [c][kb][140][4]: four layers of a g-point are one
// 32-byte sector, written by the layers' threads (lw_gas.cuh) and read by the
// g-point's
constexpr int kRt64Block = NGPT * 4;

__host__ __device__ inline size_t rt64_smem_bytes(int nlay) {   // the warps' partial sums
  return (size_t)kRt64Warps * 4 * (nlay + 1) * sizeof(double);
}

// L2 loads that keep their place among the table gathers
__device__ __forceinline__ double2 ld_stream(const double2* p) {
  double2 v;
  asm volatile("ld.global.cg.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

// four layers of a thread's g-point and band
struct Rt64In {
  double tau[4], frac[4], blay[4], plev[5];   // plev: the five levels around them
};
struct Rt64Terms {
  double tr[4], sd[4], su[4];      // clear sky: transmittance, layer sources down and up
  double trt[4], sdt[4], sut[4];   // the same in total sky
};

__global__ void __launch_bounds__(kRt64Threads, 3)
lw_rt64_kernel(const Block* __restrict__ blocks, int nblocks, const Block b0, int ncols, Flags f, Consts cs,
               Tables<double> tab, Scratch<double> sc, int NLP, const uint32_t* __restrict__ bits_g) {
  extern __shared__ __align__(16) unsigned char rt64_smem[];
  double* const part = reinterpret_cast<double*>(rt64_smem);   // [warp][down clear, down total, up clear, up total][nlp1]
  const int tid = threadIdx.x;
  auto exp_tfn = [&](int i, double& ex, double& tf) {
    asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(ex), "=d"(tf) : "l"(tab.trec + 2 * i));
  };
  const int lane = tid & 31, warp = tid >> 5;
  const int nlay = f.nlay, nlp1 = nlay + 1, nw = (nlay + 31) >> 5, nb = nlay / 4 + 1;   // blocks up to level nlay
  const bool on = tid < NGPT;
  const int g = on ? tid : NGPT - 1;
  int b = 0;
#pragma unroll
  for (int q = 1; q < NBANDS; ++q) b += g >= ns_of(q) ? 1 : 0;

  const int cc = blockIdx.x, c = sc.c0 + cc;
  const Block& B = (nblocks == 1) ? b0 : blocks[find_block(blocks, nblocks, c)];
  const double* crec = sc.col + (size_t)cc * kColRec;
  const bool mc = crec[33] != 0.0;
  const double secd = crec[b], pk0 = crec[16 + b], semis = crec[32], reflct = 1.0 - semis;
  double* tcol = sc.tau + (size_t)cc * NGPT * NLP + 4 * g;
  double* fcol = sc.frac + (size_t)cc * NGPT * NLP + 4 * g;
  const double* pcol = sc.band + ((size_t)cc * 3 * NBANDS + b) * NLP;   // pklay; pklev and taucld NBANDS rows apart
  const double* lcol = pcol + (size_t)NBANDS * NLP;
  const double* ccol = lcol + (size_t)NBANDS * NLP;
  const uint32_t* cbw = bits_g + ((size_t)c * NGPT + g) * nw;

  auto planck = [&](int kb, Rt64In& v) {
    const double2* p = reinterpret_cast<const double2*>(pcol + 4 * kb);
    const double2* l = reinterpret_cast<const double2*>(lcol + 4 * kb);
    const double2 p0 = __ldg(p), p1 = __ldg(p + 1), l0 = __ldg(l), l1 = __ldg(l + 1);
    v.blay[0] = p0.x; v.blay[1] = p0.y; v.blay[2] = p1.x; v.blay[3] = p1.y;
    v.plev[0] = l0.x; v.plev[1] = l0.y; v.plev[2] = l1.x; v.plev[3] = l1.y;
    v.plev[4] = __ldg(lcol + min(4 * kb + 4, nlay));
  };
  auto load = [&](int kb, Rt64In& v) {
    const double2* t = reinterpret_cast<const double2*>(tcol + (size_t)kb * kRt64Block);
    const double2* r = reinterpret_cast<const double2*>(fcol + (size_t)kb * kRt64Block);
    const double2 t0 = ld_stream(t), t1 = ld_stream(t + 1), r0 = ld_stream(r), r1 = ld_stream(r + 1);
    v.tau[0] = t0.x; v.tau[1] = t0.y; v.tau[2] = t1.x; v.tau[3] = t1.y;
    v.frac[0] = r0.x; v.frac[1] = r0.y; v.frac[2] = r1.x; v.frac[3] = r1.y;
    planck(kb, v);
  };
  // flags of layers 4 kb .. 4 kb + 3
  uint32_t word = 0;
  auto nibble = [&](int kb) { return (word >> (4 * kb & 31)) & 15u; };
  auto flags_of = [&](int kb) {   // no layer at or above nlay is cloudy
    const int w = kb >> 3, n = nlay - 32 * w;
    return (mc && on && w < nw) ? __ldg(cbw + w) & (n < 32 ? (1u << n) - 1u : ~0u) : 0u;
  };

  // Transmittances and sources of a block's layers (RLM:3598-3660), down
  // (through the lower level) and up (through the upper level).
  // A warp's loads return in order, so `next` (the next block's loads, which come
  // from further away) is issued behind this block's gathers (4.95 -> 4.66 ms).
  auto terms = [&](int kb, const Rt64In& v, Rt64Terms& o, auto&& next) {
    double od[4], at[4], pf[4];   // optical depth, 1 - transmittance, Pade factor
    bool thick = false;
    const uint32_t nib = nibble(kb);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      od[j] = secd * v.tau[j];
      od[j] = od[j] > 0.0 ? od[j] : 0.0;
      thick |= od[j] > 0.06;
      at[j] = fma(-0.5 * od[j], od[j], od[j]);
      o.tr[j] = 1.0 - at[j];
      pf[j] = kRec6 * od[j];
    }
    if (__any_sync(0xffffffffu, thick)) {
      double ex[4], tf[4];
      int i[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) i[j] = od[j] > 0.06 ? fp64::pade_index(od[j]) : 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) exp_tfn(i[j], ex[j], tf[j]);
      next();   // behind the gathers: a warp's loads return in order, and these come from further away
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool tk = od[j] > 0.06;
        o.tr[j] = tk ? ex[j] : o.tr[j];
        at[j] = tk ? 1.0 - ex[j] : at[j];
        pf[j] = tk ? tf[j] : pf[j];
        if (tk && ((nib >> j) & 1u)) od[j] = tbl_tau(tab.trec, i[j]);
      }
    } else {
      next();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double fa = v.frac[j] * at[j];
      o.sd[j] = fa * fma(v.plev[j] - v.blay[j], pf[j], v.blay[j]);
      o.su[j] = fa * fma(v.plev[j + 1] - v.blay[j], pf[j], v.blay[j]);
      o.trt[j] = o.tr[j];
      o.sdt[j] = o.sd[j];
      o.sut[j] = o.su[j];
    }
    if (nib) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (!((nib >> j) & 1u)) continue;
        const double odcld = secd * __ldg(ccol + 4 * kb + j);
        const double odtot = od[j] + odcld;
        double totfac, a;
        if (odtot < 0.06) {
          totfac = kRec6 * odtot;
          a = odtot - 0.5 * odtot * odtot;
        } else {
          double ex;
          exp_tfn(fp64::pade_index(odtot), ex, totfac);
          a = 1.0 - ex;
        }
        const double fa = v.frac[j] * a;
        o.trt[j] = o.tr[j] * exp(-odcld);   // clfm = 1 for a McICA cloudy sub-column
        o.sdt[j] = fa * fma(v.plev[j] - v.blay[j], totfac, v.blay[j]);
        o.sut[j] = fa * fma(v.plev[j + 1] - v.blay[j], totfac, v.blay[j]);
      }
    }
  };
  // layers at or above nlay pass the radiance on (their scratch is not written)
  auto mask = [&](int kb, Rt64In& v) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (4 * kb + j >= nlay) v.tau[j] = v.frac[j] = v.blay[j] = 0.0;
      if (4 * kb + j > nlay) v.plev[j] = 0.0;
    }
  };
  // sums of the block's levels over the warp's g-points
  const int idx = fp64::sum_index<8, 32>(lane);
  auto flush = [&](int kb, int q0, double (&v)[8]) {
    if (warp == kRt64Warps - 1)
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = on ? v[q] : 0.0;
    const double r = fp64::lane_sums<8, 32>(v, lane, 0xffffffffu);
    const int lv = 4 * kb + (idx >> 1);
    if (idx >= 0 && lv <= nlay) part[((size_t)warp * 4 + q0 + (idx & 1)) * nlp1 + lv] = r;
  };

  Rt64In nx;
  double xc = 0.0, xt = 0.0;
  // ---- down ----
  const double frac0 = __ldcg(fcol);
  load(nb - 1, nx);
  word = flags_of(nb - 1);
#pragma unroll 1
  for (int kb = nb - 1; kb >= 0; --kb) {
    Rt64In v = nx;
    if ((kb & 7) == 7) word = flags_of(kb);
    if (kb == nb - 1) mask(kb, v);
    Rt64Terms o;
    terms(kb, v, o, [&] { if (kb > 0) load(kb - 1, nx); });
    {   // the way up reads {tr, su} instead, but for the cloudy layers
      const uint32_t nib = nibble(kb);
      double a[4], e[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool cl = (nib >> j) & 1u;
        a[j] = cl ? v.tau[j] : o.tr[j];
        e[j] = cl ? v.frac[j] : o.su[j];
      }
      if (on) {
        double2* t = reinterpret_cast<double2*>(tcol + (size_t)kb * kRt64Block);
        double2* r = reinterpret_cast<double2*>(fcol + (size_t)kb * kRt64Block);
        __stcg(t, make_double2(a[0], a[1]));
        __stcg(t + 1, make_double2(a[2], a[3]));
        __stcg(r, make_double2(e[0], e[1]));
        __stcg(r + 1, make_double2(e[2], e[3]));
      }
    }
    double r[8];
#pragma unroll
    for (int j = 3; j >= 0; --j) {
      xc = fma(xc, o.tr[j], o.sd[j]);
      xt = fma(xt, o.trt[j], o.sdt[j]);
      r[2 * j] = xc;
      r[2 * j + 1] = xt;
    }
    flush(kb, 0, r);
  }
  // ---- surface emission and reflection (RLM:3682-3691) ----
  {
    const double rad0 = semis * frac0 * pk0;
    xc = fma(reflct, xc, rad0);
    xt = fma(reflct, xt, rad0);
  }
  // ---- up ----
  struct Pair { double tr[4], su[4]; } np;
  auto load_up = [&](int kb, Pair& v) {
    const double2* t = reinterpret_cast<const double2*>(tcol + (size_t)kb * kRt64Block);
    const double2* r = reinterpret_cast<const double2*>(fcol + (size_t)kb * kRt64Block);
    const double2 t0 = __ldcg(t), t1 = __ldcg(t + 1), r0 = __ldcg(r), r1 = __ldcg(r + 1);
    v.tr[0] = t0.x; v.tr[1] = t0.y; v.tr[2] = t1.x; v.tr[3] = t1.y;
    v.su[0] = r0.x; v.su[1] = r0.y; v.su[2] = r1.x; v.su[3] = r1.y;
  };
  load_up(0, np);
  word = flags_of(0);
#pragma unroll 1
  for (int kb = 0; kb < nb; ++kb) {
    const Pair v = np;
    if (kb + 1 < nb) load_up(kb + 1, np);
    if ((kb & 7) == 0) word = flags_of(kb);
    const uint32_t nib = nibble(kb);
    double r[8], trt[4], sut[4], tr[4], su[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      tr[j] = trt[j] = v.tr[j];
      su[j] = sut[j] = v.su[j];
    }
    if (__any_sync(0xffffffffu, nib != 0)) {
      Rt64In in;
      planck(kb, in);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool cl = (nib >> j) & 1u;
        in.tau[j] = cl ? v.tr[j] : 0.0;
        in.frac[j] = cl ? v.su[j] : 0.0;
      }
      Rt64Terms o;
      terms(kb, in, o, [] {});
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if ((nib >> j) & 1u) {
          tr[j] = o.tr[j];
          su[j] = o.su[j];
          trt[j] = o.trt[j];
          sut[j] = o.sut[j];
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      r[2 * j] = xc;
      r[2 * j + 1] = xt;
      xc = fma(xc, tr[j], su[j]);
      xt = fma(xt, trt[j], sut[j]);
    }
    flush(kb, 2, r);
  }
  __syncthreads();

  // ---- sums over the warps in a fixed order, fluxes ----
  const double flxfac = 0.5 * cs.fluxfac;   // wtdiff * fluxfac
  for (int q = tid; q < 4 * nlp1; q += kRt64Threads) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < kRt64Warps; ++w) t += part[(size_t)w * 4 * nlp1 + q];
    part[q] = t * flxfac;
  }
  __syncthreads();
  const double *dc = part, *dt = part + nlp1, *uc = part + 2 * nlp1, *ut = part + 3 * nlp1;
  const int i = c - B.col0;
  const size_t ld = (size_t)B.ld;
  const bool top = f.top_at_1 != 0;
  if (tid == 0) {
    B.out[O_TOPFLX][2 * i + 0] = ut[nlay];
    B.out[O_TOPFLX][2 * i + 1] = uc[nlay];
    B.out[O_SFCFLX][4 * i + 0] = ut[0];
    B.out[O_SFCFLX][4 * i + 1] = uc[0];
    B.out[O_SFCFLX][4 * i + 2] = dt[0];
    B.out[O_SFCFLX][4 * i + 3] = dc[0];
  }
  if (f.want_flxprf)
    for (int lv = tid; lv < nlp1; lv += kRt64Threads) {
      double* p = B.out[O_FLXPRF] + 4 * (i + ld * (size_t)(top ? nlp1 - lv - 1 : lv));
      p[0] = ut[lv]; p[1] = dt[lv]; p[2] = uc[lv]; p[3] = dc[lv];
    }
  for (int k = tid; k < nlay; k += kRt64Threads) {   // RLM:3754-3770
    const size_t x = i + ld * (size_t)(top ? nlay - 1 - k : k);
    const double rfdelp = cs.heatfac / B.in[F_DELPIN][x];
    B.out[O_HLWC][x] = ((ut[k] - dt[k]) - (ut[k + 1] - dt[k + 1])) * rfdelp;
    if (f.want_hlw0) B.out[O_HLW0][x] = ((uc[k] - dc[k]) - (uc[k + 1] - dc[k + 1])) * rfdelp;
  }
}

static inline cudaError_t rt64_one(const Block* blocks, int nblocks, const Block& b0, int nc, const Flags& f,
                                   const Consts& cs, const Tables<double>& tab, const Scratch<double>& sc, int NLP,
                                   const uint32_t* bits, cudaStream_t st) {
  lw_rt64_kernel<<<nc, kRt64Threads, rt64_smem_bytes(f.nlay), st>>>(blocks, nblocks, b0, nc, f, cs, tab, sc, NLP, bits);
  return cudaGetLastError();
}

}  // namespace lw
