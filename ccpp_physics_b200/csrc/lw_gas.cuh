// lw_gas.cuh -- kernel A of the RRTMG-LW path: per-layer column state,
// setcoef and the gas optics of all 140 g-points.
//
// Replaces, per column, the driver prologue of rrtmg_lw_run
// (physics/Radiation/RRTMG/radlw_main.F90, RLM:785-1050), the band cloud
// optics of cldprop (RLM:1589-1799), setcoef (RLM:2151-2406) and taumol
// (RLM:3836-6840).  One warp owns 32 layers of a column at a time, one lane one
// layer; the layer's setcoef record waits in shared memory and the bands are
// walked in order, so every table gather of a band happens while the band's
// coefficients are hot in L1/L2.
//
// Output (device scratch, read by kernel B in lw_rt.cuh or lw_rt64.cuh), per
// column c of the chunk and layer k (0-based, surface first), NLP = 32*V >= nlay+1:
//   tau  [c][g][NLP]      gas + aerosol optical depth  (taumol tautot)
//   frac [c][g][NLP]      Planck fraction              (taumol fracs)
//                         (for lw_rt64.cuh [c][k / 4][g][4])
//   band [c][0][b][NLP]   pklay(b, k+1)
//        [c][1][b][NLP]   pklev(b, k)      k = 0..nlay
//        [c][2][b][NLP]   taucld(b, k+1)
//   col  [c][48]          secdiff(16), pklay(b,0)(16), semiss, lcf1
#pragma once

#include "fp64_util.cuh"
#include "lw_bands.cuh"
#include "lw_common.cuh"
#include "lw_features.cuh"

namespace lw {

constexpr double kEps = 1.0e-6;                 // RLM:309
constexpr double kBpade = 1.0 / 0.278;          // RLM:312
constexpr double kStpfac = 296.0 / 1013.0;      // RLM:313
constexpr double kTblint = 10000.0;             // RLM:315 (ntbl)
constexpr double kRec6 = 0.166667;              // RLM:3548 (not 1/6)
constexpr double kConG = 9.80665, kConAvgd = 6.0221415e23;
constexpr double kConAmd = 28.9644, kConAmw = 18.0154, kConAmo3 = 47.9982;
constexpr double kAbsrain = 0.33e-3, kAbssnow0 = 1.5;   // radlw_datatb.f:941,944
constexpr int kColRec = 48;                     // doubles per column record

// Minimum resident CTAs per SM requested from the register allocator
// (measured on B200, 16,384 columns x 127 layers: gas optics 3 in FP64 and 4
// in FP32, transfer 4, gas optics behind the network 5).  The V = 8
// transfer kernels (128..255 layers) are left uncapped: with the caps their
// transfer kernel spilled ~1 KB per thread and an illegal address was
// observed that reading the code did not explain.
#ifndef LW_GAS_MINB
#define LW_GAS_MINB 3
#endif
// gas optics behind the learned gas optics (setcoef/taumol only for
// out-of-envelope layers): light enough for more resident CTAs
#ifndef LW_GAS_MINB_SG
#define LW_GAS_MINB_SG 5
#endif
#ifndef LW_RT_MINB
#ifdef LW_RT_MINB_SMALL
#define LW_RT_MINB (V > 4 ? 1 : LW_RT_MINB_SMALL)
#else
#define LW_RT_MINB (V > 4 ? 1 : 4)
#endif
#endif

static __device__ __constant__ double c_delwave[16] = {340., 150., 130., 70., 120., 160., 100., 100.,
                                                       210., 90., 320., 280., 170., 130., 220., 650.};
static __device__ __constant__ double c_a0[16] = {1.66, 1.55, 1.58, 1.66, 1.54, 1.454, 1.89, 1.33,
                                                  1.668, 1.66, 1.66, 1.66, 1.66, 1.66, 1.66, 1.66};
static __device__ __constant__ double c_a1[16] = {0.00, 0.25, 0.22, 0.00, 0.13, 0.446, -0.10, 0.40,
                                                  -0.006, 0.00, 0.00, 0.00, 0.00, 0.00, 0.00, 0.00};
static __device__ __constant__ double c_a2[16] = {0.00, -12.0, -11.7, 0.00, -0.72, -0.243, 0.19, -0.062,
                                                  0.414, 0.00, 0.00, 0.00, 0.00, 0.00, 0.00, 0.00};


// checked read of the FP64 coefficient tables
__device__ __forceinline__ double t64(const double* kt, long long o) {
  if (!LW_OK(o >= 0 && o < bandtab::end, 11, o)) return 0.0;
  return __ldg(kt + o);
}

// cldprop band optics of one layer and band (RLM:1589-1799), FP64.
__device__ __forceinline__ double band_taucld(int b, const Flags& f, const double* kt, double cf, double clwp,
                                              double relw, double ciwp, double reiw, double cda1, double cda3,
                                              double cda4) {
  if (!(cf > 2.2250738585072014e-308)) return 0.0;   // cfrac(k) > cldmin = tiny
  if (f.ilwcliq <= 0) return cda1;                    // diagnostic cloud optical depth
  double tauran = kAbsrain * cda1;
  double tausnw = (cda3 > 0.0 && cda4 > 10.0) ? kAbssnow0 * 1.05756 * cda3 / cda4 : 0.0;
  double tauliq = 0.0, tauice = 0.0;
  if (clwp > 0.0 && f.ilwcliq == 1) {
    double factor = relw - 1.5;
    int index = max(1, min(57, (int)factor));
    double fint = factor - (double)index;
    double a = t64(kt, lwtab::absliq1 + (index - 1) + 58 * b);
    double c = t64(kt, lwtab::absliq1 + index + 58 * b);
    tauliq = fmax(0.0, clwp * (a + fint * (c - a)));
  }
  if (ciwp > 0.0) {
    if (f.ilwcice == 1) {
      double refice = fmin(130.0, fmax(13.0, reiw));
      int ia = (int)t64(kt, lwtab::ipat + b);
      tauice = fmax(0.0, ciwp * (t64(kt, lwtab::absice1 + 2 * (ia - 1)) +
                                 t64(kt, lwtab::absice1 + 1 + 2 * (ia - 1)) / refice));
    } else if (f.ilwcice == 2) {
      double factor = (reiw - 2.0) / 3.0;
      int index = max(1, min(42, (int)factor));
      double fint = factor - (double)index;
      double a = t64(kt, lwtab::absice2 + (index - 1) + 43 * b);
      double c = t64(kt, lwtab::absice2 + index + 43 * b);
      tauice = fmax(0.0, ciwp * (a + fint * (c - a)));
    } else if (f.ilwcice == 3) {
      double dgeice = fmax(5.0, 1.0315 * reiw);
      double factor = (dgeice - 2.0) / 3.0;
      int index = max(1, min(45, (int)factor));
      double fint = factor - (double)index;
      double a = t64(kt, lwtab::absice3 + (index - 1) + 46 * b);
      double c = t64(kt, lwtab::absice3 + index + 46 * b);
      tauice = fmax(0.0, ciwp * (a + fint * (c - a)));
    }
  }
  return tauice + tauliq + tauran + tausnw;
}

// Planck integral of band b at temperature index/fraction (RLM:2251-2283)
__device__ __forceinline__ double planck_int(const double* kt, int b, int ind, double frac) {
  double p0 = t64(kt, lwtab::totplnk + (ind - 1) + 181 * b);
  double p1 = t64(kt, lwtab::totplnk + ind + 181 * b);
  return c_delwave[b] * (p0 + frac * (p1 - p0));
}

// Per-warp working arrays of gas_unit.
template <typename R>
struct GasWork {
  double* red;   // [2 NLP] coldry and h2o column amounts of the whole column
  double* cld;   // [8][32] cloud inputs of the layer
  R* lay;        // [N_LF][32] setcoef record (LayRef)
  int* li;       // [32]
  __host__ __device__ static constexpr size_t bytes(int NLP) {
    return sizeof(double) * (2 * (size_t)NLP + 8 * 32) + sizeof(R) * N_LF * 32 + sizeof(int) * 32;
  }
  __device__ __forceinline__ static GasWork at(void* base, int NLP) {
    GasWork w;
    w.red = reinterpret_cast<double*>(base);
    w.cld = w.red + 2 * NLP;
    w.lay = reinterpret_cast<R*>(w.cld + 8 * 32);
    w.li = reinterpret_cast<int*>(w.lay + N_LF * 32);
    return w;
  }
};

// dry-air and water-vapour column amounts of a layer (RLM:823-836)
struct ColAmt {
  double coldry, h2ovmr;
};
__device__ __forceinline__ ColAmt col_amounts(double q, double delp) {
  const double amdw = kConAmd / kConAmw;
  const double tem1c = 100.0 * kConG, tem2c = 1.0e-20 * 1.0e3 * kConAvgd;
  ColAmt o;
  o.h2ovmr = fmax(0.0, q * amdw / (1.0 - q));
  const double tem0 = (1.0 - o.h2ovmr) * kConAmd + o.h2ovmr * kConAmw;
  o.coldry = tem2c * delp / (tem1c * tem0 * (1.0 + o.h2ovmr));
  return o;
}

// Kernel A's work for 32 layers (segment seg) and bands b_lo .. b_hi - 1 of
// column cc of the chunk (global column sc.c0 + cc), by one warp, a lane per
// layer.  What the layers share (the split of the atmosphere, the cloudy-column
// test, the precipitable water) each warp finds for itself, so no warp waits
// for another: with a CTA per column, the warps of the upper atmosphere waited
// at every column's barrier for the one whose layers lie on both sides.
// 16,384 x 127: FP64 5.03 -> 4.40 ms; 32 x 64, in eight band groups, 100 -> 31 us.
template <typename R, bool SG>
__device__ __forceinline__ void gas_unit(int cc, int seg, int b_lo, int b_hi, int lane, int NLP, const GasWork<R>& W,
                                         const Block* __restrict__ blocks, int nblocks, const Block& b0,
                                         const Flags& f, const Tables<R>& tab, const Tables<double>& tab64,
                                         const Scratch<R>& sc, double* __restrict__ gas_taug,
                                         double* __restrict__ gas_fracs) {
  R* s_lay = W.lay;
  const int t = 32 * seg + lane;   // layer
  const bool first = b_lo == 0;    // of the segment's band groups
  const int nlay = f.nlay, nlp1 = nlay + 1;
  const double* kt64 = tab64.kt;
  {
    const int c = sc.c0 + cc;                        // global column
    const Block& B = (nblocks == 1) ? b0 : blocks[find_block(blocks, nblocks, c)];
    const int i = c - B.col0;
    const size_t ld = (size_t)B.ld;
    const bool top = f.top_at_1 != 0;
    auto IN = [&](int fld, int row) -> double {
      if (!LW_OK(row >= 0 && row <= nlay && i >= 0 && i < B.npts && B.in[fld], 12, row)) return 0.0;
      return B.in[fld][i + ld * row];
    };

    // what the column's layers share: laytrop (a count, RLM:2344-2346), any cloud
    // (RLM:1101), and for the column record the amounts of every layer
    const bool write_scratch = sc.tau != nullptr;
    const bool rec = first && seg == 0 && write_scratch;
    int laytrop = 0;
    bool lcf1 = false;
    for (int k0 = 0; k0 < nlay; k0 += 32) {
      const int k = k0 + lane;
      bool lo = false, cl = false;
      if (k < nlay) {
        const int rk = top ? nlay - 1 - k : k;
        lo = fp64::lower_atm(IN(F_PLYR, rk));
        cl = IN(F_CLDCF, rk) > kEps;
        if (rec) {
          const ColAmt ca = col_amounts(IN(F_QLYR, rk), IN(F_DELPIN, rk));
          W.red[k] = ca.coldry;
          W.red[NLP + k] = fmax(0.0, ca.coldry * ca.h2ovmr);
        }
      }
      laytrop += __popc(__ballot_sync(0xffffffffu, lo));
      lcf1 |= __any_sync(0xffffffffu, cl) != 0;
    }
    __syncwarp();

    // ------------------------------ prologue + setcoef, FP64 -------------
    double tlyrfr = 0.0, tlvlfr = 0.0;
    int indlay = 1, indlev = 1, r = 0;
    bool sg_skip = false;   // learned gas optics already wrote this layer's tau/frac
    if (t < nlay) {
      const int kref = t + 1;
      r = top ? nlp1 - kref - 1 : t;                  // 0-based input row of the layer
      const int rl = top ? nlp1 - kref - 1 : t + 1;   // 0-based input row of its top level
      double pavel = IN(F_PLYR, r), delp = IN(F_DELPIN, r), tavel = IN(F_TLYR, r), tz = IN(F_TLVL, rl);
      const double amdo3 = kConAmd / kConAmo3;
      const ColAmt ca = col_amounts(IN(F_QLYR, r), delp);
      const double h2ovmr = ca.h2ovmr, coldry = ca.coldry;
      double o3vmr = fmax(0.0, IN(F_OLYR, r) * amdo3);
      double temcol = 1.0e-12 * coldry;
      const double colh2o = fmax(0.0, coldry * h2ovmr);
      // the learned gas optics already wrote tau/frac of layers inside its training
      // envelope: they need no setcoef record and no taumol here
      if (SG) {
        float xf[SG_NFEAT];
        layer_features(pavel, tavel, h2ovmr, o3vmr, IN(F_CO2, r), IN(F_CH4, r), IN(F_N2O, r), xf);
        sg_skip = in_envelope(xf, f.sg_norm);
        if (!sg_skip && first && f.sg_fallback) atomicAdd(f.sg_fallback, 1u);
      }
      indlay = min(180, max(1, (int)(tavel - 159.0)));
      tlyrfr = tavel - (int)tavel;
      indlev = min(180, max(1, (int)(tz - 159.0)));
      tlvlfr = tz - (int)tz;
      if (!sg_skip) {
        const double plog = log(pavel);
        double colv[7], wxv[4];
        colv[0] = colh2o;
        colv[1] = fmax(temcol, coldry * IN(F_CO2, r));
        colv[2] = fmax(temcol, coldry * o3vmr);
        if (f.inc_minor_gas) {
          colv[3] = fmax(temcol, coldry * IN(F_N2O, r));
          colv[4] = fmax(temcol, coldry * IN(F_CH4, r));
          colv[5] = fmax(0.0, coldry * IN(F_O2, r));
          colv[6] = fmax(0.0, coldry * IN(F_CO, r));
          wxv[0] = fmax(0.0, coldry * IN(F_CCL4, r));
          wxv[1] = fmax(0.0, coldry * IN(F_CFC11, r));
          wxv[2] = fmax(0.0, coldry * IN(F_CFC12, r));
          wxv[3] = fmax(0.0, coldry * IN(F_CFC22, r));
        } else {
          colv[3] = colv[4] = colv[5] = colv[6] = 0.0;
          wxv[0] = wxv[1] = wxv[2] = wxv[3] = 0.0;
        }
        double summol = 0.0;
        for (int m = 1; m < 7; ++m) summol = summol + colv[m];
        double colbrd = coldry - summol;

        int jp = max(1, min(58, (int)(36.0 - 5.0 * (plog + 0.04))));
        int jp1 = jp + 1;
        double fp = fmax(0.0, fmin(1.0, 5.0 * (t64(kt64, lwtab::preflog + jp - 1) - plog)));
        double tem1 = (tavel - t64(kt64, lwtab::tref + jp - 1)) / 15.0;
        double tem2 = (tavel - t64(kt64, lwtab::tref + jp1 - 1)) / 15.0;
        int jt = max(1, min(4, (int)(3.0 + tem1)));
        int jt1 = max(1, min(4, (int)(3.0 + tem2)));
        double ft = fmax(-0.5, fmin(1.5, tem1 - (double)(jt - 3)));
        double ft1 = fmax(-0.5, fmin(1.5, tem2 - (double)(jt1 - 3)));
        tem1 = 1.0 - fp;
        double fac10 = tem1 * ft, fac00 = tem1 * (1.0 - ft), fac11 = fp * ft1, fac01 = fp * (1.0 - ft1);
        double forfac = pavel * kStpfac / (tavel * (1.0 + h2ovmr));
        double selffac = h2ovmr * forfac;
        double scaleminor = pavel / tavel;
        double scaleminorn2 = (pavel / tavel) * (colbrd / (coldry + colv[0]));
        tem1 = (tavel - 180.8) / 7.2;
        int indminor = min(18, max(1, (int)tem1));
        double minorfrac = tem1 - (double)indminor;
        int indfor, indself;
        double forfrac, selffrac;
        if (plog > 4.56) {
          tem1 = (332.0 - tavel) / 36.0;
          indfor = min(2, max(1, (int)tem1));
          forfrac = tem1 - (double)indfor;
          tem1 = (tavel - 188.0) / 7.2;
          indself = min(9, max(1, (int)tem1 - 7));
          selffrac = tem1 - (double)(indself + 7);
        } else {
          tem1 = (tavel - 188.0) / 36.0;
          indfor = 3;
          forfrac = tem1 - 1.0;
          indself = 0;
          selffrac = 0.0;
        }
        selffac = colv[0] * selffac;
        forfac = colv[0] * forfac;

        R* ls = s_lay + lane;
        ls[LF_FAC00 * 32] = R(fac00); ls[LF_FAC01 * 32] = R(fac01);
        ls[LF_FAC10 * 32] = R(fac10); ls[LF_FAC11 * 32] = R(fac11);
        ls[LF_SELFFAC * 32] = R(selffac); ls[LF_SELFFRAC * 32] = R(selffrac);
        ls[LF_FORFAC * 32] = R(forfac); ls[LF_FORFRAC * 32] = R(forfrac);
        ls[LF_MINORFRAC * 32] = R(minorfrac);
        ls[LF_SCALEMINOR * 32] = R(scaleminor); ls[LF_SCALEMINORN2 * 32] = R(scaleminorn2);
        for (int m = 0; m < 7; ++m) ls[(LF_COL1 + m) * 32] = R(colv[m]);
        ls[LF_COLDRY * 32] = R(coldry); ls[LF_COLBRD * 32] = R(colbrd);
        for (int m = 0; m < 4; ++m) ls[(LF_WX1 + m) * 32] = R(wxv[m]);
        ls[LF_PAVEL * 32] = R(pavel);
        W.li[lane] = jp | (jt << 8) | (jt1 << 12) | (indself << 16) | (indfor << 20) | (indminor << 24);
      }
      double* cl = W.cld + lane;
      cl[0 * 32] = IN(F_CLDCF, r);
      if (f.ilwcliq > 0) {
        cl[1 * 32] = IN(F_LWP, r); cl[2 * 32] = IN(F_RELIQ, r); cl[3 * 32] = IN(F_IWP, r);
        cl[4 * 32] = IN(F_REICE, r); cl[5 * 32] = IN(F_RWP, r); cl[6 * 32] = IN(F_SWP, r);
        cl[7 * 32] = IN(F_RESNOW, r);
      } else {
        cl[5 * 32] = IN(F_CLDOD, r);
      }
    }
    if (rec && LW_OK(cc < sc.cap, 18, cc)) {
      // precipitable water (RLM:910-919 / 1012-1019): sequential, reference order
      double pw = 0.0;
      if (lane == 0) {
        double tem1 = 0.0, tem2 = 0.0;
        for (int k = 0; k < nlay; ++k) {
          tem1 = tem1 + W.red[k] + W.red[NLP + k];
          tem2 = tem2 + W.red[NLP + k];
        }
        const double amdw = kConAmd / kConAmw;
        double tem0 = 10.0 * tem2 / (amdw * tem1 * kConG);
        pw = tem0 * (top ? IN(F_PLVL, nlay) : IN(F_PLVL, 0));
      }
      pw = __shfl_sync(0xffffffffu, pw, 0);
      double* crec = sc.col + (size_t)cc * kColRec;
      if (lane < NBANDS) {
        // diffusivity angle (RLM:1041-1050) and surface Planck terms (RLM:2251-2262)
        const double stemp = B.in[F_SFGTMP][i];
        crec[lane] = (lane == 0 || lane == 3 || lane == 9)
                         ? 1.66
                         : fmin(1.80, fmax(1.50, c_a0[lane] + c_a1[lane] * exp(c_a2[lane] * pw)));
        crec[16 + lane] = planck_int(kt64, lane, min(180, max(1, (int)(stemp - 159.0))), stemp - (int)stemp);   // pklay(b, 0): stemp
      }
      if (lane == 0) {
        const double sfe = B.in[F_SFEMIS][i];
        crec[32] = (sfe > kEps && sfe <= 1.0) ? sfe : 1.0;
        crec[33] = lcf1 ? 1.0 : 0.0;
      }
    }

    // ------------------------------ bands --------------------------------
    // taumol splits at the count laytrop (RLM:2344-2346)
    const LayRef<R> LR{s_lay, W.li, lane, 32, t < laytrop};
    // tau, frac: [g][NLP], or four layers per g-point (lw_rt64.cuh)
    const size_t hoff = (size_t)cc * NGPT * NLP + (sc.block4 ? (size_t)(t >> 2) * NGPT * 4 + (t & 3) : (size_t)t);
    const int hstep = sc.block4 ? 4 : NLP;
    R* tcol = write_scratch ? sc.tau + hoff : nullptr;
    R* fcol = write_scratch ? sc.frac + hoff : nullptr;
    R* bcol = write_scratch ? sc.band + (size_t)cc * 3 * NBANDS * NLP : nullptr;
    // FP64 inputs without a bound of their own, within the range of lw_rt64.cuh's table index
    const auto hold = [](double od) { return sizeof(R) == 8 ? fp64::finite_od(od) : od; };
#pragma unroll 1
    for (int b = b_lo; b < b_hi; ++b) {
      if (t < nlay) {
        double tcld = 0.0;
        if (lcf1) {
          const double* cl = W.cld + lane;
          tcld = band_taucld(b, f, kt64, cl[0], cl[32], cl[2 * 32], cl[3 * 32], cl[4 * 32], cl[5 * 32], cl[6 * 32],
                             cl[7 * 32]);
        }
        if (b == 6 && !f.gas_only && LW_OK(r < nlay && i < B.npts, 13, r)) B.out[O_CLDTAU][i + ld * r] = lcf1 ? tcld : 0.0;   // band 7 (RLM:1087-1097)
        if (bcol && LW_OK(cc < sc.cap && t + 1 < NLP, 14, cc)) {   // evict-first stores: the hand-off must not push the tables out of L2
          __stcs(bcol + (0 * NBANDS + b) * NLP + t, R(planck_int(kt64, b, indlay, tlyrfr)));
          __stcs(bcol + (1 * NBANDS + b) * NLP + t + 1, R(planck_int(kt64, b, indlev, tlvlfr)));
          __stcs(bcol + (2 * NBANDS + b) * NLP + t, R(hold(tcld)));
        }
        const size_t ab = i + ld * ((size_t)r + (size_t)nlay * b);
        R tauaer = R(0);
        if (!sg_skip && LW_OK(r < nlay && i < B.npts, 15, r)) tauaer = R(hold(B.in[F_AERAOD][ab] * (1.0 - B.in[F_AERSSA][ab])));
        const int ns = ns_of(b);
        const size_t go = ((size_t)c * nlay + t) * NGPT + ns;
        if (!sg_skip) band_gas_optics<R>(b, tab.kt, LR, [&](int g0, auto tau, auto frac) {
          if (tcol && LW_OK(cc < sc.cap && ns + g0 + 1 < NGPT, 16, ns + g0)) {
            each(tau, [&](int q, R v) { __stcs(tcol + (size_t)(ns + g0 + q) * hstep, v + tauaer); });
            each(frac, [&](int q, R v) { __stcs(fcol + (size_t)(ns + g0 + q) * hstep, v); });
          }
          if (f.gas_only && LW_OK(c < sc.ntot, 17, c)) {
            each(tau, [&](int q, R v) { gas_taug[go + g0 + q] = (double)v; });
            each(frac, [&](int q, R v) { gas_fracs[go + g0 + q] = (double)v; });
          }
        });
      }
      if (t == 0 && bcol) {   // pklev(b, 0): the level below the first layer
        const double tz0 = top ? IN(F_TLVL, nlay) : IN(F_TLVL, 0);
        __stcs(bcol + (1 * NBANDS + b) * NLP, R(planck_int(kt64, b, min(180, max(1, (int)(tz0 - 159.0))), tz0 - (int)tz0)));
      }
    }
    __syncwarp();   // the warp's next unit writes the working arrays
  }
}

constexpr int kGasWarps = 4;   // per CTA
// first bands of the nsplit band groups of a segment (about equal numbers of
// g-points), by nsplit = 1, 2, 4, 8
static __device__ __constant__ int c_gas_split[4][9] = {
    {0, 16}, {0, 5, 16}, {0, 3, 5, 9, 16}, {0, 2, 3, 4, 5, 7, 9, 12, 16}};

// Units of 32 layers x a band group, strided over the grid's warps; lsplit =
// log2 of the band groups per segment.  A column's segments are dealt out from
// another one in each round of the grid, so that a warp's share of the costlier
// lower atmosphere evens out.
template <typename R, bool SG>
__global__ void __launch_bounds__(32 * kGasWarps, SG ? LW_GAS_MINB_SG : LW_GAS_MINB)
lw_gas_kernel(const Block* __restrict__ blocks, int nblocks, const Block b0, int ncols, int NLP, int lsplit, Flags f,
              Tables<R> tab, Tables<double> tab64, Scratch<R> sc, double* __restrict__ gas_taug,
              double* __restrict__ gas_fracs) {
  extern __shared__ __align__(16) char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const GasWork<R> W = GasWork<R>::at(smem_raw + warp * GasWork<R>::bytes(NLP), NLP);
  const int nseg = (f.nlay + 31) >> 5, per = nseg << lsplit;
  const long long units = (long long)ncols * per, stride = (long long)gridDim.x * kGasWarps;
  for (long long u = (long long)blockIdx.x * kGasWarps + warp; u < units; u += stride) {
    const int cc = (int)(u / per), r = (int)(u % per), part = r / nseg;
    const int seg = (int)((r + u / per * per / stride) % nseg);   // the round of the column's first unit: the same for all of them
    gas_unit<R, SG>(cc, seg, c_gas_split[lsplit][part], c_gas_split[lsplit][part + 1], lane, NLP, W, blocks, nblocks,
                    b0, f, tab, tab64, sc, gas_taug, gas_fracs);
  }
}

}  // namespace lw
