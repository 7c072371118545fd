// sw_column.cu -- the RRTMG-SW column kernels for B200 (FP64).
//
// rrtmg_sw_run (physics/Radiation/RRTMG/radsw_main.F90:493-1379, RSM below)
// runs as four launches over a chunk of daytime columns (three with grid-mean
// clouds):
//   sw_optics_kernel  one warp per 32 layers of a column, a lane per layer: the driver's
//                     layer prologue (RSM:910-1094), setcoef (RSM:2242-2389),
//                     taumol16..29 (RSM:4094-5573; every lane runs the same
//                     band's code, so the band branches never diverge),
//                     the solar source sfluxzen, the clear/cloudy column test
//                     (RSM:1101-1125) and cldprop (RSM:1566-1938);
//   lw_mcica_kernel<112> or sw_mcica_two_set_kernel  the sub-column generator
//                     (lw_mcica.cu);
//   sw_up_kernel, sw_down_kernel  one g-point per thread: spcvrtm
//                     (RSM:3228-3942) or spcvrtc with vrtqdr (RSM:3959-4051)
//                     and the flux / heating-rate outputs (RSM:1225-1373).
//
// Built with -fmad=false: every statement that feeds a table index or a
// difference of nearly equal numbers keeps the reference's evaluation order
// and rounding; the recurrences behind them use fma() where that is exact
// enough (see sw_up_kernel).
#include <cstdint>
#include <cstdio>
#include <vector>

#include <cuda_runtime.h>

#include "fp64_util.cuh"
#include "sw_kernels.h"
#include "../data/rrtmg_sw_table_layout.h"

namespace sw {

using namespace fp64;

__constant__ int c_ng[14] = {6, 12, 8, 8, 10, 10, 2, 10, 8, 6, 6, 8, 6, 12};   // radsw_param.f NG16..29
__constant__ int c_ns[14] = {0, 6, 18, 26, 34, 44, 54, 56, 66, 74, 80, 86, 94, 100};
__constant__ int c_idxsfc[14] = {1, 1, 1, 1, 1, 1, 1, 1, 0, 2, 2, 2, 2, 1};    // RSM:362
__constant__ int c_idxebc[14] = {5, 5, 4, 4, 3, 3, 2, 2, 1, 1, 1, 1, 1, 5};    // RSM:363

constexpr double kEps = 1.0e-6, kOneMinus = 1.0 - kEps, kStpfac = 296.0 / 1013.0;
constexpr double kFtiny = 1.0e-12, kFlimit = 1.0e-20;
constexpr double kConG = 9.80665, kConAvgd = 6.0221415e23, kConAmd = 28.9644, kConAmw = 18.0154,
                 kConAmo3 = 47.9982;
constexpr double kAmdw = kConAmd / kConAmw, kAmdo3 = kConAmd / kConAmo3;
constexpr int kNtbmx = 10000;

__device__ __forceinline__ int band_of(int g) {   // NGB (radsw_param.f), 0-based band
  int b = 0;
#pragma unroll
  for (int j = 1; j < 14; ++j) b += (g >= c_ns[j]) ? 1 : 0;
  return b;
}

// ---- one layer's prologue + setcoef record -------------------------------
struct Lay {
  double colamt[6], colmol, delp;
  double fac00, fac01, fac10, fac11, forfac, forfrac, selffac, selffrac;
  int jp, jt, jt1, indfor, indself;
  bool lower_plog;   // plog > 4.56
};

// rrtmg_sw_run's layer prologue (RSM:910-946 / 1001-1040) for internal
// layer k (0-based, surface first) of caller column i, then setcoef.
__device__ void layer_record(const SwArgs& a, int i, int k, const double* __restrict__ T, Lay& L) {
  const int r = a.top_at_1 ? a.nlay - 1 - k : k;
  const size_t x = (size_t)i + (size_t)a.ld * r;
  const double tem1 = 100.0 * kConG, tem2 = 1.0e-20 * 1.0e3 * kConAvgd;
  const double pavel = a.plyr[x], tavel = a.tlyr[x], q = a.qlyr[x];
  L.delp = a.delp[x];
  const double h2ovmr = fmax(0.0, q * kAmdw / (1.0 - q));
  const double o3vmr = fmax(0.0, a.olyr[x] * kAmdo3);
  const double tem0 = (1.0 - h2ovmr) * kConAmd + h2ovmr * kConAmw;
  const double coldry = tem2 * L.delp / (tem1 * tem0 * (1.0 + h2ovmr));
  const double temcol = 1.0e-12 * coldry;
  L.colamt[0] = fmax(0.0, coldry * h2ovmr);
  L.colamt[1] = fmax(temcol, coldry * a.co2[x]);
  L.colamt[2] = fmax(0.0, coldry * o3vmr);
  if (a.inc_minor) {
    L.colamt[3] = fmax(temcol, coldry * a.n2o[x]);
    L.colamt[4] = fmax(temcol, coldry * a.ch4[x]);
    L.colamt[5] = fmax(temcol, coldry * a.o2[x]);
  } else {
    L.colamt[3] = L.colamt[4] = L.colamt[5] = temcol;
  }
  L.colmol = coldry + L.colamt[0];
  // setcoef (RSM:2242-2389)
  L.forfac = pavel * kStpfac / (tavel * (1.0 + h2ovmr));
  const double plog = log(pavel);
  L.jp = max(1, min(58, (int)(36.0 - 5.0 * (plog + 0.04))));
  const int jp1 = L.jp + 1;
  const double fp = 5.0 * (__ldg(T + swtab::preflog + L.jp - 1) - plog);
  double t1 = (tavel - __ldg(T + swtab::tref + L.jp - 1)) / 15.0;
  double t2 = (tavel - __ldg(T + swtab::tref + jp1 - 1)) / 15.0;
  L.jt = max(1, min(4, (int)(3.0 + t1)));
  L.jt1 = max(1, min(4, (int)(3.0 + t2)));
  const double ft = t1 - (double)(L.jt - 3);
  const double ft1 = t2 - (double)(L.jt1 - 3);
  const double fp1 = 1.0 - fp;
  L.fac10 = fp1 * ft;
  L.fac00 = fp1 * (1.0 - ft);
  L.fac11 = fp * ft1;
  L.fac01 = fp * (1.0 - ft1);
  L.lower_plog = plog > 4.56;
  if (L.lower_plog) {
    t1 = (332.0 - tavel) / 36.0;
    L.indfor = min(2, max(1, (int)t1));
    L.forfrac = t1 - (double)L.indfor;
    t2 = (tavel - 188.0) / 7.2;
    L.indself = min(9, max(1, (int)t2 - 7));
    L.selffrac = t2 - (double)(L.indself + 7);
    L.selffac = h2ovmr * L.forfac;
  } else {
    t1 = (tavel - 188.0) / 36.0;
    L.indfor = 3;
    L.forfrac = t1 - 1.0;
    L.indself = 0;
    L.selffrac = 0.0;
    L.selffac = 0.0;
  }
}

// ---- taumol for one layer, every g-point (RSM:4094-5573) ------------------
// Two g-points at a time: every band has an even number of them, and in the
// device copy of the k-tables (rswinit's, g-point fastest; sw_api.cu) a pair is
// one 16-byte gather from the layer's row.  With the tables as the reference
// holds them (row fastest) each g-point of a row is a sector of its own.  With
// a warp per 32 layers instead of per column: 16,384 x 127, 3.85 -> 2.6 ms; 57 x
// 127, 187 -> 74 us.
struct D2 {
  double x, y;
};
__device__ __forceinline__ D2 operator+(D2 a, D2 b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ D2 operator-(D2 a, D2 b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ D2 operator*(double a, D2 b) { return {a * b.x, a * b.y}; }
__device__ __forceinline__ D2 operator+(D2 a, double b) { return {a.x + b, a.y + b}; }

// bands 16..29 as 0..13 (radsw_param.f NG16..29, RSM:359-360)
__host__ __device__ constexpr int ng_of(int b) {
  return b == 0 ? 6 : b == 1 ? 12 : b == 2 || b == 3 ? 8 : b == 4 || b == 5 ? 10 : b == 6 ? 2 : b == 7 ? 10
       : b == 8 ? 8 : b == 9 || b == 10 ? 6 : b == 11 ? 8 : b == 12 ? 6 : 12;
}
__host__ __device__ constexpr int ns_of(int b) { return b == 0 ? 0 : ns_of(b - 1) + ng_of(b - 1); }
__host__ __device__ constexpr int nspa_of(int b) { return b == 4 || b == 7 || b == 9 || b == 11 || b == 13 ? 1 : b == 10 ? 0 : 9; }
__host__ __device__ constexpr int nspb_of(int b) {
  return b == 1 || b == 5 || b == 12 ? 5 : b == 7 || b == 9 || b == 10 ? 0 : 1;
}

// k-table view with Fortran row subscripts: the pair (j, j + 1) of row ind.
// ODD: a layer whose jp lies on the other side of the split than the layer
// itself (an inverted pressure profile, or a column without a lower layer, where
// laytrop is nlay) has rows beyond its tables; it reads what the reference's
// subscripts reach in the blob as it stands.
template <int NG, int ROWS, bool ODD>
struct Tab {
  const double* p;   // in the blob if ODD, else in its copy with the g-point fastest
  __device__ __forceinline__ D2 operator()(int ind, int j) const {
    if (ODD) return {__ldg(p + (ind - 1) + ROWS * (j - 1)), __ldg(p + (ind - 1) + ROWS * j)};
    const double2 v = __ldg(reinterpret_cast<const double2*>(p + (ind - 1) * NG + (j - 1)));
    return {v.x, v.y};
  }
};
__device__ __forceinline__ D2 pair_at(const double* p, int j) {
  const double2 v = __ldg(reinterpret_cast<const double2*>(p + (j - 1)));
  return {v.x, v.y};
}

// the eight-point binary-species interpolation (fac000*k(i01) + fac100*k(i01+1)
// + fac010*k(i01+d) + fac110*k(i01+d+1) + the same at i11), left to right
template <int NG, int ROWS, bool ODD>
__device__ __forceinline__ D2 k8(const Tab<NG, ROWS, ODD>& t, const double (&f)[8], int i01, int d, int i11, int j) {
  return f[0] * t(i01, j) + f[2] * t(i01 + 1, j) + f[1] * t(i01 + d, j) + f[3] * t(i01 + d + 1, j) +
         f[4] * t(i11, j) + f[6] * t(i11 + 1, j) + f[5] * t(i11 + d, j) + f[7] * t(i11 + d + 1, j);
}
template <int NG, int ROWS, bool ODD>
__device__ __forceinline__ D2 k4(const Tab<NG, ROWS, ODD>& t, const Lay& L, int i01, int i11, int j) {
  return L.fac00 * t(i01, j) + L.fac10 * t(i01 + 1, j) + L.fac01 * t(i11, j) + L.fac11 * t(i11 + 1, j);
}
// speccomb/specmult/js/fs and the eight weights (RSM:4386-4399)
__device__ __forceinline__ double spec8(const Lay& L, int g1, int g2, double strrat, double mult, int& js, double& fs,
                                        double (&f)[8]) {
  const double speccomb = L.colamt[g1] + strrat * L.colamt[g2];
  const double specmult = mult * fmin(kOneMinus, L.colamt[g1] / speccomb);
  js = 1 + (int)specmult;
  fs = fmod(specmult, 1.0);
  const double fs1 = 1.0 - fs;
  f[0] = fs1 * L.fac00;
  f[1] = fs1 * L.fac10;
  f[2] = fs * L.fac00;
  f[3] = fs * L.fac10;
  f[4] = fs1 * L.fac01;
  f[5] = fs1 * L.fac11;
  f[6] = fs * L.fac01;
  f[7] = fs * L.fac11;
  return speccomb;
}
template <int NG, int ROWS, bool ODD>
__device__ __forceinline__ D2 selfc(const Tab<NG, ROWS, ODD>& s, const Lay& L, int j) {
  const int a = L.indself, b = a + 1;
  return L.selffac * (s(a, j) + L.selffrac * (s(b, j) - s(a, j)));
}
template <int NG, int ROWS, bool ODD>
__device__ __forceinline__ D2 forc(const Tab<NG, ROWS, ODD>& f, const Lay& L, int j) {
  const int a = L.indfor, b = a + 1;
  return L.forfac * (f(a, j) + L.forfrac * (f(b, j) - f(a, j)));
}
// first table rows of a band (RSM:4187-4202)
template <int B>
__device__ __forceinline__ int row0(const Lay& L, bool lower) {
  return lower ? ((L.jp - 1) * 5 + (L.jt - 1)) * nspa_of(B) : ((L.jp - 13) * 5 + (L.jt - 1)) * nspb_of(B);
}
template <int B>
__device__ __forceinline__ int row1(const Lay& L, bool lower) {
  return lower ? (L.jp * 5 + (L.jt1 - 1)) * nspa_of(B) : ((L.jp - 12) * 5 + (L.jt1 - 1)) * nspb_of(B);
}
// band B's values of g-points j, j + 1
template <int B>
__device__ __forceinline__ void put(double* tg, int j, D2 v) {
  tg[kTgStride * (ns_of(B) + j - 1)] = v.x;
  tg[kTgStride * (ns_of(B) + j)] = v.y;
}

// bands 16, 17, 18, 19, 21, 22: binary species in the lower atmosphere (and
// above in 17 and 21); absa at table offset A, absb AB, selfref S, forref F
template <bool ODD, int B, int G2, int A, int AB, int S, int F>
__device__ __forceinline__ void binary_band(const Lay& L, bool lower, const double* __restrict__ T,
                                            const double* __restrict__ K, double* __restrict__ tg) {
  constexpr int ng = ng_of(B);
  constexpr double o2tem = 4.35e-4 / (350.0 * 2.0), o2adj = 1.6;
  const Tab<ng, 585, ODD> absa{K + A};
  const Tab<ng, B == 1 || B == 5 ? 1175 : 235, ODD> absb{K + AB};
  const Tab<ng, 10, ODD> selfref{K + S};
  const Tab<ng, B == 1 || B == 5 ? 4 : 3, ODD> forref{K + F};
  const int id0 = row0<B>(L, lower), id1 = row1<B>(L, lower);
  int js;
  double fs, f[8];
  if (lower) {
    const double speccomb = spec8(L, 0, G2, T[swtab::strrat + B], 8.0, js, fs, f);
    const int i01 = id0 + js, i11 = id1 + js;
    const double o2cont = o2tem * L.colamt[5];
#pragma unroll 1
    for (int j = 1; j <= ng; j += 2) {
      D2 t = speccomb * k8(absa, f, i01, 9, i11, j) + L.colamt[0] * (selfc(selfref, L, j) + forc(forref, L, j));
      if (B == 6) t = t + o2cont;
      put<B>(tg, j, t);
    }
  } else if (B == 1 || B == 5) {
    const double speccomb = spec8(L, 0, 1, T[swtab::strrat + B], 4.0, js, fs, f);
    const int i01 = id0 + js, i11 = id1 + js;
#pragma unroll 1
    for (int j = 1; j <= ng; j += 2) {
      const int a0 = L.indfor, a1 = a0 + 1;
      put<B>(tg, j, speccomb * k8(absb, f, i01, 5, i11, j) +
                        L.colamt[0] * L.forfac * (forref(a0, j) + L.forfrac * (forref(a1, j) - forref(a0, j))));
    }
  } else {
    const int i01 = id0 + 1, i11 = id1 + 1;
    const double o2cont = o2tem * L.colamt[5];
#pragma unroll 1
    for (int j = 1; j <= ng; j += 2) {
      if (B == 6) put<B>(tg, j, L.colamt[5] * o2adj * k4(absb, L, i01, i11, j) + o2cont);
      else put<B>(tg, j, L.colamt[B == 3 ? 1 : 4] * k4(absb, L, i01, i11, j));
    }
  }
}

// T = the coefficient blob, K = its copy with the g-point fastest in the k-tables (ODD: the blob itself)
template <bool ODD>
__device__ void taumol_layer(const Lay& L, bool lower, const double* __restrict__ T, const double* __restrict__ K,
                             double* __restrict__ tg, double* __restrict__ t24) {
  int js;
  double fs, f[8];
  using namespace swtab;
  binary_band<ODD, 0, 4, b16_absa, b16_absb, b16_selfref, b16_forref>(L, lower, T, K, tg);
  binary_band<ODD, 1, 1, b17_absa, b17_absb, b17_selfref, b17_forref>(L, lower, T, K, tg);
  binary_band<ODD, 2, 4, b18_absa, b18_absb, b18_selfref, b18_forref>(L, lower, T, K, tg);
  binary_band<ODD, 3, 1, b19_absa, b19_absb, b19_selfref, b19_forref>(L, lower, T, K, tg);
  binary_band<ODD, 5, 1, b21_absa, b21_absb, b21_selfref, b21_forref>(L, lower, T, K, tg);
  binary_band<ODD, 6, 5, b22_absa, b22_absb, b22_selfref, b22_forref>(L, lower, T, K, tg);
  {  // band 20: H2O, CH4
    constexpr int b = 4, ng = ng_of(b);
    const Tab<ng, 65, ODD> absa{K + b20_absa};
    const Tab<ng, 235, ODD> absb{K + b20_absb};
    const Tab<ng, 10, ODD> selfref{K + b20_selfref};
    const Tab<ng, 4, ODD> forref{K + b20_forref};
    const int i01 = row0<b>(L, lower) + 1, i11 = row1<b>(L, lower) + 1;
#pragma unroll 1
    for (int j = 1; j <= ng; j += 2) {
      const D2 ch4 = L.colamt[4] * pair_at(K + b20_absch4, j);
      if (lower) put<b>(tg, j, L.colamt[0] * (k4(absa, L, i01, i11, j) + selfc(selfref, L, j) + forc(forref, L, j)) + ch4);
      else put<b>(tg, j, L.colamt[0] * (k4(absb, L, i01, i11, j) + forc(forref, L, j)) + ch4);
    }
  }
  {  // band 23: H2O below, nothing above
    constexpr int b = 7, ng = ng_of(b);
    const Tab<ng, 65, ODD> absa{K + b23_absa};
    const Tab<ng, 10, ODD> selfref{K + b23_selfref};
    const Tab<ng, 3, ODD> forref{K + b23_forref};
    const double givfac = T[b23_givfac];
    const int i01 = row0<b>(L, lower) + 1, i11 = row1<b>(L, lower) + 1;
#pragma unroll 1
    for (int j = 1; j <= ng; j += 2)
      put<b>(tg, j, lower ? L.colamt[0] * (givfac * k4(absa, L, i01, i11, j) + selfc(selfref, L, j) + forc(forref, L, j))
                          : D2{0.0, 0.0});
  }
  {  // band 24: H2O/O2 below, O2 above; O3 both; Rayleigh from the species bin
    constexpr int b = 8, ng = ng_of(b);
    const Tab<ng, 585, ODD> absa{K + b24_absa};
    const Tab<ng, 235, ODD> absb{K + b24_absb};
    const Tab<ng, 10, ODD> selfref{K + b24_selfref};
    const Tab<ng, 3, ODD> forref{K + b24_forref};
    if (lower) {
      const double speccomb = spec8(L, 0, 5, T[strrat + b], 8.0, js, fs, f);
      const int i01 = row0<b>(L, lower) + js, i11 = row1<b>(L, lower) + js;
#pragma unroll 1
      for (int j = 1; j <= ng; j += 2) {
        put<b>(tg, j, speccomb * k8(absa, f, i01, 9, i11, j) + L.colamt[2] * pair_at(K + b24_abso3a, j) +
                          L.colamt[0] * (selfc(selfref, L, j) + forc(forref, L, j)));
        const D2 ra = pair_at(K + b24_rayla + 8 * (js - 1), j), rb = pair_at(K + b24_rayla + 8 * js, j);
        const D2 r = L.colmol * (ra + fs * (rb - ra));
        t24[j - 1] = r.x;
        t24[j] = r.y;
      }
    } else {
      const int i01 = row0<b>(L, lower) + 1, i11 = row1<b>(L, lower) + 1;
#pragma unroll 1
      for (int j = 1; j <= ng; j += 2) {
        put<b>(tg, j, L.colamt[5] * k4(absb, L, i01, i11, j) + L.colamt[2] * pair_at(K + b24_abso3b, j));
        const D2 r = L.colmol * pair_at(K + b24_raylb, j);
        t24[j - 1] = r.x;
        t24[j] = r.y;
      }
    }
  }
  {  // band 25: H2O below; O3 both
    constexpr int b = 9, ng = ng_of(b);
    const Tab<ng, 65, ODD> absa{K + b25_absa};
    const int i01 = row0<b>(L, lower) + 1, i11 = row1<b>(L, lower) + 1;
#pragma unroll 1
    for (int j = 1; j <= ng; j += 2)
      put<b>(tg, j, lower ? L.colamt[0] * k4(absa, L, i01, i11, j) + L.colamt[2] * pair_at(K + b25_abso3a, j)
                          : L.colamt[2] * pair_at(K + b25_abso3b, j));
  }
#pragma unroll
  for (int j = 1; j <= ng_of(10); j += 2) put<10>(tg, j, D2{0.0, 0.0});   // band 26: Rayleigh only
  {  // band 27: O3
    constexpr int b = 11, ng = ng_of(b);
    const Tab<ng, 65, ODD> absa{K + b27_absa};
    const Tab<ng, 235, ODD> absb{K + b27_absb};
    const int i01 = row0<b>(L, lower) + 1, i11 = row1<b>(L, lower) + 1;
#pragma unroll 1
    for (int j = 1; j <= ng; j += 2) put<b>(tg, j, L.colamt[2] * (lower ? k4(absa, L, i01, i11, j) : k4(absb, L, i01, i11, j)));
  }
  {  // band 28: O3/O2 both
    constexpr int b = 12, ng = ng_of(b);
    const Tab<ng, 585, ODD> absa{K + b28_absa};
    const Tab<ng, 1175, ODD> absb{K + b28_absb};
    const double speccomb = spec8(L, 2, 5, T[strrat + b], lower ? 8.0 : 4.0, js, fs, f);
    const int i01 = row0<b>(L, lower) + js, i11 = row1<b>(L, lower) + js;
#pragma unroll 1
    for (int j = 1; j <= ng; j += 2) put<b>(tg, j, speccomb * (lower ? k8(absa, f, i01, 9, i11, j) : k8(absb, f, i01, 5, i11, j)));
  }
  {  // band 29: H2O + CO2 below, CO2 + H2O above
    constexpr int b = 13, ng = ng_of(b);
    const Tab<ng, 65, ODD> absa{K + b29_absa};
    const Tab<ng, 235, ODD> absb{K + b29_absb};
    const Tab<ng, 10, ODD> selfref{K + b29_selfref};
    const Tab<ng, 4, ODD> forref{K + b29_forref};
    const int i01 = row0<b>(L, lower) + 1, i11 = row1<b>(L, lower) + 1;
#pragma unroll 1
    for (int j = 1; j <= ng; j += 2) {
      if (lower)
        put<b>(tg, j, L.colamt[0] * (k4(absa, L, i01, i11, j) + selfc(selfref, L, j) + forc(forref, L, j)) +
                          L.colamt[1] * pair_at(K + b29_absco2, j));
      else
        put<b>(tg, j, L.colamt[1] * k4(absb, L, i01, i11, j) + L.colamt[0] * pair_at(K + b29_absh2o, j));
    }
  }
}

// a (rows, bands) table of the cloud optics with Fortran subscripts
struct Rows {
  const double* p;
  int rows;
  __device__ __forceinline__ double operator()(int ind, int j) const { return __ldg(p + (ind - 1) + rows * (j - 1)); }
};

// ---- cldprop for one layer (RSM:1687-1903) --------------------------------
__device__ void cloud_layer(const SwArgs& a, size_t x, const double* __restrict__ T, double* __restrict__ tw,
                            double* __restrict__ sw, double* __restrict__ gw) {
  double tauliq[14], ssaliq[14], asyliq[14], tauice[14], ssaice[14], asyice[14];
  const double cf = a.cf[x];
  if (!(cf > kFtiny)) {
    for (int b = 0; b < 14; ++b) { tw[b] = 0.0; sw[b] = 1.0; gw[b] = 0.0; }
    return;
  }
  if (a.iswcliq > 0) {
    const double cldran = a.rwp[x], cldsnw = a.swp[x], refsnw = a.res[x];
    const double dgesnw = 1.0315 * refsnw;
    const double tauran = cldran * T[swtab::a0r];
    const double tausnw = (cldsnw > 0.0 && refsnw > 10.0) ? cldsnw * 1.09087 * (T[swtab::a0s] + T[swtab::a1s] / dgesnw)
                                                         : 0.0;
    const double cldliq = a.lwp[x], cldice = a.iwp[x], refliq = a.rel[x];
    double refice = a.rei[x];
    for (int b = 0; b < 14; ++b) { tauliq[b] = ssaliq[b] = asyliq[b] = tauice[b] = ssaice[b] = asyice[b] = 0.0; }
    if (cldliq > 0.0 && (a.iswcliq == 1 || a.iswcliq == 2)) {
      const double factor = refliq - 1.5;
      const int index = max(1, min(57, (int)factor));
      const double fint = factor - (double)index;
      const Rows ext{T + (a.iswcliq == 1 ? swtab::extliq1 : swtab::extliq2), 58};
      const Rows ssa{T + (a.iswcliq == 1 ? swtab::ssaliq1 : swtab::ssaliq2), 58};
      const Rows asy{T + (a.iswcliq == 1 ? swtab::asyliq1 : swtab::asyliq2), 58};
      for (int b = 0; b < 14; ++b) {
        const int c = b + 1;
        const double e = fmax(0.0, ext(index, c) + fint * (ext(index + 1, c) - ext(index, c)));
        const double s = fmax(0.0, fmin(1.0, ssa(index, c) + fint * (ssa(index + 1, c) - ssa(index, c))));
        const double g = fmax(0.0, fmin(1.0, asy(index, c) + fint * (asy(index + 1, c) - asy(index, c))));
        tauliq[b] = cldliq * e;
        ssaliq[b] = tauliq[b] * s;
        asyliq[b] = ssaliq[b] * g;
      }
    }
    if (cldice > 0.0) {
      if (a.iswcice == 1) {
        refice = fmin(130.0, fmax(13.0, refice));
        for (int b = 0; b < 14; ++b) {
          const int ia = c_idxebc[b] - 1;
          const double e = fmax(0.0, T[swtab::abari + ia] + T[swtab::bbari + ia] / refice);
          const double s = fmax(0.0, fmin(1.0, 1.0 - T[swtab::cbari + ia] - T[swtab::dbari + ia] * refice));
          const double g = fmax(0.0, fmin(1.0, T[swtab::ebari + ia] + T[swtab::fbari + ia] * refice));
          tauice[b] = cldice * e;
          ssaice[b] = tauice[b] * s;
          asyice[b] = ssaice[b] * g;
        }
      } else if (a.iswcice == 2 || a.iswcice == 3) {
        int index, rows;
        double fint;
        if (a.iswcice == 2) {
          refice = fmin(131.0, fmax(5.0, refice));
          const double factor = (refice - 2.0) / 3.0;
          index = max(1, min(42, (int)factor));
          fint = factor - (double)index;
          rows = 43;
        } else {
          const double dgeice = fmax(5.0, fmin(140.0, 1.0315 * refice));
          const double factor = (dgeice - 2.0) / 3.0;
          index = max(1, min(45, (int)factor));
          fint = factor - (double)index;
          rows = 46;
        }
        const Rows ext{T + (a.iswcice == 2 ? swtab::extice2 : swtab::extice3), rows};
        const Rows ssa{T + (a.iswcice == 2 ? swtab::ssaice2 : swtab::ssaice3), rows};
        const Rows asy{T + (a.iswcice == 2 ? swtab::asyice2 : swtab::asyice3), rows};
        for (int b = 0; b < 14; ++b) {
          const int c = b + 1;
          const double e = fmax(0.0, ext(index, c) + fint * (ext(index + 1, c) - ext(index, c)));
          const double s = fmax(0.0, fmin(1.0, ssa(index, c) + fint * (ssa(index + 1, c) - ssa(index, c))));
          const double g = fmax(0.0, fmin(1.0, asy(index, c) + fint * (asy(index + 1, c) - asy(index, c))));
          tauice[b] = cldice * e;
          ssaice[b] = tauice[b] * s;
          asyice[b] = ssaice[b] * g;
        }
      }
    }
    for (int b = 0; b < 14; ++b) {
      const double ssaran = tauran * (1.0 - T[swtab::b0r + b]);
      const double ssasnw = tausnw * (1.0 - (T[swtab::b0s + b] + T[swtab::b1s + b] * dgesnw));
      const double asyran = ssaran * T[swtab::c0r + b];
      const double asysnw = ssasnw * T[swtab::c0s + b];
      tw[b] = tauliq[b] + tauice[b] + tauran + tausnw;
      sw[b] = ssaliq[b] + ssaice[b] + ssaran + ssasnw;
      gw[b] = asyliq[b] + asyice[b] + asyran + asysnw;
    }
  } else {
    const double od = a.cod[x], ss = a.cssa[x], as = a.casy[x];
    for (int b = 0; b < 14; ++b) {
      tw[b] = od;
      sw[b] = od * ss;
      gw[b] = sw[b] * as;
    }
  }
}

// ---- Rayleigh optical depth of g-point g (RSM:4094-5573) --------------------
// colmol * coefficient, except band 24, whose coefficient depends on the
// layer's species bin: the optics kernel writes those eight values per layer.
// p[stride * k] * coef is taur of layer k in either case.
struct RaySrc {
  const double* p;
  int stride;
  double coef;
};
__device__ __forceinline__ RaySrc ray_src(const SwScratch& s, size_t pl, int nlay, int g, int b,
                                          const double* __restrict__ T) {
  if (b == 8) return {s.ray24 + pl * nlay * 8 + (g - c_ns[8]), 8, 1.0};
  const int j = g - c_ns[b];
  int off = 0;
  switch (b) {
    case 0: off = swtab::b16_rayl; break;
    case 1: off = swtab::b17_rayl; break;
    case 2: off = swtab::b18_rayl; break;
    case 3: off = swtab::b19_rayl; break;
    case 4: off = swtab::b20_rayl; break;
    case 5: off = swtab::b21_rayl; break;
    case 6: off = swtab::b22_rayl; break;
    case 7: off = swtab::b23_rayl + j; break;
    case 9: off = swtab::b25_rayl + j; break;
    case 10: off = swtab::b26_rayl + j; break;
    case 11: off = swtab::b27_rayl + j; break;
    case 12: off = swtab::b28_rayl; break;
    default: off = swtab::b29_rayl; break;
  }
  return {s.colmol + pl * nlay, 1, __ldg(T + off)};
}

// the stage entry point's outputs: taug and taur as [column][layer][112]
__global__ void sw_gas_unpack_kernel(SwScratch s, int nc, int nlay, const double* __restrict__ T,
                                     double* __restrict__ taug, double* __restrict__ taur) {
  const long long n = (long long)nc * nlay * kSwNg;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    const int g = (int)(q % kSwNg), k = (int)(q / kSwNg % nlay);
    const size_t pl = (size_t)(q / kSwNg / nlay);
    const RaySrc r = ray_src(s, pl, nlay, g, band_of(g), T);
    taug[q] = s.taug[tg_offset(nlay, pl, k, g)];
    taur[q] = r.p[(size_t)r.stride * k] * r.coef;
  }
}

// ---- kernel 1: optics ------------------------------------------------------
constexpr int kOptWarps = 4;   // per CTA
// 128 registers at 4 CTAs per SM, 16,384 x 127: 2.55 ms, against 3.69, 2.83 and
// 2.52 ms at 2, 3 and 5 (which slows 1,800 x 64 from 209 to 241 us)
constexpr int kOptPerSm = 4;

// Optics of 32 layers (segment seg) of one column by one warp, a lane per
// layer: a = the argument record of the call (or of the physics block) the
// column belongs to, j1 its 1-based column there.  Each warp finds what the
// layers share (laytrop, the cloudy fraction) for itself; segment 0 also writes
// the column's values.  s_col: kSwMaxLay doubles of the warp's.
__device__ __forceinline__ void optics_body(const SwArgs& a, const SwScratch& s, int pl, int nc, int j1, int seg,
                                            int lane, double* s_col, const double* __restrict__ T,
                                            const double* __restrict__ K) {
  const int i = j1 - 1, nlay = a.nlay, k = 32 * seg + lane;
  const size_t ld = (size_t)a.ld;
  auto row = [&](int kk) { return a.top_at_1 ? nlay - 1 - kk : kk; };
  // laytrop: the last layer with ln p > 4.56, nlay if none (RSM:2305, 2353)
  int laytrop = 0;
  for (int k0 = 0; k0 < nlay; k0 += 32) {
    const int kk = k0 + lane;
    const bool hi = kk < nlay && lower_atm(a.plyr[i + ld * row(kk)]);
    const unsigned m = __ballot_sync(0xffffffffu, hi);
    if (m) laytrop = k0 + 32 - __clz(m);
  }
  if (laytrop == 0) laytrop = nlay;

  // gas optics
  if (k < nlay) {
    Lay L;
    layer_record(a, i, k, T, L);
    s.colmol[(size_t)pl * nlay + k] = L.colmol;
    const bool lower = (k + 1) <= laytrop;
    double *tg = s.taug + tg_offset(nlay, pl, k, 0), *t24 = s.ray24 + ((size_t)pl * nlay + k) * 8;
    if (lower != (L.jp < 13)) taumol_layer<true>(L, lower, T, T, tg, t24);
    else taumol_layer<false>(L, lower, T, K, tg, t24);
  }

  // solar source per band (RSM:4225-4310), one band per lane
  if (seg == 0) {
    int* s_jp = reinterpret_cast<int*>(s_col);
    for (int kk = lane; kk < nlay; kk += 32) {
      const double plog = log(a.plyr[i + ld * row(kk)]);
      s_jp[kk] = max(1, min(58, (int)(36.0 - 5.0 * (plog + 0.04))));
    }
    __syncwarp();
    if (lane < 14) {
      const int b = lane, jb = 16 + b, ng = c_ng[b], ns = c_ns[b];
      const int ibd = (int)T[swtab::ibx + b];
      double* sf = s.sflux + (size_t)pl * kSwNg + ns;
      if (jb == 16 || jb == 20 || jb == 23 || jb == 25 || jb == 26 || jb == 29) {
        for (int j = 0; j < ng; ++j) sf[j] = T[swtab::sfluxref01 + j + 16 * (ibd - 1)];
      } else if (jb == 27) {
        for (int j = 0; j < ng; ++j) sf[j] = T[swtab::scalekur] * T[swtab::sfluxref01 + j + 16 * (ibd - 1)];
      } else {
        const int lref = (int)T[swtab::layreffr + b];
        int ks;   // 1-based
        if (jb == 17 || jb == 28) {
          ks = nlay;
          for (int kk = laytrop; kk <= nlay - 1; ++kk)
            if (s_jp[kk - 1] < lref && s_jp[kk] >= lref) { ks = kk + 1; break; }
        } else {
          ks = laytrop;
          for (int kk = 1; kk <= laytrop - 1; ++kk)
            if (s_jp[kk - 1] < lref && s_jp[kk] >= lref) { ks = kk + 1; break; }
        }
        Lay L;
        layer_record(a, i, ks - 1, T, L);
        const int m1 = (int)T[swtab::ix1 + b] - 1, m2 = (int)T[swtab::ix2 + b] - 1;
        double colm1 = 0.0, colm2 = 0.0;
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          colm1 = (m == m1) ? L.colamt[m] : colm1;
          colm2 = (m == m2) ? L.colamt[m] : colm2;
        }
        const double speccomb = colm1 + T[swtab::strrat + b] * colm2;
        const double specmult = T[swtab::specwt + b] * fmin(kOneMinus, colm1 / speccomb);
        const int js = 1 + (int)specmult;
        const double fs = fmod(specmult, 1.0);
        const bool two = (jb == 17 || jb == 28);
        const double* ref = T + (two ? swtab::sfluxref02 : swtab::sfluxref03);
        const int nbin = two ? 5 : 9;
        for (int j = 0; j < ng; ++j) {
          const double r0 = ref[j + 16 * ((js - 1) + nbin * (ibd - 1))], r1 = ref[j + 16 * (js + nbin * (ibd - 1))];
          sf[j] = r0 + fs * (r1 - r0);
        }
      }
    }
    __syncwarp();
  }

  if (a.gas_only) return;
  // clear / cloudy column (RSM:1101-1125), in layer order on lane 0 from a
  // shared copy: read from memory, its 127 dependent loads were a third of the
  // kernel's time
  for (int kk = lane; kk < nlay; kk += 32) s_col[kk] = a.cf[i + ld * row(kk)];
  __syncwarp();
  double zcf1 = 0.0;
  if (lane == 0) {
    double zcf0 = 1.0, z1 = 1.0;
    for (int kk = 0; kk < nlay; ++kk) {
      const double cf = s_col[kk];
      if (a.iovr == a.iovr_rand) {
        zcf0 = zcf0 * (1.0 - cf);
      } else if (a.iovr == a.iovr_maxrand) {
        if (cf > kFtiny) z1 = fmin(z1, 1.0 - cf);
        else if (z1 < 1.0) { zcf0 = zcf0 * z1; z1 = 1.0; }
      } else if (a.iovr >= 2) {
        zcf0 = fmin(zcf0, 1.0 - cf);
      }
    }
    if (a.iovr == a.iovr_maxrand) zcf0 = zcf0 * z1;
    if (zcf0 <= kFtiny) zcf0 = 0.0;
    if (zcf0 > kOneMinus) zcf0 = 1.0;
    zcf1 = 1.0 - zcf0;
    if (seg == 0) {
      s.zcf1[pl] = zcf1;
      s.zcf0[pl] = zcf0;
      // McICA seed: ipsdsw0 + i or icseed(i) (RSM:875-883); grid-mean clouds draw none
      s.seed[pl] = (a.isubcsw == 2) ? a.icseed[i] : 1 + a.seed0 + j1;
    }
  }
  zcf1 = __shfl_sync(0xffffffffu, zcf1, 0);
  if (k < nlay) {
    const size_t x = i + ld * row(k);
    const double cf = s_col[k];
    s.cldf[(size_t)pl + (size_t)nc * k] = (cf < kFtiny) ? 0.0 : cf;   // mcica_subcol input (RSM:1904-1908)
    if (a.isubcsw <= 0) {   // grid-mean clouds: cldfrc = cfrac / cf1 (RSM:1930-1934)
      s.aux[(size_t)pl + (size_t)nc * k] = (zcf1 > 0.0) ? cf / zcf1 : 0.0;
    } else if (a.iovr == 3) {   // fac_lcf between layers k-1 and k (RSM:2106-2108), dz in internal order
      double f = 0.0;
      if (k > 0) f = exp(-0.5 * (a.dz[x] + a.dz[i + ld * row(k - 1)]) / a.delg[i]);
      s.aux[(size_t)pl + (size_t)nc * k] = f;
    } else if (a.iovr == 4 || a.iovr == 5) {   // alpha, in the caller's row order (RSM:921, 1012)
      s.aux[(size_t)pl + (size_t)nc * k] = a.alpha[i + ld * k];
    }
    if (zcf1 > 0.0) {
      double* tw = s.taucw + ((size_t)pl * nlay + k) * 14;
      double* sw = s.ssacw + ((size_t)pl * nlay + k) * 14;
      double* gw = s.asycw + ((size_t)pl * nlay + k) * 14;
      cloud_layer(a, x, T, tw, sw, gw);
      a.cldtau[x] = tw[9];   // band 25 (RSM:1144-1152)
    }
  }
  __syncwarp();
}

__global__ void __launch_bounds__(32 * kOptWarps, kOptPerSm)
sw_optics_kernel(SwArgs a, SwScratch s, int p0, int nc, const double* __restrict__ T, const double* __restrict__ K) {
  __shared__ double s_col[kOptWarps][kSwMaxLay];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nseg = (a.nlay + 31) >> 5;
  const int u = blockIdx.x * kOptWarps + w, pl = u / nseg, seg = u - pl * nseg;
  if (pl >= nc) return;   // whole warps only: no block barrier below
  const int j1 = a.idxday[p0 + pl];
  if (j1 < 1 || j1 > a.npts) {   // idxday outside 1..npts: skip the column, report
    if (lane == 0) atomicOr(s.bad, 1);
    return;
  }
  optics_body(a, s, pl, nc, j1, seg, lane, s_col[w], T, K);
}

// many physics blocks in one launch: daytime point p is column pts[p].y of block pts[p].x
__global__ void __launch_bounds__(32 * kOptWarps, kOptPerSm)
sw_optics_blocks_kernel(const SwArgs* __restrict__ tab, const int2* __restrict__ pts, SwScratch s, int p0, int nc,
                        const double* __restrict__ T, const double* __restrict__ K) {
  __shared__ double s_col[kOptWarps][kSwMaxLay];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nseg = (tab[0].nlay + 31) >> 5;
  const int u = blockIdx.x * kOptWarps + w, pl = u / nseg, seg = u - pl * nseg;
  if (pl >= nc) return;
  const int2 q = pts[p0 + pl];
  optics_body(tab[q.x], s, pl, nc, q.y, seg, lane, s_col[w], T, K);
}

// ---- kernel 3: transfer ------------------------------------------------------
struct LayOpt {
  double rb, rd, tb, td, e3, e4;
};

// fmax / fmin with a constant: NaN gives the constant, as fmax and fmin do
__device__ __forceinline__ double at_least(double c, double x) { return x > c ? x : c; }
__device__ __forceinline__ double at_most(double c, double x) { return x < c ? x : c; }
__device__ __forceinline__ double clamp01(double x) { return at_least(0.0, at_most(1.0, x)); }

// exp_tbl in global or in shared memory
struct TblGlobal {
  const double* p;
  __device__ __forceinline__ double operator()(int i) const { return __ldg(p + i); }
};
struct TblShared {
  const double* p;   // shared memory
  __device__ __forceinline__ double operator()(int i) const { return p[i]; }
};

__device__ __forceinline__ double exp_small(double z) { return 1.0 - z + 0.5 * z * z; }
template <typename Tbl>
__device__ __forceinline__ double exp_of(const Tbl& ET, double z) {   // od_lo = 0.06
  return (z <= 0.06) ? exp_small(z) : ET(pade_index(z));
}

// The two-stream layer reflectance / transmittance of spcvrtm (RSM:3447-3600).
// Thin layers difference nearly equal numbers here, so everything up to the
// two final quotients keeps the reference's operations and their order.
template <typename Tbl>
__device__ __forceinline__ void two_stream(double ztau0, double zssa0, double zasy0, double cosz, double sntz,
                                           int iswmode, const Tbl& ET, LayOpt& o) {
  const double zcrit = 0.9999995, eps1 = 1.0e-8;
  const double zssaw = at_most(kOneMinus, div_markstein(zssa0, ztau0));
  const double zasyw = div_markstein(zasy0, at_least(kFtiny, zssa0));
  double za1 = zasyw * zasyw;
  double za2 = zssaw * za1;
  const double ztau1 = (1.0 - za2) * ztau0;
  const double zssa1 = div_markstein(zssaw - za2, 1.0 - za2);
  const double zasy1 = div_markstein(zasyw, 1.0 + zasyw);
  const double zasy3 = 0.75 * zasy1;
  double zgam1, zgam2, zgam3;
  if (iswmode == 1) {
    zgam1 = 1.75 - zssa1 * (1.0 + zasy3);
    zgam2 = -0.25 + zssa1 * (1.0 - zasy3);
    zgam3 = 0.5 - zasy3 * cosz;
  } else if (iswmode == 2) {
    zgam1 = 2.0 - zssa1 * (1.25 + zasy3);
    zgam2 = 0.75 * zssa1 * (1.0 - zasy1);
    zgam3 = 0.5 - zasy3 * cosz;
  } else {
    const double zsr3 = sqrt(3.0);
    zgam1 = zsr3 * (2.0 - zssa1 * (1.0 + zasy1)) * 0.5;
    zgam2 = zsr3 * zssa1 * (1.0 - zasy1) * 0.5;
    zgam3 = (1.0 - zsr3 * zasy1 * cosz) * 0.5;
  }
  const double zgam4 = 1.0 - zgam3;
  // direct-beam transmittance of the scaled optical depth; the layer optics
  // use it capped at 500, the beam (e3) does not
  const double zbeam = ztau1 * sntz;
  const double zexm2 = exp_of(ET, at_most(500.0, zbeam));
  o.e3 = (zbeam <= 500.0) ? zexm2 : exp_of(ET, zbeam);
  o.e4 = exp_of(ET, ztau0 * sntz);
  if (zssaw >= zcrit) {
    za1 = zgam1 * cosz - zgam3;
    za2 = zgam1 * ztau1;
    o.rb = clamp01((za2 - za1 * (1.0 - zexm2)) / (1.0 + za2));
    o.tb = clamp01(1.0 - o.rb);
    o.rd = clamp01(za2 / (1.0 + za2));
    o.td = clamp01(1.0 - o.rd);
  } else {
    za1 = zgam1 * zgam4 + zgam2 * zgam3;
    za2 = zgam1 * zgam3 + zgam2 * zgam4;
    double zrk = (zgam1 - zgam2) * (zgam1 + zgam2);
    zrk = (zrk > eps1) ? sqrt_markstein(zrk) : 0.0;
    const double zrk2 = zrk + zrk;
    const double zrp = zrk * cosz;
    const double zrp1 = 1.0 + zrp, zrm1 = 1.0 - zrp;
    const double zrpp1 = 1.0 - zrp * zrp;
    const double zrpp = copysign(at_least(kFlimit, fabs(zrpp1)), zrpp1);
    const double zrkg1 = zrk + zgam1, zrkg3 = zrk * zgam3, zrkg4 = zrk * zgam4;
    const double zr1 = zrm1 * (za2 + zrkg3);
    const double zr2 = zrp1 * (za2 - zrkg3);
    const double zr3 = zrk2 * (zgam3 - za2 * cosz);
    const double zr4 = zrpp * zrkg1;
    const double zr5 = zrpp * (zrk - zgam1);
    const double zt1 = zrp1 * (za1 + zrkg4);
    const double zt2 = zrm1 * (za1 - zrkg4);
    const double zt3 = zrk2 * (zgam4 + za1 * cosz);
    const double zexm1 = exp_of(ET, at_most(500.0, zrk * ztau1));
    const double zexp1 = div_markstein(1.0, zexm1);
    const double zexp2 = div_markstein(1.0, zexm2);
    const double ze1r45 = zr4 * zexp1 + zr5 * zexm1;
    // zden1 of the beam (zssa1 / ze1r45) and of the diffuse light
    // (zr4 / (ze1r45 zrkg1), its denominator kept eps1 from 0)
    const double zb = ze1r45 * zrkg1;
    double dbeam, ddiff;
    if (fabs(zb) > eps1 && fabs(ze1r45) > eps1) {
      const double q = recip_newton(zb);
      dbeam = zssa1 * (zrkg1 * q);
      ddiff = zr4 * q;
    } else {
      dbeam = zssa1 / ze1r45;
      ddiff = (ze1r45 >= 0.0) ? zr4 / fmax(eps1, zb) : zr4 / fmin(-eps1, zb);
    }
    if (fabs(ze1r45) <= eps1) {
      o.rb = eps1;
      o.tb = zexm2;
    } else {
      o.rb = clamp01((zr1 * zexp1 - zr2 * zexm1 - zr3 * zexm2) * dbeam);
      o.tb = clamp01(zexm2 * (1.0 - (zt1 * zexp1 - zt2 * zexm1 - zt3 * zexp2) * dbeam));
    }
    o.rd = clamp01(zgam2 * (zexp1 - zexm1) * ddiff);
    o.td = clamp01(zrk2 * ddiff);
  }
}

// spcvrtc's mixing of a cloudy layer's optics with its clear optics o
// (RSM:3039-3042, 3057, 3072): zc0 * clear + zc1 * cloudy
__device__ __forceinline__ void mix_grid(double zc1, const LayOpt& o, LayOpt& w) {
  const double zc0 = 1.0 - zc1;
  w.rb = zc0 * o.rb + zc1 * w.rb;
  w.rd = zc0 * o.rd + zc1 * w.rd;
  w.tb = zc0 * o.tb + zc1 * w.tb;
  w.td = zc0 * o.td + zc1 * w.td;
  w.e3 = zc0 * o.e3 + zc1 * w.e3;
  w.e4 = zc0 * o.e4 + zc1 * w.e4;
}

// Transfer, thread = g-point (112 per column; columns share warps, so no lane
// idles), in two kernels.
//
// sw_up_kernel, bottom to top: each layer's two-stream optics are evaluated
// once for the clear sky (and before that once more where the layer is cloudy),
// and vrtqdr's upward recurrence (RSM:4011-4020) gives the reflectances
// (zrupb, zrupd) of everything below a level.  With those known, the way down
// needs no second adding recurrence: for the beam D and the diffuse flux F
// entering a layer,
//   D' = e3 D,  F' = (td F + ((tb - e3) + e3 zrupb rd) D) / (1 - rd zrupd),
// and the level's fluxes are D + F down and zrupb D + zrupd F up, which is
// what vrtqdr's zrdnd / ztdn form (RSM:4026-4046) gives, with one quotient per
// layer and sweep in place of four.  sw_down_kernel does that and the outputs.
//
// Two kernels, because they want different things: the way up is a chain of
// FP64 operations per layer (128 registers, sixteen warps per SM, 63 % of the
// issue slots), the way down streams the stored layers (80 registers, 6.4 TB/s).
// As phases of one kernel, with a slot of the store per resident column, the
// same loops took 13.0 ms at 16,384 x 127; as two, with whole columns per CTA,
// they took 9.1 ms (a column per warp, both adding recurrences and four
// 10-shuffle sums per level took 21.3 ms).  Down at 4, 5, 6 and 7 CTAs per SM: 9.4, 9.1, 9.1 and 9.8 ms.
constexpr int kRtAhead = 2;   // layers whose stored records are in flight on the way down (even)
constexpr int kRtLay = kRtVals * kSwNg;   // store doubles of a layer

// a thread's view of its column
struct RtCol {
  const double *aod, *ssa, *asy;    // layer 0 of the g-point's band, xstep per layer
  const double *tg;                 // taug of layers 0..3
  RaySrc ray;
  ptrdiff_t xstep;
  const double *tcw, *scw, *gcw;    // cloud optics of the band, 14 per layer
  const uint32_t* bits;             // McICA flags
  const double* cfr;                // normalised cloud fraction, cfs per layer (grid-mean)
  size_t cfs;
  double* st;                       // the g-point's layer store
  double cosz, sntz;
  int nlay, nw, iswmode;
  bool cloudy;
};

// layer k is cloudy for this g-point: its McICA flag, or cldfrc > ftiny
// (RSM:2885); word = the flags of layers 32 (k / 32) ..
template <bool GRID>
__device__ __forceinline__ uint32_t flags_of(const RtCol& c, int w) {
  return (!GRID && c.cloudy && w >= 0 && w < c.nw) ? __ldg(c.bits + w) : 0u;
}
template <bool GRID>
__device__ __forceinline__ bool cloud_at(const RtCol& c, int k, uint32_t word) {
  return GRID ? (c.cloudy && c.cfr[(size_t)k * c.cfs] > kFtiny) : ((word >> (k & 31)) & 1u);
}

// all-sky optics of the cloudy layers, into store values 8..11, and what the way
// up alone needs (rb, e4) where it then leaves zrupb, zrupd (6, 7)
template <bool GRID, typename Tbl>
__device__ __forceinline__ void rt_cloudy(const RtCol& c, const Tbl& ET) {
#pragma unroll 1
  for (int w = 0; w < c.nw; ++w) {
    uint32_t m = flags_of<GRID>(c, w);
    if (GRID)
      for (int k = 32 * w; k < min(32 * w + 32, c.nlay); ++k) m |= (cloud_at<true>(c, k, 0) ? 1u : 0u) << (k & 31);
    while (m) {   // each lane its own layers: a warp's rounds are the most cloudy layers of one lane
      const int k = 32 * w + __ffs(m) - 1;
      m &= m - 1;
      const ptrdiff_t xo = c.xstep * k;
      const double tae = finite_od(__ldg(c.aod + xo)), sae = __ldg(c.ssa + xo), gae = __ldg(c.asy + xo);
      const double tr = c.ray.p[c.ray.stride * k] * c.ray.coef, tg = c.tg[(size_t)(k >> 2) * kSwNg * kTgStride + (k & 3)];
      const double ztau0 = fmax(kFtiny, tr + tg + tae);
      const double zssa0 = tr + tae * sae;
      const double zasy0 = gae * sae * tae;
      const size_t x = (size_t)k * 14;
      LayOpt v;
      const double tc = c.tcw[x], down = huge_od(tc) ? 0x1p-64 : 1.0;   // finite_od, for all three
      two_stream(ztau0 + tc * down, zssa0 + c.scw[x] * down, zasy0 + c.gcw[x] * down, c.cosz, c.sntz, c.iswmode, ET, v);
      if (GRID) {
        LayOpt o;
        two_stream(ztau0, zssa0, zasy0, c.cosz, c.sntz, c.iswmode, ET, o);
        mix_grid(c.cfr[(size_t)k * c.cfs], o, v);
      }
      double* q = c.st + (size_t)k * kRtLay;
      __stcg(q + 8 * kSwNg, v.td);
      __stcg(q + 9 * kSwNg, v.tb - v.e3);
      __stcg(q + 10 * kSwNg, v.e3);
      __stcg(q + 11 * kSwNg, v.rd);
      __stcg(q + 6 * kSwNg, v.rb);
      __stcg(q + 7 * kSwNg, v.e4);
    }
  }
}

// bottom to top from the surface's (ub, ud): store values td, tb - e3, e3, rd
// of each layer and zrupb, zrupd (clear, all-sky) below it; above the top
// layer the unscaled beam transmittances of the column and zrupb, zrupd
template <bool GRID, typename Tbl>
__device__ __forceinline__ void rt_up(const RtCol& c, const Tbl& ET, double ub, double ud) {
  double ubw = ub, udw = ud, beam0 = 1.0, beam0w = 1.0;
  const double *aod = c.aod, *ssa = c.ssa, *asy = c.asy, *ray = c.ray.p, *tgp = c.tg;
  double* st = c.st;
  struct In { double tr, tae, sae, gae; } nx;
  auto fetch = [&](In& v) {
    v.tr = *ray;
    v.tae = __ldg(aod);
    v.sae = __ldg(ssa);
    v.gae = __ldg(asy);
    ray += c.ray.stride;
    aod += c.xstep;
    ssa += c.xstep;
    asy += c.xstep;
  };
  fetch(nx);
  double2 n01 = ld_once2(tgp), n23 = ld_once2(tgp + 2);
  uint32_t word = 0, nword = flags_of<GRID>(c, 0);
#pragma unroll 1
  for (int k0 = 0; k0 < c.nlay; k0 += 4) {
    if ((k0 & 31) == 0) {
      word = nword;
      nword = flags_of<GRID>(c, (k0 >> 5) + 1);
    }
    const double2 c01 = n01, c23 = n23;
    if (k0 + 4 < c.nlay) {
      tgp += kSwNg * kTgStride;
      n01 = ld_once2(tgp);
      n23 = ld_once2(tgp + 2);
    }
#pragma unroll 1
    for (int kk = 0; kk < 4; ++kk) {
      const int k = k0 + kk;
      if (k >= c.nlay) break;
      const In cur = nx;
      if (k + 1 < c.nlay) fetch(nx);   // issued ahead of this layer's arithmetic
      const double tg = (kk & 2) ? ((kk & 1) ? c23.y : c23.x) : ((kk & 1) ? c01.y : c01.x);
      const double tr = cur.tr * c.ray.coef;
      const double tae = finite_od(cur.tae);
      LayOpt o;
      two_stream(fmax(kFtiny, tr + tg + tae), tr + tae * cur.sae, cur.gae * cur.sae * tae, c.cosz, c.sntz, c.iswmode,
                 ET, o);
      double tbd = o.tb - o.e3;
      __stcg(st, o.td);
      __stcg(st + kSwNg, tbd);
      __stcg(st + 2 * kSwNg, o.e3);
      __stcg(st + 3 * kSwNg, o.rd);
      __stcg(st + 4 * kSwNg, ub);
      __stcg(st + 5 * kSwNg, ud);
      beam0 *= o.e4;
      const double q = recip_newton(fma(-ud, o.rd, 1.0));
      ub = fma(o.td * fma(tbd, ud, o.e3 * ub), q, o.rb);
      ud = fma(o.td * o.td * ud, q, o.rd);
      if (c.cloudy) {
        if (cloud_at<GRID>(c, k, word)) {
          o.rb = __ldcg(st + 6 * kSwNg);
          o.e4 = __ldcg(st + 7 * kSwNg);
          o.td = __ldcg(st + 8 * kSwNg);
          tbd = __ldcg(st + 9 * kSwNg);
          o.e3 = __ldcg(st + 10 * kSwNg);
          o.rd = __ldcg(st + 11 * kSwNg);
        }
        __stcg(st + 6 * kSwNg, ubw);
        __stcg(st + 7 * kSwNg, udw);
        beam0w *= o.e4;
        const double qw = recip_newton(fma(-udw, o.rd, 1.0));
        ubw = fma(o.td * fma(tbd, udw, o.e3 * ubw), qw, o.rb);
        udw = fma(o.td * o.td * udw, qw, o.rd);
      }
      st += kRtLay;
    }
  }
  __stcg(st, beam0);
  __stcg(st + kSwNg, beam0w);
  __stcg(st + 4 * kSwNg, ub);
  __stcg(st + 5 * kSwNg, ud);
  __stcg(st + 6 * kSwNg, ubw);
  __stcg(st + 7 * kSwNg, udw);
}

// where the way down puts its sums: a group's [4][nlp1] up, down clear, up,
// down all-sky; with hswb also [kRtBandSlots][2][nlp1] total-sky band fluxes
struct RtSums {
  double *part, *accb;
  double cf1, cf0;
  int nlp1, grp, b, blo, nbg;   // the g-point's band, the group's first band and their number - 1 (at most 2)
};

// top to bottom from (ub, ud) at the top level: fluxes of every level, summed
// over the group's g-points two levels at a time
template <bool GRID, bool BANDS>
__device__ __forceinline__ void rt_down(const RtCol& c, double zsolar, const RtSums& S, double (&end)[4]) {
  const int half = threadIdx.x & 15;
  const unsigned hmask = 0xffffu << (threadIdx.x & 16);
  const int idx8 = sum_index<8, 16>(half), idx4 = sum_index<4, 16>(half);
  const double* st = c.st + (size_t)c.nlay * kRtLay;   // the layer at hand
  double ub = __ldcg(st + 4 * kSwNg), ud = __ldcg(st + 5 * kSwNg), ubw = __ldcg(st + 6 * kSwNg),
         udw = __ldcg(st + 7 * kSwNg), D = zsolar, F = 0.0, Dw = zsolar, Fw = 0.0;
  st -= kRtLay;
  double v[8];
  auto level = [&](int slot) {   // fluxes of the level reached into v[4 * slot ..]
    v[4 * slot + 0] = fma(F, ud, D * ub);
    v[4 * slot + 1] = D + F;
    v[4 * slot + 2] = c.cloudy ? fma(Fw, udw, Dw * ubw) : 0.0;
    v[4 * slot + 3] = c.cloudy ? Dw + Fw : 0.0;
  };
  auto flush = [&](int m, int nlev) {   // sums of levels m (slot 0) and m - 1 (slot 1)
    if (BANDS) {   // total-sky band fluxes (spcvrtc: cf1 all-sky + cf0 clear, RSM:3160-3161)
#pragma unroll 1
      for (int q = 0; q < 3; ++q) {
        double u[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const double c0 = v[4 * (e >> 1) + (e & 1)], c1 = v[4 * (e >> 1) + 2 + (e & 1)];
          const double t = c.cloudy ? (GRID ? S.cf1 * c1 + S.cf0 * c0 : c1) : c0;
          u[e] = (S.b == S.blo + q) ? t : 0.0;
        }
        const double r = lane_sums<4, 16>(u, half, hmask);
        const int lev = idx4 >> 1;
        if (q <= S.nbg && idx4 >= 0 && lev < nlev)
          S.accb[((size_t)2 * (S.blo + q + S.grp) + (idx4 & 1)) * S.nlp1 + (m - lev)] = r;
      }
    }
    const double r = lane_sums<8, 16>(v, half, hmask);
    const int lev = idx8 >> 2;
    if (idx8 >= 0 && lev < nlev) S.part[(size_t)(idx8 & 3) * S.nlp1 + (m - lev)] = r;
  };
  struct Rec { double td, tbd, e3, rd, ub, ud, ubw, udw; };
  auto load = [&](int below, Rec& r) {   // the record `below` layers under it
    const double* p = st - below * kRtLay;
    r.td = __ldcg(p);
    r.tbd = __ldcg(p + kSwNg);
    r.e3 = __ldcg(p + 2 * kSwNg);
    r.rd = __ldcg(p + 3 * kSwNg);
    r.ub = __ldcg(p + 4 * kSwNg);
    r.ud = __ldcg(p + 5 * kSwNg);
    if (c.cloudy) {
      r.ubw = __ldcg(p + 6 * kSwNg);
      r.udw = __ldcg(p + 7 * kSwNg);
    }
  };
  uint32_t word = flags_of<GRID>(c, (c.nlay - 1) >> 5), nword = flags_of<GRID>(c, ((c.nlay - 1) >> 5) - 1);
  auto step = [&](int m, const Rec& r) {   // through layer m
    if ((m & 31) == 31 && m < c.nlay - 1) {
      word = nword;
      nword = flags_of<GRID>(c, (m >> 5) - 1);
    }
    ub = r.ub;
    ud = r.ud;
    const double q = recip_newton(fma(-r.rd, ud, 1.0));
    F = fma(r.td, F, fma(r.e3 * ub, r.rd, r.tbd) * D) * q;
    D *= r.e3;
    if (c.cloudy) {
      ubw = r.ubw;
      udw = r.udw;
      double td = r.td, tbd = r.tbd, e3 = r.e3, rd = r.rd;
      if (cloud_at<GRID>(c, m, word)) {
        td = __ldcg(st + 8 * kSwNg);
        tbd = __ldcg(st + 9 * kSwNg);
        e3 = __ldcg(st + 10 * kSwNg);
        rd = __ldcg(st + 11 * kSwNg);
      }
      const double qw = recip_newton(fma(-rd, udw, 1.0));
      Fw = fma(td, Fw, fma(e3 * ubw, rd, tbd) * Dw) * qw;
      Dw *= e3;
    }
  };
  level(0);
  Rec r[kRtAhead];   // the next layers' records
#pragma unroll
  for (int q = 0; q < kRtAhead; ++q)
    if (c.nlay > q) load(q, r[q]);
#pragma unroll 1
  for (int m0 = c.nlay - 1; m0 >= 0; m0 -= kRtAhead) {
#pragma unroll
    for (int q = 0; q < kRtAhead; ++q) {
      const int m = m0 - q;
      if (m >= 0) {
        step(m, r[q]);
        if (m >= kRtAhead) load(kRtAhead, r[q]);
        st -= kRtLay;
        level((q & 1) ? 0 : 1);
        if ((q & 1) == 0) flush(m + 1, 2);
      }
    }
  }
  if ((c.nlay & 1) == 0) {   // an odd number of levels: the last one is alone in slot 0
    v[4] = v[5] = v[6] = v[7] = 0.0;
    flush(0, 1);
  }
  end[0] = D;
  end[1] = F;
  end[2] = Dw;
  end[3] = Fw;
}

// thread g's view of column j1 of record a, column pl of the chunk
__device__ __forceinline__ RtCol rt_col(const SwArgs& a, const SwScratch& s, int pl, int nc, int j1, int g, int b,
                                        const double* __restrict__ T) {
  const int nlay = a.nlay, top = a.top_at_1;
  const size_t i = (size_t)(j1 - 1), ld = (size_t)a.ld;
  RtCol c;
  const size_t xb = i + ld * ((size_t)nlay * b + (top ? nlay - 1 : 0));
  c.aod = a.aod + xb;
  c.ssa = a.ssa + xb;
  c.asy = a.asy + xb;
  c.tg = s.taug + tg_offset(nlay, pl, 0, g);
  c.ray = ray_src(s, pl, nlay, g, b, T);
  c.xstep = top ? -(ptrdiff_t)ld : (ptrdiff_t)ld;
  const size_t cx = (size_t)pl * nlay * 14 + b;
  c.tcw = s.taucw + cx;
  c.scw = s.ssacw + cx;
  c.gcw = s.asycw + cx;
  c.bits = s.bits + ((size_t)pl * kSwNg + g) * s.nw;
  c.cfr = s.aux + pl;
  c.cfs = (size_t)nc;
  c.st = s.rt_store + (size_t)pl * rt_col_store(nlay) + g;
  c.cosz = a.cosz[i];
  c.sntz = 1.0 / c.cosz;
  c.nlay = nlay;
  c.nw = s.nw;
  c.iswmode = a.iswmode;
  c.cloudy = s.zcf1[pl] > kEps;
  return c;
}

template <bool GRID, typename Tbl>
__device__ __forceinline__ void up_body(const SwArgs& a, const SwScratch& s, int pl, int nc, int j1, int g,
                                        const double* __restrict__ T, const Tbl& ET) {
  const int b = band_of(g), ibd = c_idxsfc[b];
  const size_t i = (size_t)(j1 - 1);
  const RtCol c = rt_col(a, s, pl, nc, j1, g, b, T);
  if (c.cloudy) rt_cloudy<GRID>(c, ET);
  rt_up<GRID>(c, ET, ibd ? (ibd == 1 ? a.alb_nir_dir[i] : a.alb_uvis_dir[i]) : 0.5 * (a.alb_nir_dir[i] + a.alb_uvis_dir[i]),
              ibd ? (ibd == 1 ? a.alb_nir_dif[i] : a.alb_uvis_dif[i]) : 0.5 * (a.alb_nir_dif[i] + a.alb_uvis_dif[i]));
}

template <bool GRID, bool BANDS>
__device__ __forceinline__ void down_body(const SwArgs& a, const SwScratch& s, int pl, int nc, int j1, int g,
                                          double* __restrict__ acc, const double* __restrict__ T) {
  const int nlay = a.nlay, nlp1 = nlay + 1, grp = g >> 4, top = a.top_at_1;
  double* accb = acc + (size_t)4 * kRtGroups * nlp1;
  double* sfc = accb + (BANDS ? (size_t)2 * kRtBandSlots * nlp1 : 0);   // [kRtGroups][2][5]
  const size_t i = (size_t)(j1 - 1), ld = (size_t)a.ld;
  const int b = band_of(g), ibd = c_idxsfc[b];
  const double cf1 = s.zcf1[pl], cf0 = s.zcf0[pl];
  const bool cloudy = cf1 > kEps;
  const double zsolar = a.s0fac * a.cosz[i] * s.sflux[(size_t)pl * kSwNg + g];
  double end[4];   // beam and diffuse flux at the surface, clear and all-sky
  {
    const RtCol c = rt_col(a, s, pl, nc, j1, g, b, T);
    RtSums S;
    S.part = acc + (size_t)grp * 4 * nlp1;
    S.accb = accb;
    S.cf1 = cf1;
    S.cf0 = cf0;
    S.nlp1 = nlp1;
    S.grp = grp;
    S.b = b;
    S.blo = band_of(g & ~15);
    S.nbg = band_of(g | 15) - S.blo;
    rt_down<GRID, BANDS>(c, zsolar, S, end);
  }
  const double* tops = s.rt_store + (size_t)pl * rt_col_store(nlay) + (size_t)nlay * kRtLay + g;
  const double beam[2] = {__ldcg(tops), __ldcg(tops + kSwNg)};

  // surface direct / diffuse partition (RSM:3641-3655) and UV-B (RSM:3907)
  {
    const int half = threadIdx.x & 15, idx8 = sum_index<8, 16>(half);
    const unsigned hmask = 0xffffu << (threadIdx.x & 16);
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      const double zb1 = zsolar * beam[pass], f0 = end[2 * pass] + end[2 * pass + 1], zb2 = f0 - zb1;
      double w[8] = {(ibd == 1) ? zb1 : (ibd == 0 ? 0.5 * zb1 : 0.0), (ibd == 2) ? zb1 : (ibd == 0 ? 0.5 * zb1 : 0.0),
                     (ibd == 1) ? zb2 : (ibd == 0 ? 0.5 * zb2 : 0.0), (ibd == 2) ? zb2 : (ibd == 0 ? 0.5 * zb2 : 0.0),
                     (b == 27 - 16) ? f0 : 0.0, 0.0, 0.0, 0.0};
      const double r = lane_sums<8, 16>(w, half, hmask);
      if (idx8 >= 0 && idx8 < 5) sfc[(grp * 2 + pass) * 5 + idx8] = r;
    }
  }
  __syncthreads();

  // ---- sums over the column's groups, in a fixed order ----
  for (int q = g; q < 4 * nlp1; q += kSwNg) {
    double t = 0.0;
#pragma unroll
    for (int p = 0; p < kRtGroups; ++p) t += acc[(size_t)p * 4 * nlp1 + q];
    acc[q] = t;
  }
  __syncthreads();
  double *up0 = acc, *dn0 = acc + nlp1, *upc = acc + 2 * nlp1, *dnc = acc + 3 * nlp1;
  if (cloudy && GRID) {   // spcvrtc's total-sky fluxes (RSM:3158-3178)
    for (int m = g; m < nlp1; m += kSwNg) {
      upc[m] = cf1 * upc[m] + cf0 * up0[m];
      dnc[m] = cf1 * dnc[m] + cf0 * dn0[m];
    }
  }
  if (GRID) __syncthreads();

  // outputs (RSM:1225-1373)
  const double* fu_t = cloudy ? upc : up0;
  const double* fd_t = cloudy ? dnc : dn0;
  auto row = [&](int m) { return top ? nlay - 1 - m : m; };     // internal layer -> caller row
  auto lev = [&](int k) { return top ? nlay - k : k; };         // internal level -> caller level
  for (int m = g; m < nlay; m += kSwNg) {
    const int r = row(m);
    const size_t x = i + ld * r;
    const double rfdelp = a.heatfac / a.delp[x];
    a.hswc[x] = ((fd_t[m + 1] - fu_t[m + 1]) - (fd_t[m] - fu_t[m])) * rfdelp;
    if (a.hsw0) a.hsw0[x] = ((dn0[m + 1] - up0[m + 1]) - (dn0[m] - up0[m])) * rfdelp;
    if (BANDS)
      for (int bb = 0; bb < 14; ++bb) {   // a band's g-points lie in one or two groups
        const int p0 = c_ns[bb] >> 4, p1 = (c_ns[bb] + c_ng[bb] - 1) >> 4;
        double u0 = 0.0, u1 = 0.0, d0 = 0.0, d1 = 0.0;
        for (int p = p0; p <= p1; ++p) {
          const double* bu = accb + (size_t)(2 * (bb + p)) * nlp1;
          const double* bd = bu + nlp1;
          u0 += bu[m]; u1 += bu[m + 1]; d0 += bd[m]; d1 += bd[m + 1];
        }
        a.hswb[i + ld * ((size_t)r + (size_t)nlay * bb)] = ((d1 - u1) - (d0 - u0)) * rfdelp;
      }
  }
  if (a.flxprf)
    for (int k = g; k < nlp1; k += kSwNg) {
      double* rec = a.flxprf + 4 * (i + ld * lev(k));
      rec[0] = fu_t[k];
      rec[1] = fd_t[k];
      rec[2] = up0[k];
      rec[3] = dn0[k];
    }
  if (g == 0) {
    double* tf = a.topflx + 3 * i;
    tf[0] = fu_t[nlay];
    tf[1] = dn0[nlay];
    tf[2] = up0[nlay];
    double* sf = a.sfcflx + 4 * i;
    sf[0] = fu_t[0];
    sf[1] = fd_t[0];
    sf[2] = up0[0];
    sf[3] = dn0[0];
  }
  if (a.fdncmp && g < 6) {
    // records uvbfc, uvbf0, nirbm, nirdf, visbm, visdf from the sums bm1, bm2, df1, df2, uvb
    const int from[6] = {4, 4, 0, 2, 1, 3};
    int q = from[0];
#pragma unroll
    for (int e = 1; e < 6; ++e) q = (g == e) ? from[e] : q;
    double clr = 0.0, all = 0.0;
    for (int p = 0; p < kRtGroups; ++p) {
      clr += sfc[(p * 2 + 0) * 5 + q];
      all += sfc[(p * 2 + 1) * 5 + q];
    }
    if (GRID) all = cf1 * all + cf0 * clr;
    a.fdncmp[6 * i + g] = (cloudy && g != 1) ? all : clr;
  }
}

// exp_tbl of the upward kernel: SHT in shared memory, else gathered through L1
template <bool SHT>
struct RtTable;
template <>
struct RtTable<false> {
  typedef TblGlobal type;
  static __device__ __forceinline__ type get(const double* ET, double*) { return {ET}; }
};
template <>
struct RtTable<true> {
  typedef TblShared type;
  static __device__ __forceinline__ type get(const double* ET, double* sm) {
    for (int q = threadIdx.x; q <= kNtbmx; q += blockDim.x) sm[q] = ET[q];
    __syncthreads();
    return {sm};
  }
};
template <bool SHT>
__host__ __device__ constexpr size_t rt_table_doubles() { return SHT ? kNtbmx + 1 : 0; }

// CTAs of NT threads walk the chunk's (column, g-point) pairs.  Nothing is
// shared between the g-points of a column on the way up, so the wide form
// (NT = kUpThreads) fills the four warps that a scheduler holds at 128
// registers; as whole columns, four of 3.5 warps, a call of 16,384 x 127 took
// 12.37 ms instead of 11.66 (five columns at 96 registers spilled: 13.50).
template <bool GRID, int NT, bool SHT>
__global__ void __launch_bounds__(NT, kUpThreads / NT)
sw_up_kernel(SwArgs a, SwScratch s, int p0, int nc, const double* __restrict__ T, const double* __restrict__ ET) {
  extern __shared__ double sm[];
  const auto tbl = RtTable<SHT>::get(ET, sm);
  for (int q = blockIdx.x * NT + threadIdx.x; q < nc * kSwNg; q += gridDim.x * NT) {
    const int pl = q / kSwNg, g = q - pl * kSwNg;
    const int j1 = a.idxday[p0 + pl];
    if (j1 < 1 || j1 > a.npts) continue;   // reported by the optics kernel
    up_body<GRID>(a, s, pl, nc, j1, g, T, tbl);
  }
}

template <bool GRID, int NT, bool SHT>
__global__ void __launch_bounds__(NT, kUpThreads / NT)
sw_up_blocks_kernel(const SwArgs* __restrict__ tab, const int2* __restrict__ pts, SwScratch s, int p0, int nc,
                    const double* __restrict__ T, const double* __restrict__ ET) {
  extern __shared__ double sm[];
  const auto tbl = RtTable<SHT>::get(ET, sm);
  for (int q = blockIdx.x * NT + threadIdx.x; q < nc * kSwNg; q += gridDim.x * NT) {
    const int pl = q / kSwNg, g = q - pl * kSwNg;
    const int2 at = pts[p0 + pl];
    up_body<GRID>(tab[at.x], s, pl, nc, at.y, g, T, tbl);
  }
}

// a column per CTA
template <bool GRID, bool BANDS>
__global__ void __launch_bounds__(kSwNg, BANDS ? 2 : kDownPerSm)
sw_down_kernel(SwArgs a, SwScratch s, int p0, int nc, const double* __restrict__ T) {
  extern __shared__ double sm[];
  const int j1 = a.idxday[p0 + blockIdx.x];
  if (j1 < 1 || j1 > a.npts) return;
  down_body<GRID, BANDS>(a, s, blockIdx.x, nc, j1, threadIdx.x, sm, T);
}

template <bool GRID, bool BANDS>
__global__ void __launch_bounds__(kSwNg, BANDS ? 2 : kDownPerSm)
sw_down_blocks_kernel(const SwArgs* __restrict__ tab, const int2* __restrict__ pts, SwScratch s, int p0, int nc,
                      const double* __restrict__ T) {
  extern __shared__ double sm[];
  const int2 q = pts[p0 + blockIdx.x];
  down_body<GRID, BANDS>(tab[q.x], s, blockIdx.x, nc, q.y, threadIdx.x, sm, T);
}

// Zeroes every output of every column of the physics blocks (RSM:824-845):
// column c of the concatenation is column c - colpre[b] of block b.
__global__ void sw_zero_blocks_kernel(const SwArgs* __restrict__ tab, const int* __restrict__ colpre, int nb,
                                      int total) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < total; c += gridDim.x * blockDim.x) {
    int lo = 0, hi = nb - 1;   // last block with colpre[b] <= c
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (colpre[mid] <= c) lo = mid;
      else hi = mid - 1;
    }
    const SwArgs& a = tab[lo];
    const size_t i = (size_t)(c - colpre[lo]), ld = (size_t)a.ld, nlay = (size_t)a.nlay;
    for (size_t k = 0; k < nlay; ++k) {
      a.hswc[i + ld * k] = 0.0;
      a.cldtau[i + ld * k] = 0.0;
      if (a.hsw0) a.hsw0[i + ld * k] = 0.0;
      if (a.hswb)
        for (size_t b = 0; b < 14; ++b) a.hswb[i + ld * (k + nlay * b)] = 0.0;
    }
    if (a.flxprf)
      for (size_t k = 0; k <= nlay; ++k)
        for (int q = 0; q < 4; ++q) a.flxprf[4 * (i + ld * k) + q] = 0.0;
    for (int q = 0; q < 3; ++q) a.topflx[3 * i + q] = 0.0;
    for (int q = 0; q < 4; ++q) a.sfcflx[4 * i + q] = 0.0;
    if (a.fdncmp)
      for (int q = 0; q < 6; ++q) a.fdncmp[6 * i + q] = 0.0;
  }
}

// The daytime-point table of the physics blocks: point dayp[b] + p is column
// idxday_b[p] of block b; an index outside 1..npts_b sets *bad.
__global__ void sw_points_kernel(const SwArgs* __restrict__ tab, const int* __restrict__ dayp, int nb,
                                 int2* __restrict__ pts, int* bad) {
  const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (b >= nb) return;
  const SwArgs& a = tab[b];
  for (int p = lane; p < dayp[b + 1] - dayp[b]; p += 32) {
    int j1 = a.idxday[p];
    if (j1 < 1 || j1 > a.npts) {
      atomicOr(bad, 1);
      j1 = 1;   // a valid column; the call reports the error
    }
    pts[dayp[b] + p] = make_int2(b, j1);
  }
}

// The per-layer overlap parameter of the sub-column generator for the stage
// entry point: fac_lcf between layers k-1 and k (iovr 3, RSM:2106-2108) or
// alpha (iovr 4, 5), [c + ldo*k]; inputs [c + ld*k], internal layer order.
__global__ void sw_overlap_aux_kernel(int ncols, int nlay, int ld, int iovr, const double* __restrict__ dz,
                                      const double* __restrict__ delg, const double* __restrict__ alpha,
                                      double* __restrict__ aux, int ldo) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)ncols * nlay) return;
  const int c = (int)(t % ncols), k = (int)(t / ncols);
  double v;
  if (iovr == 3)
    v = (k > 0) ? exp(-0.5 * (dz[c + (size_t)ld * k] + dz[c + (size_t)ld * (k - 1)]) / delg[c]) : 0.0;
  else
    v = alpha[c + (size_t)ld * k];
  aux[c + (size_t)ldo * k] = v;
}

cudaError_t overlap_aux_launch(int ncols, int nlay, int ld, int iovr, const double* dz, const double* delg,
                               const double* alpha, double* aux, int ldo, cudaStream_t st) {
  const long long n = (long long)ncols * nlay;
  if (n <= 0) return cudaSuccess;
  sw_overlap_aux_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(ncols, nlay, ld, iovr, dz, delg, alpha, aux, ldo);
  return cudaGetLastError();
}

cudaError_t gas_unpack_launch(const SwScratch& s, int nc, int nlay, const double* T, double* taug, double* taur,
                              cudaStream_t st) {
  sw_gas_unpack_kernel<<<1024, 256, 0, st>>>(s, nc, nlay, T, taug, taur);
  return cudaGetLastError();
}

static int optics_grid(int nc, int nlay) { return (int)(((long)nc * ((nlay + 31) / 32) + kOptWarps - 1) / kOptWarps); }

// Reorders every (rows, ng) k-table of the coefficient blob from row fastest to
// g-point fastest, in place.
void gpoint_fastest(double* blob) {
  using namespace swtab;
  const struct { int off, rows, ng; } t[] = {
      {b16_absa, 585, 6},  {b16_absb, 235, 6},  {b16_selfref, 10, 6},  {b16_forref, 3, 6},
      {b17_absa, 585, 12}, {b17_absb, 1175, 12}, {b17_selfref, 10, 12}, {b17_forref, 4, 12},
      {b18_absa, 585, 8},  {b18_absb, 235, 8},  {b18_selfref, 10, 8},  {b18_forref, 3, 8},
      {b19_absa, 585, 8},  {b19_absb, 235, 8},  {b19_selfref, 10, 8},  {b19_forref, 3, 8},
      {b20_absa, 65, 10},  {b20_absb, 235, 10}, {b20_selfref, 10, 10}, {b20_forref, 4, 10},
      {b21_absa, 585, 10}, {b21_absb, 1175, 10}, {b21_selfref, 10, 10}, {b21_forref, 4, 10},
      {b22_absa, 585, 2},  {b22_absb, 235, 2},  {b22_selfref, 10, 2},  {b22_forref, 3, 2},
      {b23_absa, 65, 10},  {b23_selfref, 10, 10}, {b23_forref, 3, 10},
      {b24_absa, 585, 8},  {b24_absb, 235, 8},  {b24_selfref, 10, 8},  {b24_forref, 3, 8},
      {b25_absa, 65, 6},   {b27_absa, 65, 8},   {b27_absb, 235, 8},
      {b28_absa, 585, 6},  {b28_absb, 1175, 6},
      {b29_absa, 65, 12},  {b29_absb, 235, 12}, {b29_selfref, 10, 12}, {b29_forref, 4, 12}};
  std::vector<double> row;
  for (const auto& q : t) {
    row.assign(blob + q.off, blob + q.off + (size_t)q.rows * q.ng);
    for (int i = 0; i < q.rows; ++i)
      for (int j = 0; j < q.ng; ++j) blob[q.off + (size_t)i * q.ng + j] = row[(size_t)j * q.rows + i];
  }
}

cudaError_t optics_launch(const SwArgs& a, const SwScratch& s, int p0, int nc, const double* T, const double* K,
                          cudaStream_t st) {
  if (nc <= 0) return cudaSuccess;
  sw_optics_kernel<<<optics_grid(nc, a.nlay), 32 * kOptWarps, 0, st>>>(a, s, p0, nc, T, K);
  return cudaGetLastError();
}

size_t down_smem(int nlay, bool hswb) { return rt_col_doubles(nlay, hswb) * sizeof(double); }
constexpr size_t kUpSmem = rt_table_doubles<true>() * sizeof(double);

cudaError_t rt_prepare(int max_smem) {
  const void* up[] = {(const void*)sw_up_kernel<false, kUpThreads, true>, (const void*)sw_up_kernel<true, kUpThreads, true>,
                      (const void*)sw_up_blocks_kernel<false, kUpThreads, true>,
                      (const void*)sw_up_blocks_kernel<true, kUpThreads, true>};
  const void* down[] = {(const void*)sw_down_kernel<false, false>,        (const void*)sw_down_kernel<true, false>,
                        (const void*)sw_down_kernel<false, true>,         (const void*)sw_down_kernel<true, true>,
                        (const void*)sw_down_blocks_kernel<false, false>, (const void*)sw_down_blocks_kernel<true, false>,
                        (const void*)sw_down_blocks_kernel<false, true>,  (const void*)sw_down_blocks_kernel<true, true>};
  cudaError_t e = cudaSuccess;
  for (const void* f : up)
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kUpSmem);
  for (const void* f : down)
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
  return e;
}

cudaError_t blocks_prepare(const SwArgs* tab, const int* colpre, const int* dayp, int nb, int total_cols,
                           int2* pts, int* bad, cudaStream_t st) {
  sw_points_kernel<<<(nb + 7) / 8, 256, 0, st>>>(tab, dayp, nb, pts, bad);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || total_cols <= 0) return e;
  sw_zero_blocks_kernel<<<min((total_cols + 127) / 128, 4096), 128, 0, st>>>(tab, colpre, nb, total_cols);
  return cudaGetLastError();
}

cudaError_t optics_blocks_launch(const SwArgs* tab, const int2* pts, const SwScratch& s, int p0, int nc, int nlay,
                                 const double* T, const double* K, cudaStream_t st) {
  if (nc <= 0) return cudaSuccess;
  sw_optics_blocks_kernel<<<optics_grid(nc, nlay), 32 * kOptWarps, 0, st>>>(tab, pts, s, p0, nc, T, K);
  return cudaGetLastError();
}

cudaError_t rt_blocks_launch(const SwArgs* tab, const int2* pts, bool grid, bool want_b, const SwScratch& s, int p0,
                             int nc, int nlay, const double* T, const double* ET, cudaStream_t st) {
  if (nc <= 0) return cudaSuccess;
  // one CTA per SM, exp_tbl in shared memory, once they have work for nearly all their threads (four columns' 448 of
  // 512); below that a column per CTA, which spreads a small call over the SMs.  A call, wide / narrow, us: 64 layers,
  // 100 columns 397 / 372, 300 420 / 405, 592 (four per SM) 447 / 454, 600 438 / 530, 1,800 922 / 1,022; 127 layers, 100
  // 544 / 505, 300 583 / 563, 592 632 / 658, 600 704 / 903, 1,800 1,596 / 1,826
  if (nc >= s.num_sms * kUpWide) {
    const auto up = grid ? sw_up_blocks_kernel<true, kUpThreads, true> : sw_up_blocks_kernel<false, kUpThreads, true>;
    up<<<s.num_sms, kUpThreads, kUpSmem, st>>>(tab, pts, s, p0, nc, T, ET);
  } else {
    const auto up = grid ? sw_up_blocks_kernel<true, kSwNg, false> : sw_up_blocks_kernel<false, kSwNg, false>;
    up<<<nc, kSwNg, 0, st>>>(tab, pts, s, p0, nc, T, ET);
  }
  const auto down = want_b ? (grid ? sw_down_blocks_kernel<true, true> : sw_down_blocks_kernel<false, true>)
                           : (grid ? sw_down_blocks_kernel<true, false> : sw_down_blocks_kernel<false, false>);
  down<<<nc, kSwNg, down_smem(nlay, want_b), st>>>(tab, pts, s, p0, nc, T);
  return cudaGetLastError();
}

cudaError_t rt_launch(const SwArgs& a, const SwScratch& s, int p0, int nc, const double* T, const double* ET,
                      cudaStream_t st) {
  if (nc <= 0) return cudaSuccess;
  const bool want_b = a.hswb != nullptr, grid = a.isubcsw <= 0;
  if (nc >= s.num_sms * kUpWide) {   // as in rt_blocks_launch
    const auto up = grid ? sw_up_kernel<true, kUpThreads, true> : sw_up_kernel<false, kUpThreads, true>;
    up<<<s.num_sms, kUpThreads, kUpSmem, st>>>(a, s, p0, nc, T, ET);
  } else {
    const auto up = grid ? sw_up_kernel<true, kSwNg, false> : sw_up_kernel<false, kSwNg, false>;
    up<<<nc, kSwNg, 0, st>>>(a, s, p0, nc, T, ET);
  }
  const auto down = want_b ? (grid ? sw_down_kernel<true, true> : sw_down_kernel<false, true>)
                           : (grid ? sw_down_kernel<true, false> : sw_down_kernel<false, false>);
  down<<<nc, kSwNg, down_smem(a.nlay, want_b), st>>>(a, s, p0, nc, T);
  return cudaGetLastError();
}

}  // namespace sw
