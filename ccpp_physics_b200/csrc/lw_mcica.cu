// lw_mcica.cu -- McICA sub-column cloud generator on the GPU, bit-exact.
//
// Restates mcica_subcol (physics/Radiation/RRTMG/radlw_main.F90, RLM:1847-
// 2107) with the GFS Mersenne twister of physics/Radiation/
// mersenne_twister.f (random_setseed_t MT:285-299, random_number_t
// MT:330-372).  One warp owns one cloudy column:
//   * seeding mt(i) = 69069^i * seed (mod 2^32): a lane starts at its power of
//     69069 and goes on in steps of 69069^32, one multiply per word;
//   * the stream lives in shared memory as its raw (untempered) sequence; a
//     twist appends the next 624 words in place, four per lane and 128 per
//     step;
//   * for max-random overlap (iovr=1) the random array is g-point major
//     (rand2d index (n-1)*nlay+k, RLM:1935-1941), so each g-point's walk
//     reads a contiguous run of the stream.  Lanes own g-points, 28 at a
//     time; the sequence ring holds one round's draws and the twist history.
// Integer arithmetic is exact; the u32 -> real conversion (u/(2^32-1)) and
// the FP64 comparisons/products of the walk are IEEE operations, so the
// sub-column flags equal the Fortran's bit for bit.
#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstdio>
#include <cuda_runtime.h>

#include "lw_common.cuh"
#include "lw_launch.h"

namespace lw {

__device__ __constant__ uint32_t c_pow69069[32];
constexpr uint32_t pow69069(int n) { return n == 0 ? 1u : 69069u * pow69069(n - 1); }
constexpr uint32_t kPow69069_32 = pow69069(32);

constexpr uint32_t kMata = 0x9908B0DFu, kUmask = 0x80000000u, kLmask = 0x7FFFFFFFu;
constexpr uint32_t kTmaskB = 0x9D2C5680u, kTmaskC = 0xEFC60000u;
// untempered word whose tempering is 2^32 - 1 (the only draw equal to 1)
constexpr uint32_t kRawAllOnes = 0x12DD9BB3u;

__device__ __forceinline__ uint32_t mt_word(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t y = (a & kUmask) | (b & kLmask);
  return c ^ (y >> 1) ^ ((y & 1u) ? kMata : 0u);
}
__device__ __forceinline__ uint32_t temper(uint32_t y) {
  y ^= y >> 11;
  y ^= (y << 7) & kTmaskB;
  y ^= (y << 15) & kTmaskC;
  y ^= y >> 18;
  return y;
}

// u / (2^32 - 1), correctly rounded, without a division (the GFS twister's
// harvest = real(y) / (2**32 - 1), mersenne_twister.f:362-369, for the
// unsigned value u of y).  1/(2^32-1) = (2^32+1)/(2^64-1), so the quotient
// is m * 2^-64 * (1 + 2^-64 + ...) with the 64-bit integer
// m = u * (2^32 + 1) = (u << 32) | u.  One FMA gives RN(m * 2^-64) exactly;
// the true quotient lies strictly above m * 2^-64 (for u > 0) but within one
// unit of m's last bit, so the two round alike except when m's discarded
// bits are exactly one half: then the quotient must round up, which ties-to-
// even misses when the kept last bit is 0.  m has 32 + L significant bits
// (L = bit length of u), so d = L - 21 bits are discarded, all from the low
// word, i.e. the low d bits of u.
__device__ __forceinline__ double u32_unit(uint32_t u) {
  const double a = (double)u * 0x1p-32;   // exact
  double r = fma(a, 0x1p-32, a);          // RN(m * 2^-64)
  const int d = (32 - __clz(u)) - 21;
  if (d >= 1) {
    const uint32_t half = 1u << (d - 1);
    if ((u & ((half << 1) - 1u)) == half && ((u >> d) & 1u) == 0u)
      r = __longlong_as_double(__double_as_longlong(r) + 1);
  }
  return r;
}

// Appends the next 624 sequence words to the ring at position jp (a
// multiple of 624; the previous block o sits just before it, cyclically)
// (MT:341-356): word t from words t, t + 1 and t + 397 of the sequence that
// starts at o, four words per lane and 128 per step, which reach back to the
// step before at the latest (word t + 3 needs word t - 224 of this block).
// t + 397 is one past a multiple of 4, so each group takes two 16-byte and two
// 4-byte reads and one 16-byte store: a word at a time, 16 accesses instead of
// five, lw_mcica_kernel took 0.38 instead of 0.29 ms at 16,384 x 127.
// With HIT, also returns whether this lane wrote the one word that tempers to
// 2^32 - 1 (kRawAllOnes).
template <bool HIT = false>
__device__ bool twist_ring(uint32_t* ring, int cap, int jp, int lane) {
  const uint32_t* o = ring + ((jp == 0 ? cap : jp) - 624);
  uint32_t* w = ring + jp;
  bool hit = false;
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int t = 4 * (lane + 32 * s);
    if (t < 624) {
      const uint4 a = *reinterpret_cast<const uint4*>(o + t);
      const uint32_t a4 = *(t + 4 < 624 ? o + t + 4 : w);
      const uint4 c = *reinterpret_cast<const uint4*>(t < 228 ? o + t + 396 : w + t - 228);
      const uint32_t c4 = *(t < 224 ? o + t + 400 : w + t - 224);
      uint4 v;
      v.x = mt_word(a.x, a.y, c.y);
      v.y = mt_word(a.y, a.z, c.z);
      v.z = mt_word(a.z, a.w, c.w);
      v.w = mt_word(a.w, a4, c4);
      *reinterpret_cast<uint4*>(w + t) = v;
      if (HIT) hit |= v.x == kRawAllOnes || v.y == kRawAllOnes || v.z == kRawAllOnes || v.w == kRawAllOnes;
    }
    __syncwarp();
  }
  return hit;
}

struct McicaArgs {
  int nlay, nw, iovr, isubclw, top_at_1;
  int cap;        // ring capacity in words (iovr 0..2)
  McicaStage st;  // stage entry point inputs (blocks == nullptr)
};

// The draw conversion h(u) = u / (2^32 - 1) (u32_unit) is strictly
// increasing (consecutive u differ by 2^-32, far above a double's spacing),
// so every comparison of a draw with a per-layer value x is a comparison of
// the tempered word u with an exact integer threshold:
//   h(u) >= x  <=>  u >= umin_ge(x),   h(u) < x  <=>  u < ulim_lt(x),
//   h(u) <= x  <=>  u <= umax_le(x).
// Thresholds are 64-bit: 2^32 / -1 / 0 mean that no word qualifies (x above
// 1, below 0, or NaN, for which every comparison is false).  x (2^32 - 1) is
// within one unit of the threshold, so a few exact steps settle it.
__device__ long long umin_ge(double x) {
  if (x <= 0.0) return 0;
  if (!(x <= 1.0)) return 4294967296LL;
  long long u = (long long)(x * 4294967295.0);
  if (u > 4294967295LL) u = 4294967295LL;
  for (int it = 0; it < 8 && u > 0 && u32_unit((uint32_t)(u - 1)) >= x; ++it) --u;
  for (int it = 0; it < 8 && u <= 4294967295LL && u32_unit((uint32_t)u) < x; ++it) ++u;
  return u;
}
__device__ long long ulim_lt(double x) { return (x != x) ? 0 : umin_ge(x); }
__device__ long long umax_le(double x) {
  if (!(x >= 0.0)) return -1;
  if (x >= 1.0) return 4294967295LL;
  long long u = (long long)(x * 4294967295.0);   // smallest u with h(u) > x, minus one
  for (int it = 0; it < 8 && u > 0 && u32_unit((uint32_t)(u - 1)) > x; ++it) --u;
  for (int it = 0; it < 8 && u32_unit((uint32_t)u) <= x; ++it) ++u;
  return u - 1;
}

// Overlaps built from two layer-major random sets (RLM:1995-2091):
//   iovr = 3, decorrelation length: top-down, layer k keeps the value of layer
//     k+1 when set2(k) <= fac_lcf(k+1), else its own set-1 draw;
//   iovr = 4/5, exponential / exponential-random: bottom-up, layer k keeps the
//     value of layer k-1 when set2(k) < alpha(k), else its own draw.
// Set 1 is stream positions [0, 140 nlay), set 2 the next 140 nlay; two
// twister states walk them in lockstep, layer by layer, surface first.
//
// Each state is the 624 words x_i..x_{i+623} themselves, updated in place:
// the next W <= 227 words depend only on words already there, so a layer's
// 140 draws of a set are computed straight into registers (five per lane) and
// stored over the words they replace, with one barrier between the reads and
// the stores of both sets.  Jumping to set 2 takes 224 words at a time.
//
// iovr 3's top-down rule is evaluated bottom-up: a layer's value is the set-1
// draw of the nearest layer at or above it whose link to the layer above is
// broken (the top layer's always is), so each g-point keeps the run of layers
// still waiting for that draw.  A break resolves a run: (g-point, run, draw)
// goes into a queue in shared memory, and 32 of them at a time are turned
// into flags, one per lane; a tenth of the g-points break at a layer, and
// resolving them on the spot ran the search with a few lanes active.  Runs
// without a cloudy layer are not queued.
//
// The tests are on tempered words against integer thresholds (above):
// clr_t[k] = umin_ge(1 - cldf(k)) for the cloud flag (RLM:2097-2103), and
// aux_t[k] = umax_le(fac_lcf(k)) (iovr 3, 0-based, aux_t[0] unused) or
// ulim_lt(alpha(k)) (iovr 4, 5).  A clear layer's flag (threshold 2^32 - 1)
// is set by the draw of all ones alone.  So once the walk is above the top
// cloudy layer and no run with a cloudy layer waits, the remaining set-1 words
// are only looked through for that draw; if one turns up, the column is done
// again to its top (walk_all).
//
// Bound by integer issue.  5,003 columns of 127 layers, iovr 3: 1.12 ms with
// 1,248-word rings read back per draw, runs resolved on the spot and 12 warps
// per SM; 0.30 ms so (12.6 KB a warp, 16 warps per SM).
constexpr int kTwoSetWarps = 2;      // per CTA, a column each; the grid holds every column, so warps are refilled as they end
constexpr int kTwoSetQueue = 192;    // 31 events left over and at most 160 of one layer
constexpr int kNoCloud = 0x7fff;     // "no cloudy layer at or above"

__device__ __forceinline__ uint32_t wrap624(uint32_t q) { return min(q, q - 624u); }   // q < 1248

// The next 32 W words of a state whose oldest word is x[pos] (W <= 7: 224 of
// the 227 that depend on present words only), lane + 32 j to r[j].
template <int W>
__device__ __forceinline__ void mt_next(const uint32_t* x, uint32_t pos, int lane, uint32_t (&r)[W]) {
#pragma unroll
  for (int j = 0; j < W; ++j) {
    const uint32_t q = pos + lane + 32 * j;
    r[j] = mt_word(x[wrap624(q)], x[wrap624(q + 1)], x[wrap624(q + 397)]);
  }
}
// Stores the first `count` of them over the words they replace.
template <int W>
__device__ __forceinline__ void mt_put(uint32_t* x, uint32_t pos, int count, int lane, const uint32_t (&r)[W]) {
#pragma unroll
  for (int j = 0; j < W; ++j)
    if (lane + 32 * j < count) x[wrap624(pos + lane + 32 * j)] = r[j];
}
// Advances by `count` words; whether this lane met the word that tempers to 2^32 - 1.
__device__ bool mt_skip(uint32_t* x, uint32_t& pos, int count, int lane) {
  bool hit = false;
  for (int left = count; left > 0; left -= 224) {
    const int n = min(left, 224);
    uint32_t r[7];
    mt_next(x, pos, lane, r);
#pragma unroll
    for (int j = 0; j < 7; ++j) hit |= lane + 32 * j < n && r[j] == kRawAllOnes;
    __syncwarp();
    mt_put(x, pos, n, lane, r);
    __syncwarp();
    pos = wrap624(pos + n);
  }
  return hit;
}

// Per-warp shared memory of the kernel below.
struct TwoSetSmem {
  long long* clr;    // [nlay] cloud thresholds
  long long* aux;    // [nlay] link thresholds
  long long* srt;    // [32 nw] per 32-layer word, the cloud thresholds in ascending order
  uint2* ev;         // [kTwoSetQueue] waiting events: draw; g-point | last layer << 8 | first layer << 16
  uint32_t* xa;      // [624] state of set 1
  uint32_t* xb;      // [624] state of set 2
  uint32_t* pm;      // [33 nw] the mask of a word's layers with the c smallest thresholds
  uint32_t* ow;      // [140 nw] flags
  int16_t* nxt;      // [32 nw + 2] lowest cloudy layer at or above
  __host__ __device__ static size_t bytes(int nlay, int nw) {
    return ((size_t)16 * nlay + 256 * nw + 8 * kTwoSetQueue + 2 * 624 * 4 + 4 * (33 * nw + NGPT * nw) +
            2 * (32 * nw + 2) + 15) & ~(size_t)15;
  }
  __device__ TwoSetSmem(char* p, int nlay, int nw) {
    clr = reinterpret_cast<long long*>(p);
    aux = clr + nlay;
    srt = aux + nlay;
    ev = reinterpret_cast<uint2*>(srt + 32 * nw);
    xa = reinterpret_cast<uint32_t*>(ev + kTwoSetQueue);
    xb = xa + 624;
    pm = xb + 624;
    ow = pm + 33 * nw;
    nxt = reinterpret_cast<int16_t*>(ow + NGPT * nw);
  }
};

// The flags of one event: per 32-layer word of its run, the layers whose
// threshold the draw reaches are a prefix of the word's sorted thresholds.
__device__ __forceinline__ void two_set_event(const TwoSetSmem& m, uint2 e, int nw) {
  const long long v = e.x;
  const int n = e.y & 255, k1 = (e.y >> 8) & 255, k0 = e.y >> 16;
  for (int w = k0 >> 5; w <= (k1 >> 5); ++w) {
    const int lo = max(k0 - 32 * w, 0), hi = min(k1 - 32 * w, 31);
    const uint32_t run = (0xFFFFFFFFu >> (31 - hi)) & (0xFFFFFFFFu << lo);
    const long long* sw = m.srt + 32 * w;
    int cnt = 0;
#pragma unroll
    for (int st = 16; st >= 1; st >>= 1)
      if (sw[cnt + st - 1] <= v) cnt += st;
    cnt += (sw[31] <= v) ? 1 : 0;   // only when all 32 qualify (then cnt was 31)
    const uint32_t f = run & m.pm[33 * w + cnt];
    if (f) atomicOr(m.ow + n * nw + w, f);   // two events of a g-point may be in flight
  }
}

__global__ void __launch_bounds__(32 * kTwoSetWarps)
lw_mcica_two_set_kernel(const Block* __restrict__ blocks, int nblocks, const Block b0, int ncols, McicaArgs a,
                        uint32_t* __restrict__ bits) {
  extern __shared__ __align__(16) char smem_raw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int nlay = a.nlay, nlp1 = nlay + 1, nw = a.nw;
  const int c = blockIdx.x * kTwoSetWarps + wib;
  if (c >= ncols) return;   // the warps share nothing
  const TwoSetSmem m(smem_raw + TwoSetSmem::bytes(nlay, nw) * wib, nlay, nw);

  // cloud and link thresholds (inputs as in lw_mcica_kernel below)
  const Block* B = (nblocks > 0) ? ((nblocks == 1) ? &b0 : &blocks[find_block(blocks, nblocks, c)]) : nullptr;
  const int i = B ? c - B->col0 : 0;
  int32_t seed;
  bool any = false;
  if (B) {
    for (int k = lane; k < nlay; k += 32) {
      const double cf = B->in[F_CLDCF][i + (size_t)B->ld * (a.top_at_1 ? nlp1 - (k + 1) - 1 : k)];
      any |= cf > 1.0e-6;
      m.clr[k] = umin_ge(1.0 - ((cf < 2.2250738585072014e-308) ? 0.0 : cf));
    }
    seed = (a.isubclw == 1) ? 140 + (B->seed0 + i + 1) : B->icseed[i];   // RLM:765-773
  } else {
    for (int k = lane; k < nlay; k += 32) m.clr[k] = umin_ge(1.0 - a.st.cldf[c + (size_t)a.st.ld * k]);
    any = true;
    seed = a.st.seed[c];
  }
  if (!__any_sync(0xffffffffu, any)) return;   // clear column: no draws
  if (a.iovr == 3) {
    // fac_lcf(k) = exp(-0.5 (dz(k) + dz(k-1)) / de_lgth), dz in the internal order (RLM:819, 2001)
    const double dl = B ? B->in[F_DELGTH][i] : a.st.delg[c];
    for (int k = 1 + lane; k < nlay; k += 32) {
      double dz0, dz1;
      if (B) {
        const int r0 = a.top_at_1 ? nlp1 - (k + 1) - 1 : k, r1 = a.top_at_1 ? nlp1 - k - 1 : k - 1;
        dz0 = B->in[F_DZLYR][i + (size_t)B->ld * r0];
        dz1 = B->in[F_DZLYR][i + (size_t)B->ld * r1];
      } else {
        dz0 = a.st.dz[c + (size_t)a.st.ld * k];
        dz1 = a.st.dz[c + (size_t)a.st.ld * (k - 1)];
      }
      m.aux[k] = umax_le(exp(-0.5 * (dz0 + dz1) / dl));
    }
  } else {
    // alpha is taken in the caller's row order, unflipped (RLM:820, 933)
    for (int k = lane; k < nlay; k += 32)
      m.aux[k] = ulim_lt(B ? B->in[F_ALPHA][i + (size_t)B->ld * k] : a.st.alpha[c + (size_t)a.st.ld * k]);
  }
  __syncwarp();
  // the next cloudy layer above each, and iovr 3's sorted thresholds and
  // prefix masks per 32-layer word (layers past nlay never qualify)
  int up = kNoCloud, ktop = -1;
  if (lane == 0) m.nxt[32 * nw] = kNoCloud;
  for (int w = nw - 1; w >= 0; --w) {
    const int k = 32 * w + lane;
    const long long th = (k < nlay) ? m.clr[k] : LLONG_MAX;
    const uint32_t cloudy = __ballot_sync(0xffffffffu, th < 0xFFFFFFFFLL);
    const uint32_t here = cloudy & (0xFFFFFFFFu << lane);
    m.nxt[k] = (int16_t)(here ? 32 * w + __ffs(here) - 1 : up);
    if (cloudy) {
      up = 32 * w + __ffs(cloudy) - 1;
      if (ktop < 0) ktop = 32 * w + 31 - __clz(cloudy);
    }
    if (a.iovr == 3) {
      int rank = 0;
      for (int o = 0; o < 32; ++o) {
        const long long t2 = __shfl_sync(0xffffffffu, th, o);
        rank += (t2 < th || (t2 == th && o < lane)) ? 1 : 0;
      }
      m.srt[32 * w + rank] = th;
      for (int q = 0; q <= 32; ++q) {
        const uint32_t b = __ballot_sync(0xffffffffu, rank < q);
        if (lane == 0) m.pm[33 * w + q] = b;
      }
    }
  }
  const uint32_t s0 = (uint32_t)(seed == 0 ? 4357 : seed);   // random_setseed_t (MT:285-299)
  const uint32_t below = (1u << lane) - 1u;

  for (bool walk_all = false;; walk_all = true) {
    // mt(i) = 69069^i seed; set 2 starts 140 nlay draws on
    uint32_t v = s0 * c_pow69069[lane];
    for (int n = lane; n < 624; n += 32) {
      m.xa[n] = m.xb[n] = v;
      v *= kPow69069_32;
    }
    for (int n = lane; n < NGPT * nw; n += 32) m.ow[n] = 0u;
    __syncwarp();
    uint32_t pa = 0, pb = 0;
    mt_skip(m.xb, pb, NGPT * nlay, lane);

    int start[5], nc[5];          // iovr 3: the waiting run's first layer and its lowest cloudy one
    uint32_t cdf[5], word[5];     // iovr 4, 5: the value carried up, the flags of this 32-layer word
    const int nc0 = m.nxt[0];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      start[j] = 0;
      nc[j] = (lane + 32 * j < NGPT) ? nc0 : kNoCloud;
      cdf[j] = word[j] = 0u;
    }
    int nev = 0, k = 0;
    for (; k < nlay; ++k) {
      if (k > ktop && !walk_all) {   // nothing cloudy from here on
        bool more = false;
#pragma unroll
        for (int j = 0; j < 5; ++j) more |= (a.iovr == 3) ? nc[j] < k : cdf[j] == 0xFFFFFFFFu;
        if (!__any_sync(0xffffffffu, more)) break;
      }
      uint32_t c1[5], c2[5];
      mt_next(m.xa, pa, lane, c1);
      mt_next(m.xb, pb, lane, c2);
      __syncwarp();
      mt_put(m.xa, pa, NGPT, lane, c1);
      mt_put(m.xb, pb, NGPT, lane, c2);
      __syncwarp();
      pa = wrap624(pa + NGPT);
      pb = wrap624(pb + NGPT);
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        c1[j] = temper(c1[j]);
        c2[j] = temper(c2[j]);
      }
      if (a.iovr == 3) {
        const bool top = (k == nlay - 1);
        const long long fk = top ? -1 : m.aux[k + 1];
        const int nc1 = m.nxt[k + 1];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          const int n = lane + 32 * j;
          const bool brk = n < NGPT && (long long)c2[j] > fk;   // not linked to the layer above
          const bool put = brk && (k >= nc[j] || c1[j] == 0xFFFFFFFFu);
          const uint32_t b = __ballot_sync(0xffffffffu, put);
          if (put) m.ev[nev + __popc(b & below)] = make_uint2(c1[j], n | (k << 8) | (start[j] << 16));
          nev += __popc(b);
          if (brk) {
            start[j] = k + 1;
            nc[j] = nc1;
          }
        }
        if (nev >= 32) {
          __syncwarp();
          do {
            nev -= 32;
            two_set_event(m, m.ev[nev + lane], nw);
          } while (nev >= 32);
          __syncwarp();
        }
      } else {
        const long long ak = m.aux[k], ck = m.clr[k];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          const int n = lane + 32 * j;
          if (n >= NGPT) continue;
          cdf[j] = (k > 0 && (long long)c2[j] < ak) ? cdf[j] : c1[j];
          if ((long long)cdf[j] >= ck) word[j] |= 1u << (k & 31);
          if ((k & 31) == 31) {
            m.ow[n * nw + (k >> 5)] = word[j];
            word[j] = 0u;
          }
        }
      }
    }
    // what the walk left out may hold the one draw that flags a clear layer
    const bool again = k < nlay && __any_sync(0xffffffffu, mt_skip(m.xa, pa, NGPT * (nlay - k), lane));
    if (again) continue;
    __syncwarp();
    if (a.iovr == 3) {
      if (lane < nev) two_set_event(m, m.ev[lane], nw);
    } else if (k & 31) {   // the last word begun
#pragma unroll
      for (int j = 0; j < 5; ++j)
        if (lane + 32 * j < NGPT) m.ow[(lane + 32 * j) * nw + (k >> 5)] = word[j];
    }
    break;
  }
  __syncwarp();
  uint32_t* out = bits + (size_t)c * NGPT * nw;
  for (int n = lane; n < NGPT * nw; n += 32) out[n] = m.ow[n];
}

// The draws of random (iovr=0) and maximum-random (iovr=1) overlap come from
// a ring that holds the raw (untempered) twister sequence itself: sequence
// index s (x_0..x_623 = the seeding, draw p = tempered x_{624+p}) sits at
// ring[s mod cap].  A twist appends the next 624 words in place,
//   x_{j+t} = mt_word(x_{j+t-624}, x_{j+t-623}, x_{j+t-227}),
// so there is no separate state array and no copy; cap is a multiple of
// 624, so neither the block being written nor the one before it wraps.
// Lanes walk g-points in rounds of kMcicaRound (5 x 28 = 140): the ring
// holds one round's draws plus the twist history.  Rounds of 20 (14 warps per
// SM instead of 12) took 0.31 ms at 16,384 x 127, of 10 (20 warps) 0.37 ms,
// of 28 0.29 ms.
constexpr int kMcicaRound = 28;

__host__ __device__ constexpr uint32_t temper_c(uint32_t y) {
  return ((((y ^ (y >> 11)) ^ (((y ^ (y >> 11)) << 7) & kTmaskB)) ^
           ((((y ^ (y >> 11)) ^ (((y ^ (y >> 11)) << 7) & kTmaskB)) << 15) & kTmaskC)) ^
          (((((y ^ (y >> 11)) ^ (((y ^ (y >> 11)) << 7) & kTmaskB)) ^
             ((((y ^ (y >> 11)) ^ (((y ^ (y >> 11)) << 7) & kTmaskB)) << 15) & kTmaskC)) >>
            18)));
}
static_assert(temper_c(kRawAllOnes) == 0xFFFFFFFFu, "kRawAllOnes tempers to 2^32 - 1");

// Per-warp shared memory: clear[nlay] = 1 - cldf (double), ring[cap].
__host__ __device__ inline size_t mcica_warp_bytes(int nlay, int cap) {
  return ((nlay * 8 + 15) & ~15) + (size_t)cap * 4;
}

constexpr int kMcicaWarps = 6;   // 6 warps x 18.5 KB (127 layers): two CTAs, twelve warps per SM

// iovr 0..2.  NG g-points per column: 140 for the longwave path (block or
// stage inputs), 112 for the shortwave path (stage inputs).
template <int NG>
__global__ void __launch_bounds__(32 * kMcicaWarps)
lw_mcica_kernel(const Block* __restrict__ blocks, int nblocks, const Block b0, int ncols, McicaArgs a,
                uint32_t* __restrict__ bits) {
  extern __shared__ __align__(16) char smem_raw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const size_t wbytes = mcica_warp_bytes(a.nlay, a.cap);
  char* my = smem_raw + wbytes * wib;
  double* clr = reinterpret_cast<double*>(my);   // 1 - cldf(k), used by every test of the walk
  uint32_t* ring = reinterpret_cast<uint32_t*>(my + ((a.nlay * 8 + 15) & ~15));
  const int nlay = a.nlay, nlp1 = nlay + 1, cap = a.cap;
  const int warps_total = gridDim.x * (blockDim.x >> 5);

  for (int c = blockIdx.x * (blockDim.x >> 5) + wib; c < ncols; c += warps_total) {
    __syncwarp();
    int32_t seed;
    bool any = false;
    if (nblocks > 0) {
      // layer cloud fraction in internal (surface-first) order, floored as
      // in cldprop (RLM:1805-1811); lcf1 test of the driver (RLM:1070-1076)
      const Block& B = (nblocks == 1) ? b0 : blocks[find_block(blocks, nblocks, c)];
      const int i = c - B.col0;
      for (int k = lane; k < nlay; k += 32) {
        int r = a.top_at_1 ? nlp1 - (k + 1) - 1 : k;
        double cf = B.in[F_CLDCF][i + (size_t)B.ld * r];
        any |= cf > 1.0e-6;
        clr[k] = 1.0 - ((cf < 2.2250738585072014e-308) ? 0.0 : cf);
      }
      seed = (a.isubclw == 1) ? 140 + (B.seed0 + i + 1) : B.icseed[i];   // RLM:765-773
    } else {
      for (int k = lane; k < nlay; k += 32) {
        clr[k] = 1.0 - a.st.cldf[c + (size_t)a.st.ld * k];
      }
      any = true;
      seed = a.st.seed[c];
    }
    if (!__any_sync(0xffffffffu, any)) continue;   // clear column: no draws
    const uint32_t s0 = (uint32_t)(seed == 0 ? 4357 : seed);   // random_setseed_t (MT:285-299)

    uint32_t* out = bits + (size_t)c * NG * a.nw;
    // seeding x_0..x_623 at ring[0..623]: mt(i) = 69069^i seed
    uint32_t x = s0 * c_pow69069[lane];
    for (int n = lane; n < 624; n += 32) {
      ring[n] = x;
      x *= kPow69069_32;
    }
    __syncwarp();
    if (a.iovr == 2) {
      // maximum overlap: one draw per g-point, the same at every layer (RLM:1981-1993)
      twist_ring(ring, cap, 624, lane);   // sequence 624..1247 at ring[624..1247] (cap >= 1248)
      for (int n = lane; n < NG; n += 32) {
        double r = u32_unit(temper(ring[624 + n]));
        for (int w = 0; w < a.nw; ++w) {
          uint32_t word = 0;
          for (int b = 0; b < 32; ++b) {
            int k = w * 32 + b;
            if (k < nlay && r >= clr[k]) word |= 1u << b;
          }
          out[n * a.nw + w] = word;
        }
      }
      continue;
    }
    // random (iovr=0) and maximum-random (iovr=1): draw n*nlay+k (RLM:1920-1941)
    long long gen = 624;       // sequence indices generated so far
    int jp = 624;              // gen mod cap
    bool hit = false;          // warp-uniform: some generated word tempers to 2^32 - 1
    static_assert(NG % kMcicaRound == 0, "whole rounds of g-points");
    for (int n0 = 0; n0 < NG; n0 += kMcicaRound) {
      const long long need = 624 + (long long)(n0 + kMcicaRound) * nlay;
      while (gen < need) {
        hit |= __any_sync(0xffffffffu, twist_ring<true>(ring, cap, jp, lane));
        gen += 624;
        jp += 624;
        if (jp == cap) jp = 0;
      }
      const int n = n0 + lane;
      if (!hit) {
        // No draw so far is 1 (only that word tempers to 2^32 - 1), so every
        // cdf stays below 1: a clear layer's flag (cdf >= 1, see below) is 0
        // and the layer after it starts afresh (cdf = r * 1).  Only the
        // cloudy layers are walked, word by word from the warp's mask of them;
        // the flags are those of the walk below, bit for bit.
        const int q0 = (int)((624 + (long long)n * nlay) % cap);
        double cdf = 0.0;
        int kprev = -2;
        for (int w = 0; w < a.nw; ++w) {
          const int kk = 32 * w + lane;
          uint32_t m = __ballot_sync(0xffffffffu, kk < nlay && clr[kk] != 1.0);   // the word's cloudy layers
          if (lane < kMcicaRound) {
            uint32_t word = 0;
            while (m) {
              const int b = __ffs(m) - 1;
              m &= m - 1;
              const int k = 32 * w + b;
              int q = q0 + k;
              if (q >= cap) q -= cap;
              const double r = u32_unit(temper(ring[q]));
              if (k == 0 || a.iovr == 0 || kprev != k - 1) {
                cdf = r;
              } else {
                const double tem1 = clr[k - 1];        // max-random walk (RLM:1949-1960)
                cdf = (cdf > tem1) ? cdf : r * tem1;
              }
              if (cdf >= clr[k]) word |= 1u << b;      // RLM:2097-2103
              kprev = k;
            }
            out[n * a.nw + w] = word;
          }
        }
        __syncwarp();
        continue;
      }
      if (lane < kMcicaRound) {
        int q = (int)((624 + (long long)n * nlay) % cap);
        double cdf = 0.0;
        uint32_t word = 0;
#pragma unroll 4   // lets the ring and cloud-fraction loads of four layers issue ahead
        for (int k = 0; k < nlay; ++k) {
          const uint32_t raw = ring[q];
          if (++q == cap) q = 0;
          const double ck = clr[k];
          if (ck == 1.0) {
            // Clear layer (the same for every lane: lanes are g-points of one layer).
            // Its flag is cdf >= 1, and every draw is <= 1 with equality only for
            // the word that tempers to 2^32 - 1, so the flag needs neither tempering
            // nor conversion: a fresh draw is 1 only for that word, an inherited cdf
            // only if it is 1, and r * tem1 < 1 when tem1 < 1.  The cdf of a clear
            // layer is never read again: the next layer compares it with
            // 1 - cldf = 1 and takes r * 1 = r instead.
            bool bit;
            if (k == 0 || a.iovr == 0) {
              bit = (raw == kRawAllOnes);
            } else {
              const double tem1 = clr[k - 1];
              bit = (tem1 == 1.0) ? (raw == kRawAllOnes) : (cdf > tem1 && cdf >= 1.0);
            }
            if (bit) word |= 1u << (k & 31);
          } else {
            const double r = u32_unit(temper(raw));
            if (k == 0 || a.iovr == 0) {
              cdf = r;
            } else {
              const double tem1 = clr[k - 1];        // max-random walk (RLM:1949-1960)
              cdf = (cdf > tem1) ? cdf : r * tem1;
            }
            if (cdf >= ck) word |= 1u << (k & 31);   // RLM:2097-2103
          }
          if ((k & 31) == 31 || k == nlay - 1) {
            out[n * a.nw + (k >> 5)] = word;
            word = 0;
          }
        }
      }
      __syncwarp();
    }
  }
}

// The raw (untempered) words of one twister stream after
// random_setseed_t(seed) (MT:285-299): out[j] is the state word that draw j
// of random_number_t (MT:330-372) tempers.  One CTA walks a stream, a ring of
// sequence words in shared memory, 227 words per barrier (word i + 624 needs
// words i, i + 1 and i + 397); tempering and the conversion to a random index
// run later, in parallel, for the words that are used (seed_index_of).
//
// The walk is a serial chain, so a longer stream is cut into segments of
// kSeedJump words and each segment's state is jumped to: the state N words on
// is the GF(2) sum of the states i = 0 .. 19936 whose bit is set in
// x^N mod p(x), and those states' words are the stream's first kSeedJump ones
// (c_seed_jump, and how it is made: data/make_mt_jump.py).  Rounds of
// kSeedSegs segments: the first segment by one CTA, the sums by many, the other
// segments a CTA each.  The seeds of a 384 x 384 face (294,912 words) take 166 us
// with one walk and 86 us so; at 82,418 words, past the line, 83 and 80 us, and
// at 61,952 words 72 and 78 us.
constexpr int kSeedThreads = 256, kSeedPhase = 227, kSeedRing = 2048;
constexpr int kSeedJump = 33 * 624, kSeedSegs = 16;
constexpr int kSeedPolyBits = 19937, kSeedChunk = 512;   // polynomial bits per CTA of the sums
constexpr int kSeedSumThreads = 160;                     // four words of the state each
constexpr int kSeedWalk = 4 * kSeedJump;                 // words up to which one CTA walks
static_assert(kSeedJump + 624 >= kSeedPolyBits + 624 && 4 * kSeedSumThreads >= 624, "words of the sums");

__device__ const uint32_t c_seed_jump[kSeedSegs - 1][624] = {
#include "../data/mt_jump.inc"
};

// n words from the state in ring[0..623]; every thread of the CTA calls it,
// after a barrier.  The state behind them is then ring[(n + q) % kSeedRing].
__device__ void seed_walk(uint32_t* ring, int n, uint32_t* __restrict__ out) {
  const int t = threadIdx.x;
  for (int b = 0; b < n; b += kSeedPhase) {
    if (t < kSeedPhase) {
      const uint32_t i = b + t;
      const uint32_t v = mt_word(ring[i % kSeedRing], ring[(i + 1) % kSeedRing], ring[(i + 397) % kSeedRing]);
      ring[(i + 624) % kSeedRing] = v;
      if (i < (uint32_t)n) out[i] = v;
    }
    __syncthreads();
  }
}

// The first segment of a round (or the whole stream): from the seed, or from
// state[kSeedSegs] where the round before ended.  Leaves its first state in
// state[0] and clears the others for the sums (state null: neither).
__global__ void __launch_bounds__(kSeedThreads)
lw_seed_stream_kernel(uint32_t seed, bool first, int n, uint32_t* __restrict__ state, uint32_t* __restrict__ out) {
  __shared__ uint32_t ring[kSeedRing];
  const int t = threadIdx.x;
  if (!first) {
    for (int q = t; q < 624; q += kSeedThreads) ring[q] = state[kSeedSegs * 624 + q];
  } else if (t < 32) {   // MT:290-296, signed wrap = unsigned multiply
    uint32_t v = seed;
    for (int q = 0; q < t; ++q) v *= 69069u;
    for (int q = t; q < 624; q += 32) {
      ring[q] = v;
      v *= kPow69069_32;
    }
  }
  __syncthreads();
  if (state) {
    for (int q = t; q < 624; q += kSeedThreads) state[q] = ring[q];
    for (int q = 624 + t; q < kSeedSegs * 624; q += kSeedThreads) state[q] = 0u;
  }
  seed_walk(ring, n, out);
}

// state[s] ^= the states of this CTA's kSeedChunk polynomial bits, s = blockIdx.y + 1
__global__ void __launch_bounds__(kSeedSumThreads)
lw_seed_jump_kernel(uint32_t* __restrict__ state, const uint32_t* __restrict__ out) {
  __shared__ uint32_t x[kSeedChunk + 4 * kSeedSumThreads];
  const int t = threadIdx.x, i0 = blockIdx.x * kSeedChunk;
  for (int q = t; q < kSeedChunk + 624; q += kSeedSumThreads) {   // sequence words i0 + q
    const int i = i0 + q;
    x[q] = i < 624 ? state[i] : out[i - 624];
  }
  __syncthreads();
  const uint32_t* g = c_seed_jump[blockIdx.y] + i0 / 32;
  uint32_t acc[4] = {0u, 0u, 0u, 0u};
  for (int w = 0; w < kSeedChunk / 32 && i0 / 32 + w < 624; ++w) {
    uint32_t m = __ldg(g + w);
    while (m) {
      const int b = 32 * w + __ffs(m) - 1;
      m &= m - 1;
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] ^= x[b + t + kSeedSumThreads * q];
    }
  }
  uint32_t* y = state + (blockIdx.y + 1) * 624;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (t + kSeedSumThreads * q < 624) atomicXor(y + t + kSeedSumThreads * q, acc[q]);
}

// segments 1 .. of a round of m words; the state behind the last of a full
// round goes to state[kSeedSegs]
__global__ void __launch_bounds__(kSeedThreads)
lw_seed_segment_kernel(int m, uint32_t* __restrict__ state, uint32_t* __restrict__ out) {
  __shared__ uint32_t ring[kSeedRing];
  const int t = threadIdx.x, s = blockIdx.x + 1, n = min(kSeedJump, m - s * kSeedJump);
  for (int q = t; q < 624; q += kSeedThreads) ring[q] = state[s * 624 + q];
  __syncthreads();
  seed_walk(ring, n, out + (size_t)s * kSeedJump);
  if (s == kSeedSegs - 1)
    for (int q = t; q < 624; q += kSeedThreads) state[kSeedSegs * 624 + q] = ring[(uint32_t)(n + q) % kSeedRing];
}

// random_index_t (MT:489-503) of one raw word: max(ceiling(h * imax), 1)
// with h = random_number_t's harvest of that word; h * imax rounds as in the
// Fortran (FP64 product, no contraction).
__device__ __forceinline__ int32_t seed_index_of(uint32_t raw, int32_t imax) {
  const double c = ceil(__dmul_rn(u32_unit(temper(raw)), (double)imax));
  return c < 1.0 ? 1 : (int32_t)c;
}

// icsdsw/icsdlw of column ix (GFS_rad_time_vary.fv3.F90:76-82): with
// p = i+isc-1 + (j+jsc-2) cnx (1-based), numrdm(p) and numrdm(p + cnx cny),
// numrdm = random_index(imax) of the face's stream.  A p outside the face
// records the smallest such column in *bad and writes nothing for it.
__global__ void lw_seed_gather_kernel(const uint32_t* __restrict__ raw, const int32_t* __restrict__ imap,
                                      const int32_t* __restrict__ jmap, int n, int isc, int jsc, int cnx,
                                      long long face, int32_t imax, int32_t* icsdsw, int32_t* icsdlw, int* bad) {
  const int ix = blockIdx.x * blockDim.x + threadIdx.x;
  if (ix >= n) return;
  const long long p = (long long)imap[ix] + isc - 1 + ((long long)jmap[ix] + jsc - 2) * cnx;
  if (p < 1 || p > face) {
    atomicMin(bad, ix);
    return;
  }
  icsdsw[ix] = seed_index_of(raw[p - 1], imax);
  icsdlw[ix] = seed_index_of(raw[p - 1 + face], imax);
}

// host side ------------------------------------------------------------------

size_t seed_state_words() { return (size_t)(kSeedSegs + 1) * 624; }

cudaError_t seed_stream_launch(int32_t seed, long long m, uint32_t* raw, uint32_t* state, cudaStream_t st) {
  if (m <= 0) return cudaSuccess;
  if (m > INT_MAX) return cudaErrorInvalidValue;
  const uint32_t s = (uint32_t)(seed == 0 ? 4357 : seed);   // MT:291
  if (m <= kSeedWalk) {
    lw_seed_stream_kernel<<<1, kSeedThreads, 0, st>>>(s, true, (int)m, nullptr, raw);
    return cudaGetLastError();
  }
  constexpr int round = kSeedSegs * kSeedJump;
  for (long long done = 0; done < m; done += round) {
    const int n = (int)std::min<long long>(round, m - done), segs = (n + kSeedJump - 1) / kSeedJump;
    uint32_t* out = raw + done;
    lw_seed_stream_kernel<<<1, kSeedThreads, 0, st>>>(s, done == 0, std::min(n, kSeedJump), state, out);
    if (segs > 1) {
      lw_seed_jump_kernel<<<dim3((kSeedPolyBits + kSeedChunk - 1) / kSeedChunk, segs - 1), kSeedSumThreads, 0, st>>>(state, out);
      lw_seed_segment_kernel<<<segs - 1, kSeedThreads, 0, st>>>(n, state, out);
    }
  }
  return cudaGetLastError();
}

cudaError_t seed_gather_launch(const uint32_t* raw, const int32_t* imap, const int32_t* jmap, int n, int isc,
                               int jsc, int cnx, long long face, int32_t imax, int32_t* icsdsw, int32_t* icsdlw,
                               int* bad, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  lw_seed_gather_kernel<<<(n + 255) / 256, 256, 0, st>>>(raw, imap, jmap, n, isc, jsc, cnx, face, imax, icsdsw,
                                                         icsdlw, bad);
  return cudaGetLastError();
}

// ring words: one round's draws plus a twist block (at least two blocks, for
// iovr 2), a multiple of 624
int mcica_ring_capacity(int nlay) {
  const long need = std::max((long)kMcicaRound * nlay + 623, 1248L);
  return (int)((need + 623) / 624 * 624);
}

cudaError_t mcica_prepare(int max_smem) {
  cudaError_t e = cudaFuncSetAttribute(lw_mcica_kernel<NGPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(lw_mcica_two_set_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(lw_mcica_kernel<kSwNgpt>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
}

cudaError_t mcica_upload_powers() {
  uint32_t pw[32];
  for (int i = 0; i < 32; ++i) pw[i] = pow69069(i);
  return cudaMemcpyToSymbol(c_pow69069, pw, sizeof(pw));
}

cudaError_t mcica_launch(const Block* blocks, int nblocks, const Block& b0, int ncols, int nlay, int iovr, int isubclw,
                         int top_at_1, const McicaStage& stage, uint32_t* bits, int num_sms, cudaStream_t st) {
  McicaArgs a;
  a.nlay = nlay;
  a.nw = (nlay + 31) / 32;
  a.iovr = iovr;
  a.isubclw = isubclw;
  a.top_at_1 = top_at_1;
  a.cap = iovr < 3 ? mcica_ring_capacity(nlay) : 0;
  a.st = stage;
  if (iovr >= 3) {
    if (ncols < 1) return cudaSuccess;
    const size_t smem = TwoSetSmem::bytes(nlay, a.nw) * kTwoSetWarps;
    lw_mcica_two_set_kernel<<<(ncols + kTwoSetWarps - 1) / kTwoSetWarps, 32 * kTwoSetWarps, smem, st>>>(
        blocks, nblocks, b0, ncols, a, bits);
    return cudaGetLastError();
  }
  const int wpb = kMcicaWarps;
  size_t smem = mcica_warp_bytes(nlay, a.cap) * wpb;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lw_mcica_kernel<NGPT>, wpb * 32, smem);
  if (per_sm < 1) per_sm = 1;
  int grid = min((ncols + wpb - 1) / wpb, num_sms * per_sm);
  if (grid < 1) return cudaSuccess;
  lw_mcica_kernel<NGPT><<<grid, wpb * 32, smem, st>>>(blocks, nblocks, b0, ncols, a, bits);
#if LW_DEBUG_CHECKS
  {
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { fprintf(stderr, "lw debug: mcica kernel failed\n"); return e; }
  }
#endif
  return cudaGetLastError();
}

// Shortwave sub-columns with decorrelation-length (iovr 3) or exponential /
// exponential-random (iovr 4, 5) overlap (radsw_main.F90:2101-2198).  Both
// random sets are g-major, set 1 = draws [0, 112 nlay) and set 2 = draws
// [112 nlay, 224 nlay) of one stream, cdfunc(k, n) = draw (n-1) nlay + k, so
// the draws of a g-point lie side by side: lanes are the layers of a 32-layer
// word.  cdfunc(k) = cdfunc(k+1) when cdfun2(k) <= fac_lcf(k+1) (iovr 3), or
// cdfunc(k-1) when cdfun2(k) < alpha(k) (iovr 4, 5): a layer's value is the
// draw of the nearest layer above (below) it that is not linked.  The ballot
// of the broken links names that lane, a shuffle brings its draw, runs that
// cross a word take the value carried from the word before, and the ballot of
// cdfunc(k) >= 1 - cldf(k) is the word of flags.  The comparisons are of
// tempered words with integer thresholds (umin_ge and its like).
// stage.alpha holds fac_lcf (iovr 3, entry k is the factor between layers k-1
// and k) or alpha (iovr 4, 5), per layer in internal order.
//
// Each set is read from its own ring of two twister blocks; set 2's runs 112
// nlay draws ahead.  A g-point needs at most 255 draws, so a block is
// overwritten only once it has been read.
//
// Bound by integer issue.  3,001 columns of 64 layers (1,800 daylit), iovr 3,
// with the kernel that forms fac_lcf: 0.25 ms with a lane per g-point (28 of
// 32 lanes, rings of 28 g-points, draws converted to FP64), 0.11 ms so.
constexpr int kSwTwoSetRing = 1248;
constexpr int kSwTwoSetWarps = 2;   // per CTA, a column each

__host__ __device__ inline size_t sw_two_set_warp_bytes(int nlay) {
  return (2 * (size_t)nlay * 8 + 2 * (size_t)kSwTwoSetRing * 4 + 15) & ~(size_t)15;
}

__global__ void __launch_bounds__(32 * kSwTwoSetWarps)
sw_mcica_two_set_kernel(int ncols, McicaArgs a, uint32_t* __restrict__ bits) {
  extern __shared__ __align__(16) char smem_raw[];
  constexpr uint32_t kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int nlay = a.nlay, nw = a.nw;
  const int c = blockIdx.x * kSwTwoSetWarps + wib;
  if (c >= ncols) return;   // the warps share nothing
  long long* clr = reinterpret_cast<long long*>(smem_raw + sw_two_set_warp_bytes(nlay) * wib);
  long long* aux = clr + nlay;   // layer k is not linked when its set-2 word is >= aux[k]
  uint32_t* ra = reinterpret_cast<uint32_t*>(aux + nlay);
  uint32_t* rb = ra + kSwTwoSetRing;
  for (int k = lane; k < nlay; k += 32) {
    clr[k] = umin_ge(1.0 - a.st.cldf[c + (size_t)a.st.ld * k]);
    if (a.iovr == 3)
      aux[k] = (k == nlay - 1) ? 0 : umax_le(a.st.alpha[c + (size_t)a.st.ld * (k + 1)]) + 1;
    else
      aux[k] = (k == 0) ? 0 : ulim_lt(a.st.alpha[c + (size_t)a.st.ld * k]);
  }
  const int32_t seed = a.st.seed[c];
  uint32_t x = (uint32_t)(seed == 0 ? 4357 : seed) * c_pow69069[lane];   // random_setseed_t (MT:285-299)
  for (int n = lane; n < 624; n += 32) {
    ra[n] = rb[n] = x;
    x *= kPow69069_32;
  }
  __syncwarp();
  // sequence indices: of the g-point's first draw in each set, and generated so far
  int sa = 624, sb = 624 + kSwNgpt * nlay, ga = 624, gb = 624;
  uint32_t* out = bits + (size_t)c * kSwNgpt * nw;
  for (int n = 0; n < kSwNgpt; ++n) {
    while (ga < sa + nlay) {
      twist_ring(ra, kSwTwoSetRing, (ga / 624) & 1 ? 624 : 0, lane);
      ga += 624;
    }
    while (gb < sb + nlay) {
      twist_ring(rb, kSwTwoSetRing, (gb / 624) & 1 ? 624 : 0, lane);
      gb += 624;
    }
    const int qa = sa % kSwTwoSetRing, qb = sb % kSwTwoSetRing;
    uint32_t carry = 0;   // the value at the edge of the word before
    for (int i = 0; i < nw; ++i) {
      const int w = (a.iovr == 3) ? nw - 1 - i : i;
      const int k = 32 * w + lane;
      const bool in = k < nlay;
      uint32_t v = 0, l = 0;
      long long lk = 0, ck = 0;
      if (in) {
        const int ia = qa + k, ib = qb + k;
        v = temper(ra[ia >= kSwTwoSetRing ? ia - kSwTwoSetRing : ia]);
        l = temper(rb[ib >= kSwTwoSetRing ? ib - kSwTwoSetRing : ib]);
        lk = aux[k];
        ck = clr[k];
      }
      const uint32_t brk = __ballot_sync(kAll, in && (long long)l >= lk);
      // the nearest broken link at or above (iovr 3) or at or below this layer
      const uint32_t at = brk & ((a.iovr == 3) ? kAll << lane : kAll >> (31 - lane));
      const int src = (a.iovr == 3) ? __ffs(at) - 1 : 31 - __clz(at);
      const uint32_t got = __shfl_sync(kAll, v, src & 31);
      const uint32_t cdf = at ? got : carry;
      const uint32_t flags = __ballot_sync(kAll, in && (long long)cdf >= ck);
      if (lane == 0) out[n * nw + w] = flags;
      carry = __shfl_sync(kAll, cdf, (a.iovr == 3) ? 0 : 31);
    }
    sa += nlay;
    sb += nlay;
    __syncwarp();   // the reads of a block before it is overwritten
  }
}

cudaError_t mcica_sw_two_set_prepare(int max_smem) {
  return cudaFuncSetAttribute(sw_mcica_two_set_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
}

cudaError_t mcica_sw_two_set_launch(int ncols, int nlay, int iovr, const McicaStage& stage, uint32_t* bits,
                                    cudaStream_t st) {
  if (iovr < 3 || iovr > 5) return cudaErrorInvalidValue;
  McicaArgs a;
  a.nlay = nlay;
  a.nw = (nlay + 31) / 32;
  a.iovr = iovr;
  a.isubclw = 2;
  a.top_at_1 = 0;
  a.cap = 0;
  a.st = stage;
  if (ncols < 1) return cudaSuccess;
  const size_t smem = sw_two_set_warp_bytes(nlay) * kSwTwoSetWarps;
  sw_mcica_two_set_kernel<<<(ncols + kSwTwoSetWarps - 1) / kSwTwoSetWarps, 32 * kSwTwoSetWarps, smem, st>>>(ncols, a,
                                                                                                           bits);
  return cudaGetLastError();
}

// Shortwave sub-columns (mcica_subcol, radsw_main.F90:1952-2212) for iovr 0
// (random), 1 (maximum-random) and 2 (maximum): the draws are g-major,
// rand2d((n-1)*nlay + k) as in the longwave generator, over 112 g-points.
// stage.cldf is the layer cloud fraction floored at ftiny = 1e-12
// (radsw_main.F90:1904-1908), internal (surface-first) order.
cudaError_t mcica_sw_launch(int ncols, int nlay, int iovr, const McicaStage& stage, uint32_t* bits, int num_sms,
                            cudaStream_t st) {
  if (iovr < 0 || iovr > 2) return cudaErrorInvalidValue;
  McicaArgs a;
  a.nlay = nlay;
  a.nw = (nlay + 31) / 32;
  a.iovr = iovr;
  a.isubclw = 2;
  a.top_at_1 = 0;
  a.cap = mcica_ring_capacity(nlay);
  a.st = stage;
  const int wpb = kMcicaWarps;
  size_t smem = mcica_warp_bytes(nlay, a.cap) * wpb;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lw_mcica_kernel<kSwNgpt>, wpb * 32, smem);
  if (per_sm < 1) per_sm = 1;
  int grid = min((ncols + wpb - 1) / wpb, num_sms * per_sm);
  if (grid < 1) return cudaSuccess;
  Block none{};
  lw_mcica_kernel<kSwNgpt><<<grid, wpb * 32, smem, st>>>(nullptr, 0, none, ncols, a, bits);
  return cudaGetLastError();
}

}  // namespace lw
