#pragma once
// pt2_epi.cuh -- k_pt2, the second of the two forward kernels: everything the
// reference does with a perturber once <I|H|Psi> and its diagonal energies are
// known (denominators, E2, norms, selection, histogram, unit-60 records:
// pert1.f:151-295, diexcit.f:304-478), for the candidates that k_cand left.
//
// A CTA owns one work unit at a time; its warps take contiguous parts of the
// unit's slots, pick the candidates among them and run the epilogue on 32 at a
// time.  What bounds it is the FP64 pipe, 16 cycles of an SM per warp
// instruction on GB300, so the epilogue is written for few of those (20 per
// root; 26 counted per 32 perturbers with one root, partly filled warps and all,
// and 55 in one kernel before): reciprocals from the hardware's approximation and
// one third-order step, and sums in fixed point -- integer adds, exact, so
// independent of the order in which warps and CTAs finish, and the E2 sums are
// the class sums' totals.  60 orbitals, S = 2001, an eighth of the generators:
// 3.08 ms, the FP64 pipe 82 % busy.
#include "pt2_kernel.cuh"

namespace cipsi_dev {
namespace {

constexpr int kWtCap = 8;  // spin-flip weights tabulated for lesp < kWtCap

// ------------------------------------------------------------ exact sums
// A lane's sum in units of 2^-kFxUnit as a two's complement integer.  Terms of
// 2^kFxMin to 2^kFxMax have no bit below that unit and are added exactly; larger
// and smaller ones go to tables of their own (fx_out), so that a sum of small
// terms keeps as many places as one of large terms.
struct Fx {
  uint32_t w[kFxWords];
};

__device__ __forceinline__ Fx fx_of(uint4 w, uint32_t top) { return Fx{{w.x, w.y, w.z, w.w, top}}; }

// adds t if 2^kFxMin <= |t| < 2^kFxMax, else nothing
__device__ __forceinline__ void fx_add(Fx& s, double t) {
  const int hi = __double2hiint(t);
  const uint32_t lo = (uint32_t)__double2loint(t);
  const int ex = (hi >> 20) & 0x7ff;
  const uint32_t m1 = ((uint32_t)hi & 0xfffffu) | 0x100000u;
  // |t| = m 2^(ex-1075); bit position of m's lowest bit in the sum
  const int sh = ex - (1075 - kFxUnit);
  const int w = sh >> 5;  // 0, 1, 2
  const uint32_t a0 = __funnelshift_l(0u, lo, sh);
  const uint32_t a1 = __funnelshift_l(lo, m1, sh);
  const uint32_t a2 = __funnelshift_l(m1, 0u, sh);
  const bool w0 = w == 0, w1 = w == 1, w2 = (unsigned)(sh - 64) < (unsigned)(kFxMax - kFxMin - 64);
  uint32_t v0 = w0 ? a0 : 0u;
  uint32_t v1 = w1 ? a0 : (w0 ? a1 : 0u);
  uint32_t v2 = w2 ? a0 : (w1 ? a1 : (w0 ? a2 : 0u));
  uint32_t v3 = w2 ? a1 : (w1 ? a2 : 0u);
  uint32_t v4 = w2 ? a2 : 0u;
  const uint32_t sg = (uint32_t)(hi >> 31);  // s + v, or s - v = s + ~v + 1
  v0 ^= sg;
  v1 ^= sg;
  v2 ^= sg;
  v3 ^= sg;
  v4 ^= sg;
  asm("{\n\t.reg .u32 t;\n\t"
      "add.cc.u32 t, %10, 0xffffffff;\n\t"
      "addc.cc.u32 %0, %0, %5;\n\t"
      "addc.cc.u32 %1, %1, %6;\n\t"
      "addc.cc.u32 %2, %2, %7;\n\t"
      "addc.cc.u32 %3, %3, %8;\n\t"
      "addc.u32 %4, %4, %9;\n\t}"
      : "+r"(s.w[0]), "+r"(s.w[1]), "+r"(s.w[2]), "+r"(s.w[3]), "+r"(s.w[4])
      : "r"(v0), "r"(v1), "r"(v2), "r"(v3), "r"(v4), "r"(sg & 1u));
}

__device__ __forceinline__ int fx_exponent(double t) { return ((__double2hiint(t) >> 20) & 0x7ff) - 1023; }
// high word of |t|; that of every term of the lanes' sums lies in [kFxHiMin, kFxHiMax)
__device__ __forceinline__ int fx_high(double t) { return __double2hiint(t) & 0x7fffffff; }
constexpr int kFxHiMin = (1023 + kFxMin) << 20, kFxHiMax = (1023 + kFxMax) << 20;

// |t| = (hi + lo 2^-64) units into the words g; its sign
__device__ void fx_words(unsigned long long* g, unsigned long long hi, unsigned long long lo, bool neg) {
  unsigned __int128 x = (unsigned __int128)hi << 64 | lo;
  if (neg) x = (unsigned __int128)0 - x;
#pragma unroll 1
  for (int i = 0; i < 3; ++i) {
    atomicAdd(&g[i], (unsigned long long)(uint32_t)x);
    x >>= 32;
  }
  atomicAdd(&g[3], (unsigned long long)(long long)(int32_t)(uint32_t)x);
}
static_assert(kFxWordsHi == 4 && kFxWordsLo == 4, "fx_words writes four");

// a term of 2^kFxMax or more to sum q's own table (exact below 2^62); plain
// FP64 beyond, for infinities and for NaN
__device__ __noinline__ void fx_big(const Params& p, int q, double t) {
  const double a = fabs(t);
  if (!(a < 0x1p62)) {
    atomicAdd(p.sums_big + q, t);
    return;
  }
  // 2^-kFxUnitHi units: the whole part above the lowest 44 bits of the words
  const unsigned long long n = (unsigned long long)a;
  const unsigned long long f = (unsigned long long)((a - trunc(a)) * 0x1p44);
  fx_words(p.sums_hi + (size_t)q * kFxWordsHi, n >> (64 - kFxUnitHi), n << kFxUnitHi | f, t < 0.0);
}
// a sum of up to 32 terms below 2^kFxMin, likewise; plain FP64 below 2^kFxMinLo
__device__ __noinline__ void fx_small(const Params& p, int q, double t) {
  if (t == 0.0) return;
  if (fx_exponent(t) < kFxMinLo) {
    atomicAdd(p.sums_big + q, t);
    return;
  }
  const double a = fabs(t) * 0x1p116;  // whole part: units of 2^64 of the words' 2^-180
  const unsigned long long n = (unsigned long long)a;
  fx_words(p.sums_lo + (size_t)q * kFxWordsLo, n, (unsigned long long)((a - (double)n) * 0x1p64), t < 0.0);
}
static_assert(kFxUnitHi == 44 && kFxUnitLo == 180 && kFxMin == -64, "fx_big and fx_small are written for these");

// The term t of each lane that has one (`mine`) to a table of sum q, if the
// lanes' sums do not take it.  Called by the whole warp.  Small terms are added
// up by sum first, in an order that only the queue decides: couplings that
// vanish but for rounding are many, and thousands of warps would wait for one
// address.
__device__ __noinline__ void fx_out(const Params& p, bool mine, int q, double t) {
  constexpr unsigned kFull = 0xffffffffu;
  const int h = fx_high(t);
  const bool small = mine && h < kFxHiMin;
  if (mine && h >= kFxHiMax) fx_big(p, q, t);
  unsigned rest = __ballot_sync(kFull, small);
#pragma unroll 1
  while (rest) {
    const int src = __ffs((int)rest) - 1;
    const int qs = __shfl_sync(kFull, q, src);
    const bool same = small && q == qs;
    rest &= ~__ballot_sync(kFull, same);
    double s = same ? t : 0.0;
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
    if ((threadIdx.x & 31) == src) fx_small(p, qs, s);
  }
}

// 1/d to within about an ulp: hardware approximation r0 (relative error below
// 2^-19), then r0 (1 + e + e^2) with e = 1 - d r0, a third-order Newton-type
// (Householder) step: error e^3 < 2^-57 before rounding.
__device__ __forceinline__ double recip(double d) {
  double r0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(d));
  const double e = fma(-d, r0, 1.0);
  return fma(r0, fma(e, e, e), r0);
}
// exponent field in [64, 1984): neither d nor 1/d comes near the range's ends
__device__ __forceinline__ bool recip_ok(double d) {
  return (((unsigned)__double2hiint(d) >> 20) & 0x7ffu) - 64u < 1920u;
}

// One perturber's terms of a root: b^2 w / d for the MP, EN and barycentric
// denominators, the norms (b/d)^2 w, and the coefficient the selection looks at
struct Terms {
  double mp, vp, b, pm, pv, c, deno;
};
__device__ __noinline__ Terms terms_by_division(double b, double wgt, double dmp, double dvp, double db) {
  Terms t;
  const double cm = b / dmp;
  t.mp = (b * cm) * wgt;
  t.pm = cm * cm * wgt;
  t.c = b / dvp;
  t.vp = (b * t.c) * wgt;
  t.pv = t.c * t.c * wgt;
  t.b = (b * (b / db)) * wgt;
  return t;
}
// the terms of root m for a coupling b
__device__ __forceinline__ Terms terms_of(const Params& p, int m, double b, double wgt, double hmpi, double hvpi) {
  Terms t;
  const double dmp = p.emp[m] - hmpi;
  if (p.yen) {
    const double dvp = p.e[m] - hvpi, db = p.eb[m] - hvpi;
    if (recip_ok(dmp) && recip_ok(dvp) && recip_ok(db)) {
      const double b2w = (b * b) * wgt;
      const double rm = recip(dmp), rv = recip(dvp);
      t.mp = b2w * rm;
      t.vp = b2w * rv;
      t.b = b2w * recip(db);
      t.pm = t.mp * rm;
      t.pv = t.vp * rv;
      t.c = b * rv;
    } else {  // a denominator at (or near) zero or huge
      t = terms_by_division(b, wgt, dmp, dvp, db);
    }
    t.deno = dvp;
    return t;
  }
  // one quotient, the coefficient that the selection looks at: by division, as
  // every other quotient of the reference (b times the reciprocal is off by up to
  // 1.4 ulp)
  t.c = b / dmp;
  t.mp = (b * t.c) * wgt;
  t.pm = t.c * t.c * wgt;
  t.vp = t.b = t.pv = 0.0;
  t.deno = dmp;
  return t;
}
// all of them fit the lanes' sums
__device__ __forceinline__ bool terms_in(const Params& p, const Terms& t, double b) {
  int lo = min(fx_high(t.mp), fx_high(t.pm)), hi = max(fx_high(t.mp), fx_high(t.pm));
  if (p.yen) {
    lo = min(min(lo, fx_high(t.vp)), min(fx_high(t.b), fx_high(t.pv)));
    hi = max(max(hi, fx_high(t.vp)), max(fx_high(t.b), fx_high(t.pv)));
  }
  return (lo >= kFxHiMin && hi < kFxHiMax) || (__double_as_longlong(b) << 1) == 0;
}
// those of root m, class ct, that do not, to the global tables (of the lanes that
// have some: `mine`); called by the whole warp
__device__ __noinline__ void odd_terms(const Params& p, bool mine, int m, int ct, double b, double wgt, double hmpi,
                                       double hvpi) {
  Terms t{};
  if (mine) t = terms_of(p, m, b, wgt, hmpi, hvpi);
  fx_out(p, mine, fx_tab(0, ct, m), t.mp);
  fx_out(p, mine, fx_acc(1, m), t.pm);
  if (!p.yen) return;
  fx_out(p, mine, fx_tab(1, ct, m), t.vp);
  fx_out(p, mine, fx_acc(0, m), t.b);
  fx_out(p, mine, fx_acc(2, m), t.pv);
}
__device__ __noinline__ double spin_weight_any(int nespf, int lesp) { return spin_weight(nespf, lesp); }

// tests of run parameters on their bits too: an FP64 compare takes as long as an
// addition
constexpr long long kBitsOne = 0x3ff0000000000000ll;
__device__ __forceinline__ bool below_zero(double x) {
  return __double_as_longlong(x) < 0 && (__double_as_longlong(x) << 1) != 0;
}

// one lane sum over the warp, added to global sum q (words of 32 bits in
// 64-bit counters: carries are resolved when the sums are converted)
__device__ __noinline__ void flush_fx(const Params& p, Fx s, int q) {
  constexpr unsigned kFull = 0xffffffffu;
  if (!__any_sync(kFull, (s.w[0] | s.w[1] | s.w[2] | s.w[3] | s.w[4]) != 0u)) return;
#pragma unroll
  for (int i = 0; i < kFxWords; ++i) {
    // 32 words summed as two 16-bit halves in 32-bit lanes
    const uint32_t x = s.w[i];
    const long long lo = (long long)__reduce_add_sync(kFull, x & 0xffffu);
    const long long hi = i < kFxWords - 1 ? (long long)__reduce_add_sync(kFull, x >> 16)
                                          : (long long)__reduce_add_sync(kFull, (int)x >> 16);
    const long long v = lo + hi * 65536;
    if ((threadIdx.x & 31) == 0 && v != 0) atomicAdd(&p.sums[(size_t)q * kFxWords + i], (unsigned long long)v);
  }
}

__device__ __noinline__ int hist_class_exact(const Params& p, double val) { return hist_class(p, val); }

// histogram class of a non-negative value, as hist_class; high words first
__device__ __forceinline__ int hist_class_hi(const Params& p, double val) {
  const int hv = __double2hiint(val);
  int c = 0;
  bool tie = false;
#pragma unroll
  for (int i = 0; i < kNClass - 1; ++i) {
    const int ha = p.aval_hi[i];
    c += hv > ha ? 1 : 0;
    tie = tie || hv == ha;
  }
  return tie ? hist_class_exact(p, val) : c;
}

struct EpiShared {
  double wt[2][kWtCap];  // 1 + fmul
  int nm[2][kWtCap];     // nmul
  uint64_t kbits[4];
  long long unit_base;   // pool segment of the unit being compacted
  int unit;
  int tmp[kWarps];
  uint32_t q_slot[kWarps][64], q_meta[kWarps][64];      // candidates awaiting their epilogue
  uint32_t hn[kWarps][(kNClass + 1) * (1 + kMaxRoots)];  // histogram counts: nom, then nam per root
};

// CTAs per SM by the registers that the sums of R roots want
template <int R>
constexpr int kEpiCtas = R <= 2 ? 3 : 2;

template <int W, int R, bool B>
__global__ void __launch_bounds__(kThreads, kEpiCtas<R>) k_pt2(Params p0, LaunchArgs la) {
  constexpr unsigned kFull = 0xffffffffu;
  // the current geometry's parameters, in shared memory (device functions
  // then read them through a shared-memory reference instead of a local
  // copy of the kernel argument)
  __shared__ Params sgeo;
  const Params& p = sgeo;
  __shared__ EpiShared sh;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const unsigned below = (1u << lane) - 1u;
  uint32_t* const q_slot = sh.q_slot[wid];
  uint32_t* const q_meta = sh.q_meta[wid];
  if (!B) {
    if (tid == 0) sgeo = p0;
    __syncthreads();
  }
  int cur_geo = -1;

  // lane sums: by class the MP and EN terms (class kNClass: terms outside the
  // histogram), then e2b, psimp, psivp
  // (the tables in local memory: four words of a sum are one access, the top
  // words of both another)
  uint4 tab[kNClass + 1][R][2];
  uint2 top[kNClass + 1][R];
  // classes that the lane has terms of; the rows of the others are not touched
  // (all of them, of all resident threads, are 50 MB to clear and to read again,
  // 270 with eight roots: 33 and 140 us of a run that has few perturbers)
  unsigned held = 0u;
  Fx acc[3][R];
  unsigned long long ietat = 0;
  unsigned int nproc = 0, nsel = 0;
  double dpivot = 0.0;
  auto zero_sums = [&]() {
    held = 0u;
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int m = 0; m < R; ++m) acc[q][m] = Fx{};
#pragma unroll 1
    for (int i = lane; i < (kNClass + 1) * (1 + R); i += 32) sh.hn[wid][i] = 0u;
    ietat = 0ull;
    nproc = nsel = 0u;
    dpivot = 0.0;
    __syncwarp();
  };
  zero_sums();

  // the warp's sums and counters into the geometry's; then zero
  auto flush_geometry = [&]() {
    const unsigned classes = __reduce_or_sync(kFull, held);
#pragma unroll 1
    for (int i = 0; i < (kNClass + 1) * R; ++i) {
      const int c = i / R, m = i % R;
      if (!((classes >> c) & 1u) || m >= p.metat) continue;
      const bool mine = (held >> c) & 1u;
      const uint2 t = mine ? top[c][m] : make_uint2(0u, 0u);
      flush_fx(p, mine ? fx_of(tab[c][m][0], t.x) : Fx{}, fx_tab(0, c, m));
      flush_fx(p, mine ? fx_of(tab[c][m][1], t.y) : Fx{}, fx_tab(1, c, m));
    }
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int m = 0; m < R; ++m)
        if (m < p.metat) flush_fx(p, acc[q][m], fx_acc(q, m));
    unsigned long long it = ietat, db = __double_as_longlong(dpivot);
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) {
      it += __shfl_xor_sync(kFull, it, o);
      const unsigned long long y = __shfl_xor_sync(kFull, db, o);
      db = y > db ? y : db;
    }
    const unsigned long long pr = (unsigned long long)__reduce_add_sync(kFull, nproc & 0xffffu) +
                                  ((unsigned long long)__reduce_add_sync(kFull, nproc >> 16) << 16);
    const unsigned long long se = (unsigned long long)__reduce_add_sync(kFull, nsel & 0xffffu) +
                                  ((unsigned long long)__reduce_add_sync(kFull, nsel >> 16) << 16);
    if (lane == 0) {
      if (it) atomicAdd(&p.counters[C_IETAT], it);
      if (pr) atomicAdd(&p.counters[C_NPROC], pr);
      if (se) atomicAdd(&p.counters[C_NSEL], se);
      if (db) atomicMax(p.dpivot_bits, db);
    }
    __syncwarp();
#pragma unroll 1
    for (int c = lane; c < p.nclass; c += 32) {
      if (sh.hn[wid][c]) atomicAdd(&p.hist_nom[c], (unsigned long long)sh.hn[wid][c]);
#pragma unroll
      for (int m = 0; m < R; ++m) {
        const uint32_t x = sh.hn[wid][(kNClass + 1) * (1 + m) + c];
        if (m < p.metat && x) atomicAdd(&p.hist_nam[c * p.metat + m], (unsigned long long)x);
      }
    }
    __syncwarp();
    zero_sums();
  };

#pragma unroll 1
  for (;;) {
    __syncthreads();
    if (tid == 0) sh.unit = atomicAdd(&la.work[1], 1);
    __syncthreads();
    int unit = sh.unit;
    if (unit >= la.nunits) break;
    const long long slot0 = la.unit_slot[unit];
    const int nslots = la.unit_nslots[unit];
    if (B) {
      const int gi = la.unit_geo[unit];
      if (gi != cur_geo) {
        if (cur_geo >= 0) flush_geometry();
        __syncthreads();
        const int* src = reinterpret_cast<const int*>(la.geo + gi);
        int* dst = reinterpret_cast<int*>(&sgeo);
#pragma unroll 1
        for (int i = tid; i < (int)(sizeof(Params) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
        __syncthreads();
        cur_geo = gi;
      }
      unit = la.unit_local[unit];
    }
    const int k = p.gens[p.unit_g[unit]];
    const int nespk = k < 0 ? 0 : p.nesp[k];
    if (tid < 2 * W) {
      const int n = min(max(p.noca - (tid % W) * 64, 0), 64);
      sh.kbits[tid] = k < 0 ? ((n >= 64) ? ~0ull : ((1ull << n) - 1ull)) : p.S[(size_t)k * 2 * W + tid];
    }
    if (tid < 2 * kWtCap) {
      const int kind = tid / kWtCap, lesp = tid % kWtCap;
      const double fm = spin_weight_any(kind ? 2 * nespk + 1 : nespk, lesp);
      sh.wt[kind][lesp] = 1.0 + fm;
      sh.nm[kind][lesp] = (int)fm;
    }
    __syncthreads();
    // ---- this warp's part of the slots (whole groups of 32)
    const int per = ((nslots + kThreads - 1) / kThreads) * 32;
    const int s1 = min(nslots, (wid + 1) * per);
    int qn = 0;
    bool anysel = false;
    // denominators, E2, selection, histogram, unit-60 record of the last cnt
    // queued candidates (pert1.f:171-295, diexcit.f:327-478)
    auto epilogue = [&](int cnt) {
      const bool live = lane < cnt;
      qn -= cnt;
      const int e = qn + (live ? lane : 0);
      const long long s = slot0 + q_slot[e];
      const uint32_t flag = q_meta[e];
      const double hmpi = live ? la.cand.mp[s] : 0.0, hvpi = live && p.yen ? la.cand.vp[s] : 0.0;
      const int lesp = (int)(flag >> 8), wk = (flag & kMWt1) ? 1 : 0;
      double wgt;
      int nmul;
      if (lesp < kWtCap) {
        wgt = sh.wt[wk][lesp];
        nmul = sh.nm[wk][lesp];
      } else {
        const double fm = spin_weight_any(wk ? 2 * nespk + 1 : nespk, lesp);
        wgt = 1.0 + fm;
        nmul = (int)fm;
      }
      double tmp[R], tvp[R], vil[R], xam = 0.0;
      bool ydeg = false;
      unsigned odd = 0u;  // roots with a term that the lane's sums do not take
#pragma unroll
      for (int m = 0; m < R; ++m) {
        tmp[m] = tvp[m] = vil[m] = 0.0;
        if (!live || m >= p.metat) continue;
        const double b = la.cand.b[m * la.cand.cap + s];
        const Terms t = terms_of(p, m, b, wgt, hmpi, hvpi);
        tmp[m] = t.mp;
        tvp[m] = t.vp;
        if (p.yen) {
          fx_add(acc[0][m], t.b);
          fx_add(acc[2][m], t.pv);
        }
        fx_add(acc[1][m], t.pm);
        if (!terms_in(p, t, b)) odd |= 1u << m;
        // comparisons of magnitudes on their IEEE bit patterns (exact for
        // non-negative doubles; NaN compares as in the reference: never below)
        const long long bdeno = __double_as_longlong(t.deno) & 0x7fffffffffffffffll;
        if (p.ywdeg && !(bdeno > kBits005 && bdeno <= kBitsInf)) {
          const long long beim = __double_as_longlong(b * t.c) & 0x7fffffffffffffffll;
          if (!(beim < kBits1em6)) ydeg = true;
        }
        double xim = fabs(t.c);
        if (p.ysele) xim = fabs(b * t.c);
        if (lt_nonneg(xim, p.teste[m])) dpivot = max_nonneg(dpivot, xim);
        if (p.ymoyen) {
          if (__double_as_longlong(p.taum[m]) != kBitsOne) xim *= p.taum[m];
          vil[m] = xim;
          xam = max_nonneg(xam, xim);
        }
      }
      // histogram (cip/isto.f; pert1 calls it always, diexcit only if ymoyen)
      const bool all = __double_as_longlong(p.teseff) <= 0;
      const bool hist = live && (!(flag & kMD2) || p.ymoyen) &&
                        (all || __double_as_longlong(xam) >= __double_as_longlong(p.teseff));
      const int cls = hist ? hist_class_hi(p, xam) : kNClass;
      auto class_of = [&](int m) { return hist && (all || !lt_nonneg(vil[m], p.teseff)) ? cls : kNClass; };
      if (live) {
        ietat += (unsigned long long)(long long)(nmul + 1);
        nproc += 1u;
        if (hist) atomicAdd(&sh.hn[wid][cls], (uint32_t)(1 + nmul));
#pragma unroll
        for (int m = 0; m < R; ++m) {
          if (m >= p.metat) continue;
          const int ct = class_of(m);
          if (ct < kNClass)
            atomicAdd(&sh.hn[wid][(kNClass + 1) * (1 + m) + (R == 1 ? cls : hist_class_hi(p, vil[m]))], (uint32_t)(1 + nmul));
          if (!((held >> ct) & 1u)) {
            held |= 1u << ct;
#pragma unroll 1
            for (int i = 0; i < R; ++i) {
              tab[ct][i][0] = tab[ct][i][1] = make_uint4(0u, 0u, 0u, 0u);
              top[ct][i] = make_uint2(0u, 0u);
            }
          }
          uint2 top2 = top[ct][m];
          Fx f = fx_of(tab[ct][m][0], top2.x);
          fx_add(f, tmp[m]);
          tab[ct][m][0] = make_uint4(f.w[0], f.w[1], f.w[2], f.w[3]);
          top2.x = f.w[4];
          if (p.yen) {
            f = fx_of(tab[ct][m][1], top2.y);
            fx_add(f, tvp[m]);
            tab[ct][m][1] = make_uint4(f.w[0], f.w[1], f.w[2], f.w[3]);
            top2.y = f.w[4];
          }
          top[ct][m] = top2;
        }
      }
      if (__any_sync(kFull, odd != 0u)) {
#pragma unroll
        for (int m = 0; m < R; ++m) {
          if (m >= p.metat) continue;
          const bool mine = (odd >> m) & 1u;
          odd_terms(p, mine, m, class_of(m), mine ? la.cand.b[m * la.cand.cap + s] : 0.0, wgt, hmpi, hvpi);
        }
      }
      if (ydeg) xam = 1.0;
      // unit-60 record (pie.f): counted; its values stay at the candidate's slot
      // until the unit is done
      const bool sel = live && p.ymoyen &&
                       (below_zero(p.tau) || __double_as_longlong(xam) > (__double_as_longlong(p.tau) & 0x7fffffffffffffffll));
      if (sel) {
        ++nsel;
        if (p.rec_mode) {
          la.cand.mp[s] = xam;
          // ENvp per root written by cipsym (cipsym/pert1.f:244): eivp*(fmul+1)
#pragma unroll
          for (int m = 0; m < R; ++m)
            if (m < p.metat) la.cand.b[m * la.cand.cap + s] = p.symvar ? tvp[m] : 0.0;
          la.cand.meta[s] = flag | kMSel;
          anysel = true;
        }
      }
      __syncwarp();
    };

    for (int s0 = wid * per; s0 < s1 || qn > 0; s0 += 32) {
      if (s0 < s1) {
        const int s = s0 + lane;
        const uint32_t meta = s < s1 ? la.cand.meta[slot0 + s] : 0u;
        const unsigned lm = __ballot_sync(kFull, meta != 0u);
        if (meta) {
          const int at = qn + __popc(lm & below);
          q_slot[at] = (uint32_t)s;
          q_meta[at] = meta;
        }
        qn += __popc(lm);
        __syncwarp();
      }
      if (qn >= 32 || (s0 + 32 >= s1 && qn > 0)) epilogue(min(qn, 32));
    }
    if (!p.rec_mode) continue;
    // ---- the unit's records, in slot order, to one segment of the pool
    // (records beyond its capacity are counted but not stored: the host sees
    // pool_count > pool_cap)
    int cnt = 0;
    if (__syncthreads_or(anysel)) {
#pragma unroll 1
      for (int s = wid * per; s < s1; s += 32)
        cnt += __popc(__ballot_sync(kFull, s + lane < s1 && (la.cand.meta[slot0 + s + lane] & kMSel)));
    }
    if (lane == 0) sh.tmp[wid] = cnt;
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      before += w < wid ? sh.tmp[w] : 0;
      total += sh.tmp[w];
    }
    if (tid == 0) {
      sh.unit_base = total ? (long long)atomicAdd(p.pool_count, (unsigned long long)total) : 0ll;
      p.unit_pool[unit] = sh.unit_base;
      p.unit_nsel[unit] = total;
    }
    __syncthreads();
    if (cnt == 0) continue;
    long long pos = sh.unit_base + before;
#pragma unroll 1
    for (int s0 = wid * per; s0 < s1; s0 += 32) {
      const bool sel = s0 + lane < s1 && (la.cand.meta[slot0 + s0 + lane] & kMSel);
      const unsigned lm = __ballot_sync(kFull, sel);
      const long long d = pos + __popc(lm & below);
      if (sel && d < p.pool_cap) {
        const long long s = slot0 + s0 + lane;
        uint64_t u[2 * W];
#pragma unroll
        for (int q = 0; q < 2 * W; ++q) u[q] = sh.kbits[q];
        const uint32_t code = la.cand.code[s];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int cc = (int)((code >> (8 * t)) & 0xffu);
          const int sp = cc >= p.norb ? 1 : 0, o = cc - sp * p.norb;
#pragma unroll
          for (int q = 0; q < 2 * W; ++q) u[q] ^= q == sp * W + (o >> 6) ? 1ull << (o & 63) : 0ull;
        }
#pragma unroll
        for (int q = 0; q < 2 * W; ++q) p.pool_bits[(size_t)d * 2 * W + q] = u[q];
        p.pool_xam[d] = la.cand.mp[s];
#pragma unroll
        for (int m = 0; m < R; ++m)
          if (m < p.metat) p.pool_evp[(size_t)d * p.metat + m] = la.cand.b[m * la.cand.cap + s];
      }
      pos += __popc(lm);
    }
  }
  if (!B || cur_geo >= 0) flush_geometry();
}

}  // namespace

template <int W, int R, bool B>
cudaError_t launch_pt2(const Params& p, const LaunchArgs& la, int sms, cudaStream_t st) {
  const int grid = min(la.nunits, sms * kEpiCtas<R>);
  if (grid < 1) return cudaSuccess;
  k_pt2<W, R, B><<<grid, kThreads, 0, st>>>(p, la);
  return cudaGetLastError();
}

}  // namespace cipsi_dev
