#pragma once
// pt2_fwd.cuh -- k_cand, the first of the two forward kernels (the work of
// cip/pertu.f + cip/diexcit.f up to a candidate's <I|H|Psi> and diagonal
// energies; k_pt2 of pt2_epi.cuh does the rest); compiled in pt2_w1.cu and
// pt2_w2.cu for 1 and 2 words per spin string.  Bitstring helpers, matrix
// elements and the adjoint kernel are in pt2_kernel.cuh.
//
// A CTA owns one work unit at a time (a generator k and a range of its
// blocks of removed electrons R); its warps then work on their own:
//
//   * a warp takes a block R, collects L_R (the determinants of S that can be
//     within two excitations of some I = K' + A, K' = k - R) in its own shared
//     memory and goes through the block row by row: a row fixes the first
//     added spin orbital a1, its columns are the second one a2.  No barrier:
//     the blocks of a unit differ by orders of magnitude in |L_R|.
//   * entries of L_R below k own the candidates they touch: the whole block, a
//     row, a column or single candidates, marked once per block, before any
//     matrix element is formed.  The entries above k are looked at once per
//     group of rows, by lanes: most touch no column, some one to three (they
//     hold a2 as well), a few all of them.  They give (candidate, determinant)
//     events, evaluated 32 at a time with the warp in step.  (Comparing every
//     candidate with every entry took 45-180 compares and 3700 warp
//     instructions per 32 candidates on the 60-orbital system.)
//   * <I|H|k> itself, the only element of most candidates, needs no
//     bitstrings: two pair indices, one or two integrals and the parities of
//     the four orbitals with respect to K'.
//   * a candidate leaves through the candidate buffer (24 + 8 roots bytes), so
//     that this kernel holds no FP64 epilogue: in one kernel the warps' code
//     did not fit the instruction cache (4 of 14 cycles per instruction waited
//     for it) and the class sums crowded L1.
#include "pt2_kernel.cuh"

namespace cipsi_dev {
namespace {

constexpr int kShareNb = 256;  // neighbours of a generator from which on a lone block's L_R is built once
constexpr int kWindow = 256;  // blocks of a unit laid out in shared memory at a time
// a column of the rows worked together: element found, one not zero, lesp
constexpr uint32_t kXHas = 0x8000u, kXNz = 0x4000u, kXLesp = 0x3fffu;

struct UnitShared {
  uint64_t kbits[4];
  uint64_t occcol[2][2];  // columns whose orbital is occupied in the reference
  uint64_t symcol[2][kMaxSym][2];
  int occ[kMaxElec];      // spin orbital code (orb + spin*norb) of k's electrons
  int nel_s[2], nvir[2];
  int unit, job, nbig, nblk, slots;
  int blk_slot[kWindow];
  int tmp[2 * kWarps + 16];
  uint16_t blk_r[kWindow];
  uint16_t big[kWindow];
  uint8_t vir[2][kMaxOrb];
  uint8_t colof[2 * kMaxOrb];  // column of an empty spin orbital, 255: occupied
};

// electrons e1 (< e2) of R block r among nel electrons
__device__ __forceinline__ void block_electrons(int r, int nel, int& e1, int& e2) {
  if (r < nel) {
    e1 = r;
    e2 = -1;
    return;
  }
  int t = r - nel;
  e1 = 0;
#pragma unroll 1
  while (t >= nel - 1 - e1) {
    t -= nel - 1 - e1;
    ++e1;
  }
  e2 = e1 + 1 + t;
}

// a real*4 widened to double with integer operations (the conversion
// instruction takes the FP64 pipe); denormals and infinities by the instruction
__device__ __forceinline__ double widen(float f) {
  const uint32_t u = __float_as_uint(f);
  const uint32_t mag = u & 0x7fffffffu;
  if (mag == 0u) return 0.0;
  if (mag - 0x00800000u >= 0x7f000000u) return (double)f;
  return __hiloint2double((int)((u & 0x80000000u) | ((mag >> 3) + 0x38000000u)), (int)(u << 29));
}

// (pq|rs) from two entries of the pair table; zero across irreps
__device__ __forceinline__ double ai_pairs(const Params& p, int pij, int pkl) {
  const int s1 = pij >> 24;
  if (s1 != (pkl >> 24)) return 0.0;
  const int a = pij & 0xFFFFFF, b = pkl & 0xFFFFFF;
  const int lo = min(a, b), hi = max(a, b);
  const int idx = lo + ((hi * (hi - 1)) >> 1) + __ldg(&p.ntttt[s1]) - 2;
  if (p.eri64) return __ldg(&p.eri64[idx]);
  return widen(__ldg(&p.eri[idx]));
}

// bit b of the result: parity of the set bits of x below b
__device__ __forceinline__ uint64_t parity_below(uint64_t x) {
  x <<= 1;
  x ^= x << 1;
  x ^= x << 2;
  x ^= x << 4;
  x ^= x << 8;
  x ^= x << 16;
  x ^= x << 32;
  return x;
}

// Out of line: what is called rarely or from several places.  The kernel's hot
// loops have to stay small (at 300 KB of code, a quarter of the issue slots
// waited for instructions).
template <int W>
struct Bits {
  uint64_t w[2 * W];
};

// <I|H|j> of two determinants one spin orbital apart, as hmat (the same terms
// in the same order) with one code site for the sum over the changed orbitals
// of the more excited one
template <int W>
__device__ __noinline__ double element_single(const Params& p, Bits<W> u, int j) {
  const int norb = p.norb;
  int rankI = 0, rankJ = 0, pp = 0, qq = 0, s = 0;
  Bits<W> v;
#pragma unroll
  for (int q = 0; q < 2 * W; ++q) {
    const int n = min(max(p.noca - (q % W) * 64, 0), 64);
    const uint64_t hf = (n >= 64) ? ~0ull : ((1ull << n) - 1ull);
    v.w[q] = __ldg(&p.S[(size_t)j * 2 * W + q]);
    rankI += __popcll(hf & ~u.w[q]);
    rankJ += __popcll(hf & ~v.w[q]);
    const uint64_t gone = v.w[q] & ~u.w[q], come = u.w[q] & ~v.w[q];
    if (gone) {
      pp = (q % W) * 64 + __ffsll((long long)gone) - 1;
      s = q / W;
    }
    if (come) qq = (q % W) * 64 + __ffsll((long long)come) - 1;
  }
  uint64_t vs[W];
  pick_spin<W>(v.w, s, vs);
  const bool odd = popc_between<W>(vs, min(pp, qq), max(pp, qq)) & 1;
  double val = __ldg(&p.F[tri(pp, qq)]);
  const int pq = __ldg(&p.pairtab[pp * norb + qq]);
#pragma unroll 1
  for (int q = 0; q < 2 * W; ++q) {
    const int n = min(max(p.noca - (q % W) * 64, 0), 64);
    const uint64_t hf = (n >= 64) ? ~0ull : ((1ull << n) - 1ull);
    const uint64_t D = rankI > rankJ ? get_word<2 * W>(u.w, q) : get_word<2 * W>(v.w, q);
    uint64_t d = D ^ hf;
#pragma unroll 1
    while (d) {
      const int b = __ffsll((long long)d) - 1;
      d &= d - 1;
      const int r = (q % W) * 64 + b;
      const bool hole = !((D >> b) & 1ull);
      const double x = ai_pairs(p, pq, __ldg(&p.pairtab[r * norb + r]));
      val = hole ? val - x : val + x;
      if (q / W == s) {
        const double y = ai_pairs(p, __ldg(&p.pairtab[pp * norb + r]), __ldg(&p.pairtab[qq * norb + r]));
        val = hole ? val + y : val - y;
      }
    }
  }
  return odd ? -val : val;
}

// An L_R entry for K': x: E = j \ K', one spin orbital code per byte, ascending
// (unused bytes repeat the first code); y: j; z: the holes H = K' \ j (up to
// two codes), |K' \ j| << 16.
template <int W>
__device__ __noinline__ uint3 make_entry(const Params& p, Bits<W> kp, int j) {
  uint32_t eb = 0, hb = 0;
  int ne = 0, nh = 0;
#pragma unroll
  for (int q = 0; q < 2 * W; ++q) {
    const uint64_t sj = __ldg(&p.S[(size_t)j * 2 * W + q]);
    const int base = (q % W) * 64 + (q / W) * p.norb;
    uint64_t d = sj ^ kp.w[q];
#pragma unroll 1
    while (d) {
      const int b = __ffsll((long long)d) - 1;
      d &= d - 1;
      if ((sj >> b) & 1ull) {
        if (ne < 4) eb |= (uint32_t)(base + b) << (8 * ne);
        ++ne;
      } else {
        if (nh < 2) hb |= (uint32_t)(base + b) << (8 * nh);
        ++nh;
      }
    }
  }
  const uint32_t first = eb & 0xffu;
  if (ne < 2) eb |= first << 8;
  if (ne < 3) eb |= first << 16;
  if (ne < 4) eb |= first << 24;
  return make_uint3(eb, (uint32_t)j, hb | (uint32_t)nh << 16);
}

struct Elem {
  double h;
  int kind;  // differences
};
// <I|H|j>, I = K' + {a1, a2} (codes; a1c < 0 in a single block) and the entry
// (E, H, m) of j.  Two differences: P = I \ j = H + (A \ E) and Q = j \ I =
// E \ A, both ascending, the sign from the parities of their positions in the
// common core K' - H + (A and E); par: parities of the electrons of K'.
template <int W>
__device__ __noinline__ Elem element_of(const Params& p, const uint64_t* par, Bits<W> kp, int a1c, int a2c, uint32_t E,
                                        uint2 jh) {
  const int norb = p.norb;
  const int m = (int)(jh.y >> 16);
  const int ne = (a1c >= 0 ? 2 : 1) + m;
  int q1 = -1, q2 = -1, nq = 0, in1 = -1, in2 = -1;
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const int code = (E >> (8 * x)) & 0xff;
    if (x < ne) {
      if (code == a1c) {
        in1 = code;
      } else if (code == a2c) {
        in2 = code;
      } else {
        q1 = nq == 0 ? code : q1;
        q2 = nq == 1 ? code : q2;
        ++nq;
      }
    }
  }
  Elem r;
  auto orb_of = [&](int c) { return c >= norb ? c - norb : c; };
  if (nq == 1) {
    if (a1c >= 0) or_word<2 * W>(kp.w, (a1c >= norb ? W : 0) + (orb_of(a1c) >> 6), 1ull << (orb_of(a1c) & 63));
    or_word<2 * W>(kp.w, (a2c >= norb ? W : 0) + (orb_of(a2c) >> 6), 1ull << (orb_of(a2c) & 63));
    r.h = element_single<W>(p, kp, (int)jh.x);
    r.kind = 1;
    return r;
  }
  r.kind = 2;
  const int h1 = m >= 1 ? (int)(jh.y & 0xffu) : -1, h2 = m >= 2 ? (int)((jh.y >> 8) & 0xffu) : -1;
  int p1 = h1, p2 = h2;
  if (m == 0) {
    p1 = a1c;
    p2 = a2c;
  } else if (m == 1) {
    p2 = a1c >= 0 && in1 < 0 ? a1c : a2c;
  }
  if (p1 > p2) {
    const int t = p1;
    p1 = p2;
    p2 = t;
  }
  auto par_of = [&](int c) -> uint32_t {
    const int o = orb_of(c);
    return (uint32_t)(par[(c >= norb ? W : 0) + (o >> 6)] >> (o & 63)) & 1u;
  };
  uint32_t odd = par_of(p1) ^ par_of(p2) ^ par_of(q1) ^ par_of(q2);
  // each hole and each common added orbital counts for the orbitals of its
  // spin above it
  auto above = [&](int c) -> uint32_t {
    const bool s = c >= norb;
    return (uint32_t)(((p1 >= norb) == s && p1 > c) ^ ((p2 >= norb) == s && p2 > c) ^ ((q1 >= norb) == s && q1 > c) ^
                      ((q2 >= norb) == s && q2 > c));
  };
  if (h1 >= 0) odd ^= above(h1);
  if (h2 >= 0) odd ^= above(h2);
  if (in1 >= 0) odd ^= above(in1);
  if (in2 >= 0) odd ^= above(in2);
  const int op1 = orb_of(p1), op2 = orb_of(p2), oq1 = orb_of(q1), oq2 = orb_of(q2);
  double v = ai_pairs(p, __ldg(&p.pairtab[oq1 * norb + op1]), __ldg(&p.pairtab[oq2 * norb + op2]));
  if ((p1 >= norb) == (p2 >= norb))
    v -= ai_pairs(p, __ldg(&p.pairtab[oq1 * norb + op2]), __ldg(&p.pairtab[oq2 * norb + op1]));
  r.h = __hiloint2double(__double2hiint(v) ^ (int)(odd << 31), __double2loint(v));
  return r;
}

// Candidate t of pertu (pertu.f:62-108: the reference and its singles, no owner
// test): false when it is none, in S or meets nothing.
template <int W, int R>
struct PertuOut {
  double bc[R], hmp, hvp;
  uint32_t code;
  unsigned n1, n2, ncmp;
  bool cand, live;
};
template <int W, int R>
__device__ __noinline__ void pertu_candidate(const Params& p, int t, PertuOut<W, R>& o) {
  const int no = p.noca, nv = p.norb - p.noca;
  uint64_t hf[2 * W];
  Bits<W> u;
#pragma unroll
  for (int q = 0; q < 2 * W; ++q) {
    const int n = min(max(p.noca - (q % W) * 64, 0), 64);
    u.w[q] = hf[q] = (n >= 64) ? ~0ull : ((1ull << n) - 1ull);
  }
  o.cand = true;
  o.code = 0;
  o.n1 = o.n2 = o.ncmp = 0;
  o.hmp = o.hvp = 0.0;
#pragma unroll
  for (int m = 0; m < R; ++m) o.bc[m] = 0.0;
  const int tt = p.pertu_ref ? t - 1 : t;  // tt < 0: the reference itself
  if (tt >= 0) {
    const int s = tt / (no * nv);
    const int rem = tt % (no * nv);
    const int h = rem / nv, v = no + rem % nv;
    o.cand = p.its[p.orbsym[h]][p.orbsym[v]] == p.isym - 1;
    clear_word<2 * W>(u.w, s * W + (h >> 6), 1ull << (h & 63));
    or_word<2 * W>(u.w, s * W + (v >> 6), 1ull << (v & 63));
    o.code = (uint32_t)(h + s * p.norb) | (uint32_t)(v + s * p.norb) << 8;
  }
  o.live = o.cand;
  if (!o.cand) return;
#pragma unroll 1
  for (int j = 0; j < p.ncf; ++j) {
    int x = 0;
#pragma unroll
    for (int q = 0; q < 2 * W; ++q) x += __popcll(u.w[q] ^ __ldg(&p.S[(size_t)j * 2 * W + q]));
    ++o.ncmp;
    if (x > 4) continue;
    if (x == 0) {
      o.live = false;
      break;
    }
    int kind;
    uint64_t v[2 * W];
    int rankI = 0, rankJ = 0;
#pragma unroll
    for (int q = 0; q < 2 * W; ++q) {
      v[q] = __ldg(&p.S[(size_t)j * 2 * W + q]);
      rankI += __popcll(hf[q] & ~u.w[q]);
      rankJ += __popcll(hf[q] & ~v[q]);
    }
    const double h = hmat<W>(p, u.w, v, rankI, rankJ, hf, kind);
    if (kind == 1) ++o.n1; else ++o.n2;
#pragma unroll
    for (int m = 0; m < R; ++m)
      if (m < p.metat) o.bc[m] += h * __ldg(&p.c[(size_t)j * p.metat + m]);
  }
  if (o.n1 + o.n2 == 0) o.live = false;
  if (o.live) diag_terms<W>(p, u.w, hf, o.hmp, o.hvp, p.yen != 0);
}

// CTAs per SM: two where shared memory allows (7.5 KB of it static and the
// system's 1 KB per CTA).  Three would fit for one-word strings, but 85
// registers a thread and 24 warps' code in the instruction cache cost more than
// the warps hide (60 orbitals, S = 2001: 55 ms against 47; 45 orbitals: 8.5
// against 6.0).
template <int W, int R>
constexpr int kCandCtas = 2 * (fwd_smem<W, R>() + 7680) <= 228 * 1024 ? 2 : 1;

template <int W, int R, bool B>
__global__ void __launch_bounds__(kThreads, kCandCtas<W, R>) k_cand(Params p0, LaunchArgs la) {
  constexpr unsigned kFull = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char dyn[];
  // the current geometry's parameters, in shared memory (device functions
  // then read them through a shared-memory reference instead of a local
  // copy of the kernel argument)
  __shared__ Params sgeo;
  const Params& p = sgeo;
  __shared__ UnitShared sh;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  WarpMem<W, R>& wm = reinterpret_cast<WarpMem<W, R>*>(dyn)[wid];
  constexpr int XN = WarpMem<W, R>::XN, CapA = WarpMem<W, R>::CapA, CapB = WarpMem<W, R>::CapB;
  const unsigned below = (1u << lane) - 1u;

  // per-geometry state
  int32_t* my_nb_j = nullptr;
  uint64_t* my_nb_em = nullptr;
  uint64_t hf[2 * W];
  auto geo_init = [&]() {
    my_nb_j = p.nb_j + (size_t)blockIdx.x * p.nb_stride;
    my_nb_em = p.nb_emask + (size_t)blockIdx.x * p.nb_stride;
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const int n = min(max(p.noca - w * 64, 0), 64);
        hf[s * W + w] = (n >= 64) ? ~0ull : ((1ull << n) - 1ull);
      }
  };
  if (!B) {
    if (tid == 0) sgeo = p0;
    __syncthreads();
    geo_init();
  }
  int cur_geo = -1;

  unsigned long long ncand = 0, ncmp = 0, np1 = 0, np2 = 0;  // the warp's, in every lane
  auto flush_geometry = [&]() {
    if (lane == 0) {
      if (ncand) atomicAdd(&p.counters[C_NCAND], ncand);
      if (ncmp) atomicAdd(&p.counters[C_NCMP], ncmp);
      if (np1) atomicAdd(&p.counters[C_NP1], np1);
      if (np2) atomicAdd(&p.counters[C_NP2], np2);
    }
    ncand = ncmp = np1 = np2 = 0ull;
    __syncwarp();
  };

  for (;;) {
    __syncthreads();
    if (tid == 0) sh.unit = atomicAdd(&la.work[0], 1);
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
        geo_init();
      }
      unit = la.unit_local[unit];
    }
    const int norb = p.norb, noca = p.noca;
    const int ur0 = p.unit_r0[unit], ur1 = p.unit_r1[unit];
    const int g = p.unit_g[unit];
    const int k = p.gens[g];
    const bool pertu = k < 0;
    const uint8_t dmask = pertu ? 0 : p.gen_dmask[g];
    const int nespk = pertu ? 0 : p.nesp[k];
    const bool yefk = pertu ? false : p.yef[k] != 0;
    int nnb = 0, nown = 0, nel = 0;

    // ------------------------------------------------ the unit's generator
    if (tid < 2 * W) sh.kbits[tid] = pertu ? get_word<2 * W>(hf, tid) : p.S[(size_t)k * 2 * W + tid];
    if (tid < 4) sh.occcol[tid >> 1][tid & 1] = 0ull;
    if (tid < 2 * kMaxSym * 2) (&sh.symcol[0][0][0])[tid] = 0ull;
    __syncthreads();
    uint64_t kb[2 * W];
#pragma unroll
    for (int q = 0; q < 2 * W; ++q) kb[q] = sh.kbits[q];
    if (!pertu) {
      // electron and virtual lists: one thread per spin orbital
#pragma unroll 1
      for (int c = tid; c < 2 * norb; c += blockDim.x) {
        const int s = c >= norb ? 1 : 0, o = c - s * norb;
        uint64_t sw[W];
        pick_spin<W>(kb, s, sw);
        const int nbel = popc_between<W>(sw, -1, o);  // electrons of this spin below o
        const bool on = (get_word<W>(sw, o >> 6) >> (o & 63)) & 1ull;
        int na = 0;
        if (s == 1)
#pragma unroll
          for (int w = 0; w < W; ++w) na += __popcll(kb[w]);
        if (on) {
          sh.occ[na + nbel] = c;
          sh.colof[c] = 255;
        } else {
          const int col = o - nbel;
          sh.vir[s][col] = (uint8_t)o;
          sh.colof[c] = (uint8_t)col;
          unsigned long long* sym = reinterpret_cast<unsigned long long*>(&sh.symcol[s][p.orbsym[o]][col >> 6]);
          atomicOr(sym, 1ull << (col & 63));
          if (o < noca)
            atomicOr(reinterpret_cast<unsigned long long*>(&sh.occcol[s][col >> 6]), 1ull << (col & 63));
        }
      }
      if (tid < 2) {
        int nes = 0;
        for (int w = 0; w < W; ++w) nes += __popcll(get_word<2 * W>(kb, tid * W + w));
        sh.nel_s[tid] = nes;
        sh.nvir[tid] = norb - nes;
      }
      // neighbours of k: what can interact with a candidate of k (degree <= 4),
      // except k and the determinants below k that are no generators (they
      // neither own a candidate nor enter its sum)
      const int2 nb = ordered_partition2(
          p.ncf,
          [&](int j) {
            int x = 0;
#pragma unroll
            for (int q = 0; q < 2 * W; ++q) x += __popcll(kb[q] ^ __ldg(&p.S[(size_t)j * 2 * W + q]));
            if (x > 8 || j == k) return -1;
            return j > k ? 1 : (p.ygen[j] ? 0 : -1);
          },
          [&](int slot, int j) {
            // electrons of k missing in j, as a mask over k's electron indices
            uint64_t em = 0;
            int base = 0;
#pragma unroll
            for (int q = 0; q < 2 * W; ++q) {
              uint64_t miss = kb[q] & ~__ldg(&p.S[(size_t)j * 2 * W + q]);
#pragma unroll 1
              while (miss) {
                const int b = __ffsll((long long)miss) - 1;
                miss &= miss - 1;
                em |= 1ull << (base + __popcll(kb[q] & ((1ull << b) - 1ull)));
              }
              base += __popcll(kb[q]);
            }
            my_nb_j[slot] = j;
            my_nb_em[slot] = em;
          },
          sh.tmp);
      nown = nb.x;  // owners (below k) first
      nnb = nb.x + nb.y;
      // (the partition's barriers publish the lists above)
      nel = sh.nel_s[0] + sh.nel_s[1];
    }

    // ------------------------------------------------ candidates
    // Phases: the reference's own perturbers (pertu.f), or windows of blocks
    // -- each first block by block on the warps alone, then the blocks whose
    // L_R a warp could not hold, one after the other on all warps.
    enum { kPhPertu, kPhWarps, kPhBig, kPhDone };
    int ph = pertu ? kPhPertu : kPhWarps;
    int w0 = ur0, slots = pertu ? ur1 - ur0 : 0, bigi = 0;
    int ws = 1;  // warps that share a block
    // the warp's block
    bool two = false, same = false, opened = false;
    int so1 = 0, so2 = 0, sr = 0, sc = 0, hfR = 0, symR = 0, bslot = 0, ncol = 0;
    int nA = 0, nB = 0, sub = 0, capA = 0, capB = 0, nlive = 0, lr0 = 0;
    const uint32_t *geA = nullptr, *geB = nullptr;  // entries beyond capA / capB
    const uint2 *gjA = nullptr, *gjB = nullptr;
    double hK = 0.0, mK = 0.0;
    Bits<W> kp;
    // its current rows
    int G = 0, nal = 0, pos = 0;
    bool hasx = false;

    auto eA_at = [&](int i) -> uint32_t { return i < capA ? wm.eA[i] : geA[i - capA]; };
    auto eB_at = [&](int i) -> uint32_t { return i < capB ? wm.eB[i] : geB[i - capB]; };
    auto orb_of = [&](int code) { return code >= norb ? code - norb : code; };
    auto spin_of = [&](int code) { return code >= norb ? 1 : 0; };
    auto par_of = [&](int s, int o) -> uint32_t { return (uint32_t)(wm.par[s * W + (o >> 6)] >> (o & 63)) & 1u; };
    auto nonzero = [](double x) { return (__double_as_longlong(x) << 1) != 0; };
    auto merge_xf = [](uint32_t o, uint32_t xf) { return (o | (xf & (kXHas | kXNz))) + (xf & kXLesp); };
    // column of a spin orbital code among the empty orbitals of spin s, or -1
    auto col_of = [&](int code, int s) -> int {
      const int c = sh.colof[code];
      return c != 255 && spin_of(code) == s ? c : -1;
    };
    auto add_coef = [&](double h, int j, double* v) {
#pragma unroll
      for (int m = 0; m < R; ++m)
        if (m < p.metat) v[m] += h * __ldg(&p.c[(size_t)j * p.metat + m]);
    };

    // block bi's orbitals
    auto block_orbitals = [&](int bi) -> uint64_t {
      int e1, e2;
      block_electrons(sh.blk_r[bi], nel, e1, e2);
      bslot = sh.blk_slot[bi];
      two = e2 >= 0;
      so1 = sh.occ[e1];
      so2 = two ? sh.occ[e2] : 0;
      const int o1 = orb_of(so1), o2 = orb_of(so2);
      sr = spin_of(so1);
      sc = two ? spin_of(so2) : sr;
      same = two && sr == sc;
      hfR = (o1 < noca ? 1 : 0) + (two && o2 < noca ? 1 : 0);
      symR = two ? p.its[p.orbsym[o1]][p.orbsym[o2]] : p.orbsym[o1];
#pragma unroll
      for (int q = 0; q < 2 * W; ++q) kp.w[q] = kb[q];
      clear_word<2 * W>(kp.w, sr * W + (o1 >> 6), 1ull << (o1 & 63));
      if (two) clear_word<2 * W>(kp.w, sc * W + (o2 >> 6), 1ull << (o2 & 63));
      ncol = sh.nvir[sc];
      return (1ull << e1) | (two ? 1ull << e2 : 0ull);
    };

    // diagonal energies of I = K' + A from those of K' (cip/hdig.f, hmp.f
    // written over occupation changes dn relative to the reference):
    //   hdig = sum_r dn_r F_rr + 1/2 sum_rs dn_r dn_s (J_rs - [same spin] K_rs)
    //   hmp  = sum_r dn_r fmpb_r
    auto block_energies = [&]() {
      int ndn = 0;
#pragma unroll 1
      for (int q = 0; q < 4 * W; ++q) {  // per word: holes, then particles
        const int w = q >> 1;
        const uint64_t kw = get_word<2 * W>(kp.w, w), hw = get_word<2 * W>(hf, w);
        uint64_t d = (q & 1) ? kw & ~hw : hw & ~kw;
#pragma unroll 1
        while (d) {
          const int b = __ffsll((long long)d) - 1;
          d &= d - 1;
          if (lane == 0) {
            wm.dn_so[ndn] = (uint8_t)((w % W) * 64 + b + (w / W) * norb);
            wm.dn_sg[ndn] = (uint8_t)(q & 1);
          }
          ++ndn;
        }
      }
      __syncwarp();
      const int nn = norb * norb;
#pragma unroll 1
      for (int s = sr; s <= sc; ++s)
#pragma unroll 1
        for (int c = lane; c < sh.nvir[s]; c += 32) {
          const int a = sh.vir[s][c];
          double x = 0.0;
#pragma unroll 2
          for (int i = 0; i < ndn; ++i) {
            const int r = wm.dn_so[i], t = r >= norb ? 1 : 0;
            const double y = __ldg(&p.jx[(s == t ? nn : 0) + (r - t * norb) * norb + a]);
            x = wm.dn_sg[i] ? x + y : x - y;
          }
          wm.vd[s][c] = __ldg(&p.F[tri(a, a)]) + x + 0.5 * __ldg(&p.jx[nn + a * norb + a]);
        }
      // the ndn + ndn^2 terms over the lanes, summed in a fixed order
      double e = 0.0, mp = 0.0;
#pragma unroll 1
      for (int t = lane; t < ndn * (ndn + 1); t += 32) {
        const int i = t < ndn ? t : (t - ndn) / ndn, j = t < ndn ? t : t - ndn - i * ndn;
        const int r = wm.dn_so[i], q = wm.dn_so[j];
        const int s1 = r >= norb ? 1 : 0, s2 = q >= norb ? 1 : 0;
        const int o1 = r - s1 * norb, o2 = q - s2 * norb;
        if (t < ndn) {
          const double f = __ldg(&p.F[tri(o1, o1)]), b = __ldg(&p.fmpb[r]);
          e = wm.dn_sg[i] ? e + f : e - f;
          mp = wm.dn_sg[i] ? mp + b : mp - b;
        } else {
          const double x = 0.5 * __ldg(&p.jx[(s1 == s2 ? nn : 0) + o1 * norb + o2]);
          e = wm.dn_sg[i] == wm.dn_sg[j] ? e + x : e - x;
        }
      }
#pragma unroll 1
      for (int o = 16; o > 0; o >>= 1) {
        e += __shfl_down_sync(kFull, e, o);
        mp += __shfl_down_sync(kFull, mp, o);
      }
      hK = __shfl_sync(kFull, e, 0);
      mK = __shfl_sync(kFull, mp, 0);
      __syncwarp();
    };

    // Block bi for this warp (rows sub, sub + ws, ...).  Neighbours with
    // m = |K' \ j| <= 2 are picked 32 at a time; those below k (owners) and in
    // S leave their marks (I = K' + A and j are m + |A \ E| apart), the others
    // are listed (lists given: they are there already).  false: too long.
    auto open_block = [&](int bi, bool listed) -> bool {
      const uint64_t rmask = block_orbitals(bi);
      const int nrows = !two ? 1 : (same ? sh.nvir[sr] - 1 : sh.nvir[sr]);
      __syncwarp();
#pragma unroll 1
      for (int i = lane; i < nrows * 2 * W; i += 32) (&wm.own[0][0])[i] = 0u;
      if (lane < 4 * W) (&wm.owncol[0][0])[lane] = 0u;
      wm.rpos[lane] = wm.rpos[32 + lane] = 0xffffffffu;
      if (lane < 2 * W) {
        const uint64_t x = get_word<2 * W>(kp.w, lane);
        uint64_t y = parity_below(x);
        if (W == 2 && (lane & 1) && (__popcll(get_word<2 * W>(kp.w, lane & ~1)) & 1)) y = ~y;
        wm.par[lane] = y;
      }
      __syncwarp();
      if (!listed) {
        capA = CapA;
        capB = CapB;
        nA = nB = 0;
      }
      const size_t wo = ((size_t)blockIdx.x * kWarps + wid) * 2 * p.lrw_cap;
      uint32_t* const ge = p.lrw_e + wo;
      uint2* const gj = p.lrw_jh + wo;
      if (!listed) {
        geA = ge;
        gjA = gj;
        geB = ge + p.lrw_cap;
        gjB = gj + p.lrw_cap;
      }
      bool dead = false, over = false;
      int nc = 0, t0 = 0;
      // (lists given: the owners, then the entries of list A)
      const int tend = listed ? nown + nA : nnb;
#pragma unroll 1
      while (!over && !dead && (t0 < tend || nc > 0)) {
#pragma unroll 1
        while (nc < 32 && t0 < tend) {
          const int t = t0 + lane;
          int m = 9;
          if (t < tend) m = listed && t >= nown ? 3 * (int)(gjA[t - nown].y >> 16) : __popcll(my_nb_em[t] & ~rmask);
          const bool in = m <= 2;
          const unsigned bm = __ballot_sync(kFull, in);
          if (in) wm.hits[nc + __popc(bm & below)] = (uint32_t)t;
          nc += __popc(bm);
          t0 += 32;
        }
        __syncwarp();
        const int take = min(nc, 32);
        const int t = lane < take ? (int)wm.hits[lane] : -1;
        const uint32_t later = wm.hits[32 + lane];
        __syncwarp();
        wm.hits[lane] = later;  // (by every lane, whatever is left: before the next lot's stores)
        __syncwarp();
        nc -= take;
        const bool owner = t < nown;  // (or no entry)
        uint3 en = make_uint3(0u, 0u, 9u << 16);
        if (t >= 0) {
          if (listed && !owner) en = make_uint3(geA[t - nown], gjA[t - nown].x, gjA[t - nown].y);
          else en = make_entry<W>(p, kp, my_nb_j[t]);
        }
        const int m = (int)(en.z >> 16);
        // every candidate of the block has this owner
        dead = __any_sync(kFull, t >= 0 && owner && (m == 0 || (!two && m == 1)));
        if (t >= 0 && (owner || m == 0)) {
          if (two && m != 1) {
            // the candidates with both orbitals in E (owned; or j itself)
#pragma unroll 1
            for (int x = 0; x < 2 + m; ++x) {
              const int r = col_of((en.x >> (8 * x)) & 0xff, sr);
#pragma unroll 1
              for (int y = same ? x + 1 : 0; y < 2 + m; ++y) {
                const int c = col_of((en.x >> (8 * y)) & 0xff, sc);
                if (r >= 0 && c >= 0) atomicOr(&wm.own[r][c >> 5], 1u << (c & 31));
              }
            }
          } else {
            // every candidate with an orbital in E (all of a single block's)
#pragma unroll 1
            for (int x = 0; x < (two ? 3 : 1 + m); ++x) {
              const int code = (en.x >> (8 * x)) & 0xff, c = sh.colof[code];
              if (c != 255) atomicOr(&wm.owncol[spin_of(code)][c >> 5], 1u << (c & 31));
            }
          }
        }
        if (!listed) {
          const unsigned m0 = __ballot_sync(kFull, m <= 1 && !owner);
          const unsigned m1 = __ballot_sync(kFull, m == 2 && !owner);
          over = nA + __popc(m0) > CapA + p.lrw_cap || nB + __popc(m1) > CapB + p.lrw_cap;
          if (!over && m <= 2 && !owner) {
            const int i = m <= 1 ? nA + __popc(m0 & below) : nB + __popc(m1 & below);
            const int cap = m <= 1 ? CapA : CapB;
            if (i < cap) {
              (m <= 1 ? wm.eA : wm.eB)[i] = en.x;
              (m <= 1 ? wm.jhA : wm.jhB)[i] = make_uint2(en.y, en.z);
            } else {
              const size_t o = (m <= 1 ? 0 : p.lrw_cap) + i - cap;
              ge[o] = en.x;
              gj[o] = make_uint2(en.y, en.z);
            }
          }
          nA += __popc(m0);
          nB += __popc(m1);
        }
      }
      __syncwarp();
      nlive = lr0 = nal = pos = 0;
      if (over && !dead) return false;
      // ---- rows, one per lane: valid columns (rank-change class, symmetry,
      // spin patterns: cip/igene.f, diexcit.f:183-194) less the owned ones
      const int mine = two ? (nrows - sub + ws - 1) / ws : 1;
      unsigned nvalid = 0;
#pragma unroll 1
      for (int i0 = 0; i0 < mine; i0 += 32) {
        const bool on = i0 + lane < mine;
        const int rw = on && two ? sub + ws * (i0 + lane) : 0;
        const int a1 = two ? sh.vir[sr][rw] : 0;
        const int d0 = two ? hfR + (a1 >= noca ? 1 : 0) : hfR + 1;  // bit of D + 2 with a reference-occupied a2
        const bool al0 = (dmask >> d0) & 1, al1 = (dmask >> (d0 + 1)) & 1;
        const int symA = two ? p.its[symR][p.orbsym[a1]] : symR;
        const bool drow = dead || (two && ((wm.owncol[sr][rw >> 5] >> (rw & 31)) & 1u));
        uint64_t sm[W];
#pragma unroll
        for (int w = 0; w < W; ++w) sm[w] = 0ull;
#pragma unroll 1
        for (int s = 0; s < p.nsym; ++s)
          if (p.its[symA][s] == 0) {
#pragma unroll
            for (int w = 0; w < W; ++w) sm[w] |= sh.symcol[sc][s][w];
          }
        bool any = false;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const uint64_t oc = sh.occcol[sc][w];
          uint64_t nv = al1 ? ~oc : 0ull;
          if (two && d0 == 3 && !yefk) {  // D = +2 with a reference-empty a2
            if (same) {
              if (sc == 1) nv = 0ull;
            } else {
              const int o1 = orb_of(so1), o2 = orb_of(so2);
              if (o1 > o2) nv = 0ull;
              if (o1 == o2) {  // a2 >= a1 only
                const int c1 = a1 - popc_between<W>(kb + W, -1, a1);
                const int lo = min(max(c1 - 64 * w, 0), 64);
                nv &= lo >= 64 ? 0ull : ~0ull << lo;
              }
            }
          }
          uint64_t x = on ? ((al0 ? oc : 0ull) | nv) & sm[w] : 0ull;
          if (same) {  // a2 > a1
            const int lo = min(max(rw + 1 - 64 * w, 0), 64);
            x &= lo >= 64 ? 0ull : ~0ull << lo;
          }
          if (!two && ws > 1) {  // a single block's columns are shared by 32s
            uint64_t m32 = 0;
            if ((2 * w) % ws == sub) m32 |= 0xffffffffull;
            if ((2 * w + 1) % ws == sub) m32 |= 0xffffffff00000000ull;
            x &= m32;
          }
          nvalid += (unsigned)__popcll(x);
          uint64_t o = (uint64_t)wm.owncol[sc][2 * w] | (uint64_t)wm.owncol[sc][2 * w + 1] << 32;
          if (two && on) o |= (uint64_t)wm.own[rw][2 * w] | (uint64_t)wm.own[rw][2 * w + 1] << 32;
          x = drow ? 0ull : x & ~o;
          if (on) {
            wm.own[rw][2 * w] = (uint32_t)x;
            wm.own[rw][2 * w + 1] = (uint32_t)(x >> 32);
          }
          any = any || x != 0ull;
        }
        const unsigned lm = __ballot_sync(kFull, any);
        if (any) {
          const int at = nlive + __popc(lm & below);
          wm.rows[at] = (uint8_t)rw;
          if (two) reinterpret_cast<uint8_t*>(wm.rpos)[a1 + sr * norb] = (uint8_t)at;
        }
        nlive += __popc(lm);
      }
      ncand += __reduce_add_sync(kFull, nvalid);
      __syncwarp();
      ncmp += (unsigned long long)nB * (unsigned)nlive;
      if (nlive > 0) block_energies();
      return true;
    };

    // the next rows of the block: surviving candidates (cols[0..nal)), the
    // other determinants' elements (xb, xf), the constants of <I|H|k>
    auto open_rows = [&]() {
      __syncwarp();  // the last rows' tables have been read by every lane
      nal = pos = 0;
      hasx = false;
      // as many rows as their candidates fit (one always does): what is done
      // once per group of rows counts less, and the batches of 32 candidates are
      // fuller, than with up to four rows by their number of columns (37
      // orbitals, four irreps, S = 334: 0.93 -> 0.80 ms; 60 orbitals, S = 2001,
      // an eighth of the generators: 6.25 -> 5.95)
      const int lrb = lr0, avail = two ? min(kMaxG, nlive - lrb) : 1;
      const int rw = lane < avail ? wm.rows[lrb + lane] : 0;
      int mine = 0;
      if (lane < avail) {
#pragma unroll
        for (int h = 0; h < 2 * W; ++h) mine += __popc(wm.own[rw][h]);
      }
      int incl = mine;
#pragma unroll
      for (int o = 1; o < kMaxG; o <<= 1) {
        const int y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
      }
      G = __popc(__ballot_sync(kFull, lane < avail && incl <= XN));
      if (lane < G) {
        wm.rfirst[lane] = incl - mine;
        wm.rrow[lane] = rw;
        if (two) {
          const int a1 = sh.vir[sr][rw], o1 = orb_of(so1), o2 = orb_of(so2);
          wm.ra1[lane] = a1;
          wm.rpA[lane] = __ldg(&p.pairtab[o1 * norb + a1]);
          wm.rpX[lane] = __ldg(&p.pairtab[o2 * norb + a1]);
          wm.rsg[lane] = par_of(sr, o1) ^ par_of(sc, o2) ^ par_of(sr, a1);
          wm.rhv[lane] = hK + wm.vd[sr][rw];
          wm.rmp[lane] = mK + __ldg(&p.fmpb[a1 + sr * norb]);
        }
      }
#pragma unroll 1
      for (int g = 0; g < G; ++g) {
        const int r = __shfl_sync(kFull, rw, g);
#pragma unroll
        for (int h = 0; h < 2 * W; ++h) {
          const uint32_t am = wm.own[r][h];
          if ((am >> lane) & 1u) wm.cols[nal + __popc(am & below)] = (uint16_t)(g << 8 | (32 * h + lane));
          nal += __popc(am);
        }
      }
      lr0 += G;
      __syncwarp();
      if (two) np2 += (unsigned)nal; else np1 += (unsigned)nal;
      // ---- the other determinants of L_R: first the entries that touch a whole
      // row, then the events, each in entry order per candidate whatever the
      // rows worked together (so the sums are those of any launch shape)
      enum { kDense, kSparseA, kSparseB, kDone };
      int stage = nA > 0 ? kDense : (nB > 0 ? kSparseB : kDone);
      int it = 0, nh = 0, nd = 0, ne = 0, ev0 = 0;
      int pat = lane, pg = 0;  // this lane's next pair of A entry and row, row after row
#pragma unroll 1
      for (;;) {
        if (stage != kDone && ne < 32 && nd <= kDenseCap - 32) {
          // the next 32 (entry, row) pairs
          bool has = false;
          uint32_t at = 0, E = 0;
          int g = 0;
          if (stage <= kSparseA) {
#pragma unroll 1
            while (pat >= nA && pg < G) {
              pat -= nA;
              ++pg;
            }
            has = pg < G;
            at = (uint32_t)pat;
            g = pg;
            if (has) E = eA_at(pat);
            pat += 32;
            it += 32;
          } else {
#pragma unroll 1
            while (nh < 32 && it < nB) {
              const bool in = it + lane < nB;
              const uint32_t e = in ? eB_at(it + lane) : 0u;
              unsigned hm = in && !two ? 1u : 0u;
              if (in && two) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  const uint32_t d = (uint32_t)reinterpret_cast<const uint8_t*>(wm.rpos)[(e >> (8 * q)) & 0xffu] - (uint32_t)lrb;
                  hm |= d < (uint32_t)G ? 1u << d : 0u;
                }
              }
              if (__any_sync(kFull, hm != 0u)) {
                // up to four rows an entry
                const int n = __popc(hm);
                const unsigned n0 = __ballot_sync(kFull, n & 1), n1 = __ballot_sync(kFull, n & 2),
                               n2 = __ballot_sync(kFull, n & 4);
                int o = nh + __popc(n0 & below) + 2 * __popc(n1 & below) + 4 * __popc(n2 & below);
                nh += __popc(n0) + 2 * __popc(n1) + 4 * __popc(n2);
#pragma unroll 1
                while (hm) {
                  const int gg = __ffs((int)hm) - 1;
                  hm &= hm - 1u;
                  wm.hits[o++] = (uint32_t)(it + lane) << 4 | (uint32_t)gg;
                }
              }
              it += 32;
            }
            __syncwarp();
            const int take = min(nh, 32);
            has = lane < take;
            const uint32_t x = wm.hits[lane];
            at = x >> 4;
            g = (int)(x & 15u);
            if (has) E = eB_at((int)at);
            nh -= take;
#pragma unroll 1
            for (int i = 0; i < nh; i += 32) {  // the rest moves to the front
              const uint32_t y = wm.hits[32 + i + lane < kHitCap2 ? 32 + i + lane : 0];
              __syncwarp();
              wm.hits[i + lane] = y;
              __syncwarp();
            }
          }
          const int a1c = two ? wm.ra1[has ? g : 0] + sr * norb : -1;
          const bool a1in = two && has_byte(E, (uint32_t)a1c * 0x01010101u);
          bool whole = false;  // (A entries)
          if (stage != kSparseB && has)
            whole = !two || a1in || (at < (uint32_t)capA ? wm.jhA[at].y : gjA[at - capA].y) < 1u << 16;
          if (stage == kDense) {
            const unsigned bm = __ballot_sync(kFull, whole);
            if (whole) wm.dense[nd + __popc(bm & below)] = at << 4 | (uint32_t)g;
            nd += __popc(bm);
          } else {
            const bool sparse = has && (stage == kSparseB || !whole);
            if (__any_sync(kFull, sparse)) {
              // the columns this entry holds, entry after entry
              const int rw = sparse ? wm.rrow[g] : 0;
              unsigned em[4], mine = 0;
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int code = (E >> (8 * q)) & 0xff;
                // (three codes but for |K' \ j| = 2 in a double block)
                const int col = code == a1c || (q == 3 && !(two && stage == kSparseB)) ? -1 : col_of(code, sc);
                const bool ev = sparse && col >= 0 && ((wm.own[rw][max(col, 0) >> 5] >> (col & 31)) & 1u);
                em[q] = __ballot_sync(kFull, ev);
                mine |= ev ? 1u << q : 0u;
              }
              int o = ev0 + ne + __popc(em[0] & below) + __popc(em[1] & below) + __popc(em[2] & below) +
                      __popc(em[3] & below);
              ne += __popc(em[0]) + __popc(em[1]) + __popc(em[2]) + __popc(em[3]);
#pragma unroll 1
              while (mine) {
                const int q = __ffs((int)mine) - 1;
                mine &= mine - 1u;
                const int col = sh.colof[(E >> (8 * q)) & 0xff];
                int x = wm.rfirst[g] + __popc(wm.own[rw][col >> 5] & ((1u << (col & 31)) - 1u));
#pragma unroll
                for (int h = 0; h < 2 * W - 1; ++h) x += h < (col >> 5) ? __popc(wm.own[rw][h]) : 0;
                wm.ev[o++ & (kEvCap - 1)] = at << 8 | (stage == kSparseB ? 128u : 0u) | (uint32_t)x;
              }
            }
          }
          __syncwarp();
        }
        if ((nd > 0 || ne > 0) && !hasx) {
          hasx = true;
#pragma unroll 1
          for (int c = lane; c < nal; c += 32) {
            wm.xf[c] = 0;
#pragma unroll
            for (int m = 0; m < R; ++m) wm.xb[m][c] = 0.0;
          }
          __syncwarp();
        }
        const bool last_dense = stage == kDense && it >= nA * G;
        if (nd > kDenseCap - 32 || (nd > 0 && last_dense)) {
          // an element for every surviving candidate of the entry's row: each lane
          // goes through its own row's entries
          if (lane <= G) {
            int lo = 0, hi = nd;
#pragma unroll 1
            while (lo < hi) {
              const int mid = (lo + hi) >> 1;
              if ((int)(wm.dense[mid] & 15u) < lane) lo = mid + 1;
              else hi = mid;
            }
            wm.dfirst[lane] = (uint8_t)lo;
          }
          __syncwarp();
#pragma unroll 1
          for (int c0 = 0; c0 < nal; c0 += 32) {
            const int x = c0 + lane;
            const bool act = x < nal;
            const int rc = act ? wm.cols[x] : 0;
            const int rg = rc >> 8, c = rc & 0xff;
            int d = act ? wm.dfirst[rg] : 0;
            const int d1 = act ? wm.dfirst[rg + 1] : 0;
            if (!__any_sync(kFull, d < d1)) continue;
            const int a1c = two ? wm.ra1[rg] + sr * norb : -1, a2c = sh.vir[sc][c] + sc * norb;
            double v[R];
#pragma unroll
            for (int m = 0; m < R; ++m) v[m] = wm.xb[m][x];
            uint32_t xf = 0;
            unsigned n1 = 0, nt = 0;
#pragma unroll 1
            for (; __any_sync(kFull, d < d1); ++d) {
              if (d < d1) {
                const int i = (int)(wm.dense[d] >> 4);
                const uint2 jh = i < capA ? wm.jhA[i] : gjA[i - capA];
                const int j = (int)jh.x;
                const Elem el = element_of<W>(p, wm.par, kp, a1c, a2c, eA_at(i), jh);
                n1 += el.kind == 1 ? 1u : 0u;
                ++nt;
                xf |= kXHas;
                if (nonzero(el.h)) xf |= kXNz;
                if (j > k && j <= k + nespk) ++xf;
                add_coef(el.h, j, v);
              }
            }
            if (xf & kXHas) {
#pragma unroll
              for (int m = 0; m < R; ++m) wm.xb[m][x] = v[m];
              wm.xf[x] = (uint16_t)merge_xf(wm.xf[x], xf);
            }
            const unsigned s1 = __reduce_add_sync(kFull, n1);
            np1 += s1;
            np2 += __reduce_add_sync(kFull, nt) - s1;
          }
          nd = 0;
          __syncwarp();
        }
        // stages in turn (a single block's A entries touch its whole row)
        if (last_dense) {
          stage = two ? kSparseA : (nB > 0 ? kSparseB : kDone);
          it = 0;
          pat = lane;
          pg = 0;
        } else if (stage == kSparseA && it >= nA * G) {
          stage = nB > 0 ? kSparseB : kDone;
          it = 0;
        } else if (stage == kSparseB && it >= nB && nh == 0) {
          stage = kDone;
        }
        if (ne >= 32 || (stage == kDone && ne > 0)) {
          const int cnt = min(ne, 32);
          const bool act = lane < cnt;
          const uint32_t e = wm.ev[(ev0 + (act ? lane : 0)) & (kEvCap - 1)];
          ne -= cnt;
          ev0 += cnt;
          const int x = (int)(e & 127u), i = (int)(e >> 8), rc = wm.cols[x], rg = rc >> 8, c = rc & 0xff;
          double v[R];
#pragma unroll
          for (int m = 0; m < R; ++m) v[m] = 0.0;
          uint32_t xf = kXHas;
          if (act) {
            const bool lb = (e & 128u) != 0u;
            const uint2 jh = lb ? (i < capB ? wm.jhB[i] : gjB[i - capB]) : (i < capA ? wm.jhA[i] : gjA[i - capA]);
            const int j = (int)jh.x;
            const Elem el = element_of<W>(p, wm.par, kp, two ? wm.ra1[rg] + sr * norb : -1,
                                          sh.vir[sc][c] + sc * norb, lb ? eB_at(i) : eA_at(i), jh);
            if (nonzero(el.h)) xf |= kXNz;
            if (j > k && j <= k + nespk) ++xf;
            add_coef(el.h, j, v);
          }
          np2 += (unsigned)cnt;
          // lanes of one candidate: the first adds all of them in lane order
          const unsigned grp = __match_any_sync(kFull, act ? (uint32_t)x : 256u + lane);
          const unsigned more = __reduce_max_sync(kFull, (unsigned)__popc(grp)) - 1u;
          const bool lead = act && (grp & below) == 0u;
          unsigned rest = lead ? grp & (grp - 1u) : 0u;
          if (lead) {
#pragma unroll
            for (int m = 0; m < R; ++m) v[m] += wm.xb[m][x];
          }
#pragma unroll 1
          for (unsigned t = 0; t < more; ++t) {
            const int src = rest ? __ffs(rest) - 1 : lane;
            const uint32_t ox = __shfl_sync(kFull, xf, src);
#pragma unroll
            for (int m = 0; m < R; ++m) {
              const double y = __shfl_sync(kFull, v[m], src);
              if (rest) v[m] += y;
            }
            if (rest) xf = merge_xf(xf, ox);
            rest &= rest - 1u;
          }
          if (lead) {
#pragma unroll
            for (int m = 0; m < R; ++m) wm.xb[m][x] = v[m];
            wm.xf[x] = (uint16_t)merge_xf(wm.xf[x], xf);
          }
          __syncwarp();
        } else if (stage == kDone) {
          break;
        }
      }
    };

    int pt0 = ur0 + wid * 32;  // pertu's candidates, 32 a warp

    // up to 32 candidates into the candidate buffer; false: nothing is left in
    // this phase
    auto produce = [&]() -> bool {
      double h = 0.0, x[R], hv = 0.0, hm = 0.0;
      uint32_t flag = 0, code = 0;
      int slot = 0;
      bool live = false, hx = false;
      if (ph == kPhPertu) {
        if (pt0 >= ur1) return false;
        const int t = pt0 + lane;
        pt0 += kThreads;
        PertuOut<W, R> o;
        o.cand = o.live = false;
        o.n1 = o.n2 = o.ncmp = 0;
        if (t < ur1) pertu_candidate<W, R>(p, t, o);
        ncand += (unsigned)__popc(__ballot_sync(kFull, o.cand));
        np1 += __reduce_add_sync(kFull, o.n1);
        np2 += __reduce_add_sync(kFull, o.n2);
        ncmp += __reduce_add_sync(kFull, o.ncmp);
        live = hx = o.live;
        if (live) {
#pragma unroll
          for (int m = 0; m < R; ++m) x[m] = o.bc[m];
          hm = o.hmp;
          hv = o.hvp;
          code = o.code;
          slot = t - ur0;
        }
      } else {
#pragma unroll 1
        while (pos >= nal) {
          if (lr0 < nlive) {
            open_rows();
            continue;
          }
          int bi;
          if (ph == kPhBig) {
            if (opened) return false;
            opened = true;
            bi = sh.big[bigi];
          } else {
            int job = 0;
            if (lane == 0) job = atomicAdd(&sh.job, 1);
            job = __shfl_sync(kFull, job, 0);
            if (job >= sh.nblk * ws) return false;
            bi = job / ws;
            sub = job - bi * ws;
          }
          if (!open_block(bi, ph == kPhBig) && sub == 0 && lane == 0)
            sh.big[atomicAdd(&sh.nbig, 1)] = (uint16_t)bi;
        }
        // the next candidates of the rows
        live = pos + lane < nal;
        const int xi = pos + lane, rc = live ? wm.cols[xi] : 0;
        pos += 32;
        if (live) {
          const int rg = rc >> 8, c = rc & 0xff;
          const int a2 = sh.vir[sc][c];
          const int o1 = orb_of(so1), o2 = orb_of(so2);
          uint32_t xf = 0;
          if (hasx) xf = wm.xf[xi];
          hx = (xf & kXHas) != 0u;
          if (hx) {
#pragma unroll
            for (int m = 0; m < R; ++m) x[m] = wm.xb[m][xi];
          }
          hv = wm.vd[sc][c];
          hm = __ldg(&p.fmpb[a2 + sc * norb]);
          if (two) {
            const int a1 = wm.ra1[rg], rw = wm.rrow[rg];
            // <k - R + A|H|k>: the pairs of o1, o2 with a1 are the row's
            h = ai_pairs(p, wm.rpA[rg], __ldg(&p.pairtab[o2 * norb + a2]));
            if (same) h -= ai_pairs(p, __ldg(&p.pairtab[o1 * norb + a2]), wm.rpX[rg]);
            h = __hiloint2double(__double2hiint(h) ^ (int)((wm.rsg[rg] ^ par_of(sc, a2)) << 31), __double2loint(h));
            hv = wm.rhv[rg] + (hv + __ldg(&p.jx[(same ? norb * norb : 0) + a1 * norb + a2]));
            hm = wm.rmp[rg] + hm;
            if (hfR == 2 && a1 >= noca && a2 >= noca) {
              flag |= kMD2;
              if (!yefk && !(!same && o1 == o2 && a1 == a2)) flag |= kMWt1;
              if (!nonzero(h) && !(xf & kXNz)) live = false;  // diexcit drops zero couplings
            }
            code = (uint32_t)so1 | (uint32_t)so2 << 8 | (uint32_t)(a1 + sr * norb) << 16 |
                   (uint32_t)(a2 + sc * norb) << 24;
            // pairs a1 < a2 of one spin in row-major order, or a1 x a2
            slot = bslot + (same ? rw * (ncol - 1) - rw * (rw - 1) / 2 + (c - rw - 1) : rw * ncol + c);
          } else {
            Bits<W> u = kp;
            or_word<2 * W>(u.w, sc * W + (a2 >> 6), 1ull << (a2 & 63));
            h = element_single<W>(p, u, k);
            hv = hK + hv;
            hm = mK + hm;
            code = (uint32_t)so1 | (uint32_t)(a2 + sc * norb) << 8;
            slot = bslot + c;
          }
          flag |= (xf & kXLesp) << 8;
        }
      }
      if (live) {
        if (slot >= nslots) {
          atomicAdd(&p.counters[C_STAGE_OVF], 1ull);  // host sizing error
        } else {
          const long long s = slot0 + slot;
#pragma unroll
          for (int m = 0; m < R; ++m) {
            if (m >= p.metat) continue;
            const double ck = pertu ? 0.0 : __ldg(&p.c[(size_t)k * p.metat + m]);
            la.cand.b[m * la.cand.cap + s] = fma(h, ck, hx ? x[m] : 0.0);
          }
          la.cand.mp[s] = hm;
          la.cand.vp[s] = hv;
          la.cand.code[s] = code;
          la.cand.meta[s] = flag | kMLive;
        }
      }
      return true;
    };

    for (;;) {
      // ---- set-up of the phase
      nlive = lr0 = nal = pos = 0;
      if (ph == kPhWarps) {
        __syncthreads();  // the generator's tables are written; the last window's are read
        const int r = w0 + tid;
        bool ok = false;
        int nc = 0;
        if (r < ur1) {
          int e1, e2;
          block_electrons(r, nel, e1, e2);
          const int c1 = sh.occ[e1], c2 = e2 >= 0 ? sh.occ[e2] : 0;
          const int s1 = c1 >= norb ? 1 : 0, s2 = c2 >= norb ? 1 : 0;
          const int nR = e2 >= 0 ? 2 : 1;
          const int hr = (orb_of(c1) < noca ? 1 : 0) + (nR == 2 && orb_of(c2) < noca ? 1 : 0);
#pragma unroll 1
          for (int aV = 0; aV <= nR; ++aV) ok = ok || ((dmask >> (hr + aV - nR + 2)) & 1);
          if (ok) nc = (int)block_candidates(nR, nR == 2 && s1 == s2, sh.nvir[s1], sh.nvir[0], sh.nvir[1]);
        }
        int incl = nc;
#pragma unroll 1
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += y;
        }
        const unsigned om = __ballot_sync(kFull, ok);
        if (lane == 31) {
          sh.tmp[wid] = incl;
          sh.tmp[kWarps + wid] = __popc(om);
        }
        __syncthreads();
        int s0 = slots, b0 = 0, ts = 0, tb = 0;
#pragma unroll 1
        for (int w = 0; w < kWarps; ++w) {
          if (w < wid) {
            s0 += sh.tmp[w];
            b0 += sh.tmp[kWarps + w];
          }
          ts += sh.tmp[w];
          tb += sh.tmp[kWarps + w];
        }
        if (ok) {
          const int bi = b0 + __popc(om & below);
          sh.blk_r[bi] = (uint16_t)r;
          sh.blk_slot[bi] = s0 + incl - nc;
        }
        // A warp takes whole blocks; only where the unit has few (the reference's
        // units hold one) several share a block, each with its own copy of L_R
        // and every second, fourth, eighth row.  Opening a block is most of the
        // work where candidates are few, so idle warps cost less than copies:
        // sharing below 16, 8, 4 blocks took 1277 us on 37 orbitals (S = 334),
        // below 8, 4, 2 1027, below 6, 3, 2 940; 60 orbitals (S = 2001) 44.7,
        // 42.1 and 41.9 ms; the other way on a two-root active space of 120
        // orbitals, 67.5 and 69.  One block and a long L_R (the reference's own):
        // all warps share one copy (45 orbitals, S = 451: its blocks took up to
        // 5.0 ms, 6 to a unit, of a launch whose work is 3.7 ms a CTA; now 0.9).
        const bool all = tb == 1 && nnb >= kShareNb;
        if (all && tid < tb) sh.big[tid] = (uint16_t)tid;
        if (tid == 0) {
          sh.job = 0;
          sh.nbig = all ? tb : 0;
          sh.nblk = all ? 0 : tb;
        }
        slots += ts;
        ws = tb >= 6 ? 1 : tb >= 3 ? 2 : tb >= 2 ? 4 : kWarps;
        __syncthreads();
      } else if (ph == kPhBig) {
        // L_R of the block by the whole CTA, in the CTA's global scratch (the
        // warps then mark the owned candidates each for itself)
        ws = kWarps;
        sub = wid;
        opened = false;
        const uint64_t rmask = block_orbitals(sh.big[bigi]);
        uint32_t* const ge = p.lr_e + (size_t)blockIdx.x * p.nb_stride;
        uint2* const gj = p.lr_jh + (size_t)blockIdx.x * p.nb_stride;
        const int2 np = ordered_partition2(
            nnb - nown,
            [&](int t) {
              const int m = __popcll(my_nb_em[nown + t] & ~rmask);
              return m <= 1 ? 0 : (m == 2 ? 1 : -1);
            },
            [&](int slot, int t) {
              const uint3 en = make_entry<W>(p, kp, my_nb_j[nown + t]);
              ge[slot] = en.x;
              gj[slot] = make_uint2(en.y, en.z);
            },
            sh.tmp);
        capA = capB = 0;
        nA = np.x;
        nB = np.y;
        geA = ge;
        gjA = gj;
        geB = ge + nA;
        gjB = gj + nA;
      }
      // ---- the warps on their own
#pragma unroll 1
      while (produce()) {
      }
      __syncthreads();
      bool next = ph == kPhBig && ++bigi == sh.nbig;
      if (ph == kPhWarps) {
        bigi = 0;
        next = sh.nbig == 0;
        ph = kPhBig;
      }
      if (next) {
        w0 += kWindow;
        ph = w0 < ur1 ? kPhWarps : kPhDone;
      }
      if (pertu) ph = kPhDone;
      if (ph == kPhDone) break;
    }
  }
  if (!B || cur_geo >= 0) flush_geometry();
}

}  // namespace

template <int W, int R>
int cand_ctas() {
  return kCandCtas<W, R>;
}
template <int W, int R, bool B>
cudaError_t launch_cand(const Params& p, const LaunchArgs& la, int grid, cudaStream_t st) {
  constexpr size_t smem = fwd_smem<W, R>();
  cudaError_t e = cudaFuncSetAttribute(k_cand<W, R, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_cand<W, R, B><<<grid, kThreads, smem, st>>>(p, la);
  return cudaGetLastError();
}

}  // namespace cipsi_dev
