// pt2_common.cuh -- types shared by the perturbation kernels (pt2_kernel.cuh,
// compiled in pt2_w1.cu / pt2_w2.cu) and the host side (cipsi_engine.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "../../include/cipsi_gb300.h"

namespace cipsi_dev {

constexpr int kNClass = CIPSI_NCLASS;
constexpr int kMaxRoots = CIPSI_MAX_ROOTS;
constexpr int kThreads = 256;
constexpr int kMaxSym = 8;
constexpr int kMaxElec = 64;
constexpr int kMaxOrb = 128;
constexpr int kRowCap = 128;  // k_pt2_one: per-warp list of |K' \ j| = 2 entries holding a1
constexpr int kHitCap = 8;    // k_pt2_one: per-thread list of scan hits awaiting their matrix elements

// counters[] slots
enum {
  C_IETAT = 0,
  C_NPROC,
  C_NSEL,
  C_NCAND,
  C_NCMP,
  C_NP1,
  C_NP2,
  C_STAGE_OVF,  // candidates whose slot lay outside their unit's (must stay 0)
  C_NCOUNTERS
};

struct Params {
  int norb, noca, nel, ncf, metat, nsym, isym;
  int ngen;
  const int32_t* gens;       // generator indices (0-based); -1 = pertu block
  const uint8_t* gen_dmask;  // allowed rank changes per generator, bit (D+2)
  int nunits;                // work units: (generator slot, range of R blocks
  const int32_t* unit_g;     //   or, for the pertu block, of candidates)
  const int32_t* unit_r0;
  const int32_t* unit_r1;
  const uint64_t* S;         // ncf x 2W words (alpha words, beta words)
  const uint8_t* ygen;
  const int32_t* nesp;
  const uint8_t* yef;
  const double* c;           // ncf x metat, canonical phase
  const float* eri;
  const int32_t* pairtab;    // norb x norb: pair index | irrep << 24
  const int32_t* ntttt;     // [irrep 1..nsym] first packed index (1-based)
  const double* F;           // packed i*(i+1)/2 + j (i >= j, 0-based)
  const double* J;
  const double* K;
  const double* jx;          // 2 x norb x norb: J (opposite spins), J - K (same spin)
  const double* fmpb;        // 2*norb by spin orbital
  const int8_t* orbsym;      // 0-based irreps
  int its[kMaxSym][kMaxSym]; // 0-based product table
  double e[kMaxRoots], eb[kMaxRoots], emp[kMaxRoots], teste[kMaxRoots], taum[kMaxRoots];
  int yen, ysele, ymoyen, ywdeg, symvar, nclass;
  double tau, teseff;
  double aval[kNClass];
  long long aval_bits[kNClass];  // bit patterns of aval (non-negative, ascending)
  int aval_hi[kNClass];          // their high words
  int pertu_ref, pertu_mono;
  // scratch
  int32_t* nb_j;             // per block: ncf entries
  uint64_t* nb_emask;
  uint64_t* lr_ent;          // per block: ncf compact L_R entries beyond lr_cap (k_pt2_one)
  uint32_t* lr_e;            // per block: L_R of a block too long for one warp (k_cand):
  uint2* lr_jh;              //   ncf entries each
  uint32_t* lrw_e;           // per block: 2 x kWarps x lrw_cap entries, the overflow of the warps' lists
  uint2* lrw_jh;
  int lrw_cap;
  int lr_cap;                // shared-memory capacity of L_R (k_pt2_one)
  int nb_stride;             // entries per block in nb_j / nb_emask / lr_ent
  // outputs
  double* gen_part;          // nunits x (5 * metat): per-unit sums (k_pt2_one)
  unsigned long long* counters;
  unsigned long long* dpivot_bits;
  unsigned long long* hist_nom;      // nclass
  unsigned long long* hist_nam;      // nclass x metat
  double* hist_tab;                  // 2 x nclass x metat (tabmp, tabvp)
  double* red;                       // 5 x metat reduced sums (k_reduce / k_finish output)
  // exact sums of the forward kernel, indexed by fx_tab / fx_acc: words of 32
  // bits in 64-bit counters, for terms of 2^-64 to 2^22, for larger and for
  // smaller ones (kFx*), and what lies beyond those or is not finite
  unsigned long long* sums;
  unsigned long long* sums_hi;
  unsigned long long* sums_lo;
  double* sums_big;
  // unit-60 records.  When k_pt2 is done with a work unit, it compacts the
  // selected candidates, in slot order, into one segment of the record pool
  // and notes the segment in the unit table.  k_gather then lays the segments
  // out in unit order, so the records come out in (unit, candidate) order
  // whatever the scheduling.
  int rec_mode;                      // 0: selection counted only; 1: records kept
  uint64_t* pool_bits;               // pool_cap x 2W
  double* pool_xam;                  // pool_cap
  double* pool_evp;                  // pool_cap x metat
  long long pool_cap;
  unsigned long long* pool_count;    // records placed in the pool (may exceed pool_cap: then not stored)
  long long* unit_pool;              // per unit: first pool record of its segment
  int32_t* unit_nsel;                // per unit: records of its segment
  int* work;                         // work counter
  // (pq|rs) as doubles: the caller's FP64 integrals (derivative checks) or
  // the real*4 ones widened on the device; null = read the real*4 `eri`
  const double* eri64;
  // adjoint launch (k_pt2_one<..., ADJ = true>): seeds dE/d e2mp[m], e2vp[m],
  // e2b[m] and the gradient outputs
  double seed_mp[kMaxRoots], seed_vp[kMaxRoots], seed_b[kMaxRoots];
  double* g_eri;    // ninte: dE/d(pq|rs) in the packed order
  double* g_F;      // n(n+1)/2: dE/dF (off-diagonal terms of one-difference elements)
  double* g_slice;  // per block: [F | J | K] packed triangles, then fmpb[2n]
  int slice_stride; // doubles per block slice (3 n(n+1)/2 + 2n)
  double* g_roots;  // 3 x metat: dE/d e, d eb, d emp
  // one-electron adjoint: no (pq|rs) gradient (g_eri unused), so only the
  // single-excitation elements (their F term) take part in the second pass
  int adj_1e;
};

static_assert(sizeof(Params) % sizeof(int) == 0, "Params is copied as ints");

// Candidates between the two forward kernels: k_cand writes each candidate that
// can be a perturber at its slot (its position in its work unit's candidate
// order, from the unit's first slot on), k_pt2 reads them in that order and
// leaves the values of a selected one's record in place.
struct CandBuf {
  double* b;       // R x cap: <I|H|Psi_m>; then ENvp of a selected one
  double* mp;      // cap: hmp(I); then its unit-60 value
  double* vp;      // cap: hdig(I)
  uint32_t* code;  // cap: the four spin orbitals toggled in the generator, a byte each
  uint32_t* meta;  // cap: kM* bits, lesp << 8; 0: no candidate
  long long cap;
};
constexpr uint32_t kMLive = 1u, kMD2 = 2u, kMWt1 = 4u, kMSel = 8u;

// One launch of a forward kernel: its work units' first slots and numbers of
// slots, the candidate buffer, the work counter.  Batched launch: many
// geometries (each with its own Params) in one persistent launch; unit u then
// belongs to geometry unit_geo[u] and is unit unit_local[u] of its unit list.
struct LaunchArgs {
  const long long* unit_slot;
  const int32_t* unit_nslots;
  CandBuf cand;
  int nunits;
  int* work;  // [0] k_cand, [1] k_pt2
  const Params* geo;
  const int32_t* unit_geo;
  const int32_t* unit_local;
};

__device__ __forceinline__ void kahan_add(double& s, double& c, double x) {
  const double y = x - c;
  const double t = s + y;
  c = (t - s) - y;
  s = t;
}

// k_pt2_one, forward: per-warp queue of perturbers that survived the interaction
// scan.  The FP64 epilogue then runs on full warps: the FP64 pipe of GB300 is
// narrow, and a warp instruction costs the same with 32 lanes or with the few
// that would be live at the candidate level.
constexpr int kQCap = 64;
template <int R>
struct WarpQueue {
  double bc[R][kQCap];
  double hmp[kQCap], hvp[kQCap], fmul[kQCap];
  int nmul[kQCap];
  unsigned char flags[kQCap];  // bit 0 ybis, bit 1 is_pert1
};

constexpr int kWarps = kThreads / 32;
constexpr int kMaxDn = 48;      // spin orbitals where K' differs from the reference
constexpr int kMaxG = 16;       // rows of a block worked together
constexpr int kDenseCap = 64;   // per-warp list of (entry, row): the entry touches the whole row
constexpr int kEvCap = 256;     // per-warp ring of (entry, row, column) events
constexpr int kHitCap2 = 32 + 32 * 4;  // per-warp list of (entry, row): the entry holds the row's a1
constexpr int kLrWarpG = 1024;  // overflow entries of each L_R list of a warp, in global scratch

// One warp's part of k_cand's shared memory.  The L_R lists are short: what
// shared memory does not take is L1, which holds their overflow.
template <int W, int R>
struct WarpMem {
  static constexpr int NC = 64 * W;                  // columns: empty orbitals of one spin
  static constexpr int XN = R <= 2 ? 128 : 64 * W;   // candidates of the rows worked together
  static constexpr int CapA = 64;                    // L_R entries with |K' \ j| <= 1
  static constexpr int CapB = R == 1 ? 96 : 64;      // and with |K' \ j| = 2
  double vd[2][NC];                      // hdig(K'+a) - hdig(K') by (spin, column)
  double xb[R][XN];                      // sums of <I|H|j> c_j over j != k
  double rhv[kMaxG], rmp[kMaxG];         // per row: hdig(K'+a1), hmp(K'+a1)
  uint64_t par[2 * W];                   // bit o: parity of the electrons of K' below o, by spin
  uint2 jhA[CapA], jhB[CapB];            // L_R entries: j; holes of K' in j, |K' \ j| << 16
  uint32_t eA[CapA], eB[CapB];           // their spin orbitals E = j \ K', one code per byte
  uint32_t own[NC][2 * W];               // candidates (row, column) owned by an earlier generator or in S;
                                         //   from the block's row pass on: those still alive
  uint32_t owncol[2][2 * W];             // orbitals (by spin, column) every candidate of which is owned
  uint32_t dense[kDenseCap];             // entry << 4 | row, rows ascending
  uint32_t ev[kEvCap];                   // entry << 8 | list << 7 | candidate
  uint32_t hits[kHitCap2];               // entry << 4 | row
  int ra1[kMaxG], rrow[kMaxG], rpA[kMaxG], rpX[kMaxG], rfirst[kMaxG];
  uint32_t rsg[kMaxG];
  uint32_t rpos[64];                     // by spin orbital code, a byte each: its place in rows[], 255: none
  uint16_t xf[XN];                       // per candidate: element found, non-zero, lesp
  uint16_t cols[XN];                     // surviving candidates: row << 8 | column
  uint8_t rows[NC];                      // the block's rows with a candidate alive
  uint8_t dfirst[kMaxG + 4];             // by row: its first place in dense[]
  uint8_t dn_so[kMaxDn], dn_sg[kMaxDn];  // where K' differs from the reference: code, 1 = added
};
template <int W, int R>
constexpr size_t fwd_smem() {
  return (size_t)kWarps * sizeof(WarpMem<W, R>);
}

// indices of the exact sums: by class (kNClass: outside the histogram) the MP
// (q = 0) and EN (q = 1) terms; e2b, psimp, psivp (q = 0, 1, 2)
__host__ __device__ constexpr int fx_tab(int q, int c, int m) { return (q * (kNClass + 1) + c) * kMaxRoots + m; }
__host__ __device__ constexpr int fx_acc(int q, int m) { return (2 * (kNClass + 1) + q) * kMaxRoots + m; }
constexpr int kFxSums = (2 * (kNClass + 1) + 3) * kMaxRoots;
// words of the three tables and their units (2^-unit): every bit of a term is
// held, whatever its size -- terms of 2^-64 to 2^22 end at 2^-116 or above,
// those up to 2^62 at 2^-30 or above, those down to 2^-127 at 2^-179 or above
constexpr int kFxWords = 5, kFxUnit = 116, kFxWordsHi = 4, kFxUnitHi = 44, kFxWordsLo = 4, kFxUnitLo = 180;
constexpr int kFxMin = -64, kFxMax = 22, kFxMinLo = -127;  // exponents: the main table's terms; the least of sums_lo

// Candidates of one block of removed electrons R: nv added orbitals for
// |R| = 1, nv(nv-1)/2 same-spin pairs, nva * nvb opposite-spin pairs (nv:
// empty orbitals of the generator in the spin(s) of R).  A work unit's
// candidate slots are numbered block after block (blocks with no allowed
// rank-change class take none), then by the candidate's index in its block:
// the added orbital, or the pair (a1 < a2) in row-major order.
__host__ __device__ inline long long block_candidates(int nR, bool same_spin, int nv1, int nva, int nvb) {
  if (nR == 1) return nv1;
  return same_spin ? (long long)nv1 * (nv1 - 1) / 2 : (long long)nva * nvb;
}

// The forward kernels, plain and batched: k_cand<W, R, B> (pt2_w1.cu,
// pt2_w2.cu) on `grid` CTAs and k_pt2<W, R, B> (pt2_epi.cu) on as many as fit,
// one after the other.
template <int W, int R, bool B>
cudaError_t launch_cand(const Params& p, const LaunchArgs& la, int grid, cudaStream_t st);
template <int W, int R, bool B>
cudaError_t launch_pt2(const Params& p, const LaunchArgs& la, int sms, cudaStream_t st);
// CTAs of k_cand<W, R, *> per SM
template <int W, int R>
int cand_ctas();
// k_pt2_one<W, R, ADJ> launched with `smem` bytes of dynamic shared memory
// (pt2_adj.cu, pt2_adj_w2.cu: adjoint; pt2_one.cu: forward)
template <int W, int R, bool ADJ>
cudaError_t launch_pt2_one(const Params& p, int grid, size_t smem, cudaStream_t st);

// The Hamiltonian over a determinant list by rows (hbuild.cu): launch_hcount
// counts, per row i, the columns j < min(i, jmax) within two excitations;
// launch_hfill writes them and their elements, in increasing j, from rowptr[i]
// on.
struct HBuildArgs {
  Params p;                 // integrals (pairtab, ntttt, eri / eri64, F) and norb
  const uint64_t* S;        // n x 2W words
  const int8_t* sigma;      // n: phase of each determinant's excitation list
  int n;                    // determinants (rows)
  int jmax;                 // columns j < min(i, jmax)
  uint64_t hf[4];           // the reference determinant (2W words)
  int seg, nseg;            // columns per segment (hscan_segment), segments
  int32_t* segcnt;          // nseg x n: hits, then their exclusive sums over the segments
  int32_t* count;           // columns per row
  const long long* rowptr;  // first pair of each row
  int32_t* col;
  double* val;
};

int hscan_segment(int n);
template <int W>
cudaError_t launch_hcount(const HBuildArgs& a, cudaStream_t st);
template <int W>
cudaError_t launch_hfill(const HBuildArgs& a, int sms, cudaStream_t st);

}  // namespace cipsi_dev
