// cipsi_engine.cu -- host side of the GB300 engine for the CIPSI second-order
// perturbation / selection step: contexts, run planning, launches, results,
// the batched multi-geometry launch and the allocation-free entry point.
// The kernels are in pt2_fwd.cuh, pt2_epi.cuh (forward runs) and pt2_kernel.cuh
// (adjoint and allocation-free run; the algorithm is described there).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "pt2_common.cuh"

using namespace cipsi_dev;

namespace {

// fixed-order Kahan reduction of the per-unit partial sums: block q sums
// column q; thread t takes a contiguous range of units, then thread 0 adds
// the per-thread sums in thread order (bitwise reproducible)
constexpr int kReduceThreads = 256;
__global__ void __launch_bounds__(kReduceThreads) k_reduce(const double* part, int nunits, int nq,
                                                           double* out) {
  __shared__ double ps[kReduceThreads], pc[kReduceThreads];
  const int q = blockIdx.x;
  const int per = (nunits + kReduceThreads - 1) / kReduceThreads;
  const int u0 = threadIdx.x * per, u1 = min(nunits, u0 + per);
  double s = 0.0, c = 0.0;
  for (int u = u0; u < u1; ++u) kahan_add(s, c, part[(long long)u * nq + q]);
  ps[threadIdx.x] = s;
  pc[threadIdx.x] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    double S = 0.0, C = 0.0;
    for (int t = 0; t < kReduceThreads; ++t) {
      kahan_add(S, C, ps[t]);
      kahan_add(S, C, -pc[t]);
    }
    out[q] = S - C;
  }
}

// One exact sum (N words of 32 bits in 64-bit counters, the top one signed, in
// units of 2^-unit) as a double, from its leading 96 bits (at least 65 of them
// significant: an error of half an ulp and 2^-11 of one at most).
template <int N>
__device__ double fx_value(const unsigned long long* g, int unit) {
  uint32_t w[N + 1];
  unsigned long long c = 0, any = 0;
  for (int i = 0; i < N; ++i) any |= g[i];
  if (any == 0) return 0.0;
  for (int i = 0; i < N - 1; ++i) {
    // the carry is below 2^32 and the counter well below 2^64 - 2^32
    const unsigned long long x = g[i] + c;
    w[i] = (uint32_t)x;
    c = x >> 32;
  }
  const long long top = (long long)(g[N - 1] + c);
  w[N - 1] = (uint32_t)top;
  w[N] = (uint32_t)((unsigned long long)top >> 32);
  const bool neg = top < 0;
  if (neg) {
    unsigned long long b = 1;
    for (int i = 0; i <= N; ++i) {
      b += (uint32_t)~w[i];
      w[i] = (uint32_t)b;
      b >>= 32;
    }
  }
  int h = N;
  while (h > 0 && w[h] == 0u) --h;
  const unsigned long long hi = ((unsigned long long)w[h] << 32) | (h >= 1 ? w[h - 1] : 0u);
  double v = (double)hi * 4294967296.0 + (double)(h >= 2 ? w[h - 2] : 0u);
  v = ldexp(v, 32 * (h - 2) - unit);
  return neg ? -v : v;
}

// The forward kernel's exact sums of geometry blockIdx.x as doubles: class
// sums to hist_tab, E2 sums and norms (every class together, and the terms
// outside the histogram) to red.  One small block per geometry: no partial
// sums per work unit are kept or added up.  The tables (22 KB, one after the
// other) come to shared memory first, all loads in flight at once: a thread
// that walks its classes' words in global memory waits for each.
constexpr int kFinishThreads = 256;
constexpr int kFxTables = (kFxWords + kFxWordsHi + kFxWordsLo + 1) * kFxSums;
__global__ void __launch_bounds__(kFinishThreads) k_finish(Params p0, const Params* geo) {
  __shared__ unsigned long long tables[kFxTables];
  const Params& p = geo ? geo[blockIdx.x] : p0;
  const int mt = p.metat, nc = p.nclass;
  const unsigned long long* from = p.sums;
#pragma unroll 11
  for (int i = threadIdx.x; i < kFxTables; i += kFinishThreads) tables[i] = from[i];
  __syncthreads();
  const unsigned long long *main = tables, *high = main + kFxWords * kFxSums, *low = high + kFxWordsHi * kFxSums;
  const double* big = reinterpret_cast<const double*>(low + kFxWordsLo * kFxSums);
  auto value = [&](const unsigned long long* s, const unsigned long long* hi, const unsigned long long* lo, double x) {
    return (fx_value<kFxWords>(s, kFxUnit) + fx_value<kFxWordsLo>(lo, kFxUnitLo)) +
           (fx_value<kFxWordsHi>(hi, kFxUnitHi) + x);
  };
  // (the E2 sums' threads have the most to do: theirs are the first warps)
  for (int i = threadIdx.x; i < 5 * mt + 2 * nc * mt; i += kFinishThreads) {
    if (i >= 5 * mt) {
      const int h = i - 5 * mt, q = h / (nc * mt), c = h / mt % nc, m = h % mt;
      const int x = fx_tab(q, c, m);
      p.hist_tab[h] = value(main + kFxWords * x, high + kFxWordsHi * x, low + kFxWordsLo * x, big[x]);
      continue;
    }
    const int q = i / mt, m = i % mt;
    unsigned long long s[kFxWords] = {}, hi[kFxWordsHi] = {}, lo[kFxWordsLo] = {};
    double b = 0.0;
    for (int c = 0; c <= (q < 2 ? kNClass : 0); ++c) {
      const int x = q < 2 ? fx_tab(q, c, m) : fx_acc(q - 2, m);
      for (int w = 0; w < kFxWords; ++w) s[w] += main[kFxWords * x + w];
      for (int w = 0; w < kFxWordsHi; ++w) hi[w] += high[kFxWordsHi * x + w];
      for (int w = 0; w < kFxWordsLo; ++w) lo[w] += low[kFxWordsLo * x + w];
      b += big[x];
    }
    p.red[i] = value(s, hi, lo, b);
  }
}

// adjoint: sum the per-block slices [F | J | K | fmpb] over blocks
__global__ void k_slice_reduce(const double* sl, int nblocks, int stride, int nt, double* gF, double* gJ,
                               double* gK, double* gf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= stride) return;
  double s = 0.0;
  for (int b = 0; b < nblocks; ++b) s += sl[(size_t)b * stride + i];
  if (i < nt) gF[i] += s;
  else if (i < 2 * nt) gJ[i - nt] = s;
  else if (i < 3 * nt) gK[i - 2 * nt] = s;
  else gf[i - 3 * nt] = s;
}

// Output offsets of the unit segments: unit_out[u] = base + the records of
// units u0..u-1 (exclusive scan of unit_nsel over [u0, u1), one block);
// *total = the records of [u0, u1).
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) k_scan_units(const int32_t* nsel, long long* out, int u0, int u1,
                                                             long long base, unsigned long long* total) {
  __shared__ long long wsum[kScanThreads / 32];
  __shared__ long long carry;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) carry = base;
  __syncthreads();
  for (int c0 = u0; c0 < u1; c0 += kScanThreads) {
    const int u = c0 + tid;
    const long long v = u < u1 ? nsel[u] : 0;
    long long incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    if (wid == 0) {
      long long w = wsum[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      wsum[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    const long long before = carry + (wid ? wsum[wid - 1] : 0) + (incl - v);
    if (u < u1) out[u] = before;
    __syncthreads();
    if (tid == 0) carry += wsum[kScanThreads / 32 - 1];
    __syncthreads();
  }
  if (tid == 0 && total) *total = (unsigned long long)(carry - base);
}

// Records of units [u0, u1) from their pool segments to the output arrays
// at unit_out[u] - out_base (unit order), with the owner (1-based generator
// index, 0 for pertu's candidates) taken from the unit; records beyond
// out_cap are dropped (the run reports an overflow).
struct GatherArgs {
  const uint64_t* pool_bits;
  const double* pool_xam;
  const double* pool_evp;
  long long pool_cap;
  const long long* unit_pool;
  const int32_t* unit_nsel;
  const long long* unit_out;
  const int32_t* unit_g;
  const int32_t* gens;
  int u0, u1, words, metat;
  long long out_base, out_cap;
  uint64_t* out_bits;
  int32_t* out_owner;
  double* out_xam;
  double* out_evp;
};
__global__ void __launch_bounds__(256) k_gather(GatherArgs a) {
  for (int u = a.u0 + blockIdx.x; u < a.u1; u += gridDim.x) {
    const int n = a.unit_nsel[u];
    if (n == 0) continue;
    const long long src = a.unit_pool[u];
    const long long dst = a.unit_out[u] - a.out_base;
    const int k = a.gens[a.unit_g[u]];
    const int owner = k < 0 ? 0 : k + 1;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const long long d = dst + i, q = src + i;
      if (d >= a.out_cap || q >= a.pool_cap) break;
      for (int w = 0; w < a.words; ++w) a.out_bits[d * a.words + w] = a.pool_bits[q * a.words + w];
      a.out_owner[d] = owner;
      a.out_xam[d] = a.pool_xam[q];
      for (int m = 0; m < a.metat; ++m) a.out_evp[d * a.metat + m] = a.pool_evp[q * a.metat + m];
    }
  }
}

// What a run accumulates into, in one allocation cleared by one call:
// counters, dpivot, histogram counts | exact sums (k_finish reads their tables
// as one array) | work counter, records in the pool (8 bytes each).
constexpr size_t kCountWords = C_NCOUNTERS + 1 + kNClass + kNClass * kMaxRoots;
constexpr size_t kZeroWords = kCountWords + (size_t)kFxTables + 2;
// a run's result on the device: reduced sums, class sums, counters
constexpr size_t kTabWord = 5 * kMaxRoots, kTabWords = 2 * kNClass * kMaxRoots;
constexpr size_t kResWords = kTabWord + kTabWords + kCountWords;
void set_zeroed(Params& p, unsigned long long* z) {
  p.counters = z;
  p.dpivot_bits = z + C_NCOUNTERS;
  p.hist_nom = z + C_NCOUNTERS + 1;
  p.hist_nam = z + C_NCOUNTERS + 1 + kNClass;
  p.sums = z + kCountWords;
  p.sums_hi = p.sums + (size_t)kFxWords * kFxSums;
  p.sums_lo = p.sums_hi + (size_t)kFxWordsHi * kFxSums;
  p.sums_big = reinterpret_cast<double*>(p.sums_lo + (size_t)kFxWordsLo * kFxSums);
  p.work = reinterpret_cast<int*>(z + kZeroWords - 2);
  p.pool_count = z + kZeroWords - 1;
}

// zero what every geometry of a batch accumulates into (block b: geometry b)
__global__ void k_batch_clear(const Params* geo) {
  unsigned long long* z = geo[blockIdx.x].counters;
  for (int i = threadIdx.x; i < (int)kZeroWords; i += blockDim.x) z[i] = 0ull;
}

}  // namespace

// =================================================================== host

struct cipsi_ctx {
  cipsi_dims d{};
  int device = 0;
  int W = 1;
  std::string err;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  bool have_int = false, have_space = false, have_roots = false;
  // host copies needed for set-up
  std::vector<int32_t> itsym, its;
  std::vector<int32_t> rank;
  std::vector<uint64_t> Sbits;
  std::vector<uint8_t> ygen, ysaut, yef1;
  std::vector<int32_t> nesp;
  std::vector<double> sigma;
  std::vector<double> croot;  // metat*ncf reference phase (column-major)
  double e[kMaxRoots]{}, eb[kMaxRoots]{}, emp[kMaxRoots]{}, teste[kMaxRoots]{}, taum[kMaxRoots]{};
  // device buffers
  uint64_t* dS = nullptr;
  uint8_t *dygen = nullptr, *dyef = nullptr;
  int32_t* dnesp = nullptr;
  double* dc = nullptr;
  float* deri = nullptr;
  double* deri64 = nullptr;  // FP64 storage of (pq|rs) (cipsi_set_integrals_f64store)
  double* deri_w = nullptr;  // the real*4 (pq|rs) widened to double (small integral sets)
  int32_t* dpairtab = nullptr;
  int32_t* dntttt = nullptr;
  double *dF = nullptr, *dJ = nullptr, *dK = nullptr, *dfmpb = nullptr;
  double* djx = nullptr;  // J and J - K as square matrices (coalesced rows)
  int8_t* dorbsym = nullptr;
  int64_t ninte = 0;
  // per-run buffers
  // the plan on the device (pack_plan): one allocation and one copy
  unsigned char* dplan = nullptr;
  size_t plan_cap = 0;
  std::vector<unsigned char> hplan;
  int nunits = 0;
  // candidate buffer of runs whose slots take up to kCandOwnBytes; those of
  // larger runs go through the device's (CandArena): cand_shared, of the last
  // run; cand_user: this context counts among its users
  unsigned char* dcand = nullptr;
  size_t cand_bytes = 0, cand_limit = 0;  // cand_limit: cipsi_set_candidate_bytes
  bool cand_shared = false, cand_user = false;
  int32_t* dnb_j = nullptr;
  uint64_t* dnb_em = nullptr;
  uint64_t* dlr_ent = nullptr;
  uint32_t *dlr_e = nullptr, *dlrw_e = nullptr;
  uint2* dlrw_jh = nullptr;
  size_t scratch_blocks = 0;
  double* dgen_part = nullptr;
  size_t gen_part_cap = 0;
  double* dgrad = nullptr;  // adjoint: small gradient buffers, grad_cap doubles
  size_t grad_cap = 0;
  unsigned long long* dcounters = nullptr;  // kZeroWords: counters, exact sums, work and pool counters
  // (dred, dhist_tab and the counters are one allocation, in this order, so
  // that a result is one copy into hres, which is pinned)
  double* dhist_tab = nullptr;
  double* dred = nullptr;
  unsigned long long* hres = nullptr;
  uint64_t* dsel_bits = nullptr;
  int32_t* dsel_owner = nullptr;
  double *dsel_xam = nullptr, *dsel_evp = nullptr;
  long long sel_cap = 0;
  // record path: the pool of unit segments, the unit table (segment, records,
  // output offset)
  uint64_t* dpool_bits = nullptr;
  double *dpool_xam = nullptr, *dpool_evp = nullptr;
  long long pool_cap = 0;
  long long* dunit_pool = nullptr;
  int32_t* dunit_nsel = nullptr;
  long long* dunit_out = nullptr;
  unsigned long long* dscan_total = nullptr;
  int unit_tab_cap = 0;
  // streamed runs (cipsi_run_pt2_stream): two device record buffers, a copy
  // stream, a ring of pinned host buffers; per-unit record counts of the
  // last run, reused to size the chunks of a run with the same plan
  uint64_t* dout_bits[2] = {nullptr, nullptr};
  int32_t* dout_owner[2] = {nullptr, nullptr};
  double* dout_xam[2] = {nullptr, nullptr};
  double* dout_evp[2] = {nullptr, nullptr};
  long long out_cap = 0;
  cudaStream_t copy_stream = nullptr;
  cudaEvent_t ev_gathered[2] = {nullptr, nullptr}, ev_copied[2] = {nullptr, nullptr};
  cudaEvent_t ev_host[2] = {nullptr, nullptr};
  void* hbuf[2] = {nullptr, nullptr};
  long long hbuf_cap = 0;
  int stream_chunks = 0;  // chunks of the last streamed run
  std::vector<int32_t> last_unit_nsel;
  unsigned long long last_plan_sig = 0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, evk = nullptr;  // evk: end of k_pt2
  long long last_launches = 0;
  // launch tuning (cipsi_set_tuning): r_chunk, from which unit_blocks takes the
  // blocks per work unit, and CTAs per SM (0 = as many as shared memory allows)
  int tune_r_chunk = 6;
  int tune_ctas = 0;
  // set by a batched run: the event that marks its end (fetch waits on it),
  // and whether ev0/ev1 time this context's own launch
  cudaEvent_t ext_done = nullptr;
  bool ev_valid = false;
  // bumped whenever a device buffer is (re)allocated: a batch built on this
  // context refuses to run after that
  unsigned long long buf_gen = 0;
  // pending run
  int ngen = 0;
  int nclass = kNClass;
  bool pending = false;
  cipsi_opts last_opts{};
  long long nsel = 0;  // records of the last fetched run
  // caller-provided record arrays in pinned host memory (cipsi_set_selection_sink):
  // the kernel writes the unit-60 records there directly
  bool sink = false;
  uint64_t* sink_bits = nullptr;
  int32_t* sink_owner = nullptr;
  double *sink_xam = nullptr, *sink_evp = nullptr;
  long long sink_cap = 0;
  void* sink_host[4] = {nullptr, nullptr, nullptr, nullptr};  // the caller's addresses
  // the Hamiltonian over the space (cipsi_hamiltonian_build): the caller's Fock
  // matrix when given, the kept workspace, pairs by rows
  double* dFraw = nullptr;
  unsigned char* dh_work = nullptr;
  size_t h_work_cap = 0;
  int32_t* dh_col = nullptr;
  double* dh_val = nullptr;
  long long h_cap = 0;
  std::vector<long long> h_rowptr;
  bool have_h = false;
  float h_ms = 0.f;
};

namespace {

int fail(cipsi_ctx* c, int code, const std::string& msg) {
  if (c) c->err = msg;
  return code;
}

#define CK(call)                                                                        \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess)                                                              \
      return fail(ctx, CIPSI_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// Integral sets up to this size are also kept widened to double on the
// device (13 MB for 60 orbitals; the 120-orbital set stays real*4 only, so
// that it still fits in L2).  The values are the real*4 ones, exactly; the
// kernel then loads a double per integral instead of converting a float.
constexpr size_t kWidenMaxBytes = (size_t)48 << 20;

__global__ void k_widen(const float* __restrict__ in, double* __restrict__ out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (double)in[i];
}

template <typename T>
int upload(cipsi_ctx* ctx, T** dptr, const T* h, size_t n) {
  if (*dptr) cudaFree(*dptr);
  *dptr = nullptr;
  ++ctx->buf_gen;
  CK(cudaMalloc((void**)dptr, std::max<size_t>(n, 1) * sizeof(T)));
  if (n) CK(cudaMemcpyAsync(*dptr, h, n * sizeof(T), cudaMemcpyHostToDevice, ctx->stream));
  return 0;
}

template <typename T>
void dfree(T*& p) {
  if (p) cudaFree(p);
  p = nullptr;
}

// The candidate buffer of large runs, one per device for all contexts of the
// process: such a run fills the device by itself, so that taking turns costs
// nothing, and a program that keeps hundreds of contexts keeps one buffer.
// `busy` is recorded after a part's kernels; whoever enqueues the next part, on
// whatever stream, waits for it there, holding the lock.  The last user frees
// the buffer.
struct CandArena {
  std::mutex mu;
  unsigned char* base = nullptr;
  size_t bytes = 0;
  cudaEvent_t busy = nullptr;
  int users = 0;
};
constexpr int kMaxDevices = 64;
CandArena g_arena[kMaxDevices];

void leave_arena(cipsi_ctx* ctx) {
  if (!ctx->cand_user) return;
  CandArena& a = g_arena[ctx->device];
  std::lock_guard<std::mutex> hold(a.mu);
  ctx->cand_user = false;
  if (--a.users > 0) return;
  if (a.base) cudaFree(a.base);  // (waits for the device)
  if (a.busy) cudaEventDestroy(a.busy);
  a.base = nullptr;
  a.bytes = 0;
  a.busy = nullptr;
}

// `want` bytes of device memory, or half as often as it takes down to `need`
cudaError_t alloc_down(unsigned char** p, size_t need, size_t want, size_t* got) {
  for (size_t b = std::max(want, need);; b = std::max(b / 2, need)) {
    const cudaError_t e = cudaMalloc((void**)p, b);
    if (e == cudaSuccess) {
      *got = b;
      return e;
    }
    *p = nullptr;
    cudaGetLastError();
    if (e != cudaErrorMemoryAllocation || b == need) return e;
  }
}

int roots_pad(int mt) { return mt <= 1 ? 1 : mt <= 2 ? 2 : mt <= 4 ? 4 : 8; }

// the forward form of k_pt2_one of class (W, R)
cudaError_t launch_one(int W, int R, const Params& p, int grid, size_t smem, cudaStream_t st) {
  if (W == 1)
    return R == 1 ? launch_pt2_one<1, 1, false>(p, grid, smem, st)
         : R == 2 ? launch_pt2_one<1, 2, false>(p, grid, smem, st)
         : R == 4 ? launch_pt2_one<1, 4, false>(p, grid, smem, st)
                  : launch_pt2_one<1, 8, false>(p, grid, smem, st);
  return R == 1 ? launch_pt2_one<2, 1, false>(p, grid, smem, st)
       : R == 2 ? launch_pt2_one<2, 2, false>(p, grid, smem, st)
       : R == 4 ? launch_pt2_one<2, 4, false>(p, grid, smem, st)
                : launch_pt2_one<2, 8, false>(p, grid, smem, st);
}

// The code and the local memory that cipsi_run_pt2_static's kernels take on the
// device, which the runtime allocates at their first launch: a context has them
// from its creation on, so that the call itself allocates nothing.
cudaError_t load_static(int W, int R, cudaStream_t st) {
  cudaFuncAttributes at;
  const cudaError_t e = cudaFuncGetAttributes(&at, k_reduce);
  return e != cudaSuccess ? e : launch_one(W, R, Params{}, 1, 0, st);  // no units: it returns at once
}

}  // namespace

extern "C" {

int cipsi_ctx_create(cipsi_ctx** out, const cipsi_dims* dims, int32_t device) {
  if (!out || !dims) return CIPSI_ERR_ARG;
  *out = nullptr;
  cipsi_ctx* ctx = new cipsi_ctx();
  ctx->d = *dims;
  ctx->device = device;
  const cipsi_dims& d = *dims;
  if (d.norb < 2 || d.norb > kMaxOrb) {
    *out = ctx;
    return fail(ctx, CIPSI_ERR_ARG, "norb must be in [2, 128]");
  }
  if (d.noca < 1 || d.noca >= d.norb || 2 * d.noca > kMaxElec) {
    *out = ctx;
    return fail(ctx, CIPSI_ERR_ARG, "noca must be in [1, min(norb-1, 32)]");
  }
  if (d.nsym < 1 || d.nsym > kMaxSym || d.isym < 1 || d.isym > d.nsym) {
    *out = ctx;
    return fail(ctx, CIPSI_ERR_ARG, "nsym must be in [1, 8] and isym in [1, nsym]");
  }
  if (d.isz != 0) {
    *out = ctx;
    return fail(ctx, CIPSI_ERR_ARG, "only isz = 0 (Ms = 0) is supported");
  }
  if (d.metat < 1 || d.metat > kMaxRoots) {
    *out = ctx;
    return fail(ctx, CIPSI_ERR_ARG, "metat must be in [1, 8]");
  }
  if (d.ncf < 1) {
    *out = ctx;
    return fail(ctx, CIPSI_ERR_ARG, "ncf must be positive");
  }
  ctx->W = d.norb <= 64 ? 1 : 2;
  *out = ctx;
  CK(cudaSetDevice(device));
  CK(cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking));
  ctx->stream = ctx->own_stream;
  CK(cudaEventCreate(&ctx->ev0));
  CK(cudaEventCreate(&ctx->ev1));
  CK(cudaEventCreate(&ctx->evk));
  CK(load_static(ctx->W, roots_pad(d.metat), ctx->stream));
  return CIPSI_OK;
}

void cipsi_ctx_destroy(cipsi_ctx* ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  if (ctx->stream) cudaStreamSynchronize(ctx->stream);
  dfree(ctx->dS); dfree(ctx->dygen); dfree(ctx->dyef); dfree(ctx->dnesp); dfree(ctx->dc);
  dfree(ctx->deri); dfree(ctx->dpairtab); dfree(ctx->dntttt); dfree(ctx->dF); dfree(ctx->dJ);
  dfree(ctx->dK); dfree(ctx->djx); dfree(ctx->dfmpb); dfree(ctx->dorbsym); dfree(ctx->dplan); dfree(ctx->dcand);
  leave_arena(ctx);
  dfree(ctx->deri64);
  dfree(ctx->deri_w);
  dfree(ctx->dnb_j); dfree(ctx->dnb_em); dfree(ctx->dlr_ent); dfree(ctx->dgen_part); dfree(ctx->dgrad);
  dfree(ctx->dlr_e); dfree(ctx->dlrw_e); dfree(ctx->dlrw_jh);
  dfree(ctx->dred);
  if (ctx->hres) cudaFreeHost(ctx->hres);
 
  dfree(ctx->dsel_bits); dfree(ctx->dsel_owner); dfree(ctx->dsel_xam); dfree(ctx->dsel_evp);
  dfree(ctx->dpool_bits); dfree(ctx->dpool_xam); dfree(ctx->dpool_evp);
  dfree(ctx->dunit_pool); dfree(ctx->dunit_nsel); dfree(ctx->dunit_out); dfree(ctx->dscan_total);
  dfree(ctx->dFraw); dfree(ctx->dh_work);
  dfree(ctx->dh_col); dfree(ctx->dh_val);
  for (int i = 0; i < 2; ++i) {
    dfree(ctx->dout_bits[i]); dfree(ctx->dout_owner[i]); dfree(ctx->dout_xam[i]); dfree(ctx->dout_evp[i]);
    if (ctx->hbuf[i]) cudaFreeHost(ctx->hbuf[i]);
    for (cudaEvent_t e : {ctx->ev_gathered[i], ctx->ev_copied[i], ctx->ev_host[i]})
      if (e) cudaEventDestroy(e);
  }
  if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
  if (ctx->ev0) cudaEventDestroy(ctx->ev0);
  if (ctx->ev1) cudaEventDestroy(ctx->ev1);
  if (ctx->evk) cudaEventDestroy(ctx->evk);
  if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
  delete ctx;
}

const char* cipsi_last_error(const cipsi_ctx* ctx) { return ctx ? ctx->err.c_str() : "null context"; }

int cipsi_set_stream(cipsi_ctx* ctx, void* stream) {
  if (!ctx) return CIPSI_ERR_ARG;
  ctx->stream = stream ? (cudaStream_t)stream : ctx->own_stream;
  return CIPSI_OK;
}

static int set_integrals_common(cipsi_ctx* ctx, const int32_t* itsym, const int32_t* its,
                                const double* f, const double* aj, const double* ak,
                                const int16_t* ij0, const int32_t* ntttt, int64_t ninte) {
  const int n = ctx->d.norb, ns = ctx->d.nsym;
  if (!itsym || !its || !f || !aj || !ak || !ij0 || !ntttt || ninte < 1)
    return fail(ctx, CIPSI_ERR_ARG, "set_integrals: null array or empty integral list");
  CK(cudaSetDevice(ctx->device));
  ctx->itsym.assign(itsym, itsym + n);
  ctx->its.assign(its, its + ns * ns);
  std::vector<int8_t> orbsym(n);
  for (int i = 0; i < n; ++i) {
    if (itsym[i] < 1 || itsym[i] > ns) return fail(ctx, CIPSI_ERR_ARG, "itsym out of range");
    orbsym[i] = (int8_t)(itsym[i] - 1);
  }
  for (int i = 0; i < ns * ns; ++i)
    if (its[i] < 1 || its[i] > ns) return fail(ctx, CIPSI_ERR_ARG, "its out of range");
  // pair table: pair index (1-based) | irrep (1-based) << 24, as cip/ai.f reads ij0
  std::vector<int32_t> pt((size_t)n * n);
  auto IJ0 = [&](int i, int j) -> int { return ij0[(size_t)(j - 1) * n + (i - 1)]; };
  for (int i = 1; i <= n; ++i)
    for (int j = 1; j <= n; ++j) {
      const int mi = std::min(i, j), ma = std::max(i, j);
      const int pidx = IJ0(mi, ma);
      const int irr = (mi == ma) ? 1 : IJ0(ma, mi);
      if (pidx < 1 || irr < 1 || irr > ns)
        return fail(ctx, CIPSI_ERR_ARG, "ij0 holds an invalid pair index or irrep");
      pt[(size_t)(i - 1) * n + (j - 1)] = pidx | (irr << 24);
    }
  std::vector<int32_t> nt(ns + 1, 0);
  for (int s = 0; s < ns; ++s) nt[s + 1] = ntttt[s];
  const size_t nter = (size_t)n * (n + 1) / 2;
  std::vector<double> F(f, f + nter);
  // cip/ijkf.f:34-37 zeroes |F| < 1e-10
  for (auto& x : F)
    if (std::fabs(x) < 1.0e-10) x = 0.0;
  int rc;
  if ((rc = upload(ctx, &ctx->dorbsym, orbsym.data(), orbsym.size()))) return rc;
  if ((rc = upload(ctx, &ctx->dpairtab, pt.data(), pt.size()))) return rc;
  if ((rc = upload(ctx, &ctx->dntttt, nt.data(), nt.size()))) return rc;
  if ((rc = upload(ctx, &ctx->dF, F.data(), F.size()))) return rc;
  if ((rc = upload(ctx, &ctx->dJ, aj, nter))) return rc;
  if ((rc = upload(ctx, &ctx->dK, ak, nter))) return rc;
  std::vector<double> jx((size_t)2 * n * n);
  for (int i = 0; i < n; ++i)
    for (int j = 0; j <= i; ++j) {
      const size_t t = (size_t)i * (i + 1) / 2 + j;
      jx[(size_t)i * n + j] = jx[(size_t)j * n + i] = aj[t];
      jx[(size_t)n * n + (size_t)i * n + j] = jx[(size_t)n * n + (size_t)j * n + i] = aj[t] - ak[t];
    }
  if ((rc = upload(ctx, &ctx->djx, jx.data(), jx.size()))) return rc;
  CK(cudaStreamSynchronize(ctx->stream));  // pt, nt, F, jx leave scope
  ctx->ninte = ninte;
  return CIPSI_OK;
}

int cipsi_set_integrals(cipsi_ctx* ctx, const int32_t* itsym, const int32_t* its, const double* f,
                        const double* aj, const double* ak, const int16_t* ij0,
                        const int32_t* ntttt, const float* bijkl, int64_t ninte) {
  if (!ctx) return CIPSI_ERR_ARG;
  int rc = set_integrals_common(ctx, itsym, its, f, aj, ak, ij0, ntttt, ninte);
  if (rc) return rc;
  if (!bijkl) return fail(ctx, CIPSI_ERR_ARG, "bijkl is null");
  if ((rc = upload(ctx, &ctx->deri, bijkl, (size_t)ninte))) return rc;
  if (ctx->deri64) {
    ++ctx->buf_gen;
    dfree(ctx->deri64);
  }
  dfree(ctx->deri_w);
  if ((size_t)ninte * sizeof(double) <= kWidenMaxBytes) {
    CK(cudaMalloc((void**)&ctx->deri_w, (size_t)ninte * sizeof(double)));
    const int grid = (int)std::min<int64_t>((ninte + 255) / 256, 4096);
    k_widen<<<grid, 256, 0, ctx->stream>>>(ctx->deri, ctx->deri_w, ninte);
    CK(cudaGetLastError());
  }
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->have_int = true;
  return CIPSI_OK;
}

int cipsi_set_integrals_fp64(cipsi_ctx* ctx, const int32_t* itsym, const int32_t* its,
                             const double* f, const double* aj, const double* ak,
                             const int16_t* ij0, const int32_t* ntttt, const double* pqrs,
                             int64_t ninte) {
  if (!ctx) return CIPSI_ERR_ARG;
  if (!pqrs) return fail(ctx, CIPSI_ERR_ARG, "pqrs is null");
  std::vector<float> b((size_t)ninte);
  for (int64_t i = 0; i < ninte; ++i) b[i] = (float)pqrs[i];  // real*8 -> real*4 (RN)
  return cipsi_set_integrals(ctx, itsym, its, f, aj, ak, ij0, ntttt, b.data(), ninte);
}

int cipsi_set_integrals_f64store(cipsi_ctx* ctx, const int32_t* itsym, const int32_t* its,
                                 const double* f, const double* aj, const double* ak,
                                 const int16_t* ij0, const int32_t* ntttt, const double* pqrs,
                                 int64_t ninte) {
  if (!ctx) return CIPSI_ERR_ARG;
  if (!pqrs) return fail(ctx, CIPSI_ERR_ARG, "pqrs is null");
  int rc = set_integrals_common(ctx, itsym, its, f, aj, ak, ij0, ntttt, ninte);
  if (rc) return rc;
  if ((rc = upload(ctx, &ctx->deri64, pqrs, (size_t)ninte))) return rc;
  dfree(ctx->deri_w);
  if (!ctx->deri) {
    const float zero = 0.f;
    if ((rc = upload(ctx, &ctx->deri, &zero, 1))) return rc;
  }
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->have_int = true;
  return CIPSI_OK;
}

int cipsi_set_space(cipsi_ctx* ctx, const int32_t* ne, const int32_t* nd, const int32_t* trou,
                    const int32_t* part, int64_t ntp, const uint8_t* ygen, const uint8_t* ysaut,
                    const int32_t* nesp, const uint8_t* yef1) {
  if (!ctx) return CIPSI_ERR_ARG;
  if (!ne || !nd || !trou || !part || !ygen || !ysaut || !nesp || !yef1)
    return fail(ctx, CIPSI_ERR_ARG, "set_space: null array");
  const int ncf = ctx->d.ncf, n = ctx->d.norb, W = ctx->W, noca = ctx->d.noca;
  CK(cudaSetDevice(ctx->device));
  ctx->Sbits.assign((size_t)ncf * 2 * W, 0ull);
  ctx->rank.assign(ncf, 0);
  ctx->sigma.assign(ncf, 1.0);
  for (int k = 0; k < ncf; ++k) {
    const int nec = ne[k];
    if (nec < 0 || nec > 16 || (nec > 0 && (nd[k] < 0 || nd[k] + nec > ntp)))
      return fail(ctx, CIPSI_ERR_ARG, "set_space: bad ne/nd at determinant " + std::to_string(k + 1));
    // reference determinant bits over 2*norb spin orbitals
    std::vector<uint64_t> full(4, 0ull);  // spin orbital so (0-based) -> bit so
    auto setb = [&](int so, bool on) {
      if (on) full[so >> 6] |= 1ull << (so & 63);
      else full[so >> 6] &= ~(1ull << (so & 63));
    };
    auto getb = [&](int so) { return (full[so >> 6] >> (so & 63)) & 1ull; };
    for (int o = 0; o < noca; ++o) {
      setb(o, true);
      setb(o + n, true);
    }
    int sign = 1;
    for (int i = 0; i < nec; ++i) {
      const int h = trou[nd[k] + i], pp = part[nd[k] + i];
      if (h < 1 || h > 2 * n || pp < 1 || pp > 2 * n)
        return fail(ctx, CIPSI_ERR_ARG, "set_space: spin orbital out of range");
      const int h0 = h - 1, p0 = pp - 1;
      if (!getb(h0) || getb(p0))
        return fail(ctx, CIPSI_ERR_ARG, "set_space: invalid excitation list at determinant " +
                                            std::to_string(k + 1));
      // phase of a+_p a_h on the canonical string (reference pair convention)
      const int lo = std::min(h0, p0), hi = std::max(h0, p0);
      int cnt = 0;
      for (int so = lo + 1; so < hi; ++so) cnt += (int)getb(so);
      if (cnt & 1) sign = -sign;
      setb(h0, false);
      setb(p0, true);
    }
    ctx->sigma[k] = sign;
    ctx->rank[k] = nec;
    int nal = 0, nbe = 0;
    for (int o = 0; o < n; ++o) {
      if (getb(o)) {
        ctx->Sbits[(size_t)k * 2 * W + (o >> 6)] |= 1ull << (o & 63);
        ++nal;
      }
      if (getb(o + n)) {
        ctx->Sbits[(size_t)k * 2 * W + W + (o >> 6)] |= 1ull << (o & 63);
        ++nbe;
      }
    }
    if (nal != noca || nbe != noca)
      return fail(ctx, CIPSI_ERR_ARG, "set_space: determinant with Ms != 0");
  }
  ctx->ygen.assign(ygen, ygen + ncf);
  ctx->ysaut.assign(ysaut, ysaut + ncf);
  ctx->yef1.assign(yef1, yef1 + ncf);
  ctx->nesp.assign(nesp, nesp + ncf);
  for (int k = 0; k < ncf; ++k) {
    ctx->ygen[k] = ctx->ygen[k] ? 1 : 0;
    ctx->ysaut[k] = ctx->ysaut[k] ? 1 : 0;
    ctx->yef1[k] = ctx->yef1[k] ? 1 : 0;
  }
  int rc;
  if ((rc = upload(ctx, &ctx->dS, ctx->Sbits.data(), ctx->Sbits.size()))) return rc;
  if ((rc = upload(ctx, &ctx->dygen, ctx->ygen.data(), ctx->ygen.size()))) return rc;
  if ((rc = upload(ctx, &ctx->dyef, ctx->yef1.data(), ctx->yef1.size()))) return rc;
  if ((rc = upload(ctx, &ctx->dnesp, ctx->nesp.data(), ctx->nesp.size()))) return rc;
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->have_space = true;
  ctx->have_roots = false;  // coefficients need the phases of this space
  return CIPSI_OK;
}

int cipsi_set_roots(cipsi_ctx* ctx, const double* c, const double* e, const double* eb,
                    const double* emp, const double* teste, const double* taum,
                    const double* fmpb) {
  if (!ctx) return CIPSI_ERR_ARG;
  if (!ctx->have_space) return fail(ctx, CIPSI_ERR_STATE, "set_roots before set_space");
  if (!c || !e || !eb || !emp || !teste || !taum || !fmpb)
    return fail(ctx, CIPSI_ERR_ARG, "set_roots: null array");
  const int ncf = ctx->d.ncf, mt = ctx->d.metat, n = ctx->d.norb;
  CK(cudaSetDevice(ctx->device));
  std::vector<double> cc((size_t)ncf * mt);
  for (int k = 0; k < ncf; ++k)
    for (int m = 0; m < mt; ++m) cc[(size_t)k * mt + m] = ctx->sigma[k] * c[(size_t)m * ncf + k];
  for (int m = 0; m < mt; ++m) {
    ctx->e[m] = e[m];
    ctx->eb[m] = eb[m];
    ctx->emp[m] = emp[m];
    ctx->teste[m] = teste[m];
    ctx->taum[m] = taum[m];
  }
  int rc;
  if ((rc = upload(ctx, &ctx->dc, cc.data(), cc.size()))) return rc;
  if ((rc = upload(ctx, &ctx->dfmpb, fmpb, (size_t)2 * n))) return rc;
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->have_roots = true;
  return CIPSI_OK;
}

}  // extern "C"

namespace {

int check_run_args(cipsi_ctx* ctx, const cipsi_opts* o) {
  if (!ctx || !o) return CIPSI_ERR_ARG;
  if (!ctx->have_int || !ctx->have_space || !ctx->have_roots)
    return fail(ctx, CIPSI_ERR_STATE, "run before set_integrals / set_space / set_roots");
  if (o->nclass < 2 || o->nclass > kNClass) return fail(ctx, CIPSI_ERR_ARG, "nclass must be in [2, 10]");
  for (int i = 0; i + 1 < o->nclass; ++i)
    if (!(o->aval[i] >= 0.0) || (i > 0 && !(o->aval[i] > o->aval[i - 1])))
      return fail(ctx, CIPSI_ERR_ARG, "aval must be non-negative and increasing");
  return CIPSI_OK;
}

// Generators, their allowed rank changes and the work units of one run.
struct RunPlan {
  std::vector<int32_t> gens;   // generator indices (0-based); -1 = pertu block
  std::vector<uint8_t> gmask;  // allowed rank changes, bit (D + 2)
  std::vector<int32_t> ug, ur0, ur1;
  std::vector<long long> uslots;  // candidate slots per unit (block_candidates over its allowed blocks)
  long long max_slots = 0, all_slots = 0;
  bool pertu_ref = false, pertu_mono = false;
};

// of the singles of the reference: a block a warp (60 orbitals, S = 2001: 41.2 ms at 4, 41.7 at 6,
// 39.7 at 8, 40.5 at 12; 45 orbitals, S = 451: 4.12, 4.16, 3.88, 4.08)
constexpr int kLowChunk = 8;

// Blocks of removed electrons per work unit of the forward kernels.  k_cand's
// warps take the blocks of a unit on their own, so a unit wants a few per warp:
// 16 at the default r_chunk of 6 (2.7 r_chunk above it; r_chunk itself below,
// where the caller asks for fine units).  From 6 on, when the run has few
// blocks, no more than leaves six units per CTA, down to two blocks (37
// orbitals, S = 334: 940 us at six, 1027 at eight).
// (60 orbitals, S = 2001: 45.8 ms at 24, 45.5 at 16, 47.3 at 8, 55 at 60; one
// shard of 120 orbitals: 57, 55, 54 ms.)
int unit_blocks(int r_chunk, long long run_blocks, int sms) {
  if (r_chunk < 6) return r_chunk;
  return (int)std::max(2ll, std::min<long long>(8ll * r_chunk / 3, run_blocks / (12ll * sms)));
}
// all blocks of a run, about: generators times pairs of electrons
long long run_blocks(const cipsi_ctx* ctx, const cipsi_opts* o) {
  const long long nel = 2 * ctx->d.noca;
  long long n = 0;
  for (int k = 0; k < ctx->d.ncf; ++k)
    if (ctx->ygen[k] && !ctx->ysaut[k] && !(o->gen_mask && !o->gen_mask[k])) ++n;
  return n * (nel * (nel + 1) / 2);
}

// r_chunk: allowed R blocks per work unit; low_chunk: of the reference and its
// singles, which meet most of S
void plan_run(const cipsi_ctx* ctx, const cipsi_opts* o, int r_chunk, int low_chunk, RunPlan& pl) {
  const int ncf = ctx->d.ncf, W = ctx->W;
  // flags on the content of S (pertu.f:52-61)
  bool yd = false, ym = false, yf = false;
  for (int k = 0; k < ncf; ++k) {
    if (ctx->rank[k] == 1) ym = true;
    if (ctx->rank[k] == 0) yd = true;
    if (ctx->rank[k] == 2) yf = true;
  }
  if (ym) yf = true;
  std::vector<int32_t>& gens = pl.gens;
  std::vector<uint8_t>& gmask = pl.gmask;
  const bool pertu_ref = yf && !yd && ctx->d.isym == 1;  // isz == 0, !yion
  const bool pertu_mono = yf && ym;
  pl.pertu_ref = pertu_ref;
  pl.pertu_mono = pertu_mono;
  if (o->run_pertu && (pertu_ref || pertu_mono)) {
    gens.push_back(-1);
    gmask.push_back(0);
  }
  for (int k = 0; k < ncf; ++k) {
    if (!ctx->ygen[k] || ctx->ysaut[k]) continue;
    if (o->gen_mask && !o->gen_mask[k]) continue;
    const int nec = ctx->rank[k];
    // allowed rank changes, bit (D + 2); D = +2 (diexcit) always
    // (igene.f:34-35, 89-90, 199-200, 296-298)
    uint8_t m = 1u << 4;
    if (!((nec == 0 && ym) || (nec == 1 && yd))) {
      m |= 1u << 3;  // +1
      const bool stop1 = nec < 1 || (ym && nec == 1) || (nec == 2 && yd);
      if (!stop1) {
        m |= 1u << 2;  // 0
        if (!((nec == 3 && yd) || (nec == 2 && ym))) {
          m |= 1u << 1;  // -1
          if (!((nec == 2 && (yd || yf)) || (nec == 3 && ym) || (nec == 4 && yd))) m |= 1u << 0;
        }
      }
    }
    gens.push_back(k);
    gmask.push_back(m);
  }
  const int ngen = (int)gens.size();
  // work units: a generator's R blocks that have an allowed rank-change class
  // are split into chunks (one block per unit for rank 0, up to kLowChunk for rank 1,
  // which meet most of S; r_chunk blocks for the others), so one heavy
  // generator does not serialise on one SM; low-rank generators are queued
  // first.
  const int kRChunkHigh = std::max(1, r_chunk);
  constexpr int kPertuChunk = 128;
  std::vector<int32_t>& ug = pl.ug;
  std::vector<int32_t>& ur0 = pl.ur0;
  std::vector<int32_t>& ur1 = pl.ur1;
  const int n = ctx->d.norb, noca = ctx->d.noca, nel = 2 * noca;
  const int nR = nel + nel * (nel - 1) / 2;
  std::vector<int> order(ngen);
  for (int g = 0; g < ngen; ++g) order[g] = g;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    const int ra = gens[a] < 0 ? -1 : ctx->rank[gens[a]];
    const int rb = gens[b] < 0 ? -1 : ctx->rank[gens[b]];
    return ra < rb;
  });
  std::vector<int> hfe(nel), spe(nel);
  auto push = [&](int g, int a, int b, long long slots) {
    ug.push_back(g);
    ur0.push_back(a);
    ur1.push_back(b);
    pl.uslots.push_back(slots);
    pl.max_slots = std::max(pl.max_slots, slots);
    pl.all_slots += slots;
  };
  for (int g : order) {
    const int k = gens[g];
    if (k < 0) {
      const int ntot = (pertu_ref ? 1 : 0) + (pertu_mono ? 2 * noca * (n - noca) : 0);
      for (int t = 0; t < ntot; t += kPertuChunk) push(g, t, std::min(ntot, t + kPertuChunk), std::min(ntot, t + kPertuChunk) - t);
      continue;
    }
    // electrons of k: alpha orbitals ascending, then beta; HF-occupied?
    int ne = 0, nes[2] = {0, 0};
    for (int sp = 0; sp < 2; ++sp)
      for (int orb = 0; orb < n; ++orb)
        if ((ctx->Sbits[(size_t)k * 2 * W + sp * W + (orb >> 6)] >> (orb & 63)) & 1ull) {
          spe[ne] = sp;
          hfe[ne++] = orb < noca;
          ++nes[sp];
        }
    const int nv[2] = {n - nes[0], n - nes[1]};
    const uint8_t m = gmask[g];
    // rank-change class allowed for block r?  Its candidates (slots).
    auto block = [&](int r, long long& cands) {
      int hfR, nRr, e1, e2 = -1;
      if (r < nel) {
        e1 = r;
        hfR = hfe[r];
        nRr = 1;
      } else {
        int t = r - nel;
        e1 = 0;
        while (t >= nel - 1 - e1) {
          t -= nel - 1 - e1;
          ++e1;
        }
        e2 = e1 + 1 + t;
        hfR = hfe[e1] + hfe[e2];
        nRr = 2;
      }
      cands = block_candidates(nRr, e2 >= 0 && spe[e1] == spe[e2], nv[spe[e1]], nv[0], nv[1]);
      for (int aV = 0; aV <= nRr; ++aV)
        if (m & (1u << (hfR + aV - nRr + 2))) return true;
      return false;
    };
    const int kRChunk = ctx->rank[k] == 0 ? 1 : ctx->rank[k] == 1 ? low_chunk : kRChunkHigh;
    int cnt = 0, start = -1, last = -1;
    long long slots = 0;
    for (int r = 0; r < nR; ++r) {
      long long c;
      if (!block(r, c)) continue;
      if (start < 0) start = r;
      last = r;
      slots += c;
      if (++cnt == kRChunk) {
        push(g, start, r + 1, slots);
        cnt = 0;
        start = -1;
        slots = 0;
      }
    }
    if (start >= 0) push(g, start, last + 1, slots);
  }
}

// CTAs per SM of k_cand: ctas 0 = as many as fit, 1 or 2 = at most that many
int fwd_blocks_per_sm(int W, int R, int ctas) {
  const int fit = W == 1 ? (R == 1 ? cand_ctas<1, 1>() : R == 2 ? cand_ctas<1, 2>() : R == 4 ? cand_ctas<1, 4>()
                                                                                           : cand_ctas<1, 8>())
                         : (R == 1 ? cand_ctas<2, 1>() : R == 2 ? cand_ctas<2, 2>() : R == 4 ? cand_ctas<2, 4>()
                                                                                           : cand_ctas<2, 8>());
  return ctas == 0 ? fit : std::min(fit, ctas);
}

// Bytes of a candidate's slot, the most that the device's candidate buffer
// takes (runs with more slots go through it in parts), and the most that a
// context keeps for itself.
constexpr size_t cand_slot_bytes(int R) { return 8 * (size_t)R + 8 + 8 + 4 + 4; }
constexpr size_t kCandMaxBytes = (size_t)8 << 30;
constexpr size_t kCandOwnBytes = (size_t)256 << 20;
CandBuf cand_views(unsigned char* base, long long cap, int R) {
  CandBuf c;
  c.cap = cap;
  c.b = reinterpret_cast<double*>(base);
  c.mp = c.b + (size_t)R * cap;
  c.vp = c.mp + cap;
  c.code = reinterpret_cast<uint32_t*>(c.vp + cap);
  c.meta = c.code + cap;
  return c;
}

// A share of the device's free memory for a candidate buffer of up to `want`
// bytes: a quarter, the rest stays for records and for others
size_t cand_share(size_t want) {
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
    cudaGetLastError();
    return want;
  }
  return std::min(want, fr / 4);
}

// Room for a run's candidates: *cap slots, all of them or enough for the
// largest unit at least.
int reserve_cand(cipsi_ctx* ctx, long long max_slots, long long all_slots, long long* cap) {
  const size_t sb = cand_slot_bytes(roots_pad(ctx->d.metat));
  auto bytes = [&](long long slots) { return (size_t)((std::max(slots, 1ll) + 63) / 64 * 64) * sb; };
  const size_t need = bytes(max_slots), all = bytes(all_slots);
  const size_t own = ctx->cand_limit ? ctx->cand_limit : kCandOwnBytes;
  ctx->cand_shared = !ctx->cand_limit && all > own && ctx->device < kMaxDevices;
  // larger when it has to be, or when the memory for it is free
  auto grows = [&](size_t bytes, size_t want) {
    return bytes < need || (bytes < want && cand_share(want) > bytes);
  };
  cudaError_t e = cudaSuccess;
  size_t have;
  if (!ctx->cand_shared) {
    const size_t want = std::max(need, std::min(all, own));
    if (grows(ctx->cand_bytes, want)) {
      dfree(ctx->dcand);
      ctx->cand_bytes = 0;
      e = alloc_down(&ctx->dcand, need, cand_share(want), &ctx->cand_bytes);
    }
    have = ctx->cand_bytes;
  } else {
    CandArena& a = g_arena[ctx->device];
    std::lock_guard<std::mutex> hold(a.mu);
    if (!ctx->cand_user) {
      if (!a.busy) CK(cudaEventCreateWithFlags(&a.busy, cudaEventDisableTiming));
      ctx->cand_user = true;
      ++a.users;
    }
    const size_t want = std::min(all, kCandMaxBytes);
    if (grows(a.bytes, want)) {
      const size_t least = std::max(need, a.bytes);  // runs under way count on what it was
      CK(cudaEventSynchronize(a.busy));
      dfree(a.base);
      a.bytes = 0;
      e = alloc_down(&a.base, least, cand_share(want), &a.bytes);
    }
    have = a.bytes;
  }
  if (e != cudaSuccess)
    return fail(ctx, CIPSI_ERR_CUDA,
                "candidate buffer of " + std::to_string(need) + " bytes: " + cudaGetErrorString(e));
  *cap = (long long)(have / sb) / 64 * 64;
  return CIPSI_OK;
}

// Blocks per work unit where `cap` slots at a time go through the buffer: units
// of `ub`, or as many fewer as it takes to have three for every CTA (a part ends
// with its last unit: an active space of 120 orbitals, two roots, through 1 GB
// takes 111 ms, and 173 with units of 16 blocks, of which a part has half as many
// as CTAs; through 8 GB 67 ms).
int fitted_blocks(int ub, const RunPlan& pl, long long cap, int ctas) {
  const long long nu = (long long)pl.ug.size();
  if (cap >= pl.all_slots || nu == 0) return ub;
  const long long units = cap / std::max(1ll, pl.all_slots / nu);
  return units >= 3ll * ctas ? ub : (int)std::max(1ll, ub * units / (3ll * ctas));
}

// Units in parts whose slots add up to at most cap (a unit's own slots fit):
// the parts' first units, then the number of units; slot0: each unit's first
// slot in its part.
std::vector<int> cut_units(const std::vector<long long>& slots, long long cap, std::vector<long long>& slot0) {
  std::vector<int> cut{0};
  slot0.resize(slots.size());
  long long acc = 0;
  for (int u = 0; u < (int)slots.size(); ++u) {
    if (acc + slots[u] > cap && u > cut.back()) {
      cut.push_back(u);
      acc = 0;
    }
    slot0[u] = acc;
    acc += slots[u];
  }
  if (cut.back() != (int)slots.size()) cut.push_back((int)slots.size());
  return cut;
}

// k_pt2_one's shared-memory L_R capacity, dynamic shared memory and CTAs per
// SM.  ctas: 1 = one CTA per SM with a long list, else two: the part of a longer
// list is read from the block's global scratch, 8 bytes per entry, which costs
// less than halving the resident warps.  `total` and one CTA's static shared
// memory (up to 32 KB) fit an SM twice; `queues` of it are not the list's.
struct LaunchShape {
  int lr_cap;
  size_t smem;
  int blocks_per_sm;
};
LaunchShape list_shape(int ncf_max, size_t total, size_t queues, int blocks) {
  const size_t per_entry = 8;  // compact L_R entry
  LaunchShape ls;
  ls.lr_cap = (int)std::min<size_t>((size_t)ncf_max, (total - queues - 16) / per_entry);
  ls.smem = (((size_t)ls.lr_cap * per_entry + 15) & ~(size_t)15) + queues + 16;
  ls.blocks_per_sm = blocks;
  return ls;
}
// the adjoint form, which has no queues and 4 KB more of static sums
LaunchShape adj_shape(int ncf_max, int ctas) {
  return list_shape(ncf_max, (size_t)(ctas == 1 ? 188 : 78) * 1024, 0, ctas == 1 ? 1 : 2);
}
// the forward form, with its warps' epilogue queues
LaunchShape one_shape(int R, int ncf_max) {
  const size_t q = R == 1   ? sizeof(WarpQueue<1>)
                   : R == 2 ? sizeof(WarpQueue<2>)
                   : R == 4 ? sizeof(WarpQueue<4>)
                            : sizeof(WarpQueue<8>);
  return list_shape(ncf_max, (size_t)82 * 1024, kWarps * q, 2);
}

// The record pool (unit segments), for `cap` records.
int grow_pool(cipsi_ctx* ctx, long long cap) {
  const int W = ctx->W, mt = ctx->d.metat;
  ++ctx->buf_gen;
  dfree(ctx->dpool_bits); dfree(ctx->dpool_xam); dfree(ctx->dpool_evp);
  ctx->pool_cap = 0;
  CK(cudaMalloc(&ctx->dpool_bits, (size_t)cap * 2 * W * sizeof(uint64_t)));
  CK(cudaMalloc(&ctx->dpool_xam, (size_t)cap * sizeof(double)));
  CK(cudaMalloc(&ctx->dpool_evp, (size_t)cap * mt * sizeof(double)));
  ctx->pool_cap = cap;
  return CIPSI_OK;
}

// The device record arrays (cipsi_selection_get / raw), for `cap` records.
int grow_sel(cipsi_ctx* ctx, long long cap) {
  const int W = ctx->W, mt = ctx->d.metat;
  ++ctx->buf_gen;
  dfree(ctx->dsel_bits); dfree(ctx->dsel_owner); dfree(ctx->dsel_xam); dfree(ctx->dsel_evp);
  ctx->sel_cap = 0;
  CK(cudaMalloc(&ctx->dsel_bits, (size_t)cap * 2 * W * sizeof(uint64_t)));
  CK(cudaMalloc(&ctx->dsel_owner, (size_t)cap * sizeof(int32_t)));
  CK(cudaMalloc(&ctx->dsel_xam, (size_t)cap * sizeof(double)));
  CK(cudaMalloc(&ctx->dsel_evp, (size_t)cap * mt * sizeof(double)));
  ctx->sel_cap = cap;
  return CIPSI_OK;
}

// A plan as the kernels read it: per unit its first slot in the candidate
// buffer (8 bytes), generator slot, block range and number of slots (4 each);
// the generators and their masks.  Appended to `out` at a multiple of 64 bytes.
size_t pack_plan(const RunPlan& pl, const std::vector<long long>& slot0, std::vector<unsigned char>& out) {
  const size_t base = (out.size() + 63) / 64 * 64, ngen = pl.gens.size(), nu = pl.ug.size();
  out.resize(base + nu * (8 + 4 * 4) + ngen * 5);
  size_t off = base;
  auto put = [&](const void* src, size_t n) {
    if (n) std::memcpy(out.data() + off, src, n);
    off += n;
  };
  const std::vector<int32_t> ns(pl.uslots.begin(), pl.uslots.end());
  put(slot0.data(), nu * 8);
  put(pl.ug.data(), nu * 4);
  put(pl.ur0.data(), nu * 4);
  put(pl.ur1.data(), nu * 4);
  put(ns.data(), nu * 4);
  put(pl.gens.data(), ngen * 4);
  put(pl.gmask.data(), ngen);
  return base;
}
// the kernels' parameters of a packed plan at device address d
void set_plan(Params& p, const unsigned char* d, int nunits, int ngen) {
  const int32_t* u = reinterpret_cast<const int32_t*>(d + (size_t)nunits * 8);
  p.nunits = nunits;
  p.ngen = ngen;
  p.unit_g = u;
  p.unit_r0 = u + nunits;
  p.unit_r1 = u + 2 * (size_t)nunits;
  p.gens = u + 4 * (size_t)nunits;
  p.gen_dmask = reinterpret_cast<const uint8_t*>(p.gens + ngen);
}

// Device buffers of one run on ctx (counters, histogram, records; the plan,
// uploaded on stream st, unless the caller keeps it: slot0 null), sized for it;
// the unit tables for `units` at least.  (buf_gen counts what a batch's graph
// refers to: not the plan.)
int prepare_run(cipsi_ctx* ctx, const RunPlan& pl, const std::vector<long long>* slot0, cudaStream_t st,
                int units = 0) {
  const int nunits = (int)pl.ug.size();
  if (slot0) {
    ctx->hplan.clear();
    pack_plan(pl, *slot0, ctx->hplan);
    const size_t bytes = ctx->hplan.size();
    if (bytes > ctx->plan_cap || !ctx->dplan) {
      dfree(ctx->dplan);
      ctx->plan_cap = 0;
      CK(cudaMalloc(&ctx->dplan, std::max<size_t>(bytes, 64)));
      ctx->plan_cap = std::max<size_t>(bytes, 64);
    }
    ctx->nunits = nunits;
    ctx->ngen = (int)pl.gens.size();
    if (bytes) CK(cudaMemcpyAsync(ctx->dplan, ctx->hplan.data(), bytes, cudaMemcpyHostToDevice, st));
  }
  if (!ctx->dcounters) {
    ++ctx->buf_gen;
    if (!ctx->hres) CK(cudaMallocHost(&ctx->hres, kResWords * sizeof(unsigned long long)));
    CK(cudaMalloc(&ctx->dred, (kTabWord + kTabWords + kZeroWords) * sizeof(unsigned long long)));
    ctx->dhist_tab = ctx->dred + kTabWord;
    ctx->dcounters = reinterpret_cast<unsigned long long*>(ctx->dhist_tab + kTabWords);
  }
  if (ctx->pool_cap == 0) {
    const int rc = grow_pool(ctx, 1 << 20);
    if (rc) return rc;
  }
  if (ctx->sel_cap == 0) {
    const int rc = grow_sel(ctx, 1 << 20);
    if (rc) return rc;
  }
  units = std::max(units, nunits);
  if (units > ctx->unit_tab_cap) {
    ++ctx->buf_gen;
    dfree(ctx->dunit_pool); dfree(ctx->dunit_nsel); dfree(ctx->dunit_out);
    CK(cudaMalloc(&ctx->dunit_pool, (size_t)units * sizeof(long long)));
    CK(cudaMalloc(&ctx->dunit_nsel, (size_t)units * sizeof(int32_t)));
    CK(cudaMalloc(&ctx->dunit_out, (size_t)units * sizeof(long long)));
    ctx->unit_tab_cap = units;
  }
  if (!ctx->dscan_total) {
    ++ctx->buf_gen;
    CK(cudaMalloc(&ctx->dscan_total, sizeof(unsigned long long)));
  }
  return CIPSI_OK;
}

// Kernel parameters of one run on ctx (everything but the neighbour scratch
// and the L_R capacity).
void fill_params(const cipsi_ctx* ctx, const cipsi_opts* o, const RunPlan& pl, Params& p) {
  const int mt = ctx->d.metat, nunits = (int)pl.ug.size();
  p.norb = ctx->d.norb;
  p.noca = ctx->d.noca;
  p.nel = 2 * ctx->d.noca;
  p.ncf = ctx->d.ncf;
  p.metat = mt;
  p.nsym = ctx->d.nsym;
  p.isym = ctx->d.isym;
  set_plan(p, ctx->dplan, nunits, (int)pl.gens.size());
  p.S = ctx->dS;
  p.ygen = ctx->dygen;
  p.nesp = ctx->dnesp;
  p.yef = ctx->dyef;
  p.c = ctx->dc;
  p.eri = ctx->deri;
  p.eri64 = ctx->deri64 ? ctx->deri64 : ctx->deri_w;
  p.pairtab = ctx->dpairtab;
  p.ntttt = ctx->dntttt;
  p.F = ctx->dF;
  p.J = ctx->dJ;
  p.K = ctx->dK;
  p.jx = ctx->djx;
  p.fmpb = ctx->dfmpb;
  p.orbsym = ctx->dorbsym;
  for (int i = 0; i < ctx->d.nsym; ++i)
    for (int j = 0; j < ctx->d.nsym; ++j) p.its[i][j] = ctx->its[(size_t)j * ctx->d.nsym + i] - 1;
  for (int m = 0; m < mt; ++m) {
    p.e[m] = ctx->e[m];
    p.eb[m] = ctx->eb[m];
    p.emp[m] = ctx->emp[m];
    p.teste[m] = ctx->teste[m];
    p.taum[m] = ctx->taum[m];
  }
  p.yen = o->yen;
  p.ysele = o->ysele;
  p.ymoyen = o->ymoyen;
  p.ywdeg = o->ywdeg;
  p.symvar = o->sym_variant;
  p.nclass = o->nclass;
  p.tau = o->tau;
  p.teseff = o->teseff;
  for (int i = 0; i < kNClass; ++i) {
    p.aval[i] = o->aval[i];
    std::memcpy(&p.aval_bits[i], &o->aval[i], 8);
    p.aval_hi[i] = i + 1 < o->nclass ? (int)(p.aval_bits[i] >> 32) : 0x7fffffff;
  }
  p.pertu_ref = pl.pertu_ref ? 1 : 0;
  p.pertu_mono = pl.pertu_mono ? 1 : 0;
  set_zeroed(p, ctx->dcounters);
  p.hist_tab = ctx->dhist_tab;
  p.red = ctx->dred;
  p.rec_mode = 1;
  p.pool_bits = ctx->dpool_bits;
  p.pool_xam = ctx->dpool_xam;
  p.pool_evp = ctx->dpool_evp;
  p.pool_cap = ctx->pool_cap;
  p.unit_pool = ctx->dunit_pool;
  p.unit_nsel = ctx->dunit_nsel;
}

// Output arrays of a run's records: the caller's pinned sink or the
// context's device arrays.
void record_target(const cipsi_ctx* ctx, GatherArgs& a) {
  if (ctx->sink) {
    a.out_bits = ctx->sink_bits;
    a.out_owner = ctx->sink_owner;
    a.out_xam = ctx->sink_xam;
    a.out_evp = ctx->sink_evp;
    a.out_cap = ctx->sink_cap;
  } else {
    a.out_bits = ctx->dsel_bits;
    a.out_owner = ctx->dsel_owner;
    a.out_xam = ctx->dsel_xam;
    a.out_evp = ctx->dsel_evp;
    a.out_cap = ctx->sel_cap;
  }
}

// Scan + gather of units [u0, u1) of run `p` (records at output offset
// out_base.. of the target in `a`), enqueued on st.
cudaError_t enqueue_gather(const cipsi_ctx* ctx, const Params& p, int u0, int u1, long long out_base, GatherArgs a,
                           cudaStream_t st, int dev_sms) {
  if (u1 <= u0) return cudaSuccess;
  k_scan_units<<<1, kScanThreads, 0, st>>>(p.unit_nsel, ctx->dunit_out, u0, u1, out_base, ctx->dscan_total);
  a.pool_bits = p.pool_bits;
  a.pool_xam = p.pool_xam;
  a.pool_evp = p.pool_evp;
  a.pool_cap = p.pool_cap;
  a.unit_pool = p.unit_pool;
  a.unit_nsel = p.unit_nsel;
  a.unit_out = ctx->dunit_out;
  a.unit_g = p.unit_g;
  a.gens = p.gens;
  a.u0 = u0;
  a.u1 = u1;
  a.words = 2 * ctx->W;
  a.metat = ctx->d.metat;
  a.out_base = out_base;
  const int grid = std::max(1, std::min(u1 - u0, 4 * dev_sms));
  k_gather<<<grid, 256, 0, st>>>(a);
  return cudaGetLastError();
}

// entries of a warp's L_R overflow lists for S of ncf determinants
int lrw_entries(int ncf) { return std::min(kLrWarpG, ncf); }

// Per-CTA neighbour and L_R scratch for `grid` CTAs.
int ensure_neighbour_scratch(cipsi_ctx* ctx, int grid) {
  if ((size_t)grid <= ctx->scratch_blocks && ctx->dnb_j) return CIPSI_OK;
  const int ncf = ctx->d.ncf;
  // two CTAs per SM, the most that any run launches: a later run with more units
  // finds room (and a batch of this context stays valid)
  int sms = 0;
  CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
  grid = std::max(grid, 2 * sms);
  ++ctx->buf_gen;
  dfree(ctx->dnb_j); dfree(ctx->dnb_em); dfree(ctx->dlr_ent);
  dfree(ctx->dlr_e); dfree(ctx->dlrw_e); dfree(ctx->dlrw_jh);
  ctx->scratch_blocks = 0;
  const size_t nw = (size_t)grid * kWarps * 2 * lrw_entries(ncf);
  CK(cudaMalloc(&ctx->dlr_e, (size_t)grid * ncf * sizeof(uint32_t)));
  CK(cudaMalloc(&ctx->dlrw_e, nw * sizeof(uint32_t)));
  CK(cudaMalloc(&ctx->dlrw_jh, nw * sizeof(uint2)));
  CK(cudaMalloc(&ctx->dnb_j, (size_t)grid * ncf * sizeof(int32_t)));
  CK(cudaMalloc(&ctx->dnb_em, (size_t)grid * ncf * sizeof(uint64_t)));
  CK(cudaMalloc(&ctx->dlr_ent, (size_t)grid * ncf * sizeof(uint64_t)));
  ctx->scratch_blocks = grid;
  return CIPSI_OK;
}

// the context's neighbour and L_R scratch into the kernel's parameters
void set_scratch(const cipsi_ctx* ctx, Params& p) {
  p.nb_j = ctx->dnb_j;
  p.nb_emask = ctx->dnb_em;
  p.lr_ent = ctx->dlr_ent;
  p.lr_jh = reinterpret_cast<uint2*>(ctx->dlr_ent);
  p.lr_e = ctx->dlr_e;
  p.lrw_e = ctx->dlrw_e;
  p.lrw_jh = ctx->dlrw_jh;
  p.lrw_cap = lrw_entries(ctx->d.ncf);
  p.nb_stride = ctx->d.ncf;
}

// both forward kernels of class (W, R) on the units of `la`: the candidate
// buffer's marks cleared, then k_cand on `grid` CTAs and k_pt2
template <bool B>
cudaError_t launch_forward(const Params& p, const LaunchArgs& la, int W, int R, int grid, int sms, long long slots,
                           cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(la.cand.meta, 0, (size_t)slots * sizeof(uint32_t), st);
  if (e != cudaSuccess) return e;
#define CIPSI_FORWARD(W_, R_)                                  \
  if (W == W_ && R == R_) {                                    \
    e = launch_cand<W_, R_, B>(p, la, grid, st);               \
    return e != cudaSuccess ? e : launch_pt2<W_, R_, B>(p, la, sms, st); \
  }
  CIPSI_FORWARD(1, 1)
  CIPSI_FORWARD(1, 2)
  CIPSI_FORWARD(1, 4)
  CIPSI_FORWARD(1, 8)
  CIPSI_FORWARD(2, 1)
  CIPSI_FORWARD(2, 2)
  CIPSI_FORWARD(2, 4)
  CIPSI_FORWARD(2, 8)
#undef CIPSI_FORWARD
  return cudaErrorInvalidValue;
}

// units [u0, u1) of the context's plan
LaunchArgs plan_args(const cipsi_ctx* ctx, const Params& p, int u0, int u1) {
  LaunchArgs la{};
  la.unit_slot = reinterpret_cast<const long long*>(ctx->dplan) + u0;
  la.unit_nslots = reinterpret_cast<const int32_t*>(ctx->dplan + (size_t)ctx->nunits * 8) + 3 * (size_t)ctx->nunits + u0;
  la.nunits = u1 - u0;
  la.work = p.work;
  return la;
}
// the parameters of a launch over units u0.. of the plan
Params part_params(const Params& p, int u0) {
  Params q = p;
  q.unit_g += u0;
  q.unit_r0 += u0;
  q.unit_r1 += u0;
  q.unit_pool += u0;
  q.unit_nsel += u0;
  return q;
}

// both forward kernels over units [u0, u1) of the context's plan, `slots` in all
int launch_part(cipsi_ctx* ctx, const Params& p, int u0, int u1, int grid, int sms, long long slots) {
  const int R = roots_pad(ctx->d.metat);
  const size_t sb = cand_slot_bytes(R);
  LaunchArgs la = plan_args(ctx, p, u0, u1);
  auto launch = [&](unsigned char* base, size_t bytes) {
    la.cand = cand_views(base, (long long)(bytes / sb) / 64 * 64, R);
    return slots <= la.cand.cap ? launch_forward<false>(part_params(p, u0), la, ctx->W, R, grid, sms, slots, ctx->stream)
                                : cudaErrorMemoryAllocation;
  };
  cudaError_t e;
  if (!ctx->cand_shared) {
    e = launch(ctx->dcand, ctx->cand_bytes);
  } else {
    CandArena& a = g_arena[ctx->device];
    std::lock_guard<std::mutex> hold(a.mu);
    e = cudaStreamWaitEvent(ctx->stream, a.busy, 0);
    if (e == cudaSuccess) {
      e = launch(a.base, a.bytes);
      const cudaError_t r = cudaEventRecord(a.busy, ctx->stream);  // whatever was enqueued
      if (e == cudaSuccess) e = r;
    }
  }
  if (e != cudaSuccess)
    return fail(ctx, CIPSI_ERR_CUDA, std::string("k_cand / k_pt2 launch: ") + cudaGetErrorString(e));
  return CIPSI_OK;
}

}  // namespace

extern "C" {

int cipsi_set_tuning(cipsi_ctx* ctx, int32_t r_chunk, int32_t ctas_per_sm) {
  if (!ctx) return CIPSI_ERR_ARG;
  if (r_chunk < 1 || r_chunk > 4096) return fail(ctx, CIPSI_ERR_ARG, "r_chunk must be in [1, 4096]");
  if (ctas_per_sm < 0 || ctas_per_sm > 2) return fail(ctx, CIPSI_ERR_ARG, "ctas_per_sm must be 0, 1 or 2");
  ctx->tune_r_chunk = r_chunk;
  ctx->tune_ctas = ctas_per_sm;
  return CIPSI_OK;
}

int cipsi_set_candidate_bytes(cipsi_ctx* ctx, int64_t bytes) {
  if (!ctx) return CIPSI_ERR_ARG;
  if (bytes < 0) return fail(ctx, CIPSI_ERR_ARG, "candidate bytes must not be negative");
  if (ctx->pending) return fail(ctx, CIPSI_ERR_STATE, "an asynchronous run is pending: fetch its result first");
  ctx->cand_limit = (size_t)bytes;
  dfree(ctx->dcand);
  ctx->cand_bytes = 0;
  return CIPSI_OK;
}

int cipsi_set_selection_sink(cipsi_ctx* ctx, uint64_t* bits, int32_t* owner, double* xam, double* evp,
                             int64_t capacity) {
  if (!ctx) return CIPSI_ERR_ARG;
  if (ctx->pending) return fail(ctx, CIPSI_ERR_STATE, "an asynchronous run is pending: fetch its result first");
  ++ctx->buf_gen;
  if (!bits) {
    ctx->sink = false;
    ctx->sink_bits = nullptr;
    ctx->sink_owner = nullptr;
    ctx->sink_xam = ctx->sink_evp = nullptr;
    ctx->sink_cap = 0;
    ctx->nsel = 0;
    return CIPSI_OK;
  }
  if (!owner || !xam || !evp || capacity < 1)
    return fail(ctx, CIPSI_ERR_ARG, "selection sink: null array or capacity < 1");
  CK(cudaSetDevice(ctx->device));
  void* host[4] = {bits, owner, xam, evp};
  void* dev[4] = {nullptr, nullptr, nullptr, nullptr};
  for (int i = 0; i < 4; ++i) {
    cudaPointerAttributes a{};
    CK(cudaPointerGetAttributes(&a, host[i]));
    if (a.type != cudaMemoryTypeHost)
      return fail(ctx, CIPSI_ERR_ARG, "selection sink: arrays must be pinned host memory (cudaHostAlloc or "
                                      "cudaHostRegister)");
    CK(cudaHostGetDevicePointer(&dev[i], host[i], 0));
  }
  ctx->sink = true;
  ctx->sink_bits = static_cast<uint64_t*>(dev[0]);
  ctx->sink_owner = static_cast<int32_t*>(dev[1]);
  ctx->sink_xam = static_cast<double*>(dev[2]);
  ctx->sink_evp = static_cast<double*>(dev[3]);
  ctx->sink_cap = capacity;
  for (int i = 0; i < 4; ++i) ctx->sink_host[i] = host[i];
  ctx->nsel = 0;
  return CIPSI_OK;
}

int cipsi_run_pt2_async(cipsi_ctx* ctx, const cipsi_opts* o) {
  int rc = check_run_args(ctx, o);
  if (rc) return rc;
  CK(cudaSetDevice(ctx->device));
  const int W = ctx->W, mt = ctx->d.metat;
  int dev_sms = 0;
  CK(cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, ctx->device));
  RunPlan pl;
  const int ub = unit_blocks(ctx->tune_r_chunk, run_blocks(ctx, o), dev_sms);
  plan_run(ctx, o, ub, std::min(ub, kLowChunk), pl);
  const int ctas = dev_sms * fwd_blocks_per_sm(W, roots_pad(mt), ctx->tune_ctas);
  long long cap = 0;
  rc = reserve_cand(ctx, pl.max_slots, pl.all_slots, &cap);
  if (rc) return rc;
  const int fit = fitted_blocks(ub, pl, cap, ctas);
  if (fit < ub) plan_run(ctx, o, fit, std::min(fit, kLowChunk), pl = RunPlan{});
  const int nunits = (int)pl.ug.size();
  const int grid = std::max(1, std::min(nunits, ctas));
  rc = ensure_neighbour_scratch(ctx, grid);
  if (rc) return rc;
  std::vector<long long> slot0;
  const std::vector<int> cut = cut_units(pl.uslots, cap, slot0);
  rc = prepare_run(ctx, pl, &slot0, ctx->stream);
  if (rc) return rc;
  CK(cudaMemsetAsync(ctx->dcounters, 0, kZeroWords * sizeof(unsigned long long), ctx->stream));

  Params p{};
  fill_params(ctx, o, pl, p);
  set_scratch(ctx, p);

  CK(cudaEventRecord(ctx->ev0, ctx->stream));
  if (nunits > 0) {
    for (size_t c = 0; c + 1 < cut.size(); ++c) {
      const int u0 = cut[c], u1 = cut[c + 1];
      if (c) CK(cudaMemsetAsync(p.work, 0, 2 * sizeof(int), ctx->stream));
      rc = launch_part(ctx, p, u0, u1, std::min(grid, u1 - u0), dev_sms, slot0[u1 - 1] + pl.uslots[u1 - 1]);
      if (rc) return rc;
    }
    CK(cudaEventRecord(ctx->evk, ctx->stream));
    ctx->last_launches = 2 * (long long)(cut.size() - 1) + 3;  // and the unit scan, the gather, k_finish
    GatherArgs ga{};
    record_target(ctx, ga);
    const cudaError_t e = enqueue_gather(ctx, p, 0, nunits, 0, ga, ctx->stream, dev_sms);
    if (e != cudaSuccess) return fail(ctx, CIPSI_ERR_CUDA, std::string("record gather: ") + cudaGetErrorString(e));
  } else {
    CK(cudaEventRecord(ctx->evk, ctx->stream));
    ctx->last_launches = 1;
  }
  k_finish<<<1, kFinishThreads, 0, ctx->stream>>>(p, nullptr);
  CK(cudaGetLastError());
  CK(cudaEventRecord(ctx->ev1, ctx->stream));
  ctx->ev_valid = true;
  ctx->nclass = o->nclass;
  ctx->pending = true;
  ctx->last_opts = *o;
  return CIPSI_OK;
}

int cipsi_fetch_result(cipsi_ctx* ctx, cipsi_result* r) {
  if (!ctx || !r) return CIPSI_ERR_ARG;
  if (!ctx->pending) return fail(ctx, CIPSI_ERR_STATE, "fetch_result without a run");
  CK(cudaSetDevice(ctx->device));
  if (ctx->ext_done) {
    CK(cudaEventSynchronize(ctx->ext_done));
    ctx->ext_done = nullptr;
  }
  // (one copy and one wait; with three blocking copies a call on the 20-orbital
  // system took 286 us instead of 258)
  CK(cudaMemcpyAsync(ctx->hres, ctx->dred, kResWords * sizeof(unsigned long long), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->pending = false;
  const int mt = ctx->d.metat;
  memset(r, 0, sizeof(*r));
  const double* red = reinterpret_cast<const double*>(ctx->hres);
  for (int m = 0; m < mt; ++m) {
    r->e2mp[m] = red[0 * mt + m];
    r->e2vp[m] = red[1 * mt + m];
    r->e2b[m] = red[2 * mt + m];
    r->psimp[m] = red[3 * mt + m];
    r->psivp[m] = red[4 * mt + m];
  }
  const double* tab = red + kTabWord;
  const unsigned long long* cnt = ctx->hres + kTabWord + kTabWords;
  r->ietat = (int64_t)cnt[C_IETAT];
  r->n_processed = (int64_t)cnt[C_NPROC];
  r->n_candidates = (int64_t)cnt[C_NCAND];
  r->n_compares = (int64_t)cnt[C_NCMP];
  r->n_pairs_1 = (int64_t)cnt[C_NP1];
  r->n_pairs_2 = (int64_t)cnt[C_NP2];
  {
    unsigned long long b = cnt[C_NCOUNTERS];
    double dp;
    memcpy(&dp, &b, 8);
    r->dpivot = dp;
  }
  const int nc = ctx->nclass;
  for (int i = 0; i < nc; ++i) r->nom[i] = (int64_t)cnt[C_NCOUNTERS + 1 + i];
  for (int c = 0; c < nc; ++c)
    for (int m = 0; m < mt; ++m) {
      r->nam[c * kMaxRoots + m] = (int64_t)cnt[C_NCOUNTERS + 1 + kNClass + c * mt + m];
      r->tabmp[c * kMaxRoots + m] = tab[c * mt + m];
      r->tabvp[c * kMaxRoots + m] = tab[nc * mt + c * mt + m];
    }
  // algorithmic bytes of the E2 loop (per interacting pair: metat coefficients
  // + integrals as stored; per perturber: diagonal terms), see the docs
  const double avg_rank = 4.0;
  r->alg_bytes = (int64_t)(cnt[C_NP2] * (8.0 * mt + 2 * 4.0 + 8.0) +
                           cnt[C_NP1] * (8.0 * mt + 8.0 + 2.0 * avg_rank * 2 * 4.0) +
                           cnt[C_NPROC] * (8.0 * avg_rank + 8.0 * (avg_rank + avg_rank * avg_rank) + 8.0 * mt));
  float ms = -1.f, mk = -1.f;  // batched runs: the batch's time is reported by the batch
  if (ctx->ev_valid) {
    CK(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    CK(cudaEventElapsedTime(&mk, ctx->ev0, ctx->evk));
  }
  r->kernel_ms = ms;
  r->pt2_ms = mk;
  r->launches = ctx->ev_valid ? ctx->last_launches : 0;
  // selection: records stay on the device (or in the sink) until
  // cipsi_selection_get/raw
  const long long nsel = (long long)cnt[C_NSEL];
  r->n_selected = nsel;
  if (cnt[C_STAGE_OVF])
    return fail(ctx, CIPSI_ERR_CUDA, "internal error: a candidate's slot lay outside its work unit");
  // the records are valid when every unit segment found room in the pool;
  // the output arrays then hold the first out_cap of them, in unit order
  const long long out_cap = ctx->sink ? ctx->sink_cap : ctx->sel_cap;
  ctx->nsel = nsel > ctx->pool_cap ? 0 : std::min(nsel, out_cap);
  if (nsel > ctx->pool_cap || nsel > out_cap)
    return fail(ctx, CIPSI_ERR_OVERFLOW,
                "selection buffer overflow: " + std::to_string(nsel) + " records > capacity " +
                    std::to_string(std::min(out_cap, ctx->pool_cap)) +
                    (nsel > ctx->pool_cap ? " (counted only; cipsi_run_pt2 grows the buffers and reruns)"
                     : ctx->sink         ? " (the sink holds the first records; the rest were counted only)"
                                         : " (cipsi_run_pt2 grows the buffer and reruns)"));
  return CIPSI_OK;
}

int cipsi_run_pt2(cipsi_ctx* ctx, const cipsi_opts* opts, cipsi_result* res) {
  for (int attempt = 0; attempt < 4; ++attempt) {
    int rc = cipsi_run_pt2_async(ctx, opts);
    if (rc) return rc;
    rc = cipsi_fetch_result(ctx, res);
    if (rc != CIPSI_ERR_OVERFLOW) return rc;
    // grow the pool (and the device record arrays) to what the run needed
    // and redo; a caller's sink that is too small stays the caller's
    const long long nsel = res->n_selected;
    const long long cap = nsel + nsel / 8 + 1024;
    if (nsel <= ctx->pool_cap && ctx->sink) return rc;
    if (nsel > ctx->pool_cap && (rc = grow_pool(ctx, cap))) return rc;
    if (!ctx->sink && nsel > ctx->sel_cap && (rc = grow_sel(ctx, cap))) return rc;
  }
  return fail(ctx, CIPSI_ERR_OVERFLOW, "selection buffer could not be grown");
}

}  // extern "C"

// ------------------------------------------------------- streamed records
// cipsi_run_pt2_stream: the run in chunks of consecutive work units whose
// candidate slots fit the record pool (a unit never selects more records
// than it has slots), so any selection size runs in bounded device memory.
// Per chunk, on the context stream: k_cand and k_pt2 over its units, the unit
// scan and the gather into one of two device record buffers; the copy
// stream then brings the chunk to a ring of two pinned host buffers piece
// by piece, and the caller's consumer gets each piece, in record order,
// while the GPU computes the next chunk.

namespace {

int ensure_stream_buffers(cipsi_ctx* ctx, long long cap, bool host, long long hb_cap) {
  const int W = ctx->W, mt = ctx->d.metat;
  if (cap > ctx->out_cap) {
    ++ctx->buf_gen;
    for (int i = 0; i < 2; ++i) {
      dfree(ctx->dout_bits[i]); dfree(ctx->dout_owner[i]); dfree(ctx->dout_xam[i]); dfree(ctx->dout_evp[i]);
    }
    ctx->out_cap = 0;
    for (int i = 0; i < 2; ++i) {
      CK(cudaMalloc(&ctx->dout_bits[i], (size_t)cap * 2 * W * sizeof(uint64_t)));
      CK(cudaMalloc(&ctx->dout_owner[i], (size_t)cap * sizeof(int32_t)));
      CK(cudaMalloc(&ctx->dout_xam[i], (size_t)cap * sizeof(double)));
      CK(cudaMalloc(&ctx->dout_evp[i], (size_t)cap * mt * sizeof(double)));
    }
    ctx->out_cap = cap;
  }
  if (!ctx->copy_stream) {
    CK(cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
    for (int i = 0; i < 2; ++i) {
      CK(cudaEventCreateWithFlags(&ctx->ev_gathered[i], cudaEventDisableTiming));
      CK(cudaEventCreateWithFlags(&ctx->ev_copied[i], cudaEventDisableTiming));
      CK(cudaEventCreateWithFlags(&ctx->ev_host[i], cudaEventDisableTiming));
    }
  }
  if (host && hb_cap > ctx->hbuf_cap) {
    for (int i = 0; i < 2; ++i)
      if (ctx->hbuf[i]) {
        cudaFreeHost(ctx->hbuf[i]);
        ctx->hbuf[i] = nullptr;
      }
    ctx->hbuf_cap = 0;
    const size_t bytes = (size_t)hb_cap * (2 * W * 8 + 8 + 8 + mt * 8);
    for (int i = 0; i < 2; ++i) CK(cudaHostAlloc(&ctx->hbuf[i], bytes, cudaHostAllocDefault));
    ctx->hbuf_cap = hb_cap;
  }
  return CIPSI_OK;
}

// the counters, histogram and sums of a finished run into *r (as
// cipsi_fetch_result), reading on the context stream
int read_results(cipsi_ctx* ctx, int nclass, cipsi_result* r) {
  const int mt = ctx->d.metat;
  const size_t ncount = kCountWords;
  std::vector<double> red(5 * mt), tab(2 * kNClass * kMaxRoots);
  std::vector<unsigned long long> cnt(ncount);
  CK(cudaMemcpyAsync(red.data(), ctx->dred, red.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaMemcpyAsync(cnt.data(), ctx->dcounters, ncount * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                     ctx->stream));
  CK(cudaMemcpyAsync(tab.data(), ctx->dhist_tab, tab.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  memset(r, 0, sizeof(*r));
  for (int m = 0; m < mt; ++m) {
    r->e2mp[m] = red[0 * mt + m];
    r->e2vp[m] = red[1 * mt + m];
    r->e2b[m] = red[2 * mt + m];
    r->psimp[m] = red[3 * mt + m];
    r->psivp[m] = red[4 * mt + m];
  }
  r->ietat = (int64_t)cnt[C_IETAT];
  r->n_processed = (int64_t)cnt[C_NPROC];
  r->n_candidates = (int64_t)cnt[C_NCAND];
  r->n_compares = (int64_t)cnt[C_NCMP];
  r->n_pairs_1 = (int64_t)cnt[C_NP1];
  r->n_pairs_2 = (int64_t)cnt[C_NP2];
  r->n_selected = (int64_t)cnt[C_NSEL];
  {
    const unsigned long long b = cnt[C_NCOUNTERS];
    memcpy(&r->dpivot, &b, 8);
  }
  for (int i = 0; i < nclass; ++i) r->nom[i] = (int64_t)cnt[C_NCOUNTERS + 1 + i];
  for (int c = 0; c < nclass; ++c)
    for (int m = 0; m < mt; ++m) {
      r->nam[c * kMaxRoots + m] = (int64_t)cnt[C_NCOUNTERS + 1 + kNClass + c * mt + m];
      r->tabmp[c * kMaxRoots + m] = tab[c * mt + m];
      r->tabvp[c * kMaxRoots + m] = tab[nclass * mt + c * mt + m];
    }
  const double avg_rank = 4.0;
  r->alg_bytes = (int64_t)(cnt[C_NP2] * (8.0 * mt + 2 * 4.0 + 8.0) +
                           cnt[C_NP1] * (8.0 * mt + 8.0 + 2.0 * avg_rank * 2 * 4.0) +
                           cnt[C_NPROC] * (8.0 * avg_rank + 8.0 * (avg_rank + avg_rank * avg_rank) + 8.0 * mt));
  if (cnt[C_STAGE_OVF])
    return fail(ctx, CIPSI_ERR_CUDA, "internal error: a candidate's slot lay outside its work unit");
  return CIPSI_OK;
}

}  // namespace

extern "C" {

int cipsi_run_pt2_stream(cipsi_ctx* ctx, const cipsi_opts* o, int64_t chunk_records, cipsi_record_fn fn,
                         void* user, cipsi_result* r) {
  int rc = check_run_args(ctx, o);
  if (rc) return rc;
  if (!r) return fail(ctx, CIPSI_ERR_ARG, "run_pt2_stream: null result");
  if (ctx->pending) return fail(ctx, CIPSI_ERR_STATE, "an asynchronous run is pending: fetch its result first");
  CK(cudaSetDevice(ctx->device));
  const int W = ctx->W, mt = ctx->d.metat;
  int dev_sms = 0;
  CK(cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, ctx->device));
  RunPlan pl;
  const int ub = unit_blocks(ctx->tune_r_chunk, run_blocks(ctx, o), dev_sms);
  plan_run(ctx, o, ub, std::min(ub, kLowChunk), pl);
  const int ctas = dev_sms * fwd_blocks_per_sm(W, roots_pad(mt), ctx->tune_ctas);
  // chunk capacity: what was asked, else what about half the free device
  // memory holds (pool + two record buffers), at most 2^29 records; at
  // least the largest unit's slots
  const long long rec_bytes = 2 * W * 8 + 8 + 8 * mt;
  long long cap = chunk_records;
  if (cap <= 0) {
    size_t fr = 0, tot = 0;
    CK(cudaMemGetInfo(&fr, &tot));
    const double have = (double)fr + (double)(ctx->pool_cap + 2 * ctx->out_cap) * (rec_bytes + 4);
    cap = std::min<long long>(1ll << 29, (long long)(0.45 * have / (3.0 * (rec_bytes + 4))));
    // with a consumer, about eight chunks once the run has more than 8M
    // slots: each chunk's records are delivered while the next computes,
    // so only the last chunk's delivery follows the kernels
    if (fn) {
      long long total = 0;
      for (long long x : pl.uslots) total += x;
      cap = std::min(cap, std::max<long long>(total / 8 + 1, 1ll << 20));
    }
  }
  cap = std::max(cap, std::max<long long>(pl.max_slots, 1024));
  // a chunk's candidates have to fit their buffer too
  long long cand_cap = 0;
  if ((rc = reserve_cand(ctx, pl.max_slots, std::min(cap, pl.all_slots), &cand_cap))) return rc;
  cap = std::min(cap, cand_cap);
  const int fit = fitted_blocks(ub, pl, cap, ctas);
  if (fit < ub) plan_run(ctx, o, fit, std::min(fit, kLowChunk), pl = RunPlan{});
  const int nunits = (int)pl.ug.size();
  const int grid = std::max(1, std::min(nunits, ctas));
  if ((rc = ensure_neighbour_scratch(ctx, grid))) return rc;
  std::vector<long long> slot0;
  const std::vector<int> cut = cut_units(pl.uslots, cap, slot0);
  if ((rc = prepare_run(ctx, pl, &slot0, ctx->stream))) return rc;
  if (ctx->pool_cap < cap && (rc = grow_pool(ctx, cap))) return rc;
  const long long hb_cap = std::min<long long>(cap, 1ll << 24);
  if ((rc = ensure_stream_buffers(ctx, cap, fn != nullptr, hb_cap))) return rc;
  const int nchunks = (int)cut.size() - 1;
  // per chunk: records gathered and records placed in the pool (pinned)
  unsigned long long* hcnt = nullptr;
  CK(cudaHostAlloc((void**)&hcnt, (size_t)std::max(1, 2 * nchunks) * sizeof(unsigned long long),
                   cudaHostAllocDefault));
  struct HostFree {
    unsigned long long* p;
    ~HostFree() { if (p) cudaFreeHost(p); }
  } hold{hcnt};

  CK(cudaMemsetAsync(ctx->dcounters, 0, kZeroWords * sizeof(unsigned long long), ctx->stream));
  Params p{};
  fill_params(ctx, o, pl, p);
  set_scratch(ctx, p);
  const size_t words = 2 * (size_t)W;

  long long delivered = 0;  // records handed to the consumer so far
  long long piece_no = 0;
  auto deliver = [&](int c) -> int {
    const int b = c & 1;
    CK(cudaEventSynchronize(ctx->ev_gathered[b]));
    const long long n = (long long)hcnt[2 * c];
    if ((long long)hcnt[2 * c + 1] > ctx->pool_cap)
      return fail(ctx, CIPSI_ERR_OVERFLOW, "internal error: a chunk's records overflowed the pool");
    CK(cudaStreamWaitEvent(ctx->copy_stream, ctx->ev_gathered[b], 0));
    const long long npieces = (n + hb_cap - 1) / hb_cap;
    for (long long j = 0; j <= npieces; ++j) {
      if (j < npieces) {
        const long long off = j * hb_cap, cnt = std::min(hb_cap, n - off);
        unsigned char* hb = static_cast<unsigned char*>(ctx->hbuf[(piece_no + j) & 1]);
        CK(cudaMemcpyAsync(hb, ctx->dout_bits[b] + off * words, (size_t)cnt * words * 8, cudaMemcpyDeviceToHost,
                           ctx->copy_stream));
        hb += (size_t)hb_cap * words * 8;
        CK(cudaMemcpyAsync(hb, ctx->dout_owner[b] + off, (size_t)cnt * 4, cudaMemcpyDeviceToHost, ctx->copy_stream));
        hb += (size_t)hb_cap * 8;
        CK(cudaMemcpyAsync(hb, ctx->dout_xam[b] + off, (size_t)cnt * 8, cudaMemcpyDeviceToHost, ctx->copy_stream));
        hb += (size_t)hb_cap * 8;
        CK(cudaMemcpyAsync(hb, ctx->dout_evp[b] + off * mt, (size_t)cnt * mt * 8, cudaMemcpyDeviceToHost,
                           ctx->copy_stream));
        CK(cudaEventRecord(ctx->ev_host[(piece_no + j) & 1], ctx->copy_stream));
      }
      if (j >= 1) {
        const long long off = (j - 1) * hb_cap, cnt = std::min(hb_cap, n - off);
        const int hbi = (int)((piece_no + j - 1) & 1);
        CK(cudaEventSynchronize(ctx->ev_host[hbi]));
        const unsigned char* hb = static_cast<const unsigned char*>(ctx->hbuf[hbi]);
        const uint64_t* hbits = reinterpret_cast<const uint64_t*>(hb);
        const int32_t* hown = reinterpret_cast<const int32_t*>(hb + (size_t)hb_cap * words * 8);
        const double* hxam = reinterpret_cast<const double*>(hb + (size_t)hb_cap * (words * 8 + 8));
        const double* hevp = reinterpret_cast<const double*>(hb + (size_t)hb_cap * (words * 8 + 16));
        if (fn(user, delivered, cnt, (int32_t)words, mt, hbits, hown, hxam, hevp) != 0) {
          cudaStreamSynchronize(ctx->copy_stream);
          return fail(ctx, CIPSI_ERR_ARG, "run_pt2_stream: the record consumer returned an error");
        }
        delivered += cnt;
      }
    }
    piece_no += npieces;
    CK(cudaEventRecord(ctx->ev_copied[b], ctx->copy_stream));
    return CIPSI_OK;
  };

  // both kernels of each chunk timed by a pair of events
  std::vector<cudaEvent_t> kev(2 * (size_t)nchunks, nullptr);
  struct EvFree {
    std::vector<cudaEvent_t>& v;
    ~EvFree() {
      for (cudaEvent_t e : v)
        if (e) cudaEventDestroy(e);
    }
  } evhold{kev};
  for (auto& e : kev) CK(cudaEventCreate(&e));
  CK(cudaEventRecord(ctx->ev0, ctx->stream));
  for (int c = 0; c < nchunks; ++c) {
    const int u0 = cut[c], u1 = cut[c + 1], b = c & 1;
    // the record buffer of this chunk was last read by chunk c - 2's copies
    if (c >= 2 && fn) CK(cudaStreamWaitEvent(ctx->stream, ctx->ev_copied[b], 0));
    // work counter and pool count (next to each other)
    CK(cudaMemsetAsync(p.work, 0, 2 * sizeof(unsigned long long), ctx->stream));
    CK(cudaEventRecord(kev[2 * c], ctx->stream));
    if ((rc = launch_part(ctx, p, u0, u1, std::min(grid, u1 - u0), dev_sms, slot0[u1 - 1] + pl.uslots[u1 - 1])))
      return rc;
    CK(cudaEventRecord(kev[2 * c + 1], ctx->stream));
    GatherArgs ga{};
    ga.out_bits = ctx->dout_bits[b];
    ga.out_owner = ctx->dout_owner[b];
    ga.out_xam = ctx->dout_xam[b];
    ga.out_evp = ctx->dout_evp[b];
    ga.out_cap = ctx->out_cap;
    const cudaError_t e = enqueue_gather(ctx, p, u0, u1, 0, ga, ctx->stream, dev_sms);
    if (e != cudaSuccess) return fail(ctx, CIPSI_ERR_CUDA, std::string("record gather: ") + cudaGetErrorString(e));
    CK(cudaMemcpyAsync(&hcnt[2 * c], ctx->dscan_total, 8, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaMemcpyAsync(&hcnt[2 * c + 1], p.pool_count, 8, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaEventRecord(ctx->ev_gathered[b], ctx->stream));
    if (fn && c >= 1 && (rc = deliver(c - 1))) return rc;
  }
  if (fn && nchunks >= 1 && (rc = deliver(nchunks - 1))) return rc;
  k_finish<<<1, kFinishThreads, 0, ctx->stream>>>(p, nullptr);
  CK(cudaGetLastError());
  CK(cudaEventRecord(ctx->ev1, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  if (fn) CK(cudaStreamSynchronize(ctx->copy_stream));
  if ((rc = read_results(ctx, o->nclass, r))) return rc;
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  r->kernel_ms = ms;
  double pt2 = 0.0;
  for (int c = 0; c < nchunks; ++c) {
    float t = 0.f;
    CK(cudaEventElapsedTime(&t, kev[2 * c], kev[2 * c + 1]));
    pt2 += t;
  }
  r->pt2_ms = pt2;
  r->launches = 4ll * nchunks + 1;
  for (int c = 0; c < nchunks; ++c)
    if ((long long)hcnt[2 * c + 1] > ctx->pool_cap)
      return fail(ctx, CIPSI_ERR_OVERFLOW, "internal error: a chunk's records overflowed the pool");
  if (fn && delivered != r->n_selected)
    return fail(ctx, CIPSI_ERR_CUDA, "internal error: " + std::to_string(delivered) + " records delivered of " +
                                         std::to_string(r->n_selected) + " selected");
  ctx->nsel = 0;  // the streamed records are the consumer's; none stay readable
  ctx->stream_chunks = nchunks;
  return CIPSI_OK;
}

// Order-sensitive digest of streamed records (a record consumer): per
// field array (bits, owner, xam, evp) a Fletcher-style pair of 64-bit sums
// over its words in record order, s1 = sum w_i and s2 = sum of the running
// s1, continued across calls; big pieces are split over host threads and
// the per-slice pairs combined in order.
int cipsi_record_digest(void* user, int64_t first, int64_t count, int32_t words, int32_t metat,
                        const uint64_t* bits, const int32_t* owner, const double* xam, const double* evp) {
  cipsi_digest* d = static_cast<cipsi_digest*>(user);
  if (!d || first != d->records) return -1;
  struct Pair {
    uint64_t s1 = 0, s2 = 0, n = 0;
  };
  auto fold = [](Pair& acc, const Pair& x) {
    acc.s2 += x.s2 + acc.s1 * x.n;
    acc.s1 += x.s1;
    acc.n += x.n;
  };
  // word i of a field array as a 64-bit integer
  auto run = [&](int field, uint64_t n) {
    auto word = [&](uint64_t i) -> uint64_t {
      if (field == 0) return bits[i];
      if (field == 1) return (uint64_t)(uint32_t)owner[i];
      uint64_t v;
      memcpy(&v, field == 2 ? &xam[i] : &evp[i], 8);
      return v;
    };
    auto slice = [&](uint64_t a, uint64_t b_) {
      Pair x;
      for (uint64_t i = a; i < b_; ++i) {
        x.s1 += word(i);
        x.s2 += x.s1;
      }
      x.n = b_ - a;
      return x;
    };
    const int nt = std::max(1, std::min<int>(d->threads > 0 ? d->threads : 1, (int)(n / 65536 + 1)));
    std::vector<Pair> part(nt);
    std::vector<std::thread> th;
    for (int t = 1; t < nt; ++t)
      th.emplace_back([&, t]() { part[t] = slice(n * t / nt, n * (t + 1) / nt); });
    part[0] = slice(0, n / nt);
    for (auto& x : th) x.join();
    Pair acc{d->s1[field], d->s2[field], 0};
    for (const Pair& x : part) fold(acc, x);
    d->s1[field] = acc.s1;
    d->s2[field] = acc.s2;
  };
  if (count > 0) {
    run(0, (uint64_t)count * (uint64_t)words);
    run(1, (uint64_t)count);
    run(2, (uint64_t)count);
    run(3, (uint64_t)count * (uint64_t)metat);
  }
  d->records += count;
  return 0;
}

}  // extern "C"

namespace {

// gradient buffers up to this size stay with the context
constexpr size_t kGradKeptBytes = (size_t)16 << 20;

// The adjoint launch behind cipsi_run_pt2_adjoint (geri given) and
// cipsi_run_pt2_adjoint_1e (geri null: no (pq|rs) gradient, the second pass
// over singles only).  e2, when given, receives the E2 sums of the same pass.
int run_adjoint(cipsi_ctx* ctx, const cipsi_opts* o, const double* seed, double* e2, double* gF, double* gJ,
                double* gK, double* geri, double* gfmpb, double* groots) {
  int rc = 0;
  if (ctx->pending) return fail(ctx, CIPSI_ERR_STATE, "an asynchronous run is pending: fetch its result first");
  CK(cudaSetDevice(ctx->device));
  const int ncf = ctx->d.ncf, W = ctx->W, mt = ctx->d.metat, n = ctx->d.norb;
  const int nt = n * (n + 1) / 2;
  RunPlan pl;
  plan_run(ctx, o, ctx->tune_r_chunk, 1, pl);
  const int nunits = (int)pl.ug.size();
  int dev_sms = 0;
  CK(cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, ctx->device));
  const int R = roots_pad(mt);
  const LaunchShape ls = adj_shape(ncf, ctx->tune_ctas);
  const int grid = std::max(1, std::min(nunits, dev_sms * ls.blocks_per_sm));
  rc = ensure_neighbour_scratch(ctx, grid);
  if (rc) return rc;
  const std::vector<long long> slot0(pl.ug.size(), 0);  // no candidate buffer
  rc = prepare_run(ctx, pl, &slot0, ctx->stream);
  if (rc) return rc;
  const size_t nq = (size_t)5 * mt;
  if ((size_t)std::max(nunits, 1) * nq > ctx->gen_part_cap) {  // per-unit partial sums
    dfree(ctx->dgen_part);
    ctx->gen_part_cap = 0;
    CK(cudaMalloc(&ctx->dgen_part, (size_t)std::max(nunits, 1) * nq * sizeof(double)));
    ctx->gen_part_cap = (size_t)std::max(nunits, 1) * nq;
  }
  CK(cudaMemsetAsync(ctx->dcounters, 0, kZeroWords * sizeof(unsigned long long), ctx->stream));
  CK(cudaMemsetAsync(ctx->dgen_part, 0, (size_t)std::max(nunits, 1) * nq * sizeof(double), ctx->stream));
  // gradient buffers, one after the other; those cleared come first.  A small
  // set is kept for the next call: allocated and freed each time, it can take
  // memory of the device's own for itself each time (16 orbitals, S = 60: 690 us
  // a call, 560 with other small buffers beside it)
  const int stride = 3 * nt + 2 * n;
  const bool one_e = geri == nullptr;
  auto part = [](size_t doubles) { return (doubles + 31) / 32 * 32; };
  const size_t n_eri = one_e ? 0 : part(ctx->ninte), n_t = part(nt), n_sl = part((size_t)grid * stride), n_r = part(3 * mt);
  const size_t zeroed = n_eri + n_t + n_sl + n_r, all = zeroed + 2 * n_t + part(2 * n);
  const bool kept = all * sizeof(double) <= kGradKeptBytes;
  double* mem = nullptr;
  auto release = [&]() {
    if (!kept) dfree(mem);
  };
  auto ck = [&](cudaError_t e, const char* what) {
    if (e == cudaSuccess) return 0;
    release();
    return fail(ctx, CIPSI_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  };
  if (kept && ctx->grad_cap < all) {
    dfree(ctx->dgrad);
    ctx->grad_cap = 0;
    CK(cudaMalloc(&ctx->dgrad, all * sizeof(double)));
    ctx->grad_cap = all;
  }
  if (!kept && (rc = ck(cudaMalloc(&mem, all * sizeof(double)), "cudaMalloc"))) return rc;
  double* const d_eri = kept ? ctx->dgrad : mem;
  double *const d_F = d_eri + n_eri, *const d_sl = d_F + n_t, *const d_roots = d_sl + n_sl;
  double *const d_J = d_roots + n_r, *const d_K = d_J + n_t, *const d_f = d_K + n_t;
  if ((rc = ck(cudaMemsetAsync(d_eri, 0, zeroed * sizeof(double), ctx->stream), "memset"))) return rc;

  Params p{};
  fill_params(ctx, o, pl, p);
  set_scratch(ctx, p);
  p.lr_cap = ls.lr_cap;
  p.rec_mode = 0;  // no records from an adjoint launch
  p.gen_part = ctx->dgen_part;
  for (int m = 0; m < mt; ++m) {
    p.seed_mp[m] = seed[m];
    p.seed_vp[m] = seed[mt + m];
    p.seed_b[m] = seed[2 * mt + m];
  }
  p.g_eri = d_eri;
  p.g_F = d_F;
  p.g_slice = d_sl;
  p.slice_stride = stride;
  p.g_roots = d_roots;
  p.adj_1e = one_e ? 1 : 0;
  if (nunits > 0) {
    cudaError_t e;
    if (W == 1) {
      e = R == 1 ? launch_pt2_one<1, 1, true>(p, grid, ls.smem, ctx->stream)
        : R == 2 ? launch_pt2_one<1, 2, true>(p, grid, ls.smem, ctx->stream)
        : R == 4 ? launch_pt2_one<1, 4, true>(p, grid, ls.smem, ctx->stream)
                 : launch_pt2_one<1, 8, true>(p, grid, ls.smem, ctx->stream);
    } else {
      e = R == 1 ? launch_pt2_one<2, 1, true>(p, grid, ls.smem, ctx->stream)
        : R == 2 ? launch_pt2_one<2, 2, true>(p, grid, ls.smem, ctx->stream)
        : R == 4 ? launch_pt2_one<2, 4, true>(p, grid, ls.smem, ctx->stream)
                 : launch_pt2_one<2, 8, true>(p, grid, ls.smem, ctx->stream);
    }
    if ((rc = ck(e, "adjoint k_pt2_one launch"))) return rc;
    k_reduce<<<(unsigned)nq, kReduceThreads, 0, ctx->stream>>>(ctx->dgen_part, nunits, (int)nq, ctx->dred);
  } else {
    if ((rc = ck(cudaMemsetAsync(ctx->dred, 0, nq * sizeof(double), ctx->stream), "memset"))) return rc;
  }
  k_slice_reduce<<<(stride + 255) / 256, 256, 0, ctx->stream>>>(d_sl, grid, stride, nt, d_F, d_J, d_K, d_f);
  if ((rc = ck(cudaGetLastError(), "k_slice_reduce"))) return rc;
  struct Out {
    double* host;
    const double* dev;
    size_t n;
  } outs[] = {{geri, d_eri, (size_t)ctx->ninte}, {gF, d_F, (size_t)nt}, {gJ, d_J, (size_t)nt},
              {gK, d_K, (size_t)nt}, {gfmpb, d_f, (size_t)2 * n}, {groots, d_roots, (size_t)3 * mt},
              {e2, ctx->dred, (size_t)3 * mt}};
  for (const Out& x : outs)
    if (x.host && (rc = ck(cudaMemcpyAsync(x.host, x.dev, x.n * sizeof(double), cudaMemcpyDeviceToHost,
                                           ctx->stream), "copy gradients")))
      return rc;
  if ((rc = ck(cudaStreamSynchronize(ctx->stream), "adjoint run"))) return rc;
  release();
  return CIPSI_OK;
}

}  // namespace

extern "C" {

int cipsi_run_pt2_adjoint(cipsi_ctx* ctx, const cipsi_opts* o, const double* seed, double* gF,
                          double* gJ, double* gK, double* geri, double* gfmpb, double* groots) {
  const int rc = check_run_args(ctx, o);
  if (rc) return rc;
  if (!seed || !gF || !gJ || !gK || !geri || !gfmpb || !groots)
    return fail(ctx, CIPSI_ERR_ARG, "run_pt2_adjoint: null seed or gradient array");
  return run_adjoint(ctx, o, seed, nullptr, gF, gJ, gK, geri, gfmpb, groots);
}

int cipsi_run_pt2_adjoint_1e(cipsi_ctx* ctx, const cipsi_opts* o, const double* seed, double* e2, double* gF,
                             double* gJ, double* gK, double* gfmpb, double* groots) {
  const int rc = check_run_args(ctx, o);
  if (rc) return rc;
  if (!seed || !e2 || !gF || !gJ || !gK || !gfmpb || !groots)
    return fail(ctx, CIPSI_ERR_ARG, "run_pt2_adjoint_1e: null seed, energy or gradient array");
  return run_adjoint(ctx, o, seed, e2, gF, gJ, gK, nullptr, gfmpb, groots);
}

int cipsi_selection_raw(cipsi_ctx* ctx, int64_t first, int64_t count, uint64_t* bits,
                        int32_t* owner, double* xam, double* evp) {
  if (!ctx) return CIPSI_ERR_ARG;
  if (first < 0 || count < 0 || first + count > ctx->nsel)
    return fail(ctx, CIPSI_ERR_ARG, "selection: range outside the selection");
  if (count == 0) return CIPSI_OK;
  CK(cudaSetDevice(ctx->device));
  const int W = ctx->W, mt = ctx->d.metat;
  if (ctx->sink) {
    // the records are already in host memory
    auto cp = [](void* dst, const void* src, size_t n) {
      if (dst && dst != src) std::memcpy(dst, src, n);
    };
    cp(bits, static_cast<const uint64_t*>(ctx->sink_host[0]) + (size_t)first * 2 * W, (size_t)count * 2 * W * 8);
    cp(owner, static_cast<const int32_t*>(ctx->sink_host[1]) + first, (size_t)count * 4);
    cp(xam, static_cast<const double*>(ctx->sink_host[2]) + first, (size_t)count * 8);
    cp(evp, static_cast<const double*>(ctx->sink_host[3]) + (size_t)first * mt, (size_t)count * mt * 8);
    return CIPSI_OK;
  }
  if (bits)
    CK(cudaMemcpyAsync(bits, ctx->dsel_bits + (size_t)first * 2 * W, (size_t)count * 2 * W * 8,
                       cudaMemcpyDeviceToHost, ctx->stream));
  if (owner)
    CK(cudaMemcpyAsync(owner, ctx->dsel_owner + first, (size_t)count * 4, cudaMemcpyDeviceToHost, ctx->stream));
  if (xam) CK(cudaMemcpyAsync(xam, ctx->dsel_xam + first, (size_t)count * 8, cudaMemcpyDeviceToHost, ctx->stream));
  if (evp)
    CK(cudaMemcpyAsync(evp, ctx->dsel_evp + (size_t)first * mt, (size_t)count * mt * 8,
                       cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  return CIPSI_OK;
}

int cipsi_selection_get(cipsi_ctx* ctx, int64_t first, int64_t count, int32_t* nec, int32_t* holes,
                        int32_t* parts, double* xam, double* evp, int32_t* owner) {
  if (!ctx) return CIPSI_ERR_ARG;
  const int W = ctx->W, n = ctx->d.norb, noca = ctx->d.noca;
  std::vector<uint64_t> bits((size_t)std::max<int64_t>(count, 0) * 2 * W);
  int rc = cipsi_selection_raw(ctx, first, count, bits.data(), owner, xam, evp);
  if (rc) return rc;
  for (int64_t i = 0; i < count; ++i) {
    int nh = 0, np = 0;
    int32_t* h = holes ? holes + i * 8 : nullptr;
    int32_t* pp = parts ? parts + i * 8 : nullptr;
    for (int q = 0; q < 8; ++q) {
      if (h) h[q] = 0;
      if (pp) pp[q] = 0;
    }
    for (int s = 0; s < 2; ++s)
      for (int w = 0; w < W; ++w) {
        const uint64_t word = bits[(size_t)i * 2 * W + s * W + w];
        const int lo = w * 64;
        const int nref = std::min(std::max(noca - lo, 0), 64);
        const uint64_t ref = nref >= 64 ? ~0ull : ((1ull << nref) - 1ull);
        uint64_t hm = ref & ~word, pm = word & ~ref;
        while (hm) {
          const int b = __builtin_ctzll(hm);
          hm &= hm - 1;
          if (h && nh < 8) h[nh] = lo + b + 1 + s * n;
          ++nh;
        }
        while (pm) {
          const int b = __builtin_ctzll(pm);
          pm &= pm - 1;
          if (pp && np < 8) pp[np] = lo + b + 1 + s * n;
          ++np;
        }
      }
    if (nh > 8) return fail(ctx, CIPSI_ERR_OVERFLOW, "selected determinant with excitation degree > 8");
    if (nec) nec[i] = nh;
  }
  return CIPSI_OK;
}


// ------------------------------------------------------ batched geometries
// One persistent launch per (words per spin string, roots) class runs the
// work units of many contexts (Autocip grid geometries of different sizes);
// the launches of all classes, the clearing and the reductions are captured
// once in a CUDA graph and replayed by cipsi_batch_run.

}  // extern "C"

struct cipsi_batch {
  int device = 0;
  std::string err;
  cudaStream_t stream = nullptr;
  std::vector<cipsi_ctx*> ctxs;
  std::vector<cipsi_opts> opts;
  std::vector<unsigned long long> buf_gen;
  Params* dgeo = nullptr;
  unsigned char* dplan = nullptr;  // every geometry's plan
  struct Class {
    int W = 1, R = 1;
    std::vector<int> geos;
    int nunits = 0, grid = 0, ncf_max = 0;
    int32_t* dunit_geo = nullptr;
    int32_t* dunit_local = nullptr;
    int* dwork = nullptr;
    int32_t* dnb_j = nullptr;
    uint64_t* dnb_em = nullptr;
    uint64_t* dlr_ent = nullptr;
    uint32_t *dlr_e = nullptr, *dlrw_e = nullptr;
    uint2* dlrw_jh = nullptr;
    // the units' slots and the candidate buffer, shared by the class's geometries
    unsigned char* dunit_slot = nullptr;
    unsigned char* dcand = nullptr;
    size_t cand_bytes = 0;
    std::vector<int> cut;
    std::vector<long long> part_slots;
    cudaStream_t st = nullptr;
    cudaEvent_t ev_join = nullptr;
  };
  std::vector<Class> classes;
  cudaEvent_t ev_fork = nullptr, ev0 = nullptr, ev1 = nullptr, done = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  bool pending = false;
};

namespace {

int bfail(cipsi_batch* b, int code, const std::string& msg) {
  if (b) b->err = msg;
  return code;
}

#define BCK(call)                                                                       \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess)                                                              \
      return bfail(b, CIPSI_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

void batch_free(cipsi_batch* b) {
  cudaSetDevice(b->device);
  if (b->stream) cudaStreamSynchronize(b->stream);
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  for (auto& c : b->classes) {
    dfree(c.dunit_geo); dfree(c.dunit_local); dfree(c.dwork);
    dfree(c.dnb_j); dfree(c.dnb_em); dfree(c.dlr_ent);
    dfree(c.dlr_e); dfree(c.dlrw_e); dfree(c.dlrw_jh);
    dfree(c.dunit_slot); dfree(c.dcand);
    if (c.st) cudaStreamDestroy(c.st);
    if (c.ev_join) cudaEventDestroy(c.ev_join);
  }
  dfree(b->dgeo);
  dfree(b->dplan);
  for (cudaEvent_t e : {b->ev_fork, b->ev0, b->ev1, b->done})
    if (e) cudaEventDestroy(e);
  if (b->stream) cudaStreamDestroy(b->stream);
}

}  // namespace

extern "C" {

int cipsi_batch_create(cipsi_batch** out, cipsi_ctx* const* ctxs, int32_t n, const cipsi_opts* opts,
                       int32_t r_chunk, int32_t ctas_per_sm) {
  if (!out) return CIPSI_ERR_ARG;
  *out = nullptr;
  cipsi_batch* b = new cipsi_batch();
  *out = b;
  if (!ctxs || !opts || n < 1) return bfail(b, CIPSI_ERR_ARG, "batch needs at least one context and its options");
  if (r_chunk < 1 || r_chunk > 4096 || ctas_per_sm < 0 || ctas_per_sm > 2)
    return bfail(b, CIPSI_ERR_ARG, "r_chunk must be in [1, 4096] and ctas_per_sm 0, 1 or 2");
  b->device = ctxs[0] ? ctxs[0]->device : 0;
  for (int i = 0; i < n; ++i) {
    cipsi_ctx* ctx = ctxs[i];
    if (!ctx) return bfail(b, CIPSI_ERR_ARG, "null context in batch");
    if (ctx->device != b->device) return bfail(b, CIPSI_ERR_ARG, "all contexts of a batch must use one device");
    if (ctx->pending) return bfail(b, CIPSI_ERR_STATE, "a context of the batch has a pending run");
    for (int j = 0; j < i; ++j)
      if (ctxs[j] == ctx) return bfail(b, CIPSI_ERR_ARG, "a context appears twice in the batch");
    const int rc = check_run_args(ctx, &opts[i]);
    if (rc) return bfail(b, rc, "context " + std::to_string(i) + ": " + ctx->err);
  }
  BCK(cudaSetDevice(b->device));
  BCK(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
  for (cudaEvent_t* e : {&b->ev_fork, &b->done})
    BCK(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  BCK(cudaEventCreate(&b->ev0));
  BCK(cudaEventCreate(&b->ev1));
  int dev_sms = 0;
  BCK(cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, b->device));

  // plan every geometry; per-context buffers as for a plain run
  std::vector<Params> P(n);
  std::vector<long long> work(n);
  std::vector<std::vector<long long>> uslots(n);
  std::vector<unsigned char> hplan;
  std::vector<size_t> plan_at(n);
  std::vector<int> plan_gens(n);
  b->ctxs.assign(ctxs, ctxs + n);
  b->opts.assign(opts, opts + n);
  long long all_blocks = 0;
  for (int i = 0; i < n; ++i) all_blocks += run_blocks(ctxs[i], &opts[i]);
  const int ub = unit_blocks(r_chunk, all_blocks, dev_sms);
  for (int i = 0; i < n; ++i) {
    cipsi_ctx* ctx = ctxs[i];
    b->opts[i].gen_mask = nullptr;  // used by the plan below only
    RunPlan pl;
    plan_run(ctx, &opts[i], ub, std::min(ub, kLowChunk), pl);
    // the plan is the batch's own: the context's is replaced by every plain run
    plan_at[i] = pack_plan(pl, std::vector<long long>(pl.ug.size(), 0), hplan);
    plan_gens[i] = (int)pl.gens.size();
    // a batch's units are larger than those of its contexts' own runs, which
    // should not outgrow the unit tables
    RunPlan own;
    const int oub = unit_blocks(ctx->tune_r_chunk, run_blocks(ctx, &opts[i]), dev_sms);
    if (oub < ub) plan_run(ctx, &opts[i], oub, std::min(oub, kLowChunk), own);
    if (prepare_run(ctx, pl, nullptr, b->stream, (int)own.ug.size())) return bfail(b, CIPSI_ERR_CUDA, "context " + std::to_string(i) + ": " + ctx->err);
    fill_params(ctx, &opts[i], pl, P[i]);
    uslots[i] = pl.uslots;
    work[i] = (long long)pl.ug.size() * ctx->d.ncf;
    const int W = ctx->W, R = roots_pad(ctx->d.metat);
    int c = 0;
    while (c < (int)b->classes.size() && !(b->classes[c].W == W && b->classes[c].R == R)) ++c;
    if (c == (int)b->classes.size()) {
      b->classes.emplace_back();
      b->classes[c].W = W;
      b->classes[c].R = R;
    }
    b->classes[c].geos.push_back(i);
  }
  BCK(cudaMalloc(&b->dplan, std::max<size_t>(hplan.size(), 64)));
  if (!hplan.empty()) BCK(cudaMemcpy(b->dplan, hplan.data(), hplan.size(), cudaMemcpyHostToDevice));
  for (int i = 0; i < n; ++i) set_plan(P[i], b->dplan + plan_at[i], P[i].nunits, plan_gens[i]);

  // per class: unit order (heaviest geometry first), launch shape, scratch
  for (auto& c : b->classes) {
    std::stable_sort(c.geos.begin(), c.geos.end(), [&](int x, int y) { return work[x] > work[y]; });
    std::vector<int32_t> ugeo, ulocal;
    std::vector<long long> slots;
    for (int i : c.geos) {
      c.ncf_max = std::max(c.ncf_max, ctxs[i]->d.ncf);
      for (int u = 0; u < P[i].nunits; ++u) {
        ugeo.push_back(i);
        ulocal.push_back(u);
        slots.push_back(uslots[i][u]);
      }
    }
    long long max_slots = 0, all_slots = 0;
    for (long long x : slots) {
      max_slots = std::max(max_slots, x);
      all_slots += x;
    }
    // the graph holds its address, so the buffer is the batch's own
    const size_t sb = cand_slot_bytes(c.R);
    auto bytes = [&](long long x) { return (size_t)((std::max(x, 1ll) + 63) / 64 * 64) * sb; };
    size_t want = std::min(bytes(all_slots), kCandMaxBytes);
    for (int i : c.geos)
      if (ctxs[i]->cand_limit) want = std::min(want, ctxs[i]->cand_limit);
    BCK(alloc_down(&c.dcand, bytes(max_slots), cand_share(want), &c.cand_bytes));
    const long long cap = (long long)(c.cand_bytes / sb) / 64 * 64;
    std::vector<long long> slot0;
    c.cut = cut_units(slots, cap, slot0);
    for (size_t q = 0; q + 1 < c.cut.size(); ++q) c.part_slots.push_back(slot0[c.cut[q + 1] - 1] + slots[c.cut[q + 1] - 1]);
    {
      const std::vector<int32_t> ns(slots.begin(), slots.end());
      BCK(cudaMalloc(&c.dunit_slot, std::max<size_t>(12 * slots.size(), 64)));
      if (!slots.empty()) {
        BCK(cudaMemcpy(c.dunit_slot, slot0.data(), 8 * slots.size(), cudaMemcpyHostToDevice));
        BCK(cudaMemcpy(c.dunit_slot + 8 * slots.size(), ns.data(), 4 * slots.size(), cudaMemcpyHostToDevice));
      }
    }
    c.nunits = (int)ugeo.size();
    c.grid = std::max(1, std::min(c.nunits, dev_sms * fwd_blocks_per_sm(c.W, c.R, ctas_per_sm)));
    BCK(cudaMalloc(&c.dunit_geo, (size_t)std::max(c.nunits, 1) * sizeof(int32_t)));
    BCK(cudaMalloc(&c.dunit_local, (size_t)std::max(c.nunits, 1) * sizeof(int32_t)));
    BCK(cudaMalloc(&c.dwork, 2 * sizeof(int)));
    BCK(cudaMalloc(&c.dnb_j, (size_t)c.grid * c.ncf_max * sizeof(int32_t)));
    BCK(cudaMalloc(&c.dnb_em, (size_t)c.grid * c.ncf_max * sizeof(uint64_t)));
    BCK(cudaMalloc(&c.dlr_ent, (size_t)c.grid * c.ncf_max * sizeof(uint64_t)));
    BCK(cudaMalloc(&c.dlr_e, (size_t)c.grid * c.ncf_max * sizeof(uint32_t)));
    const size_t nw = (size_t)c.grid * kWarps * 2 * lrw_entries(c.ncf_max);
    BCK(cudaMalloc(&c.dlrw_e, nw * sizeof(uint32_t)));
    BCK(cudaMalloc(&c.dlrw_jh, nw * sizeof(uint2)));
    if (c.nunits) {
      BCK(cudaMemcpy(c.dunit_geo, ugeo.data(), (size_t)c.nunits * sizeof(int32_t), cudaMemcpyHostToDevice));
      BCK(cudaMemcpy(c.dunit_local, ulocal.data(), (size_t)c.nunits * sizeof(int32_t), cudaMemcpyHostToDevice));
    }
    for (int i : c.geos) {
      P[i].nb_j = c.dnb_j;
      P[i].nb_emask = c.dnb_em;
      P[i].lr_ent = c.dlr_ent;
      P[i].lr_jh = reinterpret_cast<uint2*>(c.dlr_ent);
      P[i].lr_e = c.dlr_e;
      P[i].lrw_e = c.dlrw_e;
      P[i].lrw_jh = c.dlrw_jh;
      P[i].lrw_cap = lrw_entries(c.ncf_max);
      P[i].nb_stride = c.ncf_max;
    }
    BCK(cudaStreamCreateWithFlags(&c.st, cudaStreamNonBlocking));
    BCK(cudaEventCreateWithFlags(&c.ev_join, cudaEventDisableTiming));
  }
  BCK(cudaMalloc(&b->dgeo, (size_t)n * sizeof(Params)));
  BCK(cudaMemcpy(b->dgeo, P.data(), (size_t)n * sizeof(Params), cudaMemcpyHostToDevice));
  for (int i = 0; i < n; ++i) b->buf_gen.push_back(ctxs[i]->buf_gen);

  // capture: clear, the class launches side by side, the reductions
  BCK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeRelaxed));
  k_batch_clear<<<n, 256, 0, b->stream>>>(b->dgeo);
  BCK(cudaEventRecord(b->ev_fork, b->stream));
  for (auto& c : b->classes) {
    BCK(cudaStreamWaitEvent(c.st, b->ev_fork, 0));
    for (size_t q = 0; q + 1 < c.cut.size(); ++q) {
      const int u0 = c.cut[q], u1 = c.cut[q + 1];
      LaunchArgs la{};
      la.unit_slot = reinterpret_cast<const long long*>(c.dunit_slot) + u0;
      la.unit_nslots = reinterpret_cast<const int32_t*>(c.dunit_slot + 8 * (size_t)c.nunits) + u0;
      la.cand = cand_views(c.dcand, (long long)(c.cand_bytes / cand_slot_bytes(c.R)) / 64 * 64, c.R);
      la.nunits = u1 - u0;
      la.work = c.dwork;
      la.geo = b->dgeo;
      la.unit_geo = c.dunit_geo + u0;
      la.unit_local = c.dunit_local + u0;
      BCK(cudaMemsetAsync(c.dwork, 0, 2 * sizeof(int), c.st));
      const cudaError_t e = launch_forward<true>(P[c.geos[0]], la, c.W, c.R, std::min(c.grid, u1 - u0), dev_sms,
                                                 c.part_slots[q], c.st);
      if (e != cudaSuccess) {
        cudaGraph_t g = nullptr;
        cudaStreamEndCapture(b->stream, &g);
        if (g) cudaGraphDestroy(g);
        return bfail(b, CIPSI_ERR_CUDA, std::string("batched k_cand / k_pt2 launch: ") + cudaGetErrorString(e));
      }
    }
    BCK(cudaEventRecord(c.ev_join, c.st));
    BCK(cudaStreamWaitEvent(b->stream, c.ev_join, 0));
  }
  k_finish<<<(unsigned)n, kFinishThreads, 0, b->stream>>>(P[0], b->dgeo);
  // every geometry's records, in its unit order
  for (int i = 0; i < n; ++i) {
    GatherArgs ga{};
    record_target(ctxs[i], ga);
    const cudaError_t e = enqueue_gather(ctxs[i], P[i], 0, P[i].nunits, 0, ga, b->stream, dev_sms);
    if (e != cudaSuccess) {
      cudaGraph_t g = nullptr;
      cudaStreamEndCapture(b->stream, &g);
      if (g) cudaGraphDestroy(g);
      return bfail(b, CIPSI_ERR_CUDA, std::string("batched record gather: ") + cudaGetErrorString(e));
    }
  }
  BCK(cudaStreamEndCapture(b->stream, &b->graph));
  BCK(cudaGraphInstantiate(&b->exec, b->graph, 0));
  return CIPSI_OK;
}

int cipsi_batch_run(cipsi_batch* b) {
  if (!b || !b->exec) return CIPSI_ERR_ARG;
  for (size_t i = 0; i < b->ctxs.size(); ++i) {
    const cipsi_ctx* ctx = b->ctxs[i];
    if (ctx->buf_gen != b->buf_gen[i])
      return bfail(b, CIPSI_ERR_STATE, "context " + std::to_string(i) +
                                           " reallocated its buffers after the batch was built; rebuild the batch");
    // a result left pending by this batch's previous run is simply replaced
    if (ctx->pending && ctx->ext_done != b->done)
      return bfail(b, CIPSI_ERR_STATE, "context " + std::to_string(i) + " has a pending run");
  }
  BCK(cudaSetDevice(b->device));
  BCK(cudaEventRecord(b->ev0, b->stream));
  BCK(cudaGraphLaunch(b->exec, b->stream));
  BCK(cudaEventRecord(b->ev1, b->stream));
  BCK(cudaEventRecord(b->done, b->stream));
  for (size_t i = 0; i < b->ctxs.size(); ++i) {
    cipsi_ctx* ctx = b->ctxs[i];
    ctx->ext_done = b->done;
    ctx->ev_valid = false;
    ctx->nclass = b->opts[i].nclass;
    ctx->last_opts = b->opts[i];
    ctx->pending = true;
  }
  b->pending = true;
  return CIPSI_OK;
}

int cipsi_batch_wait(cipsi_batch* b, double* ms) {
  if (!b) return CIPSI_ERR_ARG;
  if (!b->pending) return bfail(b, CIPSI_ERR_STATE, "batch_wait without batch_run");
  BCK(cudaSetDevice(b->device));
  BCK(cudaEventSynchronize(b->done));
  b->pending = false;
  float t = 0.f;
  BCK(cudaEventElapsedTime(&t, b->ev0, b->ev1));
  if (ms) *ms = t;
  return CIPSI_OK;
}

const char* cipsi_batch_last_error(const cipsi_batch* b) { return b ? b->err.c_str() : "null batch"; }

void cipsi_batch_destroy(cipsi_batch* b) {
  if (!b) return;
  batch_free(b);
  for (cipsi_ctx* ctx : b->ctxs)
    if (ctx && ctx->ext_done == b->done) {
      ctx->ext_done = nullptr;
      ctx->pending = false;
    }
  delete b;
}

// ------------------------------------------------- run without allocation
// cipsi_run_pt2_static runs k_pt2_one + k_reduce with every per-run buffer taken
// from one file-scope device array instead of cudaMalloc'd context buffers.
// The two forward kernels do not fit it: their candidate buffer wants gigabytes
// (through 128 MB, in parts that left most of the device idle, this entry took
// 49, 409 and 574 ms at 60, 100 and 124 orbitals, S = 1001, 2001 and 2501; one
// kernel takes 36, 212 and 249).
// Layout of the array (each region 256-byte aligned): counters + dpivot +
// histogram counts | histogram sums | reduced sums | work counter |
// generator list | generator masks | work units | per-unit partial sums |
// per-block neighbour scratch (nb_j, nb_emask, lr_ent).  The generator and
// unit lists are staged in file-scope host arrays of fixed size.

}  // extern "C"

namespace {

constexpr size_t kStaticScratchBytes = (size_t)32 << 20;  // 32 MiB
constexpr int kStaticMaxUnits = 1 << 18;
constexpr int kStaticMaxGens = 1 << 17;
constexpr int kStaticMaxDevices = 64;

static __device__ __align__(256) unsigned char g_pt2_scratch[kStaticScratchBytes];

// host staging of the generator and unit lists (copied to the device array)
static int32_t g_static_gens[kStaticMaxGens];
static uint8_t g_static_gmask[kStaticMaxGens];
static int32_t g_static_units[3 * kStaticMaxUnits];

// device address of g_pt2_scratch, looked up once per device
static unsigned char* g_static_ptr[kStaticMaxDevices];
static bool g_static_ready[kStaticMaxDevices];

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

extern "C" {

int cipsi_run_pt2_static(cipsi_ctx* ctx, const cipsi_opts* o, cipsi_result* r) {
  if (!ctx || !o || !r) return CIPSI_ERR_ARG;
  if (!ctx->have_int || !ctx->have_space || !ctx->have_roots)
    return fail(ctx, CIPSI_ERR_STATE, "run before set_integrals / set_space / set_roots");
  if (ctx->pending)
    return fail(ctx, CIPSI_ERR_STATE, "an asynchronous run is pending: fetch its result first");
  if (o->nclass < 2 || o->nclass > kNClass) return fail(ctx, CIPSI_ERR_ARG, "nclass must be in [2, 10]");
  for (int i = 0; i + 1 < o->nclass; ++i)
    if (!(o->aval[i] >= 0.0) || (i > 0 && !(o->aval[i] > o->aval[i - 1])))
      return fail(ctx, CIPSI_ERR_ARG, "aval must be non-negative and increasing");
  if (ctx->device < 0 || ctx->device >= kStaticMaxDevices)
    return fail(ctx, CIPSI_ERR_ARG, "device ordinal out of range for the static scratch table");
  CK(cudaSetDevice(ctx->device));
  // set-up, once per device, with that device current
  if (!g_static_ready[ctx->device]) {
    void* ptr = nullptr;
    CK(cudaGetSymbolAddress(&ptr, g_pt2_scratch));
    g_static_ptr[ctx->device] = static_cast<unsigned char*>(ptr);
    g_static_ready[ctx->device] = true;
  }
  unsigned char* base = g_static_ptr[ctx->device];
  const int ncf = ctx->d.ncf, W = ctx->W, mt = ctx->d.metat;

  // generators and their allowed rank changes (pertu.f:52-61, igene.f:34-35,
  // 89-90, 199-200, 296-298; same rules as cipsi_run_pt2_async)
  bool yd = false, ym = false, yf = false;
  int maxrank = 0;
  for (int k = 0; k < ncf; ++k) {
    if (ctx->rank[k] == 1) ym = true;
    if (ctx->rank[k] == 0) yd = true;
    if (ctx->rank[k] == 2) yf = true;
    maxrank = std::max(maxrank, ctx->rank[k]);
  }
  if (ym) yf = true;
  const bool pertu_ref = yf && !yd && ctx->d.isym == 1;
  const bool pertu_mono = yf && ym;
  int ngen = 0;
  auto too_many_gens = [&]() {
    return fail(ctx, CIPSI_ERR_OVERFLOW,
                "cipsi_run_pt2_static: more than " + std::to_string(kStaticMaxGens) + " generators");
  };
  if (o->run_pertu && (pertu_ref || pertu_mono)) {
    g_static_gens[ngen] = -1;
    g_static_gmask[ngen++] = 0;
  }
  for (int k = 0; k < ncf; ++k) {
    if (!ctx->ygen[k] || ctx->ysaut[k]) continue;
    if (o->gen_mask && !o->gen_mask[k]) continue;
    const int nec = ctx->rank[k];
    uint8_t m = 1u << 4;
    if (!((nec == 0 && ym) || (nec == 1 && yd))) {
      m |= 1u << 3;
      const bool stop1 = nec < 1 || (ym && nec == 1) || (nec == 2 && yd);
      if (!stop1) {
        m |= 1u << 2;
        if (!((nec == 3 && yd) || (nec == 2 && ym))) {
          m |= 1u << 1;
          if (!((nec == 2 && (yd || yf)) || (nec == 3 && ym) || (nec == 4 && yd))) m |= 1u << 0;
        }
      }
    }
    if (ngen == kStaticMaxGens) return too_many_gens();
    g_static_gens[ngen] = k;
    g_static_gmask[ngen++] = m;
  }

  // work units in the order of cipsi_run_pt2_async: generators by rank
  // (pertu block first), each split into chunks of at most 6 allowed R blocks
  constexpr int kRChunk = 6;
  constexpr int kPertuChunk = 128;
  const int n = ctx->d.norb, noca = ctx->d.noca, nel = 2 * noca;
  const int nR = nel + nel * (nel - 1) / 2;
  int nunits = 0;
  int32_t* ug = g_static_units;
  int32_t* ur0 = g_static_units + kStaticMaxUnits;
  int32_t* ur1 = g_static_units + 2 * kStaticMaxUnits;
  auto push_unit = [&](int g, int a, int b) {
    if (nunits == kStaticMaxUnits) return false;
    ug[nunits] = g;
    ur0[nunits] = a;
    ur1[nunits] = b;
    ++nunits;
    return true;
  };
  auto too_many_units = [&]() {
    return fail(ctx, CIPSI_ERR_OVERFLOW,
                "cipsi_run_pt2_static: more than " + std::to_string(kStaticMaxUnits) + " work units");
  };
  int hfe[2 * 128];
  for (int rk = -1; rk <= maxrank; ++rk) {
    for (int g = 0; g < ngen; ++g) {
      const int k = g_static_gens[g];
      if ((k < 0 ? -1 : ctx->rank[k]) != rk) continue;
      if (k < 0) {
        const int ntot = (pertu_ref ? 1 : 0) + (pertu_mono ? 2 * noca * (n - noca) : 0);
        for (int t = 0; t < ntot; t += kPertuChunk)
          if (!push_unit(g, t, std::min(ntot, t + kPertuChunk))) return too_many_units();
        continue;
      }
      int ne = 0;
      for (int sp = 0; sp < 2; ++sp)
        for (int orb = 0; orb < n; ++orb)
          if ((ctx->Sbits[(size_t)k * 2 * W + sp * W + (orb >> 6)] >> (orb & 63)) & 1ull)
            hfe[ne++] = orb < noca;
      const uint8_t m = g_static_gmask[g];
      int cnt = 0, start = -1;
      for (int rb = 0; rb < nR; ++rb) {
        int hfR, nRr;
        if (rb < nel) {
          hfR = hfe[rb];
          nRr = 1;
        } else {
          int t = rb - nel, e1 = 0;
          while (t >= nel - 1 - e1) {
            t -= nel - 1 - e1;
            ++e1;
          }
          hfR = hfe[e1] + hfe[e1 + 1 + t];
          nRr = 2;
        }
        bool ok = false;
        for (int aV = 0; aV <= nRr; ++aV)
          if (m & (1u << (hfR + aV - nRr + 2))) ok = true;
        if (!ok) continue;
        if (start < 0) start = rb;
        if (++cnt == kRChunk) {
          if (!push_unit(g, start, rb + 1)) return too_many_units();
          cnt = 0;
          start = -1;
        }
      }
      if (start >= 0 && !push_unit(g, start, nR)) return too_many_units();
    }
  }

  // launch shape as in cipsi_run_pt2_async, then fewer blocks if the
  // per-block neighbour scratch would not fit in the array
  int dev_sms = 0;
  CK(cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, ctx->device));
  const int R = mt <= 1 ? 1 : mt <= 2 ? 2 : mt <= 4 ? 4 : 8;
  const LaunchShape ls = one_shape(R, ncf);
  const int lr_cap = ls.lr_cap;
  const size_t smem = ls.smem;
  const int blocks_per_sm = ls.blocks_per_sm;
  const size_t nq = (size_t)5 * mt;
  const size_t ncount = C_NCOUNTERS + 1 + kNClass + kNClass * kMaxRoots;
  const size_t off_counters = 0;
  const size_t off_tab = align256(off_counters + ncount * sizeof(unsigned long long));
  const size_t off_red = align256(off_tab + 2 * kNClass * kMaxRoots * sizeof(double));
  const size_t off_work = align256(off_red + 5 * kMaxRoots * sizeof(double));
  const size_t off_gens = align256(off_work + sizeof(int));
  const size_t off_gmask = align256(off_gens + (size_t)std::max(ngen, 1) * sizeof(int32_t));
  const size_t off_units = align256(off_gmask + (size_t)std::max(ngen, 1));
  const size_t off_part = align256(off_units + (size_t)3 * std::max(nunits, 1) * sizeof(int32_t));
  const size_t off_nb = align256(off_part + (size_t)std::max(nunits, 1) * nq * sizeof(double));
  const size_t per_block = 3 * align256((size_t)ncf * sizeof(uint64_t));
  int grid = std::max(1, std::min(nunits, dev_sms * blocks_per_sm));
  if (off_nb + per_block > kStaticScratchBytes)
    return fail(ctx, CIPSI_ERR_OVERFLOW,
                "cipsi_run_pt2_static: the run needs " + std::to_string(off_nb + per_block) +
                    " bytes of scratch, more than the static " + std::to_string(kStaticScratchBytes) +
                    " (ncf = " + std::to_string(ncf) + ", work units = " + std::to_string(nunits) +
                    "); use cipsi_run_pt2");
  grid = (int)std::min<size_t>((size_t)grid, (kStaticScratchBytes - off_nb) / per_block);
  const size_t nb_stride = align256((size_t)ncf * sizeof(uint64_t));
  unsigned char* nb0 = base + off_nb;

  // zero what the kernels accumulate into; upload the lists
  CK(cudaMemsetAsync(base, 0, off_gens, ctx->stream));
  CK(cudaMemsetAsync(base + off_part, 0, (size_t)std::max(nunits, 1) * nq * sizeof(double), ctx->stream));
  if (ngen) {
    CK(cudaMemcpyAsync(base + off_gens, g_static_gens, (size_t)ngen * sizeof(int32_t),
                       cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(base + off_gmask, g_static_gmask, (size_t)ngen, cudaMemcpyHostToDevice, ctx->stream));
  }
  int32_t* dunits = reinterpret_cast<int32_t*>(base + off_units);
  if (nunits) {
    CK(cudaMemcpyAsync(dunits, ug, (size_t)nunits * sizeof(int32_t), cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(dunits + nunits, ur0, (size_t)nunits * sizeof(int32_t), cudaMemcpyHostToDevice,
                       ctx->stream));
    CK(cudaMemcpyAsync(dunits + 2 * nunits, ur1, (size_t)nunits * sizeof(int32_t), cudaMemcpyHostToDevice,
                       ctx->stream));
  }

  Params p{};
  p.norb = ctx->d.norb;
  p.noca = ctx->d.noca;
  p.nel = nel;
  p.ncf = ncf;
  p.metat = mt;
  p.nsym = ctx->d.nsym;
  p.isym = ctx->d.isym;
  p.ngen = ngen;
  p.gens = reinterpret_cast<const int32_t*>(base + off_gens);
  p.gen_dmask = base + off_gmask;
  p.nunits = nunits;
  p.unit_g = dunits;
  p.unit_r0 = dunits + nunits;
  p.unit_r1 = dunits + 2 * nunits;
  p.S = ctx->dS;
  p.ygen = ctx->dygen;
  p.nesp = ctx->dnesp;
  p.yef = ctx->dyef;
  p.c = ctx->dc;
  p.eri = ctx->deri;
  p.eri64 = ctx->deri64 ? ctx->deri64 : ctx->deri_w;
  p.pairtab = ctx->dpairtab;
  p.ntttt = ctx->dntttt;
  p.F = ctx->dF;
  p.J = ctx->dJ;
  p.K = ctx->dK;
  p.fmpb = ctx->dfmpb;
  p.orbsym = ctx->dorbsym;
  for (int i = 0; i < ctx->d.nsym; ++i)
    for (int j = 0; j < ctx->d.nsym; ++j) p.its[i][j] = ctx->its[(size_t)j * ctx->d.nsym + i] - 1;
  for (int m = 0; m < mt; ++m) {
    p.e[m] = ctx->e[m];
    p.eb[m] = ctx->eb[m];
    p.emp[m] = ctx->emp[m];
    p.teste[m] = ctx->teste[m];
    p.taum[m] = ctx->taum[m];
  }
  p.yen = o->yen;
  p.ysele = o->ysele;
  p.ymoyen = o->ymoyen;
  p.ywdeg = o->ywdeg;
  p.symvar = o->sym_variant;
  p.nclass = o->nclass;
  p.tau = o->tau;
  p.teseff = o->teseff;
  for (int i = 0; i < kNClass; ++i) {
    p.aval[i] = o->aval[i];
    std::memcpy(&p.aval_bits[i], &o->aval[i], 8);
  }
  p.pertu_ref = pertu_ref ? 1 : 0;
  p.pertu_mono = pertu_mono ? 1 : 0;
  // nb_j, nb_emask, lr_ent: grid x ncf entries each (k_pt2_one indexes block b at
  // b * ncf), in three regions of grid * nb_stride >= grid * ncf * 8 bytes
  p.nb_j = reinterpret_cast<int32_t*>(nb0);
  p.nb_emask = reinterpret_cast<uint64_t*>(nb0 + (size_t)grid * nb_stride);
  p.lr_ent = reinterpret_cast<uint64_t*>(nb0 + (size_t)2 * grid * nb_stride);
  p.lr_cap = lr_cap;
  p.nb_stride = ncf;
  p.gen_part = reinterpret_cast<double*>(base + off_part);
  unsigned long long* dcounters = reinterpret_cast<unsigned long long*>(base + off_counters);
  p.counters = dcounters;
  p.dpivot_bits = dcounters + C_NCOUNTERS;
  p.hist_nom = dcounters + C_NCOUNTERS + 1;
  p.hist_nam = dcounters + C_NCOUNTERS + 1 + kNClass;
  p.hist_tab = reinterpret_cast<double*>(base + off_tab);
  // no record storage: selected perturbers are counted only
  p.rec_mode = 0;
  p.work = reinterpret_cast<int*>(base + off_work);
  double* dred = reinterpret_cast<double*>(base + off_red);

  CK(cudaEventRecord(ctx->ev0, ctx->stream));
  if (nunits > 0) {
    const cudaError_t e = launch_one(W, R, p, grid, smem, ctx->stream);
    if (e != cudaSuccess) return fail(ctx, CIPSI_ERR_CUDA, std::string("k_pt2_one launch: ") + cudaGetErrorString(e));
    k_reduce<<<(unsigned)nq, kReduceThreads, 0, ctx->stream>>>(p.gen_part, nunits, (int)nq, dred);
    CK(cudaGetLastError());
  }
  CK(cudaEventRecord(ctx->ev1, ctx->stream));

  // results (same fields as cipsi_fetch_result; no records are kept), read
  // on the context's stream: a legacy-stream cudaMemcpy would also wait for
  // every other blocking stream of the device
  double red[5 * kMaxRoots];
  unsigned long long cnt[C_NCOUNTERS + 1 + kNClass + kNClass * kMaxRoots];
  double tab[2 * kNClass * kMaxRoots];
  CK(cudaMemcpyAsync(red, dred, nq * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaMemcpyAsync(cnt, dcounters, ncount * sizeof(unsigned long long), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaMemcpyAsync(tab, p.hist_tab, 2 * kNClass * kMaxRoots * sizeof(double), cudaMemcpyDeviceToHost,
                     ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  memset(r, 0, sizeof(*r));
  for (int m = 0; m < mt; ++m) {
    r->e2mp[m] = red[0 * mt + m];
    r->e2vp[m] = red[1 * mt + m];
    r->e2b[m] = red[2 * mt + m];
    r->psimp[m] = red[3 * mt + m];
    r->psivp[m] = red[4 * mt + m];
  }
  r->ietat = (int64_t)cnt[C_IETAT];
  r->n_processed = (int64_t)cnt[C_NPROC];
  r->n_candidates = (int64_t)cnt[C_NCAND];
  r->n_compares = (int64_t)cnt[C_NCMP];
  r->n_pairs_1 = (int64_t)cnt[C_NP1];
  r->n_pairs_2 = (int64_t)cnt[C_NP2];
  {
    const unsigned long long b = cnt[C_NCOUNTERS];
    double dp;
    memcpy(&dp, &b, 8);
    r->dpivot = dp;
  }
  const int nc = o->nclass;
  for (int i = 0; i < nc; ++i) r->nom[i] = (int64_t)cnt[C_NCOUNTERS + 1 + i];
  for (int c = 0; c < nc; ++c)
    for (int m = 0; m < mt; ++m) {
      r->nam[c * kMaxRoots + m] = (int64_t)cnt[C_NCOUNTERS + 1 + kNClass + c * mt + m];
      r->tabmp[c * kMaxRoots + m] = tab[c * mt + m];
      r->tabvp[c * kMaxRoots + m] = tab[nc * mt + c * mt + m];
    }
  const double avg_rank = 4.0;
  r->alg_bytes = (int64_t)(cnt[C_NP2] * (8.0 * mt + 2 * 4.0 + 8.0) +
                           cnt[C_NP1] * (8.0 * mt + 8.0 + 2.0 * avg_rank * 2 * 4.0) +
                           cnt[C_NPROC] * (8.0 * avg_rank + 8.0 * (avg_rank + avg_rank * avg_rank) + 8.0 * mt));
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  r->kernel_ms = ms;
  r->pt2_ms = ms;
  r->launches = nunits > 0 ? 2 : 0;
  r->n_selected = (int64_t)cnt[C_NSEL];
  return CIPSI_OK;
}

}  // extern "C"

// ================================================ Hamiltonian over the space
// cipsi_hamiltonian_build / cipsi_hamiltonian_get: the lower triangle of H
// over the determinants given to cipsi_set_space, by rows, as moy writes it
// to its unit 1 (moy/moy.f:117-199) -- row i: the columns j < min(i, jmax)
// within two excitations, in increasing j, with <i|H|j> in the phase of the
// excitation lists.  The elements moy drops (|h| < 1e-10) are kept here;
// the caller filters them when it writes the file.
extern "C" {

int cipsi_hamiltonian_build(cipsi_ctx* ctx, const double* fock, int32_t jmax, int64_t* npairs) {
  if (!ctx || !npairs) return CIPSI_ERR_ARG;
  if (!ctx->have_int || !ctx->have_space)
    return fail(ctx, CIPSI_ERR_STATE, "hamiltonian_build needs set_integrals and set_space");
  if (ctx->pending) return fail(ctx, CIPSI_ERR_STATE, "a run is pending: fetch its result first");
  CK(cudaSetDevice(ctx->device));
  const int n = ctx->d.ncf, W = ctx->W, norb = ctx->d.norb;
  *npairs = 0;
  ctx->have_h = false;
  // workspace of the build, kept for the next one: row offsets, counts by
  // segment and by row, phases
  const int seg = hscan_segment(n), nseg = (n + seg - 1) / seg;
  const size_t off_seg = ((size_t)n + 1) * 8, off_cnt = off_seg + (size_t)nseg * n * 4, off_sg = off_cnt + (size_t)n * 4;
  const size_t work = off_sg + (size_t)n;
  if (work > ctx->h_work_cap) {
    dfree(ctx->dh_work);
    ctx->h_work_cap = 0;
    CK(cudaMalloc((void**)&ctx->dh_work, work));
    ctx->h_work_cap = work;
  }
  std::vector<int8_t> sg(n);
  for (int k = 0; k < n; ++k) sg[k] = ctx->sigma[k] < 0 ? -1 : 1;
  CK(cudaMemcpyAsync(ctx->dh_work + off_sg, sg.data(), sg.size(), cudaMemcpyHostToDevice, ctx->stream));
  const double* dF = ctx->dF;
  if (fock) {
    const int rc = upload(ctx, &ctx->dFraw, fock, (size_t)norb * (norb + 1) / 2);
    if (rc) return rc;
    dF = ctx->dFraw;
  }
  HBuildArgs a{};
  a.p.norb = norb;
  a.p.noca = ctx->d.noca;
  a.p.nsym = ctx->d.nsym;
  a.p.eri = ctx->deri;
  a.p.eri64 = ctx->deri64 ? ctx->deri64 : ctx->deri_w;
  a.p.pairtab = ctx->dpairtab;
  a.p.ntttt = ctx->dntttt;
  a.p.F = dF;
  a.S = ctx->dS;
  a.sigma = reinterpret_cast<const int8_t*>(ctx->dh_work + off_sg);
  a.seg = seg;
  a.nseg = nseg;
  a.segcnt = reinterpret_cast<int32_t*>(ctx->dh_work + off_seg);
  a.n = n;
  a.jmax = jmax < 0 ? n : std::min(jmax, n);
  for (int q = 0; q < 4; ++q) a.hf[q] = 0ull;
  for (int o = 0; o < ctx->d.noca; ++o) {
    a.hf[o >> 6] |= 1ull << (o & 63);
    a.hf[W + (o >> 6)] |= 1ull << (o & 63);
  }
  a.count = reinterpret_cast<int32_t*>(ctx->dh_work + off_cnt);
  CK(cudaEventRecord(ctx->ev0, ctx->stream));
  cudaError_t e = W == 1 ? launch_hcount<1>(a, ctx->stream) : launch_hcount<2>(a, ctx->stream);
  if (e != cudaSuccess) return fail(ctx, CIPSI_ERR_CUDA, std::string("k_hscan (count): ") + cudaGetErrorString(e));
  std::vector<int32_t> cnt(n);
  CK(cudaMemcpyAsync(cnt.data(), a.count, (size_t)n * sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->h_rowptr.assign((size_t)n + 1, 0);
  for (int i = 0; i < n; ++i) ctx->h_rowptr[i + 1] = ctx->h_rowptr[i] + cnt[i];
  const long long total = ctx->h_rowptr[n];
  CK(cudaMemcpyAsync(ctx->dh_work, ctx->h_rowptr.data(), ctx->h_rowptr.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
  if (total > ctx->h_cap || !ctx->dh_col) {
    dfree(ctx->dh_col);
    dfree(ctx->dh_val);
    ++ctx->buf_gen;
    CK(cudaMalloc((void**)&ctx->dh_col, (size_t)std::max(total, 1ll) * sizeof(int32_t)));
    CK(cudaMalloc((void**)&ctx->dh_val, (size_t)std::max(total, 1ll) * sizeof(double)));
    ctx->h_cap = std::max(total, 1ll);
  }
  a.rowptr = reinterpret_cast<const long long*>(ctx->dh_work);
  a.col = ctx->dh_col;
  a.val = ctx->dh_val;
  int dev_sms = 0;
  CK(cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, ctx->device));
  e = W == 1 ? launch_hfill<1>(a, dev_sms, ctx->stream) : launch_hfill<2>(a, dev_sms, ctx->stream);
  if (e != cudaSuccess) return fail(ctx, CIPSI_ERR_CUDA, std::string("k_hscan (fill): ") + cudaGetErrorString(e));
  CK(cudaEventRecord(ctx->ev1, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  CK(cudaEventElapsedTime(&ctx->h_ms, ctx->ev0, ctx->ev1));
  ctx->have_h = true;
  *npairs = total;
  return CIPSI_OK;
}

int cipsi_hamiltonian_get(cipsi_ctx* ctx, int32_t row0, int32_t nrows, int64_t* rowptr, int32_t* col,
                          double* val) {
  if (!ctx) return CIPSI_ERR_ARG;
  if (!ctx->have_h) return fail(ctx, CIPSI_ERR_STATE, "hamiltonian_get before hamiltonian_build");
  const int n = ctx->d.ncf;
  if (row0 < 0 || nrows < 0 || row0 + (long long)nrows > n)
    return fail(ctx, CIPSI_ERR_ARG, "hamiltonian_get: rows out of range");
  const long long a = ctx->h_rowptr[row0], b = ctx->h_rowptr[row0 + nrows];
  if (rowptr)
    for (int r = 0; r <= nrows; ++r) rowptr[r] = ctx->h_rowptr[row0 + r] - a;
  CK(cudaSetDevice(ctx->device));
  if (b > a && (col || val)) {
    if (col)
      CK(cudaMemcpyAsync(col, ctx->dh_col + a, (size_t)(b - a) * sizeof(int32_t), cudaMemcpyDeviceToHost,
                         ctx->stream));
    if (val)
      CK(cudaMemcpyAsync(val, ctx->dh_val + a, (size_t)(b - a) * sizeof(double), cudaMemcpyDeviceToHost,
                         ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
  }
  return CIPSI_OK;
}

float cipsi_hamiltonian_ms(const cipsi_ctx* ctx) { return ctx ? ctx->h_ms : 0.f; }

}  // extern "C"
