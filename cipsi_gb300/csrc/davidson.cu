// davidson.cu -- the lowest eigenpairs of the CI matrix that moy writes to
// unit 1 (the work of bd, CIPSI_sources/bd/bigdia.f), on the GPU.
//
// The matrix is H = L + L^T, L being the elements moy stores (row i: the
// columns j < i, then the diagonal as half its value, moy/moy.f:150-190,
// as bd/getmat.f rebuilds it).  It is assembled once as a full CSR matrix in
// device memory; the iteration is a block Davidson method:
//
//   V (n x k) orthonormal, W = H V;  Rayleigh-Ritz on V^T W (host, k <= 64);
//   Ritz vectors X = V S, residuals R = W S - X Theta;  converged when every
//   residual norm is below `tol`;  corrections T = R / (theta - diag(H))
//   (the diagonal preconditioner of Davidson's method), made orthogonal to
//   V twice and orthonormalised through their Gram matrix; V grows by T
//   until it would exceed kmax columns, then restarts from the Ritz vectors.
//
// Kernels: k_spmm (H times a block of vectors: one warp per row, the row's
// nonzeros over the lanes, a shuffle reduction per vector), k_gram (V^T T:
// one CTA per output element, fixed-order sums, so results are reproducible
// run to run), k_combine (X = V S), k_residual, k_precond.  Each product reads
// the 12 bytes of every nonzero once, and the vectors (8 bytes per row and
// vector) stay L2-resident up to ~10^6 rows.  At a few thousand rows an
// iteration is some twenty launches of a few microseconds: what it waits for is
// the host, so the small matrices travel as kernel arguments or stay on the
// device, and the host waits four times an iteration (6,001 rows, 240,000
// elements, 14 iterations: 6.2 ms with a wait after every product and copies
// between the work vectors, k_gram 14 us and k_combine 8.5 us each; now 4.6 ms).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/cipsi_gb300.h"
#include "symeig.h"

namespace {

constexpr int kMaxBlock = 16;  // vectors per block product

template <int NV>
__global__ void __launch_bounds__(256) k_spmm(int n, const long long* __restrict__ rowptr,
                                              const int32_t* __restrict__ col, const double* __restrict__ val,
                                              const double* __restrict__ X, int ldx, double* __restrict__ Y,
                                              int ldy, int nv) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < n; row += warps) {
    double acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
    const long long a = rowptr[row], b = rowptr[row + 1];
    for (long long t = a + lane; t < b; t += 32) {
      const int c = __ldg(&col[t]);
      const double h = __ldg(&val[t]);
#pragma unroll
      for (int v = 0; v < NV; ++v)
        if (v < nv) acc[v] = fma(h, __ldg(&X[(size_t)v * ldx + c]), acc[v]);
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      double x = acc[v];
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (lane == 0 && v < nv) Y[(size_t)v * ldy + row] = x;
    }
  }
}

// G[a * kb + b] = sum_i A[a * lda + i] * B[b * ldb + i]; one CTA per (a, b) --
// or, with norms, G[a] = the (a, a) elements alone.  Bound by the latency of
// its loads (a thread reads n / 256 pairs): four independent chains.
__global__ void __launch_bounds__(256) k_gram(int n, const double* __restrict__ A, int lda,
                                              const double* __restrict__ B, int ldb, int kb, int norms,
                                              double* __restrict__ G) {
  __shared__ double red[8];
  const int a = norms ? blockIdx.x : blockIdx.x / kb, b = norms ? blockIdx.x : blockIdx.x % kb;
  const double* x = A + (size_t)a * lda;
  const double* y = B + (size_t)b * ldb;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  int i = threadIdx.x;
  for (; i + 768 < n; i += 1024) {
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] = fma(__ldg(&x[i + 256 * q]), __ldg(&y[i + 256 * q]), s[q]);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (i + 256 * q < n) s[q] = fma(__ldg(&x[i + 256 * q]), __ldg(&y[i + 256 * q]), s[q]);
  double t = (s[0] + s[1]) + (s[2] + s[3]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    t = red[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) t += red[w];
    G[blockIdx.x] = t;
  }
}

// a small matrix as a kernel argument: at most (4 nb) x nb, nb = 10
struct Small {
  double s[400];
};

// Y[:, b] = beta * Y[:, b] + sum_a A[:, a] S[a * kb + b]   (S: ka x kb, row-major;
// with D, S = -D of the device).  A thread takes a row; with few rows each
// column b has its own threads (grid.y = kb), else a thread goes through the
// columns, so that A is read once (its rows stay in L1).
__global__ void __launch_bounds__(256) k_combine(int n, const double* __restrict__ A, int lda, int ka,
                                                 const __grid_constant__ Small S, const double* __restrict__ D, int kb,
                                                 double beta, double* __restrict__ Y, int ldy) {
  __shared__ double sS[400];
  for (int i = threadIdx.x; i < ka * kb; i += blockDim.x) sS[i] = D ? -D[i] : S.s[i];
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    for (int b = blockIdx.y; b < kb; b += gridDim.y) {
      double y = beta == 0.0 ? 0.0 : beta * Y[(size_t)b * ldy + i];
#pragma unroll 8
      for (int a = 0; a < ka; ++a) y = fma(__ldg(&A[(size_t)a * lda + i]), sS[a * kb + b], y);
      Y[(size_t)b * ldy + i] = y;
    }
  }
}

struct Theta {
  double theta[kMaxBlock];
  int from[kMaxBlock];
};
// T[:, b] = AX[:, b] - theta_b X[:, b]
__global__ void k_residual(int n, const double* __restrict__ AX, const double* __restrict__ X,
                           const __grid_constant__ Theta th, int nx, double* __restrict__ T) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int b = blockIdx.y; b < nx; b += gridDim.y)
      T[(size_t)b * n + i] = fma(X[(size_t)b * n + i], -th.theta[b], AX[(size_t)b * n + i]);
}

// T[:, b] = R[:, from_b] / (theta_b - d_i), the denominator kept away from zero
__global__ void k_precond(int n, const double* __restrict__ R, const double* __restrict__ diag,
                          const __grid_constant__ Theta th, int kb, double* __restrict__ T) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int b = blockIdx.y; b < kb; b += gridDim.y) {
      double den = th.theta[b] - diag[i];
      if (std::fabs(den) < 1e-8) den = den < 0.0 ? -1e-8 : 1e-8;
      T[(size_t)b * n + i] = R[(size_t)th.from[b] * n + i] / den;
    }
}

// V[:, b] = the unit vector at row from_b (V zeroed)
__global__ void k_units(int n, const __grid_constant__ Theta th, int nb, double* __restrict__ V) {
  if ((int)threadIdx.x < nb) V[(size_t)threadIdx.x * n + th.from[threadIdx.x]] = 1.0;
}

struct Dev {
  std::string err;
  bool ok = true;
  bool check(cudaError_t e, const char* what) {
    if (e != cudaSuccess && ok) {
      ok = false;
      err = std::string(what) + ": " + cudaGetErrorString(e);
    }
    return e == cudaSuccess;
  }
};

void seterr(char* errbuf, int32_t errlen, const std::string& m) {
  if (errbuf && errlen > 0) std::snprintf(errbuf, (size_t)errlen, "%s", m.c_str());
}

}  // namespace

extern "C" int cipsi_davidson(int32_t n, int64_t nel, const int32_t* itab, const int32_t* jtab, const double* val,
                              int32_t nroots, double tol, int32_t maxiter, int32_t device, double* evals,
                              double* evecs, int32_t* iters, double* resid, char* errbuf, int32_t errlen) {
  using cipsi_host::sym_eig;
  if (n < 1 || nel < 0 || nroots < 1 || nroots > n || !itab || !jtab || !val || !evals || !evecs) {
    seterr(errbuf, errlen, "cipsi_davidson: bad arguments");
    return CIPSI_ERR_ARG;
  }
  if (nroots > 8) {
    seterr(errbuf, errlen, "cipsi_davidson: at most 8 roots");
    return CIPSI_ERR_ARG;
  }
  // full CSR of H = L + L^T (host), diagonal kept for the preconditioner
  std::vector<long long> rowptr((size_t)n + 1, 0);
  std::vector<double> diag(n, 0.0);
  for (int64_t t = 0; t < nel; ++t) {
    const int i = itab[t] - 1, j = jtab[t] - 1;
    if (i < 0 || i >= n || j < 0 || j >= n || j > i) {
      seterr(errbuf, errlen, "cipsi_davidson: element " + std::to_string(t + 1) + " outside the lower triangle");
      return CIPSI_ERR_ARG;
    }
    if (i == j) {
      diag[i] += 2.0 * val[t];
      continue;
    }
    ++rowptr[i + 1];
    ++rowptr[j + 1];
  }
  for (int i = 0; i < n; ++i) rowptr[i + 1] += rowptr[i] + 1;  // + the diagonal slot
  std::vector<long long> fill(rowptr.begin(), rowptr.end() - 1);
  const long long nnz = rowptr[n];
  std::vector<int32_t> col((size_t)nnz);
  std::vector<double> hv((size_t)nnz);
  for (int i = 0; i < n; ++i) {
    col[fill[i]] = i;
    hv[fill[i]++] = diag[i];
  }
  for (int64_t t = 0; t < nel; ++t) {
    const int i = itab[t] - 1, j = jtab[t] - 1;
    if (i == j) continue;
    col[fill[i]] = j;
    hv[fill[i]++] = val[t];
    col[fill[j]] = i;
    hv[fill[j]++] = val[t];
  }
  // block size and subspace limit
  const int nb = std::min(n, std::min(kMaxBlock, nroots + 2));
  const int kmax = std::min(n, std::max(4 * nb, 24));
  Dev d;
  d.check(cudaSetDevice(device), "cudaSetDevice");
  cudaStream_t st = nullptr;
  d.check(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking), "cudaStreamCreate");
  long long* drow = nullptr;
  int32_t* dcol = nullptr;
  double *dval = nullptr, *ddiag = nullptr, *V = nullptr, *Wm = nullptr, *X = nullptr, *AX = nullptr, *T = nullptr,
         *AT = nullptr, *dG = nullptr, *hG = nullptr;
  // one allocation, cut into parts of whole 256 bytes
  const size_t gsz = (size_t)kmax * kmax * 8;
  unsigned char* mem = nullptr;
  {
    size_t off = 0;
    struct Part {
      void** p;
      size_t bytes, at;
    } part[] = {{(void**)&drow, rowptr.size() * 8, 0}, {(void**)&dcol, (size_t)nnz * 4, 0},
                {(void**)&dval, (size_t)nnz * 8, 0},   {(void**)&ddiag, (size_t)n * 8, 0},
                {(void**)&V, (size_t)n * kmax * 8, 0}, {(void**)&Wm, (size_t)n * kmax * 8, 0},
                {(void**)&X, (size_t)n * nb * 8, 0},   {(void**)&AX, (size_t)n * nb * 8, 0},
                {(void**)&T, (size_t)n * nb * 8, 0},   {(void**)&AT, (size_t)n * nb * 8, 0},
                {(void**)&dG, 2 * gsz, 0}};
    for (Part& q : part) {
      q.at = off;
      off += (q.bytes + 255) / 256 * 256;
    }
    d.check(cudaMalloc((void**)&mem, off), "cudaMalloc");
    d.check(cudaMallocHost((void**)&hG, 2 * gsz), "cudaMallocHost");
    if (d.ok)
      for (Part& q : part) *q.p = mem + q.at;
  }
  if (d.ok) {
    d.check(cudaMemcpyAsync(drow, rowptr.data(), rowptr.size() * 8, cudaMemcpyHostToDevice, st), "copy");
    d.check(cudaMemcpyAsync(dcol, col.data(), (size_t)nnz * 4, cudaMemcpyHostToDevice, st), "copy");
    d.check(cudaMemcpyAsync(dval, hv.data(), (size_t)nnz * 8, cudaMemcpyHostToDevice, st), "copy");
    d.check(cudaMemcpyAsync(ddiag, diag.data(), (size_t)n * 8, cudaMemcpyHostToDevice, st), "copy");
  }
  int sms = 0;
  d.check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "attr");
  const int ewgrid = std::max(1, std::min((n + 255) / 256, 8 * sms));
  // columns side by side while the rows alone leave the device part empty
  auto ew = [&](int kb) { return dim3((unsigned)ewgrid, ewgrid < 4 * sms ? (unsigned)kb : 1u); };
  const int spgrid = std::max(1, std::min((n * 32 + 255) / 256, 32 * sms));
  auto spmm = [&](const double* Xin, double* Yout, int nv) {
    for (int v0 = 0; v0 < nv && d.ok; v0 += kMaxBlock) {
      const int m = std::min(kMaxBlock, nv - v0);
      if (m <= 1)
        k_spmm<1><<<spgrid, 256, 0, st>>>(n, drow, dcol, dval, Xin + (size_t)v0 * n, n, Yout + (size_t)v0 * n, n, m);
      else if (m <= 4)
        k_spmm<4><<<spgrid, 256, 0, st>>>(n, drow, dcol, dval, Xin + (size_t)v0 * n, n, Yout + (size_t)v0 * n, n, m);
      else if (m <= 8)
        k_spmm<8><<<spgrid, 256, 0, st>>>(n, drow, dcol, dval, Xin + (size_t)v0 * n, n, Yout + (size_t)v0 * n, n, m);
      else
        k_spmm<16><<<spgrid, 256, 0, st>>>(n, drow, dcol, dval, Xin + (size_t)v0 * n, n, Yout + (size_t)v0 * n, n, m);
      d.check(cudaGetLastError(), "k_spmm");
    }
  };
  // A^T B into part `at` of the device's and the host's small matrices; the host
  // may look after sync()
  auto gram = [&](const double* A, int ka, const double* B, int kb, bool norms, bool host, int at) {
    if (!d.ok || ka == 0 || kb == 0) return;
    const int m = norms ? ka : ka * kb;
    double* g = dG + at * (gsz / 8);
    k_gram<<<m, 256, 0, st>>>(n, A, n, B, n, kb, norms ? 1 : 0, g);
    d.check(cudaGetLastError(), "k_gram");
    if (host) d.check(cudaMemcpyAsync(hG + at * (gsz / 8), g, (size_t)m * 8, cudaMemcpyDeviceToHost, st), "copy G");
  };
  auto sync = [&]() {
    if (d.ok) d.check(cudaStreamSynchronize(st), "sync");
  };
  Small sm;
  auto combine = [&](const double* A, int ka, const double* S, int kb, double beta, double* Y, const double* D) {
    if (!d.ok || kb == 0) return;
    if (S) std::memcpy(sm.s, S, (size_t)ka * kb * 8);
    k_combine<<<ew(kb), 256, 0, st>>>(n, A, n, ka, sm, D, kb, beta, Y, n);
    d.check(cudaGetLastError(), "k_combine");
  };
  // T less its components along V; the coefficients stay on the device
  auto project = [&](int k, int nt) {
    if (k == 0) return;
    gram(V, k, T, nt, false, false, 0);
    combine(V, k, nullptr, nt, 1.0, T, dG);
  };
  // T (nt columns): remove the components along V (two passes), then make
  // the columns orthonormal through their Gram matrix, dropping directions
  // with no weight left; returns the columns kept (written back into T)
  auto orthonormalise = [&](int k, int nt) -> int {
    // the scale of the corrections before projection: a direction is
    // dropped when projecting leaves less than 1e-10 of that scale
    gram(T, nt, T, nt, true, true, 1);
    for (int pass = 0; pass < 2; ++pass) project(k, nt);
    gram(T, nt, T, nt, false, true, 0);
    sync();
    if (!d.ok) return 0;
    double scale2 = 0.0;
    for (int q = 0; q < nt; ++q) scale2 = std::max(scale2, hG[gsz / 8 + q]);
    std::vector<double> w, U;
    sym_eig(nt, std::vector<double>(hG, hG + nt * nt), w, U);
    std::vector<int> keep;
    for (int q = nt - 1; q >= 0; --q)
      if (w[q] > 1e-20 * scale2 && w[q] > 0.0) keep.push_back(q);
    const int nk = (int)keep.size();
    if (nk == 0) return 0;
    std::vector<double> Sx((size_t)nt * nk);
    for (int c = 0; c < nk; ++c)
      for (int r = 0; r < nt; ++r) Sx[(size_t)r * nk + c] = U[(size_t)r * nt + keep[c]] / std::sqrt(w[keep[c]]);
    combine(T, nt, Sx.data(), nk, 0.0, AT, nullptr);
    std::swap(T, AT);
    // once more against V: the Gram step can bring back rounding-level overlap
    if (k > 0) {
      project(k, nk);
      gram(T, nk, T, nk, false, true, 0);
      sync();
      if (!d.ok) return 0;
      sym_eig(nk, std::vector<double>(hG, hG + nk * nk), w, U);
      std::vector<double> S2((size_t)nk * nk);
      for (int c = 0; c < nk; ++c)
        for (int r = 0; r < nk; ++r) S2[(size_t)r * nk + c] = U[(size_t)r * nk + c] / std::sqrt(std::max(w[c], 1e-300));
      combine(T, nk, S2.data(), nk, 0.0, AT, nullptr);
      std::swap(T, AT);
    }
    return nk;
  };
  // start: unit vectors on the nb smallest diagonal elements
  {
    std::vector<int> ord(n);
    for (int i = 0; i < n; ++i) ord[i] = i;
    std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return diag[a] < diag[b]; });
    Theta u{};
    for (int b = 0; b < nb; ++b) u.from[b] = ord[b];
    if (d.ok) {
      d.check(cudaMemsetAsync(V, 0, (size_t)n * nb * 8, st), "clear V0");
      k_units<<<1, 32, 0, st>>>(n, u, nb, V);
      d.check(cudaGetLastError(), "k_units");
    }
    spmm(V, Wm, nb);
  }
  int k = nb, it = 0;
  std::vector<double> theta, Sm, res(nroots, 0.0);
  bool converged = false;
  for (it = 1; it <= std::max(1, maxiter) && d.ok; ++it) {
    std::vector<double> w, U;
    gram(V, k, Wm, k, false, true, 0);
    sync();
    if (!d.ok) break;
    std::vector<double> Hs(hG, hG + (size_t)k * k);
    for (int a = 0; a < k; ++a)  // symmetrise (rounding)
      for (int b = a + 1; b < k; ++b) Hs[(size_t)a * k + b] = Hs[(size_t)b * k + a] = 0.5 * (Hs[(size_t)a * k + b] + Hs[(size_t)b * k + a]);
    sym_eig(k, Hs, w, U);
    const int nx = std::min(nb, k);
    Sm.assign((size_t)k * nx, 0.0);
    for (int a = 0; a < k; ++a)
      for (int b = 0; b < nx; ++b) Sm[(size_t)a * nx + b] = U[(size_t)a * k + b];
    theta.assign(w.begin(), w.begin() + nx);
    combine(V, k, Sm.data(), nx, 0.0, X, nullptr);
    combine(Wm, k, Sm.data(), nx, 0.0, AX, nullptr);
    // residuals R = AX - X theta (into T)
    Theta th{};
    for (int b = 0; b < nx; ++b) th.theta[b] = theta[b];
    if (d.ok) {
      k_residual<<<ew(nx), 256, 0, st>>>(n, AX, X, th, nx, T);
      d.check(cudaGetLastError(), "k_residual");
    }
    gram(T, nx, T, nx, true, true, 0);
    sync();
    if (!d.ok) break;
    double worst = 0.0;
    for (int b = 0; b < nroots; ++b) {
      res[b] = std::sqrt(std::max(hG[b], 0.0));
      worst = std::max(worst, res[b]);
    }
    if (worst <= tol) {
      converged = true;
      break;
    }
    // restart from the Ritz vectors when V is full
    if (k + nx > kmax) {
      d.check(cudaMemcpyAsync(V, X, (size_t)n * nx * 8, cudaMemcpyDeviceToDevice, st), "restart V");
      d.check(cudaMemcpyAsync(Wm, AX, (size_t)n * nx * 8, cudaMemcpyDeviceToDevice, st), "restart W");
      k = nx;
    }
    // corrections of the roots not yet converged (the extra block vectors
    // always): their residual columns, divided by theta - diag(H)
    std::vector<int> todo;
    for (int b = 0; b < nx; ++b)
      if (b >= nroots || res[b] > tol) todo.push_back(b);
    const int nu = (int)todo.size();
    for (int c = 0; c < nu; ++c) {
      th.from[c] = todo[c];
      th.theta[c] = theta[todo[c]];
    }
    k_precond<<<ew(nu), 256, 0, st>>>(n, T, ddiag, th, nu, AT);
    d.check(cudaGetLastError(), "k_precond");
    std::swap(T, AT);
    const int nt = std::min(orthonormalise(k, nu), kmax - k);
    if (nt <= 0) break;  // the space is exhausted (n small)
    d.check(cudaMemcpyAsync(V + (size_t)k * n, T, (size_t)n * nt * 8, cudaMemcpyDeviceToDevice, st), "append V");
    spmm(V + (size_t)k * n, Wm + (size_t)k * n, nt);
    k += nt;
  }
  std::vector<double> xo((size_t)n * nb);
  if (d.ok) {
    d.check(cudaMemcpyAsync(xo.data(), X, (size_t)n * std::min(nb, k) * 8, cudaMemcpyDeviceToHost, st), "copy X");
    d.check(cudaStreamSynchronize(st), "sync");
  }
  if (mem) cudaFree(mem);
  if (hG) cudaFreeHost(hG);
  if (st) cudaStreamDestroy(st);
  if (!d.ok) {
    seterr(errbuf, errlen, "cipsi_davidson: " + d.err);
    return CIPSI_ERR_CUDA;
  }
  // each vector's largest component made positive (a fixed sign convention)
  for (int b = 0; b < nroots; ++b) {
    double* x = xo.data() + (size_t)b * n;
    int imax = 0;
    for (int i = 1; i < n; ++i)
      if (std::fabs(x[i]) > std::fabs(x[imax])) imax = i;
    const double sg = x[imax] < 0.0 ? -1.0 : 1.0;
    for (int i = 0; i < n; ++i) evecs[(size_t)b * n + i] = sg * x[i];
    evals[b] = theta[b];
    if (resid) resid[b] = res[b];
  }
  if (iters) *iters = it;
  if (!converged) {
    seterr(errbuf, errlen, "cipsi_davidson: not converged after " + std::to_string(maxiter) + " iterations");
    return CIPSI_ERR_OVERFLOW;
  }
  return CIPSI_OK;
}
