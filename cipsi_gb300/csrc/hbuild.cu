// hbuild.cu -- the Hamiltonian over a list of determinants, lower triangle by
// rows, as moy builds it for the S + selected list (moy/moy.f:117-199):
// row i holds every column j < min(i, jmax) within two excitations of i,
// in increasing j, with <i|H|j> in the phase of the reference's excitation
// lists (the value moy's hntd returns).
//
//   k_hscan<W, false>  counts the hits (degree <= 2) of every row in every
//                      segment of columns;
//   k_hrows            per row: the segments' offsets and the row's total;
//   k_hscan<W, true>   writes the hits' columns (rowptr: scan of the totals);
//   k_hvalues          the elements, a warp per row, one per lane.
//
// The pair scan: one thread owns one row; a CTA owns kHRows consecutive rows
// and one segment of columns, which it streams through shared memory in
// tiles, so every lane of a warp reads the same column (a broadcast).  The
// degree test is XOR + popcount over the 2W words of the two bitstrings; four
// population counts per pair are what bounds it.  Segments make enough CTAs of
// the triangle (63 CTAs of 256 whole rows left most SMs idle at 16,000
// determinants: 0.55 ms a scan), and elements evaluated row by row keep the
// warps full (inside the scan they took 2.5 ms).
//
// Matrix elements: hmat() of the perturbation kernel (canonical alpha-then-
// beta string phase, the one-difference sum taken over the holes and
// particles of the more excited determinant -- the column when the ranks
// are equal, as moy/hntd.f picks it), times sigma_i * sigma_j, the
// excitation-list phases of the two determinants.  Identical determinants
// (popcount 0) give 0, as hntd does.
#include "pt2_kernel.cuh"

namespace cipsi_dev {
namespace {

constexpr int kHRows = 128;  // rows (threads) per CTA of the scan
constexpr int kHTile = 256;  // columns per shared-memory tile

template <int W, bool FILL>
__global__ void __launch_bounds__(kHRows) k_hscan(HBuildArgs a) {
  __shared__ uint64_t tile[kHTile * 2 * W];
  // heavy (high) row blocks first: row i scans i columns
  const int row0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * kHRows;
  const int i = row0 + (int)threadIdx.x;
  const bool row_ok = i < a.n;
  const int c0 = (int)blockIdx.y * a.seg;
  const int jend = min(row_ok ? min(i, a.jmax) : 0, c0 + a.seg);
  const int jblock = min(min(min(row0 + kHRows - 1, a.n - 1), a.jmax), c0 + a.seg);  // the block's largest jend
  uint64_t u[2 * W];
#pragma unroll
  for (int q = 0; q < 2 * W; ++q) u[q] = row_ok ? a.S[(size_t)i * 2 * W + q] : 0ull;
  const size_t cell = (size_t)blockIdx.y * a.n + i;
  int cnt = 0;
  long long out = FILL && row_ok ? a.rowptr[i] + a.segcnt[cell] : 0;
  for (int j0 = c0; j0 < jblock; j0 += kHTile) {
    const int nt = min(kHTile, jblock - j0);
    __syncthreads();
    for (int x = threadIdx.x; x < nt * 2 * W; x += kHRows) tile[x] = __ldg(&a.S[(size_t)j0 * 2 * W + x]);
    __syncthreads();
#pragma unroll 4
    for (int t = 0; t < nt; ++t) {
      int d = 0;
#pragma unroll
      for (int q = 0; q < 2 * W; ++q) d += __popcll(u[q] ^ tile[t * 2 * W + q]);
      if (d <= 4 && j0 + t < jend) {
        if (FILL)
          a.col[out++] = j0 + t;
        else
          ++cnt;
      }
    }
  }
  if (!FILL && row_ok) a.segcnt[cell] = cnt;
}

// per row: exclusive sums over its segments, and the total
__global__ void __launch_bounds__(256) k_hrows(HBuildArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  int s = 0;
  for (int g = 0; g < a.nseg; ++g) {
    const size_t cell = (size_t)g * a.n + i;
    const int c = a.segcnt[cell];
    a.segcnt[cell] = s;
    s += c;
  }
  a.count[i] = s;
}

template <int W>
__global__ void __launch_bounds__(256) k_hvalues(HBuildArgs a) {
  __shared__ Params sp;
  if (threadIdx.x == 0) sp = a.p;
  __syncthreads();
  const Params& p = sp;
  const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
  uint64_t hf[2 * W];
#pragma unroll
  for (int q = 0; q < 2 * W; ++q) hf[q] = a.hf[q];
#pragma unroll 1
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < a.n; i += warps) {
    const long long b = a.rowptr[i], e = a.rowptr[i + 1];
    uint64_t u[2 * W];
    int rankI = 0;
#pragma unroll
    for (int q = 0; q < 2 * W; ++q) {
      u[q] = __ldg(&a.S[(size_t)i * 2 * W + q]);
      rankI += __popcll(hf[q] & ~u[q]);
    }
    const double sgi = (double)__ldg(&a.sigma[i]);
#pragma unroll 1
    for (long long t = b + lane; t < e; t += 32) {
      const int j = a.col[t];
      uint64_t v[2 * W];
      int diff = 0, rankJ = 0;
#pragma unroll
      for (int q = 0; q < 2 * W; ++q) {
        v[q] = __ldg(&a.S[(size_t)j * 2 * W + q]);
        diff += __popcll(u[q] ^ v[q]);
        rankJ += __popcll(hf[q] & ~v[q]);
      }
      double h = 0.0;
      if (diff != 0) {
        int kind;
        h = hmat<W>(p, u, v, rankI, rankJ, hf, kind);
      }
      a.val[t] = sgi * (double)__ldg(&a.sigma[j]) * h;
    }
  }
}

}  // namespace

// columns per segment: whole tiles, at most 64 segments (the counts then take
// 256 bytes per row at most)
int hscan_segment(int n) {
  const int seg = std::max(4 * kHTile, (n + 63) / 64);
  return (seg + kHTile - 1) / kHTile * kHTile;
}

template <int W>
cudaError_t launch_hcount(const HBuildArgs& a, cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  const dim3 grid((a.n + kHRows - 1) / kHRows, a.nseg);
  k_hscan<W, false><<<grid, kHRows, 0, st>>>(a);
  k_hrows<<<(a.n + 255) / 256, 256, 0, st>>>(a);
  return cudaGetLastError();
}
template <int W>
cudaError_t launch_hfill(const HBuildArgs& a, int sms, cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  const dim3 grid((a.n + kHRows - 1) / kHRows, a.nseg);
  k_hscan<W, true><<<grid, kHRows, 0, st>>>(a);
  k_hvalues<W><<<std::min((a.n + 7) / 8, 8 * sms), 256, 0, st>>>(a);
  return cudaGetLastError();
}

template cudaError_t launch_hcount<1>(const HBuildArgs&, cudaStream_t);
template cudaError_t launch_hcount<2>(const HBuildArgs&, cudaStream_t);
template cudaError_t launch_hfill<1>(const HBuildArgs&, int, cudaStream_t);
template cudaError_t launch_hfill<2>(const HBuildArgs&, int, cudaStream_t);

}  // namespace cipsi_dev
