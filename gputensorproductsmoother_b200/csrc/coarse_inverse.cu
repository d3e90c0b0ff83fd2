// Dense FP64 inverse of the coarsest level's interior operator on the device
// (no reference counterpart: the reference's coarsest level is one patch).
//
// The operator (n <= 4096 rows) is assembled entry by entry, then inverted in
// place by blocked Gauss-Jordan elimination without pivoting, which needs
// none for a symmetric positive definite matrix: the pivots are those of its
// Cholesky factorisation, and one that is not positive is reported.  One
// launch per block of 32 columns, out of place between two buffers: with the
// diagonal block D, its row panel R and column panel C,
//   A_kk <- D^-1, A_kj <- D^-1 R_j, A_ik <- -C_i D^-1, A_ij <- A_ij - C_i D^-1 R_j.
// Every CTA inverts the 32 x 32 diagonal block itself, which saves a launch and
// its hand-over per block, and updates a 64 x 64 tile.
//
// What bounds it: the chain of n / 32 launches, each the 32 eliminations of a block
// deep, three barriers apiece (25 to 30 us a launch up to 361 rows, 50 at 1331, where
// three CTAs share an SM; the matrix stays in L2: DRAM 3 %, shared-memory pipe 55 %
// of its wavefront peak).  It replaces a Cholesky inverse on the host:
// measured for 1331 rows (a kappa update at Q4, 3^3 coarse cells) 76 ms there,
// 2.1 ms here.
#include "coarse_inverse.cuh"

#include "launch.cuh"

namespace tps {
namespace {

constexpr int kNB = 32, kTile = 64, kThreads = 256;

struct SweepSmem {
  double d[kNB][kNB + 1];    // the diagonal block, then its inverse
  double c[kTile][kNB + 1];  // column panel of the tile's rows
  double r[kNB][kTile];      // row panel of the tile's columns, old, then D^-1 times it
  double piv[kNB];           // the column being eliminated
};

// D <- D^-1 in shared memory; false where a pivot is not positive
__device__ bool invert_block(SweepSmem &s)
{
  bool ok = true;
  for (int p = 0; p < kNB; ++p) {
    if (threadIdx.x < kNB) s.piv[threadIdx.x] = s.d[threadIdx.x][p];
    __syncthreads();
    const double pv = s.piv[p];
    ok = ok && pv > 0.0;
    const double ip = 1.0 / pv;
    double v[kNB * kNB / kThreads];
#pragma unroll
    for (int u = 0; u < kNB * kNB / kThreads; ++u) {
      const int e = threadIdx.x + u * kThreads, i = e / kNB, j = e % kNB;
      const double row = (j == p ? 1.0 : s.d[p][j]) * ip;  // the scaled pivot row
      v[u] = i == p ? row : (j == p ? 0.0 : s.d[i][j]) - s.piv[i] * row;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kNB * kNB / kThreads; ++u) {
      const int e = threadIdx.x + u * kThreads;
      s.d[e / kNB][e % kNB] = v[u];
    }
    __syncthreads();
  }
  return ok;
}

__global__ void __launch_bounds__(kThreads)
    gauss_jordan_step_kernel(double *__restrict__ out, const double *__restrict__ a, int n, int kb, int *bad)
{
  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SweepSmem &s = *reinterpret_cast<SweepSmem *>(smem_raw);
  const int i0 = blockIdx.y * kTile, j0 = blockIdx.x * kTile, tid = threadIdx.x;
  const int nb = n - kb < kNB ? n - kb : kNB;  // rows past the end: an identity block
  for (int e = tid; e < kNB * kNB; e += kThreads) {
    const int i = e / kNB, j = e % kNB;
    s.d[i][j] = i < nb && j < nb ? a[static_cast<int64_t>(kb + i) * n + kb + j] : (i == j ? 1.0 : 0.0);
  }
  for (int e = tid; e < kTile * kNB; e += kThreads) {
    const int i = e / kNB, j = e % kNB;
    s.c[i][j] = i0 + i < n && j < nb ? a[static_cast<int64_t>(i0 + i) * n + kb + j] : 0.0;
  }
  for (int e = tid; e < kNB * kTile; e += kThreads) {
    const int i = e / kTile, j = e % kTile;
    s.r[i][j] = i < nb && j0 + j < n ? a[static_cast<int64_t>(kb + i) * n + j0 + j] : 0.0;
  }
  __syncthreads();
  const bool ok = invert_block(s);
  if (!ok && blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) *bad = 1;
  // R <- D^-1 R; its columns inside the diagonal block become D^-1 itself
  double rn[kNB * kTile / kThreads];
#pragma unroll
  for (int u = 0; u < kNB * kTile / kThreads; ++u) {
    const int e = tid + u * kThreads, i = e / kTile, j = e % kTile, jk = j0 + j - kb;
    double t = 0.0;
    if (jk >= 0 && jk < kNB) {
      t = s.d[i][jk];
    } else {
#pragma unroll 8
      for (int p = 0; p < kNB; ++p) t = fma(s.d[i][p], s.r[p][j], t);
    }
    rn[u] = t;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kNB * kTile / kThreads; ++u) {
    const int e = tid + u * kThreads;
    s.r[e / kTile][e % kTile] = rn[u];
  }
  __syncthreads();
  // a 4 x 4 block per thread: rows ty + 16 u, columns tx + 16 v
  const int tx = tid % 16, ty = tid / 16;
  double acc[4][4] = {};
#pragma unroll 8
  for (int p = 0; p < kNB; ++p) {
    double cv[4], rv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      cv[u] = s.c[ty + 16 * u][p];
      rv[u] = s.r[p][tx + 16 * u];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[u][v] = fma(cv[u], rv[v], acc[u][v]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int li = ty + 16 * u, lj = tx + 16 * v, i = i0 + li, j = j0 + lj;
      if (i >= n || j >= n) continue;
      const int ik = i - kb, jk = j - kb;
      const int64_t at = static_cast<int64_t>(i) * n + j;
      double w;
      if (ik >= 0 && ik < kNB)
        w = s.r[ik][lj];
      else
        w = (jk >= 0 && jk < kNB ? 0.0 : a[at]) - acc[u][v];
      out[at] = w;
    }
}

// out = (a + a^T) / 2 (elimination leaves the halves a rounding apart)
__global__ void symmetrize_kernel(double *out, const double *a, int n)
{
  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  const int j = blockIdx.x * 32 + threadIdx.x, i = blockIdx.y * 8 + threadIdx.y;
  if (i >= n || j < i || j >= n) return;
  const int64_t ij = static_cast<int64_t>(i) * n + j, ji = static_cast<int64_t>(j) * n + i;
  const double v = 0.5 * (a[ij] + a[ji]);
  out[ij] = v;
  out[ji] = v;
}

// entry (i, j) of the interior operator: the sum over the cells that hold both
// nodes, in a fixed order
__global__ void __launch_bounds__(kThreads) assemble_coarse_kernel(double *a, CoarseOperator q, int ni)
{
  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  const int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (e >= static_cast<int64_t>(ni) * ni) return;
  const int i = static_cast<int>(e / ni), j = static_cast<int>(e - static_cast<int64_t>(i) * ni);
  const int m1 = q.n * q.k - 1, np = q.k + 1;
  const int ci[3] = {1 + i % m1, 1 + (i / m1) % m1, 1 + i / (m1 * m1)};
  const int cj[3] = {1 + j % m1, 1 + (j / m1) % m1, 1 + j / (m1 * m1)};
  // cells along direction d that hold both coordinates: lo[d] .. hi[d]
  int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
  for (int d = 0; d < q.dim; ++d) {
    const int a0 = min(ci[d], cj[d]), a1 = max(ci[d], cj[d]);
    lo[d] = max(0, (a1 - 1) / q.k);  // the first cell whose last node is >= a1
    hi[d] = min(q.n - 1, a0 / q.k);  // the last cell whose first node is <= a0
  }
  double s = 0.0;
  for (int cz = lo[2]; cz <= hi[2]; ++cz)
    for (int cy = lo[1]; cy <= hi[1]; ++cy)
      for (int cx = lo[0]; cx <= hi[0]; ++cx) {
        const int c3[3] = {cx, cy, cz};
        double m[3], l[3];
        for (int d = 0; d < q.dim; ++d) {
          const int r = (ci[d] - c3[d] * q.k) * np + cj[d] - c3[d] * q.k;
          m[d] = q.cmass[r];
          l[d] = q.clap[r];
        }
        const double v = q.dim == 2 ? l[1] * m[0] + m[1] * l[0]
                                    : l[2] * m[1] * m[0] + m[2] * l[1] * m[0] + m[2] * m[1] * l[0];
        const double kc = q.kappa ? q.kappa[(static_cast<int64_t>(cz) * q.n + cy) * q.n + cx] : 1.0;
        s += kc * q.scale * v;
      }
  a[e] = s;
}

}  // namespace

cudaError_t launch_assemble_coarse(double *a, const CoarseOperator &q, int ni, cudaStream_t s)
{
  const int64_t count = static_cast<int64_t>(ni) * ni;
  TPS_LAUNCH((assemble_coarse_kernel), static_cast<unsigned>((count + kThreads - 1) / kThreads), kThreads, 0, s, a, q,
             ni);
  return cudaGetLastError();
}

cudaError_t launch_spd_inverse(double *a, double *tmp, int n, int *bad, cudaStream_t s)
{
  cudaError_t e = cudaFuncSetAttribute(gauss_jordan_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(sizeof(SweepSmem)));
  if (e != cudaSuccess) return e;
  const unsigned t = static_cast<unsigned>((n + kTile - 1) / kTile);
  double *src = a, *dst = tmp;
  for (int kb = 0; kb < n; kb += kNB) {
    TPS_LAUNCH((gauss_jordan_step_kernel), dim3(t, t), kThreads, sizeof(SweepSmem), s, dst, src, n, kb, bad);
    double *o = src;
    src = dst;
    dst = o;
  }
  // one thread per pair of entries: in place where the result already is in a
  TPS_LAUNCH((symmetrize_kernel), dim3((n + 31) / 32, (n + 7) / 8), dim3(32, 8), 0, s, a, src, n);
  return cudaGetLastError();
}

}  // namespace tps
