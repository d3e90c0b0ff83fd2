// Right-hand-side assembly on the device: b_i = sum over cells and QGauss(k+1)
// points of f(x_q) phi_i(x_q) JxW_q, the loop of
// LaplaceOperator::compute_residual (include/laplace_operator.cuh:118-181, run
// on the host through deal.II's FEValues there) for a general f given at the
// quadrature points.
//
// Layout of f: cells lexicographic (x fastest), then the (k+1)^dim Gauss
// points of the cell lexicographic (x fastest).  On a uniform mesh the
// cell integral is a sum factorisation with the 1D table w_q phi_i(x_q)
// (qwshape) and the factor h^dim.  FP64, deterministic, no atomics: every node
// is gathered by one thread; Dirichlet rows are written as zero.
//
// A CTA owns the nodes of a tile of TX x TY cells (its lower-left ones; about
// 32 x 16 nodes) and marches through cell layers in z.  Per plane of Gauss
// points: x lines of the tile's cells and of one row of cells below and left of
// it (their shared nodes belong to the tile) are contracted from global memory
// into shared memory, the next plane's lines being loaded meanwhile; the y
// stage sums the two cells of a vertex column on reading and contracts y; the
// z stage sums the two cells of a vertex row and accumulates the column's k+1
// z nodes in registers, the last of which opens the next layer.
//
// What bounds it: the latency of the two barriers per plane and of the loads
// between them at 19 warps per SM (3.1 cycles each of 12.9 per issue at Q4 48^3), then
// the shared-memory pipe (59 % of its wavefront peak; FP64 pipe 26 %, DRAM 24 %);
// f is read once from HBM and its halo from L2.  Measured, us, one thread per cell in 2^dim colour launches
// / now: 3D Q4 48^3 448 / 87, Q2 96^3 292 / 108, Q5 32^3 772 / 68, Q7 16^3 4974 /
// 70, Q4 8^3 277 / 18; 2D Q4 512^2 149 / 31, Q7 256^2 124 / 46.
#pragma once

#include "tps_common.cuh"

namespace tps {

template <int DIM, int K>
struct Asm {
  static constexpr int NP = K + 1;
  static constexpr int TX = 32 / K, TY = K == 1 ? 16 : K == 2 ? 8 : K <= 4 ? 4 : K == 5 ? 3 : 2;
  static constexpr int GX = TX * K, GY = TY * K;  // nodes owned by a CTA
  static constexpr int NT = 256;
  static constexpr int XTASKS = (TX + 1) * (TY + 1) * NP, XPT = (XTASKS + NT - 1) / NT;
  static constexpr int YTASKS = (TY + 1) * GX;
  static constexpr int COLS = GX * GY, CPT = (COLS + NT - 1) / NT;
  static constexpr int NQ = DIM == 3 ? NP * NP * NP : NP * NP;  // Gauss points of a cell
  static constexpr int PLANES = DIM == 3 ? NP : 1;              // planes of them in z
  static constexpr int T1 = XTASKS * NP, T2 = YTASKS * NP;
  static constexpr size_t BYTES = sizeof(double) * (T1 + T2);
};

template <int DIM, int K>
__global__ void __launch_bounds__(Asm<DIM, K>::NT)
    assemble_rhs_kernel(double *__restrict__ b, const double *__restrict__ fq, int n, int64_t sy, int64_t sz,
                        int layers, double hd)
{
  using A = Asm<DIM, K>;
  constexpr int NP = A::NP, NT = A::NT, GX = A::GX;
  const DegreeTables<K, double> &tb = c_tables<K, double>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *T1 = reinterpret_cast<double *>(smem_raw), *T2 = T1 + A::T1;  // [cy][cx][qy][ix], [cy][iy][gx]
  const int tid = threadIdx.x;
  const int cx0 = blockIdx.x * A::TX, cy0 = blockIdx.y * A::TY;
  const int N1 = n * K + 1;
  const int z0 = DIM == 3 ? blockIdx.z * layers : 0, z1 = DIM == 3 ? (z0 + layers < n ? z0 + layers : n) : 1;
  griddep_wait();

  // x tasks of this thread: the Gauss line (cell, qy) of the current plane
  int64_t src[A::XPT];  // its place in f at plane 0 of layer 0, or -1 outside the mesh
#pragma unroll
  for (int u = 0; u < A::XPT; ++u) {
    const int t = tid + u * NT, c = t / NP, qy = t - c * NP;
    const int ly = c / (A::TX + 1), cx = cx0 - 1 + (c - ly * (A::TX + 1)), cy = cy0 - 1 + ly;
    const bool in = t < A::XTASKS && cx >= 0 && cx < n && cy >= 0 && cy < n;
    src[u] = in ? (int64_t(cy) * n + cx) * A::NQ + qy * NP : -1;
  }
  double f[A::XPT][NP];
  auto load = [&](int z, int qz) {
    const int64_t off = DIM == 3 ? int64_t(z) * n * n * A::NQ + qz * NP * NP : 0;
#pragma unroll
    for (int u = 0; u < A::XPT; ++u)
#pragma unroll
      for (int q = 0; q < NP; ++q) f[u][q] = src[u] >= 0 ? fq[src[u] + off + q] : 0.0;
  };
  // one node, and the Dirichlet nodes beyond the last column and row
  auto store = [&](int gx, int gy, int64_t zoff, double v) {
    double *d = b + zoff + int64_t(gy) * sy + gx;
    *d = gx == 0 || gy == 0 ? 0.0 : v;
    if (gx == N1 - 2) d[1] = 0.0;
    if (gy == N1 - 2) {
      d[sy] = 0.0;
      if (gx == N1 - 2) d[sy + 1] = 0.0;
    }
  };

  constexpr int NZ = DIM == 3 ? NP : 1;
  double acc[A::CPT][NZ];
#pragma unroll
  for (int u = 0; u < A::CPT; ++u)
#pragma unroll
    for (int i = 0; i < NZ; ++i) acc[u][i] = 0.0;
  // the layer below the first one contributes its upper node plane
  const int zs = z0 > 0 ? z0 - 1 : z0;
  load(zs, 0);
  for (int z = zs; z < z1; ++z) {
#pragma unroll
    for (int qz = 0; qz < A::PLANES; ++qz) {
      // ---- x ----
#pragma unroll
      for (int u = 0; u < A::XPT; ++u) {
        const int t = tid + u * NT;
        if (t < A::XTASKS) {
#pragma unroll
          for (int i = 0; i < NP; ++i) {
            double s = tb.qwshape[i] * f[u][0];
#pragma unroll
            for (int q = 1; q < NP; ++q) s = fmadd(tb.qwshape[q * NP + i], f[u][q], s);
            T1[t * NP + i] = s;
          }
        }
      }
      __syncthreads();
      if (qz + 1 < A::PLANES) load(z, qz + 1);
      else if (z + 1 < z1) load(z + 1, 0);
      // ---- y ----
      for (int t = tid; t < A::YTASKS; t += NT) {
        const int cy = t / GX, gx = t - cy * GX, cl = gx / K, ix = gx - cl * K;
        const double *p = T1 + ((cy * (A::TX + 1) + cl + 1) * NP) * NP + ix;
        double v[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) v[q] = p[q * NP];
        if (ix == 0) {
#pragma unroll
          for (int q = 0; q < NP; ++q) v[q] += p[q * NP - NP * NP + K];  // the left cell's last node
        }
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          double s = tb.qwshape[i] * v[0];
#pragma unroll
          for (int q = 1; q < NP; ++q) s = fmadd(tb.qwshape[q * NP + i], v[q], s);
          T2[(cy * NP + i) * GX + gx] = s;
        }
      }
      __syncthreads();
      // ---- z ----
#pragma unroll
      for (int u = 0; u < A::CPT; ++u) {
        const int t = tid + u * NT;
        if (t < A::COLS) {
          const int gy = t / GX, gx = t - gy * GX, cl = gy / K, iy = gy - cl * K;
          double v = T2[((cl + 1) * NP + iy) * GX + gx];
          if (iy == 0) v += T2[(cl * NP + K) * GX + gx];  // the lower cell's last node
          if constexpr (DIM == 2) {
            acc[u][0] = v;
          } else {
#pragma unroll
            for (int i = 0; i < NP; ++i) acc[u][i] = fmadd(tb.qwshape[qz * NP + i], v, acc[u][i]);
          }
        }
      }
    }
    // ---- the layer's nodes; its upper plane opens the next layer ----
#pragma unroll
    for (int u = 0; u < A::CPT; ++u) {
      const int t = tid + u * NT, ly = t / GX, gx = cx0 * K + t - ly * GX, gy = cy0 * K + ly;
      if (t < A::COLS && gx < N1 - 1 && gy < N1 - 1) {
        if constexpr (DIM == 2) {
          store(gx, gy, 0, hd * acc[u][0]);
        } else if (z >= z0) {
#pragma unroll
          for (int i = 0; i < K; ++i) {
            const int gz = z * K + i;
            store(gx, gy, gz * sz, gz == 0 ? 0.0 : hd * acc[u][i]);
          }
          if (z == n - 1) store(gx, gy, int64_t(N1 - 1) * sz, 0.0);
        }
      }
      if constexpr (DIM == 3) {
        acc[u][0] = acc[u][K];
#pragma unroll
        for (int i = 1; i < NP; ++i) acc[u][i] = 0.0;
      }
    }
  }
}

}  // namespace tps
