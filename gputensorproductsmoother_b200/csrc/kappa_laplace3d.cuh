// 3D operator with a per-cell coefficient, dst = A(kappa) src or rhs - A(kappa)
// src on the interior rows and 0 on the Dirichlet rows, in one pass (sm_100a).
// No reference counterpart (its operator has a unit coefficient).
//
// A CTA owns the nodes of a tile of TX x TY cells (its lower-left ones) and
// marches through cell layers in z, computing the tile's cells and the row of
// cells below and left of it, whose products share the tile's first nodes.  Per
// node plane: x lines are contracted with M and L from global memory into one
// of two plane buffers (the next plane's lines are loaded meanwhile); a thread
// per (cell, x node) contracts y in registers and accumulates its (k+1)^2 (z, y)
// rows.  A layer's cell products, scaled by kappa, go through shared memory
// once, to be gathered by the tile's nodes in a fixed order (deterministic, no
// atomics); the layer's upper node plane is carried in registers.
//
// What bounds it: the FP64 pipe (46 % active at Q4 48^3) and the shared-memory pipe
// (58 % of its wavefront peak) at the 15 warps per SM that 128 registers leave,
// which do not cover the load latency (3.1 of 7.4 cycles per issue); each plane is
// read about 1.4 times (L2) and every dst entry written once.  It replaces 8
// colour launches with a read-modify-write of dst each, a fill and a finishing
// pass.  Measured, us per vmult, before / now: Q4 48^3 FP64 232 / 115, FP32 217 /
// 58; Q4 6^3 38 / 14; Q3 48^3 FP64 152 / 54; Q2 64^3 FP64 274 / 35; Q5 32^3 FP64
// 151 / 121; Q7 16^3 FP64 71 / 63.
#pragma once

#include "tps_common.cuh"

namespace tps {

template <int K, typename T>
struct Kl3 {
  static constexpr int NP = K + 1;
  static constexpr int TX = K == 1 ? 16 : K == 2 ? 8 : K == 3 ? 5 : K == 4 ? 4 : 3;
  static constexpr int TY = K == 1 ? 8 : TX;
  static constexpr int CX = TX + 1, CY = TY + 1, CELLS = CX * CY;  // cells computed
  static constexpr int NT = (CELLS * NP + 31) / 32 * 32;
  static constexpr int YN = CY * K + 1;                            // node rows of a plane
  static constexpr int XTASKS = YN * CX;
  static constexpr int RP = NP % 2 ? NP : NP + 1;                  // odd pitch of a contracted line
  static constexpr int PLANE = XTASKS * RP;
  static constexpr int GX = TX * K, GY = TY * K, COLS = GX * GY, CPT = (COLS + NT - 1) / NT;
  // products of a cell [z][y][x], padded so that the cells' x rows fall on
  // consecutive banks
  static constexpr int BANKS = 128 / static_cast<int>(sizeof(T));
  static constexpr int c_stride()
  {
    int s = NP * NP * NP;
    while (s % BANKS != NP % BANKS) ++s;
    return s;
  }
  static constexpr int CS = c_stride();
  static constexpr size_t BYTES = sizeof(T) * (4 * PLANE + CELLS * CS);
  // the planes of a layer, unrolled where the (k+1)^2 accumulators leave the
  // registers for it (unrolled in FP64 at degrees 5 and 7 they spilled: Q5 32^3
  // 290 us, Q7 16^3 87)
  static constexpr int UNROLL = sizeof(T) == 8 && K >= 5 ? 1 : NP;
  // CTAs per SM that the registers are bounded for
  static constexpr int MINB = sizeof(T) == 4 && K <= 5 ? 512 / NT : K <= 4 ? 512 / NT : K == 5 ? 4 : 2;
  static_assert(XTASKS <= NT || K == 1, "one x line per thread");
};

template <int K, typename T, bool RESIDUAL>
__global__ void __launch_bounds__(Kl3<K, T>::NT, Kl3<K, T>::MINB)
    kappa_laplace3d_kernel(T *__restrict__ dst, const T *__restrict__ src, const T *__restrict__ rhs,
                           const T *__restrict__ kappa, int n, int64_t sy, int64_t sz, int layers, T scale)
{
  using S = Kl3<K, T>;
  constexpr int NP = S::NP, NT = S::NT, CX = S::CX, RP = S::RP;
  const DegreeTables<K, T> &tb = c_tables<K, T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *PL = reinterpret_cast<T *>(smem_raw);  // two plane buffers of M x and L x lines
  T *C = PL + 4 * S::PLANE;
  const int tid = threadIdx.x;
  const int cx0 = blockIdx.x * S::TX - 1, cy0 = blockIdx.y * S::TY - 1;  // the first cell computed
  const int N1 = n * K + 1;
  const int z0 = blockIdx.z * layers, z1 = z0 + layers < n ? z0 + layers : n;
  const int zs = z0 > 0 ? z0 - 1 : 0;  // the layer below contributes its upper node plane

  // x task: node row xr of the plane, cell xc of the row
  const int xr = tid / CX, xc = tid - xr * CX;
  const int gy_x = cy0 * K + xr, gc_x = cx0 + xc;
  const bool xin = tid < S::XTASKS && gy_x >= 0 && gy_x < N1 && gc_x >= 0 && gc_x < n;
  const T *line = src + int64_t(gy_x) * sy + int64_t(gc_x) * K;
  // yz task: cell, x node
  const int yc = tid / NP, yi = tid - yc * NP;
  const int ycy = yc / CX, ycx = yc - ycy * CX;
  const int kx = cx0 + ycx, ky = cy0 + ycy;
  const bool yin = yc < S::CELLS && kx >= 0 && kx < n && ky >= 0 && ky < n;
  const int yoff = yc < S::CELLS ? (ycy * K * CX + ycx) * RP + yi : 0;
  const T *kp = kappa + int64_t(ky) * n + kx;

  T f[NP];
  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  auto load = [&](int plane) {
#pragma unroll
    for (int q = 0; q < NP; ++q) f[q] = xin ? line[int64_t(plane) * sz + q] : T(0);
  };
  // contract the loaded line into the plane's buffer
  auto contract_x = [&](int plane) {
    if (tid < S::XTASKS) {
      T *m = PL + (plane & 1) * 2 * S::PLANE + tid * RP, *l = m + S::PLANE;
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        T a = tb.cmass[i * NP] * f[0], c = tb.clap[i * NP] * f[0];
#pragma unroll
        for (int q = 1; q < NP; ++q) {
          a = fmadd(tb.cmass[i * NP + q], f[q], a);
          c = fmadd(tb.clap[i * NP + q], f[q], c);
        }
        m[i] = a;
        l[i] = c;
      }
    }
  };

  T acc[NP][NP];  // [z][y]
  T carry[S::CPT];
#pragma unroll
  for (int u = 0; u < S::CPT; ++u) carry[u] = T(0);
  load(zs * K);
  contract_x(zs * K);
  __syncthreads();
  load(zs * K + 1);
  for (int z = zs; z < z1; ++z) {
    const T kap = yin ? scale * kp[int64_t(z) * n * n] : T(0);
#pragma unroll
    for (int i = 0; i < NP; ++i)
#pragma unroll
      for (int r = 0; r < NP; ++r) acc[i][r] = T(0);
#pragma unroll(S::UNROLL)
    for (int zq = 0; zq < NP; ++zq) {
      const int plane = z * K + zq;
      if (zq > 0) {  // plane 0 was the last one of the layer below
        contract_x(plane);
        __syncthreads();
        if (plane < z1 * K) load(plane + 1);
      }
      const T *m = PL + (plane & 1) * 2 * S::PLANE + yoff, *l = m + S::PLANE;
      T a[NP], b[NP];
#pragma unroll
      for (int y = 0; y < NP; ++y) {
        a[y] = m[y * CX * RP];
        b[y] = l[y * CX * RP];
      }
#pragma unroll
      for (int r = 0; r < NP; ++r) {
        T p = tb.cmass[r * NP] * a[0], w = tb.clap[r * NP] * a[0];
        w = fmadd(tb.cmass[r * NP], b[0], w);
#pragma unroll
        for (int y = 1; y < NP; ++y) {
          p = fmadd(tb.cmass[r * NP + y], a[y], p);
          w = fmadd(tb.clap[r * NP + y], a[y], w);
          w = fmadd(tb.cmass[r * NP + y], b[y], w);
        }
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          acc[i][r] = fmadd(tb.clap[i * NP + zq], p, acc[i][r]);
          acc[i][r] = fmadd(tb.cmass[i * NP + zq], w, acc[i][r]);
        }
      }
    }
    // the cells' products (the previous layer's were gathered before the
    // barriers of this layer's planes)
    if (yc < S::CELLS) {
      T *c = C + yc * S::CS + yi;
#pragma unroll
      for (int i = 0; i < NP; ++i)
#pragma unroll
        for (int r = 0; r < NP; ++r) c[(i * NP + r) * NP] = kap * acc[i][r];
    }
    __syncthreads();
    // the tile's nodes: a vertex row or column sums its two cells
#pragma unroll
    for (int u = 0; u < S::CPT; ++u) {
      const int t = tid + u * NT;
      if (t < S::COLS) {
        const int ly = t / S::GX, lx = t - ly * S::GX;
        const int cx = lx / K, ix = lx - cx * K, cy = ly / K, iy = ly - cy * K;
        const T *c = C + ((cy + 1) * CX + cx + 1) * S::CS + iy * NP + ix;
        T v[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) v[i] = c[i * NP * NP];
        if (ix == 0) {
#pragma unroll
          for (int i = 0; i < NP; ++i) v[i] += c[i * NP * NP - S::CS + K];
        }
        if (iy == 0) {
          const T *d = c - CX * S::CS + K * NP;
#pragma unroll
          for (int i = 0; i < NP; ++i) v[i] += d[i * NP * NP];
          if (ix == 0) {
#pragma unroll
            for (int i = 0; i < NP; ++i) v[i] += d[i * NP * NP - S::CS + K];
          }
        }
        v[0] += carry[u];
        carry[u] = v[K];
        const int gx = (cx0 + 1) * K + lx, gy = (cy0 + 1) * K + ly;
        if (z >= z0 && gx < N1 - 1 && gy < N1 - 1) {
          const bool edge = gx == 0 || gy == 0;
          // one node, and the Dirichlet nodes beyond the last column and row
          auto store = [&](int64_t at, T w) {
            dst[at] = w;
            if (gx == N1 - 2) dst[at + 1] = T(0);
            if (gy == N1 - 2) {
              dst[at + sy] = T(0);
              if (gx == N1 - 2) dst[at + sy + 1] = T(0);
            }
          };
#pragma unroll
          for (int i = 0; i < K; ++i) {
            const int64_t at = gx + gy * sy + int64_t(z * K + i) * sz;
            const bool bnd = edge || (i == 0 && z == 0);
            store(at, bnd ? T(0) : RESIDUAL ? rhs[at] - v[i] : v[i]);
          }
          if (z == n - 1) store(gx + gy * sy + int64_t(N1 - 1) * sz, T(0));
        }
      }
    }
  }
}

}  // namespace tps
