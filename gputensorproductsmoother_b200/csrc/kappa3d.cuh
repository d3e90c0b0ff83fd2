// 3D vertex-patch smoother with a per-cell coefficient (sm_100a), one colour
// per launch, one patch per CTA.  No reference counterpart (the reference's
// Poisson path has a unit coefficient).  The algebra is that of the 2D kernel
// in kappa.cuh: the box residual b - A(kappa) x with the true coefficient of
// the patch's 8 cells, the local solve by the unit-coefficient fast
// diagonalisation scaled by the patch-averaged coefficient per DoF,
// D^-1/2 FD^-1 D^-1/2, and x_I <- omega (x_I + delta).
//
// The 8 cells are reflections of one another about the patch centre, and the
// 1D cell matrices are centro-symmetric.  Counted from the outer box boundary
// inward (node 0 outside, node k the patch centre), every cell therefore uses
// the same rows 1..k of the same matrices, so that one thread per (cell, x
// node) runs with compile-time constant-bank coefficients and the cells
// differ in addresses only:
//   x stage:  M_x x and L_x x of every box line and half, 2 k (k+1)
//             multiply-adds per half line, into TA and TB;
//   yz stage: a thread walks the k+1 z planes of its cell, contracts the k+1
//             entries in y in registers and accumulates its k x k (z, y) rows:
//             one pass through shared memory instead of one per direction;
//   solve:    the first stage gathers a line of interior nodes from the (up to
//             8) cells that share each node; then five line stages.
// D^-1/2 takes 27 values per patch (a node lies below, on or above the centre
// plane in each direction), formed by 27 threads.
//
// What bounds it: shared-memory wavefronts (78 % of their peak at Q4 48^3 FP64; issue
// 57 %, FP64 pipe 37 %, 36 % of the warps by shared memory), although the yz stage
// does about 460 multiply-adds per 50 shared loads there.  The kernel
// before it ran the stages cell by cell with three shared-memory exchanges and
// two square roots and divisions per node.  Measured, us per sweep on caller
// vectors, before / now: Q4 48^3 FP64 3084 / 618, FP32 1416 / 430; Q4 12^3 FP64
// 73 / 40; Q3 48^3 FP64 1061 / 263; Q2 64^3 FP64 1605 / 300; Q5 32^3 FP64 2274 / 377;
// Q7 16^3 FP64 793 / 214.  The x box is copied asynchronously (plain loads one
// after the other: 752 at Q4 48^3); b copied to shared memory as well, or loaded
// before the yz stage, measured slower (646 and more: fewer resident patches).
#pragma once

#include "ptx.cuh"
#include "smoother3d.cuh"
#include "smoother3d_warp.cuh"  // wp_max
#include "tps_common.cuh"

namespace tps {

// Paddings of the shared arrays, from an exhaustive search for the fewest
// wavefronts of the warp-wide accesses below (entries; [FP64, FP32][degree]):
// of TA and TB's y halves and x nodes, of the cell results' rows and planes, and
// the largest stride of the y-contracted lines.
struct Ks3Pad {
  int ty, td, cr, cp, ca;
};
template <int K, typename T>
constexpr Ks3Pad ks3_pad()
{
  constexpr Ks3Pad pad[2][8] = {{{},
                                 {0, 1, 0, 0, 1},
                                 {0, 2, 4, 4, 9},
                                 {0, 2, 2, 6, 33},
                                 {0, 0, 0, 4, 49},
                                 {0, 1, 4, 13, 81},
                                 {0, 6, 0, 0, 129},
                                 {2, 3, 0, 0, 177}},
                                {{},
                                 {0, 0, 0, 0, 1},
                                 {7, 3, 0, 8, 9},
                                 {0, 5, 0, 4, 25},
                                 {0, 0, 8, 8, 65},
                                 {0, 1, 6, 10, 97},
                                 {0, 14, 4, 12, 129},
                                 {0, 2, 2, 7, 177}}};
  return pad[sizeof(T) == 8 ? 0 : 1][K];
}

template <int K, typename T>
struct Ks3 {
  static constexpr int NP = K + 1, N1 = 2 * K + 1, M = 2 * K - 1;
  static constexpr Ks3Pad PAD = ks3_pad<K, T>();
  // a group of G lanes (8 cells x k x-nodes, whole warps) holds YS-th of the y
  // rows; YS groups share a patch where one group's lanes would leave the
  // other stages (2 (k+1) (2k+1) half lines, (2k-1)^2 lines) short of threads
  static constexpr int G = (8 * K + 31) / 32 * 32;
  static constexpr int YS = K >= 4 ? 2 : 1;
  static constexpr int NT = G * YS;
  static constexpr int YR = (K + YS - 1) / YS;  // y rows of a group
  static constexpr int BOX = N1 * N1 * N1;
  // TA, TB: [z][x from outside][half in y][y from outside][half in x]; the
  // centre line of y is kept in both halves
  static constexpr int TO = 2 * NP + PAD.ty, TD = 2 * TO + PAD.td, TZ = K * TD, TSZ = N1 * TZ;
  // cell results on the 2k nodes per direction (the centre once per half): [z][y][x]
  static constexpr int CR = 2 * K + PAD.cr, CP = 2 * K * CR + PAD.cp, CSZ = 2 * K * CP;
  // lines contracted in y, written and read across x and y: strides (2k-1, 1,
  // SX) of (z, y, x); the arrays between the x and z stages are dense
  static constexpr int SX = PAD.ca, SSZ = (M - 1) * (M + 1 + SX) + 1;
  static constexpr int RA = wp_max(wp_max(TSZ, CSZ), wp_max(SSZ, M * M * M));
  static constexpr int ELEMS = BOX + 2 * RA;
  static constexpr size_t BYTES = sizeof(T) * ELEMS;
};

// rows Y0+1 .. Y0+NY (y) and 1..k (z) of the cell product of one thread:
// acc[z][y] = L_z M_y TA + M_z (L_y TA + M_y TB); ta, tb point at the cell's
// outermost (z, y) entry of this x node, dz and dy step inward
template <int K, typename T, int Y0, int NY, int NA>
__device__ __forceinline__ void ks3_planes(const T *ta, const T *tb, int dz, int dy, T (&acc)[K][NA])
{
  constexpr int NP = K + 1;
  const DegreeTables<K, T> &c = c_tables<K, T>;
#pragma unroll
  for (int i = 0; i < K; ++i)
#pragma unroll
    for (int q = 0; q < NY; ++q) acc[i][q] = T(0);
#pragma unroll
  for (int z = 0; z < NP; ++z) {
    T a[NP], b[NP];
#pragma unroll
    for (int y = 0; y < NP; ++y) {
      a[y] = ta[z * dz + y * dy];
      b[y] = tb[z * dz + y * dy];
    }
#pragma unroll
    for (int q = 0; q < NY; ++q) {
      const int r = (Y0 + q + 1) * NP;
      T p = c.cmass[r] * a[0], w = c.clap[r] * a[0];
      w = fmadd(c.cmass[r], b[0], w);
#pragma unroll
      for (int y = 1; y < NP; ++y) {
        p = fmadd(c.cmass[r + y], a[y], p);
        w = fmadd(c.clap[r + y], a[y], w);
        w = fmadd(c.cmass[r + y], b[y], w);
      }
#pragma unroll
      for (int i = 0; i < K; ++i) {
        acc[i][q] = fmadd(c.clap[(i + 1) * NP + z], p, acc[i][q]);
        acc[i][q] = fmadd(c.cmass[(i + 1) * NP + z], w, acc[i][q]);
      }
    }
  }
}

template <int K, typename T>
__global__ void __launch_bounds__(Ks3<K, T>::NT)
    kappa_smoother3d_kernel(T *__restrict__ x, const T *__restrict__ b, const T *__restrict__ kappa, int n,
                            int colour, int nx_c, int ny_c, int64_t sy, int64_t sz, T s, T fd_scale, T omega)
{
  using S = Ks3<K, T>;
  constexpr int NP = S::NP, N1 = S::N1, M = S::M, NT = S::NT;
  const DegreeTables<K, T> &tb = c_tables<K, T>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ T dsq[27];  // D^-1/2 per node class (below, on, above the centre in x, y, z)
  T *X = reinterpret_cast<T *>(smem_raw);
  T *TA = X + S::BOX, *TB = TA + S::RA;
  const int tid = threadIdx.x;
  auto sync = [&]() {
    if constexpr (NT == 32) __syncwarp();
    else __syncthreads();
  };
  const int j = blockIdx.x;
  const int px = (colour & 1) + 2 * (j % nx_c), py = ((colour >> 1) & 1) + 2 * ((j / nx_c) % ny_c);
  const int pz = ((colour >> 2) & 1) + 2 * (j / (nx_c * ny_c));
  const int64_t first = int64_t(px) * K + int64_t(py) * K * sy + int64_t(pz) * K * sz;
  const T *kc = kappa + px + int64_t(py) * n + int64_t(pz) * n * n;  // the patch's first cell
  const int sy32 = static_cast<int>(sy);
  // cell of this thread in the yz stage
  const int grp = tid / S::G, gl = tid - grp * S::G;
  const bool cell_lane = gl < 8 * K;
  const int o = cell_lane ? gl / K : 0, d = cell_lane ? gl - o * K : 0;
  const int ox = o & 1, oy = (o >> 1) & 1, oz = o >> 2;
  // before the wait: no kernel writes kappa (read after it, a sweep took 1.5 to 2
  // us more: Q4 48^3 FP64 613.6 / 615.1, Q7 16^3 208.3 / 210.6)
  const T kap = s * kc[ox + oy * n + int64_t(oz) * n * n];
  T kd[8];
  if (tid < 27) {
#pragma unroll
    for (int q = 0; q < 8; ++q) kd[q] = kc[(q & 1) + ((q >> 1) & 1) * n + int64_t(q >> 2) * n * n];
  }

  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  for (int l = tid; l < S::BOX; l += NT) {
    const int r = l / N1, lx = l - r * N1, lz = r / N1, ly = r - lz * N1;
    cp_async_zfill<sizeof(T)>(X + l, x + first + lx + ly * sy32 + int64_t(lz) * sz, true);
  }
  cp_async_commit();  // all of a thread's copies in flight at once
  if (tid < 27) {
    const int c3[3] = {tid % 3, (tid / 3) % 3, tid / 9};  // 0 below, 1 on, 2 above
    T acc = T(0);
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      bool in = true;
#pragma unroll
      for (int dd = 0; dd < 3; ++dd) in = in && c3[dd] != (((q >> dd) & 1) ? 0 : 2);
      if (in) {
        acc += kd[q];
        ++cnt;
      }
    }
    dsq[tid] = T(1) / sqrt(acc / T(cnt));
  }
  cp_async_wait_all();
  sync();
  // x stage: task = (z, half in y, y from outside, half in x)
  for (int t = tid; t < N1 * 2 * NP * 2; t += NT) {
    const int hx = t & 1, r = t >> 1;  // r = (z, half in y, y)
    const int z = r / (2 * NP), ry = r - z * (2 * NP);
    const int y = ry < NP ? ry : 2 * K - (ry - NP);
    const T *src = X + (z * N1 + y) * N1 + (hx ? 2 * K : 0);
    T v[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) v[q] = src[hx ? -q : q];
    const int at = z * S::TZ + (ry < NP ? 2 * ry : S::TO + 2 * (ry - NP)) + hx;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      T a = tb.cmass[(i + 1) * NP] * v[0], c = tb.clap[(i + 1) * NP] * v[0];
#pragma unroll
      for (int q = 1; q < NP; ++q) {
        a = fmadd(tb.cmass[(i + 1) * NP + q], v[q], a);
        c = fmadd(tb.clap[(i + 1) * NP + q], v[q], c);
      }
      TA[at + i * S::TD] = a;
      TB[at + i * S::TD] = c;
    }
  }
  sync();
  // yz stage
  {
    const int base = (oz ? 2 * K : 0) * S::TZ + d * S::TD + oy * S::TO + ox;
    const int dz = oz ? -S::TZ : S::TZ;
    T *c0 = TA + (oz ? (2 * K - 1) * S::CP : 0) + (oy ? (2 * K - 1) * S::CR : 0) + (ox ? 2 * K - 1 - d : d);
    const int cz = oz ? -S::CP : S::CP, cy = oy ? -S::CR : S::CR;
    // the y halves are stored from the outside inward: both step forward.  A
    // group has its own rows of constant-bank coefficients, so its own code; the
    // barrier between the reads and the writes is one for the CTA
    T acc[K][S::YR];
    if (cell_lane) {
      if (grp == 0)
        ks3_planes<K, T, 0, S::YR>(TA + base, TB + base, dz, 2, acc);
      else if constexpr (S::YS == 2)
        ks3_planes<K, T, S::YR, K - S::YR>(TA + base, TB + base, dz, 2, acc);
    }
    sync();  // TA and TB are read
    if (cell_lane) {
      c0 += grp * S::YR * cy;
#pragma unroll
      for (int q = 0; q < S::YR; ++q)
        if (q < K - S::YR || grp == 0) {
#pragma unroll
          for (int i = 0; i < K; ++i) c0[i * cz + q * cy] = kap * acc[i][q];
        }
    }
  }
  sync();
  // residual line by line in y (b is read along x), D^-1/2, S^T along y: C (TA) -> TB
  constexpr int PM = M * M;
  for (int t = tid; t < PM; t += NT) {
    const int zi = t / M, xi = t - zi * M;  // interior indices
    const T *bg = b + first + 1 + xi + sy + int64_t(zi + 1) * sz;
    T r[M];
#pragma unroll
    for (int i = 0; i < M; ++i) r[i] = bg[i * sy32];
    // the cells that share the line: below / above the centre plane (class 0
    // and 2), or both on it; their nodes: node index, plus one above the centre
    const int zc = zi < K - 1 ? 0 : zi == K - 1 ? 1 : 2, xc = xi < K - 1 ? 0 : xi == K - 1 ? 1 : 2;
    const int zl = zc == 2 ? zi + 1 : zi, xl = xc == 2 ? xi + 1 : xi;
    for (int az = 0; az <= (zc == 1 ? 1 : 0); ++az)
      for (int ax = 0; ax <= (xc == 1 ? 1 : 0); ++ax) {
        const T *c = TA + (zl + az) * S::CP + xl + ax;
#pragma unroll
        for (int i = 0; i < K; ++i) r[i] -= c[i * S::CR];
#pragma unroll
        for (int i = K - 1; i < M; ++i) r[i] -= c[(i + 1) * S::CR];
      }
    const T *dq = dsq + xc + 9 * zc;
#pragma unroll
    for (int i = 0; i < M; ++i) r[i] *= dq[i < K - 1 ? 0 : i == K - 1 ? 3 : 6];
    T q[M];
    evec_apply<K, T, true>(r, q);
    T *dst = TB + zi * M + xi * S::SX;
#pragma unroll
    for (int i = 0; i < M; ++i) dst[i] = q[i];
  }
  sync();
  // S^T along x: TB -> TA
  for (int t = tid; t < PM; t += NT) {
    const int zi = t / M, yi = t - zi * M;
    T v[M], q[M];
#pragma unroll
    for (int i = 0; i < M; ++i) v[i] = TB[zi * M + yi + i * S::SX];
    evec_apply<K, T, true>(v, q);
#pragma unroll
    for (int i = 0; i < M; ++i) TA[t * M + i] = q[i];
  }
  sync();
  // S^T along z, eigenvalue scaling, S along z: TA -> TB
  for (int t = tid; t < PM; t += NT) {
    T v[M], q[M];
#pragma unroll
    for (int i = 0; i < M; ++i) v[i] = TA[i * PM + t];
    evec_apply<K, T, true>(v, q);
#pragma unroll
    for (int i = 0; i < M; ++i) q[i] *= fd_scale * g_lane_tables<K, T>.rlam3[i * PM + t];
    evec_apply<K, T, false>(q, v);
#pragma unroll
    for (int i = 0; i < M; ++i) TB[i * PM + t] = v[i];
  }
  sync();
  // S along x: TB -> TA
  for (int t = tid; t < PM; t += NT) {
    const int zi = t / M, yi = t - zi * M;
    T v[M], q[M];
#pragma unroll
    for (int i = 0; i < M; ++i) v[i] = TB[t * M + i];
    evec_apply<K, T, false>(v, q);
#pragma unroll
    for (int i = 0; i < M; ++i) TA[zi * M + yi + i * S::SX] = q[i];
  }
  sync();
  // S along y and the update of x_I
  T *xp = x + first + 1 + sy + sz;
  for (int t = tid; t < PM; t += NT) {
    const int zi = t / M, xi = t - zi * M;
    T v[M], q[M];
#pragma unroll
    for (int i = 0; i < M; ++i) v[i] = TA[zi * M + i + xi * S::SX];
    evec_apply<K, T, false>(v, q);
    const int xc = xi < K - 1 ? 0 : xi == K - 1 ? 1 : 2, zc = zi < K - 1 ? 0 : zi == K - 1 ? 1 : 2;
    const T *dq = dsq + xc + 9 * zc;
    const T *xo = X + (zi + 1) * N1 * N1 + N1 + xi + 1;
    T *xg = xp + xi + int64_t(zi) * sz;
#pragma unroll
    for (int i = 0; i < M; ++i)
      xg[i * sy32] = omega * fmadd(dq[i < K - 1 ? 0 : i == K - 1 ? 3 : 6], q[i], xo[i * N1]);
  }
}

}  // namespace tps
