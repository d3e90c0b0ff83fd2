// One coloured patch sweep as one launch, for small levels (sm_100a).
//
// Reference behaviour: PatchSmootherImpl::step_impl's loop over the colours
// (include/patch_smoother.cuh:185-292), one kernel per colour there.
//
// On a level of few patches a colour's launch is one patch solve deep: 2.4 to 4
// us with programmatic launches.  Here one CTA (2D), or one thread-block cluster
// of up to 8 (3D), runs all 2^d colours, with the cluster barrier between two
// colours (release and acquire at cluster scope) in place of the launch
// boundary.  x is read from L2 (other SMs wrote it earlier in the kernel); b and
// the tables are constant.  The patch solves are those of the per-colour
// kernels, operation for operation, so the sweeps are bit-identical.
//
// What bounds it: the latency of a patch solve (the teams wait 27 of 36 cycles per
// issue at the barriers between their stages, 3D Q4 4^3 FP32) and, between CTAs, of
// the cluster barrier and the trip through L2, 1 to 2 us a colour together, which is
// why only the smallest levels gain (the rule and its measurements: sweep_pays).
//
// 2D: warps of Sm2Lane (smoother2d.cuh).  3D: teams of threads, one line of
// every stage per thread (the widest stage sets the team: (2k-1)(2k+1) lines),
// the z stage reading its ring lines straight from global memory.
#pragma once

#include "smoother2d.cuh"
#include "smoother3d_warp.cuh"  // WpLayout

namespace tps {

__device__ __forceinline__ void cluster_sync()
{
  asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory");
}

struct SweepArgs {
  int n;            // cells per direction
  int reverse;      // colours in descending order
  int zero_x;       // x == 0 on entry: the first colour reads no x (3D)
  int64_t sy, sz;   // pitches
  uint32_t m0, s0, m1, s1;  // multiply-shift of the colour lattice's row length, parity 0 and 1
};

// patches per direction of a colour's parity
__device__ __forceinline__ int colour_extent(int n, int parity) { return n - 1 > parity ? (n - parity) / 2 : 0; }

template <int K, typename T>
struct Sw2 {
  // the registers of a lane (its rows of M and L) bound the warps of a CTA
  static constexpr int WARPS = (K >= 6 || (K >= 4 && sizeof(T) == 8)) ? 8 : 16;
  static constexpr size_t BYTES = Sm2<K, T>::WARP_BYTES * WARPS;
  static constexpr int PER_CTA = Sm2<K, T>::P * WARPS;  // patches at a time
};

template <int K, typename T>
__global__ void __launch_bounds__(32 * Sw2<K, T>::WARPS)
    sweep2d_kernel(T *x, const T *__restrict__ b, const SweepArgs a, T scale, T fd_scale)
{
  using S = Sm2<K, T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  Sm2Lane<K, T> lane(smem_raw + warp * S::WARP_BYTES, fd_scale);
  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  for (int i = 0; i < 4; ++i) {
    if (i > 0) cluster_sync();
    const int c = a.reverse ? 3 - i : i;
    Sm2Args q;
    q.cx = c & 1;
    q.cy = c >> 1;
    q.nx_c = colour_extent(a.n, q.cx);
    q.count = q.nx_c * colour_extent(a.n, q.cy);
    q.sy = a.sy;
    q.mx = q.cx ? a.m1 : a.m0;
    q.sx = q.cx ? a.s1 : a.s0;
    for (int w = blockIdx.x * warps + warp; w * S::P < q.count; w += gridDim.x * warps)
      lane.template solve<true>(x, b, q, scale, w);
  }
}

template <int K, typename T>
struct Sw3 {
  using L = WpLayout<K, static_cast<int>(sizeof(T))>;
  static constexpr int N1 = 2 * K + 1, M = 2 * K - 1;
  static constexpr int RING = N1 * N1 - M * M, IPAIR = (M * M + 1) / 2;
  static constexpr int NZT = RING + IPAIR, NYT = M * N1, NQT = M * M;
  static constexpr int TEAM = (wp_max(NYT, NZT) + 31) / 32 * 32;  // threads per patch
  static constexpr int ZEXT = (M - 1) * L::PZ + (N1 - 1) * L::RZ + N1;
  static constexpr int VEXT = (M - 1) * L::PV + (M - 1) * L::RV + N1;
  static constexpr int ext(Str3 s) { return (M - 1) * (s.p + s.r + s.c) + 1; }
  static constexpr int QBUF1 = wp_max(ext(L::QA), ext(L::QC)), QBUF2 = wp_max(ext(L::QB), ext(L::QD));
  // per team: [Z1 | Z2, later QA/QC | QB/QD] [V1 | V2]; per CTA the table of
  // fd_scale / (lambda_x + lambda_y + lambda_z)
  static constexpr int ELEMS = wp_max(2 * ZEXT, QBUF1 + QBUF2) + 2 * VEXT;
  static constexpr int RL = M * M * M;
  static constexpr int BY_THREADS = (sizeof(T) == 8 ? 384 : 512) / TEAM, BY_SMEM = (200 * 1024 / static_cast<int>(sizeof(T)) - RL) / ELEMS;
  static constexpr int TEAMS = BY_THREADS < BY_SMEM ? BY_THREADS : BY_SMEM;  // patches of a CTA at a time
  static constexpr int NT = TEAM * TEAMS;
  static constexpr size_t BYTES = sizeof(T) * (static_cast<size_t>(RL) + static_cast<size_t>(ELEMS) * TEAMS);
  static_assert(TEAMS >= 1 && TEAMS <= 16, "one named barrier per team");
};

template <int K, typename T>
__global__ void __launch_bounds__(Sw3<K, T>::NT)
    sweep3d_kernel(T *x, const T *__restrict__ b, const SweepArgs a, T scale, T fd_scale)
{
  using S = Sw3<K, T>;
  using Lo = typename S::L;
  using P2 = typename Pair<T>::type;
  constexpr int N1 = S::N1, M = S::M;
  constexpr Str3 QA = Lo::QA, QB = Lo::QB, QC = Lo::QC, QD = Lo::QD;
  const DegreeTables<K, T> &tb = c_tables<K, T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *RL = reinterpret_cast<T *>(smem_raw);
  const int team = threadIdx.x / S::TEAM, t = threadIdx.x - team * S::TEAM;
  T *Z1 = RL + S::RL + team * S::ELEMS, *Z2 = Z1 + S::ZEXT;
  T *V1 = Z1 + wp_max(2 * S::ZEXT, S::QBUF1 + S::QBUF2), *V2 = V1 + S::VEXT;
  T *QAb = Z1, *QBb = Z1 + S::QBUF1;
  auto team_sync = [&]() {
    if constexpr (S::TEAM == 32) __syncwarp();
    else named_bar(1 + team, S::TEAM);
  };
  for (int l = threadIdx.x; l < S::RL; l += S::NT)
    RL[l] = fd_scale / (tb.eval[l % M] + tb.eval[(l / M) % M] + tb.eval[l / (M * M)]);
  // this thread's z-stage line: a ring line (y, xx), or a pair of interior ones
  int zy = 0, zx = 0;
  if (t < N1) {
    zx = t;
  } else if (t < 2 * N1) {
    zy = N1 - 1;
    zx = t - N1;
  } else if (t < S::RING) {
    const int q = t - 2 * N1;
    zy = 1 + (q >> 1);
    zx = (q & 1) ? N1 - 1 : 0;
  }
  const int zi_y = t % M, xx_y = t / M;            // y stage: (zi, x)
  const int hi = t / M, lo = t - hi * M;           // the other stages: two line coordinates
  const int sy = static_cast<int>(a.sy), sz = static_cast<int>(a.sz);
  __syncthreads();
  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  const int teams = S::TEAMS * gridDim.x;
  for (int i = 0; i < 8; ++i) {
    if (i > 0) cluster_sync();
    const int c = a.reverse ? 7 - i : i;
    const int cx = c & 1, cy = (c >> 1) & 1, cz = c >> 2;
    const int nx = colour_extent(a.n, cx), ny = colour_extent(a.n, cy);
    const int count = nx * ny * colour_extent(a.n, cz);
    const bool zero = a.zero_x && i == 0;
    // consecutive patches go to different CTAs, so that few patches use all of them
    for (int j = team * gridDim.x + blockIdx.x; j < count; j += teams) {
      const int row = fast_div(j, cx ? a.m1 : a.m0, cx ? a.s1 : a.s0), jx = j - row * nx;
      const int jz = fast_div(row, cy ? a.m1 : a.m0, cy ? a.s1 : a.s0), jy = row - jz * ny;
      const int64_t first =
          int64_t((cx + 2 * jx) * K) + int64_t((cy + 2 * jy) * K) * a.sy + int64_t((cz + 2 * jz) * K) * a.sz;
      T bq[M];
      if (t < S::NQT) {
        const T *bb = b + first + 1 + int64_t(lo + 1) * a.sy + int64_t(hi + 1) * a.sz;
#pragma unroll
        for (int q = 0; q < M; ++q) bq[q] = bb[q];
      }
      if (!zero) {
        // ---- z: Z1 = M_z x~, Z2 = L_z x~ ----
        const T *box = x + first;
        if (t < S::RING) {
          T v[N1], ec, r1[M], r2[M];
          P2 eo[K > 1 ? K : 1];
          const T *src = box + zy * sy + zx;
#pragma unroll
          for (int z = 0; z < N1; ++z) v[z] = __ldcg(src + int64_t(z) * sz);
          fold_pairs<K, T>(v, eo, ec);
          rows_mass<K, T>(eo, ec, r1);
          rows_lap<K, T>(eo, ec, r2);
          T *d1 = Z1 + zy * Lo::RZ + zx, *d2 = Z2 + zy * Lo::RZ + zx;
#pragma unroll
          for (int q = 0; q < M; ++q) {
            d1[q * Lo::PZ] = r1[q];
            d2[q * Lo::PZ] = r2[q];
          }
        } else if (t < S::NZT) {
          const int r0 = 2 * (t - S::RING);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = r0 + h;
            if (r < M * M) {
              const int y = 1 + r / M, xx = 1 + r % M;
              const T *src = box + y * sy + xx;
              const T v0 = __ldcg(src), vn = __ldcg(src + int64_t(N1 - 1) * sz);
              T *d1 = Z1 + y * Lo::RZ + xx, *d2 = Z2 + y * Lo::RZ + xx;
#pragma unroll
              for (int q = 0; q < M; ++q) {
                d1[q * Lo::PZ] = fmadd(tb.pmass[(q + 1) * N1 + N1 - 1], vn, tb.pmass[(q + 1) * N1] * v0);
                d2[q * Lo::PZ] = fmadd(tb.plap[(q + 1) * N1 + N1 - 1], vn, tb.plap[(q + 1) * N1] * v0);
              }
            }
          }
        }
        team_sync();
        // ---- y: V1 = M_y Z2 + L_y Z1, V2 = M_y Z1 ----
        if (t < S::NYT) {
          const T *s1 = Z1 + zi_y * Lo::PZ + xx_y, *s2 = Z2 + zi_y * Lo::PZ + xx_y;
          T v[N1], ec1, ec2;
          P2 eo1[K > 1 ? K : 1], eo2[K > 1 ? K : 1];
#pragma unroll
          for (int q = 0; q < N1; ++q) v[q] = s1[q * Lo::RZ];
          fold_pairs<K, T>(v, eo1, ec1);
#pragma unroll
          for (int q = 0; q < N1; ++q) v[q] = s2[q * Lo::RZ];
          fold_pairs<K, T>(v, eo2, ec2);
          T ra[M], rc[M];
          rows_mass_lap<K, T>(eo2, ec2, eo1, ec1, ra);
          rows_mass<K, T>(eo1, ec1, rc);
          T *d1 = V1 + zi_y * Lo::PV + xx_y, *d2 = V2 + zi_y * Lo::PV + xx_y;
#pragma unroll
          for (int q = 0; q < M; ++q) {
            d1[q * Lo::RV] = ra[q];
            d2[q * Lo::RV] = rc[q];
          }
        }
        team_sync();
      }
      // ---- x: r = b - s (M_x V1 + L_x V2), then S^T along x -> QA ----
      if (t < S::NQT) {
        T res[M], q[M];
        if (!zero) {
          const T *s1 = V1 + hi * Lo::PV + lo * Lo::RV, *s2 = V2 + hi * Lo::PV + lo * Lo::RV;
          T v[N1], ec1, ec2;
          P2 eo1[K > 1 ? K : 1], eo2[K > 1 ? K : 1];
#pragma unroll
          for (int u = 0; u < N1; ++u) v[u] = s1[u];
          fold_pairs<K, T>(v, eo1, ec1);
#pragma unroll
          for (int u = 0; u < N1; ++u) v[u] = s2[u];
          fold_pairs<K, T>(v, eo2, ec2);
          T ra[M];
          rows_mass_lap<K, T>(eo1, ec1, eo2, ec2, ra);
#pragma unroll
          for (int u = 0; u < M; ++u) res[u] = bq[u] - scale * ra[u];
        } else {
#pragma unroll
          for (int u = 0; u < M; ++u) res[u] = bq[u];
        }
        evec_apply<K, T, true>(res, q);
        T *d = QAb + hi * QA.p + lo * QA.r;
#pragma unroll
        for (int u = 0; u < M; ++u) d[u * QA.c] = q[u];
      }
      team_sync();
      // ---- S^T along y: QA -> QB ----
      if (t < S::NQT) {
        const T *s = QAb + hi * QA.p + lo * QA.c;
        T v[M], q[M];
#pragma unroll
        for (int u = 0; u < M; ++u) v[u] = s[u * QA.r];
        evec_apply<K, T, true>(v, q);
        T *d = QBb + hi * QB.p + lo * QB.c;
#pragma unroll
        for (int u = 0; u < M; ++u) d[u * QB.r] = q[u];
      }
      team_sync();
      // ---- S^T along z, eigenvalue scaling, S along z: QB -> QC ----
      if (t < S::NQT) {
        const T *s = QBb + hi * QB.r + lo * QB.c;
        T v[M], q[M];
#pragma unroll
        for (int u = 0; u < M; ++u) v[u] = s[u * QB.p];
        evec_apply<K, T, true>(v, q);
#pragma unroll
        for (int u = 0; u < M; ++u) q[u] *= RL[u * M * M + t];
        evec_apply<K, T, false>(q, v);
        T *d = QAb + hi * QC.r + lo * QC.c;
#pragma unroll
        for (int u = 0; u < M; ++u) d[u * QC.p] = v[u];
      }
      team_sync();
      // ---- S along x: QC -> QD ----
      if (t < S::NQT) {
        const T *s = QAb + hi * QC.p + lo * QC.r;
        T v[M], q[M];
#pragma unroll
        for (int u = 0; u < M; ++u) v[u] = s[u * QC.c];
        evec_apply<K, T, false>(v, q);
        T *d = QBb + hi * QD.p + lo * QD.r;
#pragma unroll
        for (int u = 0; u < M; ++u) d[u * QD.c] = q[u];
      }
      team_sync();
      // ---- S along y and store x_I ----
      if (t < S::NQT) {
        const T *s = QBb + hi * QD.p + lo * QD.c;
        T v[M], q[M];
#pragma unroll
        for (int u = 0; u < M; ++u) v[u] = s[u * QD.r];
        evec_apply<K, T, false>(v, q);
        T *xp = x + first + 1 + lo + a.sy + int64_t(hi + 1) * a.sz;
#pragma unroll
        for (int u = 0; u < M; ++u) xp[u * sy] = q[u];
      }
      team_sync();  // the Q buffers (over Z) are read before the next patch's z stage
    }
  }
}

}  // namespace tps
