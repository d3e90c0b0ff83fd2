// 2D fused vertex-patch smoother, one launch per colour (sm_100a).
//
// Reference behaviour: LevelVertexPatch::patch_loop_fused with
// loop_kernel_fused_l + LocalSmoother<FUSED_L> (include/loop_kernel.cuh:786-884,
// include/evaluate_kernel.cuh:255-323, 1026-1113, 1890-1971): for every patch p
// of the colour,  x_I(p) <- omega (x_I(p) + A_II^{-1} (b - A_p x)_I).
//
// As in the 3D kernels, omega (x_I + A_II^{-1}(b_I - A_II x_I - A_IB x_B)) =
// omega A_II^{-1}(b_I - A_IB x_B): only the ring of the box is read.  In 2D
// the ring term has rank 8.  With the ring's two rows r0, rn (corners
// included) and columns c0, cn (corners zero),
//   (A_IB x_B)(y, x) =   L[y,0] (M r0)[x] + M[y,0] (L r0)[x]   (and y = 2k with rn)
//                      + M[x,0] (L c0)[y] + L[x,0] (M c0)[y]   (and x = 2k with cn),
// so a patch needs the products of four lines with M and L, one output entry
// per lane with its row of both matrices in registers, and 8 multiply-adds per
// interior DoF.
//
// A patch is solved by 2k-1 lanes, lane l = interior column l, and a warp
// holds 32 / (2k-1) patches.  Nothing is shared between warps, so stages are
// separated by the warp's own barrier:
//   ring -> shared, the four line products; column l: residual, S^T_y
//   -> row l (one transposition through shared memory): S^T_x, 1/lambda, S_x
//   -> column l: S_y, store (lanes along x).
//
// What bounds it: the latency of these stages on small levels; on large ones the
// shared-memory pipe (54 % of its wavefront peak at Q5 384^2 FP32) and the wait for
// global loads (3.7 of 9.6 cycles per issue), with the 20 warps per SM that 85
// registers leave (issue 48 %, DRAM 18 %).  The kernel before it held a stage's 1D lines of 4 to 16
// patches on a CTA of 128 threads (36 busy lanes of 128 at degree 5) between
// CTA barriers and contracted the full box.  Measured, us per sweep, before /
// now: Q5 384^2 FP32 226 / 53, FP64 286 / 95; Q7 320^2 FP32 300 / 84, FP64 466 /
// 173; Q2 512^2 FP32 55 / 20; Q1 1024^2 FP32 65 / 25; Q5 16^2 FP32 23 / 19.
#pragma once

#include "intdiv.cuh"
#include "smoother3d.cuh"  // evec_apply
#include "tps_common.cuh"

namespace tps {

template <typename T>
struct alignas(16) Quad {
  T v[4];
};

template <int K, typename T>
struct Sm2 {
  static constexpr int N1 = 2 * K + 1, M = 2 * K - 1;
  static constexpr int P = 32 / M;  // patches per warp
  // per patch: ring (N1 quads) | line products (M quads) | transposition M x M
  // (odd row pitch M: conflict-free), rounded to quads
  static constexpr int QX = (M * M + 3) / 4;
  static constexpr int PATCH_QUADS = N1 + M + QX;
  static constexpr size_t WARP_BYTES = sizeof(Quad<T>) * PATCH_QUADS * P;
  // a CTA's warps: four share a CTA where that leaves at least one CTA per SM
  static constexpr int MAX_WARPS = 4;
};

struct Sm2Args {
  int nx_c, count;   // patches of the colour per row, and in all
  int cx, cy;        // colour parities
  int64_t sy;        // row pitch
  uint32_t mx, sx;   // n / nx_c == (n * mx) >> sx
};

// What a lane keeps from patch to patch: its place in the warp's patches, its
// rows of M and L, its 1 / lambda sums, and its patch's buffers.
template <int K, typename T>
struct Sm2Lane {
  using S = Sm2<K, T>;
  using Q = Quad<T>;
  static constexpr int N1 = S::N1, M = S::M, P = S::P;
  bool own;  // lanes past the last patch repeat lane 0 of patch 0 and write nothing
  int p, l;
  Q *ring, *line;
  T *tr;
  T rm[N1], rl[N1], rlam[M];

  __device__ __forceinline__ Sm2Lane(unsigned char *warp_smem, T fd_scale)
  {
    const int lane = threadIdx.x & 31;
    own = lane < P * M;
    p = own ? lane / M : 0;
    l = own ? lane - p * M : 0;
    ring = reinterpret_cast<Q *>(warp_smem) + p * S::PATCH_QUADS;
    line = ring + N1;
    tr = reinterpret_cast<T *>(line + M);
#pragma unroll
    for (int j = 0; j < N1; ++j) {
      rm[j] = g_lane_tables<K, T>.prows2[j * M + l];
      rl[j] = g_lane_tables<K, T>.prows2[(N1 + j) * M + l];
    }
#pragma unroll
    for (int j = 0; j < M; ++j) rlam[j] = fd_scale * g_lane_tables<K, T>.rlam2[j * M + l];  // symmetric
  }

  // One warp-load of patches (the w-th P patches of the colour).  COHERENT: x
  // was written by other SMs earlier in this kernel, so it is read from L2.
  template <bool COHERENT>
  __device__ __forceinline__ void solve(T *x, const T *__restrict__ b, const Sm2Args &a, T scale, int w)
  {
    const DegreeTables<K, T> &tb = c_tables<K, T>;
    const int sy = static_cast<int>(a.sy);  // a patch spans less than 2^31 entries
    auto ld = [](const T *q) { return COHERENT ? __ldcg(q) : *q; };
    const int j0 = w * P + p;
    const bool valid = own && j0 < a.count;
    const int jp = valid ? j0 : w * P;
    const int jy = fast_div(jp, a.mx, a.sx), jx = jp - jy * a.nx_c;
    const int64_t first = int64_t((a.cx + 2 * jx) * K) + int64_t((a.cy + 2 * jy) * K) * a.sy;
    // ---- the ring and this lane's column of b ----
    const T *xb = x + first;
    const T *bb = b + first + a.sy + 1 + l;
    T r[M];
#pragma unroll
    for (int i = 0; i < M; ++i) r[i] = bb[i * sy];
#pragma unroll
    for (int u = 0; u < (N1 + M - 1) / M; ++u) {
      const int j = l + u * M;
      if (j < N1) {
        const bool corner = j == 0 || j == N1 - 1;
        Q q;
        q.v[0] = ld(xb + j);
        q.v[1] = ld(xb + j + (N1 - 1) * a.sy);
        q.v[2] = corner ? T(0) : ld(xb + j * a.sy);
        q.v[3] = corner ? T(0) : ld(xb + j * a.sy + N1 - 1);
        if (own) ring[j] = q;
      }
    }
    __syncwarp();
    // ---- entry l of M and L times the four lines ----
    T m[4], s[4];
    {
      const Q q = ring[0];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        m[c] = rm[0] * q.v[c];
        s[c] = rl[0] * q.v[c];
      }
    }
#pragma unroll
    for (int j = 1; j < N1; ++j) {
      const Q q = ring[j];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        m[c] = fmadd(rm[j], q.v[c], m[c]);
        s[c] = fmadd(rl[j], q.v[c], s[c]);
      }
    }
    if (own) line[l] = Q{{s[2], m[2], s[3], m[3]}};
    __syncwarp();
    // ---- column l: residual, S^T along y ----
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const Q q = line[i];
      T t = tb.plap[(i + 1) * N1] * m[0];
      t = fmadd(tb.pmass[(i + 1) * N1], s[0], t);
      t = fmadd(tb.plap[(i + 1) * N1 + N1 - 1], m[1], t);
      t = fmadd(tb.pmass[(i + 1) * N1 + N1 - 1], s[1], t);
      t = fmadd(rm[0], q.v[0], t);
      t = fmadd(rl[0], q.v[1], t);
      t = fmadd(rm[N1 - 1], q.v[2], t);
      t = fmadd(rl[N1 - 1], q.v[3], t);
      r[i] = fmadd(-scale, t, r[i]);
    }
    T v[M];
    evec_apply<K, T, true>(r, v);
    if (own) {
#pragma unroll
      for (int i = 0; i < M; ++i) tr[i * M + l] = v[i];
    }
    __syncwarp();
    // ---- mode row l: S^T along x, 1 / lambda, S along x ----
#pragma unroll
    for (int i = 0; i < M; ++i) r[i] = tr[l * M + i];
    evec_apply<K, T, true>(r, v);
#pragma unroll
    for (int i = 0; i < M; ++i) v[i] *= rlam[i];
    evec_apply<K, T, false>(v, r);
    if (own) {
#pragma unroll
      for (int i = 0; i < M; ++i) tr[l * M + i] = r[i];
    }
    __syncwarp();
    // ---- column l: S along y, store ----
#pragma unroll
    for (int i = 0; i < M; ++i) r[i] = tr[i * M + l];
    evec_apply<K, T, false>(r, v);
    if (valid) {
      T *xo = x + first + a.sy + 1 + l;
#pragma unroll
      for (int i = 0; i < M; ++i) xo[i * sy] = v[i];
    }
    __syncwarp();  // the ring and transposition buffers are read before the next patch
  }
};

template <int K, typename T>
__global__ void __launch_bounds__(32 * Sm2<K, T>::MAX_WARPS)
    smoother2d_kernel(T *x, const T *__restrict__ b, const Sm2Args a, T scale, T fd_scale)
{
  using S = Sm2<K, T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  Sm2Lane<K, T> lane(smem_raw + warp * S::WARP_BYTES, fd_scale);
  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  for (int w = blockIdx.x * warps + warp; w * S::P < a.count; w += gridDim.x * warps)
    lane.template solve<false>(x, b, a, scale, w);
}

}  // namespace tps
