// Geometric MG transfer between a level with n_c cells per direction and its
// uniform refinement (2 n_c cells), sm_100a.
//
// Reference behaviour: MGTransferCUDA::prolongate_and_add / restrict_and_add
// (include/cuda_mg_transfer.template.cuh:575-671) with mg_kernel
// (:21-369): per coarse cell, embed the (k+1)^d coarse values into the
// (2k+1)^d child DoFs with the 1D prolongation, weight by 1/valence (0 on the
// Dirichlet boundary), atomicAdd; restriction is the transpose.  Coarse
// Dirichlet DoFs are zeroed before prolongation and after restriction.
//
// B200 design: the weighted per-cell scatter equals exact nodal interpolation
// P = P1 (x) P1 (x) P1 restricted to interior DoFs, so both directions are
// written as gathers (no atomics, deterministic):
//   fine(i)   = sum_j P1(i_z,j_z) P1(i_y,j_y) P1(i_x,j_x) coarse(j)
//   coarse(j) = sum_i P1(i_z,j_z) P1(i_y,j_y) P1(i_x,j_x) fine(i)
// A prolongation is one pass over tiles of the fine level.  A 3D restriction is
// one 2D pass per xy-plane plus one 1D pass along z; the intermediate (fine z x
// coarse y x coarse x, a quarter of the fine level) lives in a per-level scratch
// buffer.
#pragma once

#include "ptx.cuh"
#include "tps_common.cuh"

namespace tps {

enum class XYOut { AddInterior = 0, SetInterior = 1, SetAll = 2 };

template <int K>
struct XYTile {
  // restriction: coarse cells per CTA and direction, 8 (k <= 4) or 4, so
  // that the second pass of a 256-thread CTA has a task per thread and the
  // fine-plane halo costs (2k(C+1)+1)^2 / (2kC)^2 = 1.3x at k = 4 (1.6x with
  // 4 cells; measured at 3D Q4 64^3: FP32 85 -> 70 us, FP64 124 -> 113 us)
  static constexpr int C = K <= 4 ? 8 : 4;
  static constexpr int NT = 256;
};

// 2D prolongation: coarse cells per CTA and direction.  Measured, us per
// prolongate-and-add in FP32, 8 / 4 cells: Q1 1024^2 12.3 / 13.1, Q4 512^2 12.5 /
// 12.4; FP64 tiles of 8 cells need more than 48 KB at degree 4.
template <int K, typename T>
struct ProlTile {
  static constexpr int C = (sizeof(T) == 4 && K <= 4) ? 8 : K <= 4 ? 4 : 2;
};

// 1D prolongation of one coarse cell: v[0..k] coarse nodes -> out[0..2k-1]
// fine nodes 2k*c + f (the node 2k*(c+1) belongs to the next cell).
template <int K, typename T>
__device__ __forceinline__ void prol_cell(const T (&v)[K + 1], T (&out)[2 * K])
{
  const DegreeTables<K, T> &tb = c_tables<K, T>;
#pragma unroll
  for (int f = 0; f < 2 * K; ++f) {
    T s = T(0);
#pragma unroll
    for (int b = 0; b <= K; ++b) s += tb.prol[f * (K + 1) + b] * v[b];
    out[f] = s;
  }
}

// 1D restriction to the k coarse nodes c*k+b, b < k, from the fine nodes
// v[0..4k] = 2k(c-1) .. 2k(c+1).
template <int K, typename T>
__device__ __forceinline__ void restr_cell(const T (&v)[4 * K + 1], T (&out)[K])
{
  const DegreeTables<K, T> &tb = c_tables<K, T>;
#pragma unroll
  for (int b = 0; b < K; ++b) {
    T s = T(0);
#pragma unroll
    for (int f = 0; f <= 2 * K; ++f) s += tb.prol[f * (K + 1) + b] * v[2 * K + f];
    if (b == 0) {
      // left cell; its last child node 2k is the shared vertex counted above
#pragma unroll
      for (int f = 0; f < 2 * K; ++f) s += tb.prol[f * (K + 1) + K] * v[f];
    }
    out[b] = s;
  }
}

// ---------------------------------------------------------------------------
// 2D prolongation: fine interior += P coarse for a tile of C x C coarse cells
// (rows c_sy / f_sy apart).  Coarse boundary entries read as zero (MASK) or as
// they are.
template <int K, typename T, bool MASK>
__global__ void __launch_bounds__(XYTile<K>::NT)
    prolong2d_kernel(T *__restrict__ fine, const T *__restrict__ coarse, int N1c, int N1f, int64_t c_sy, int64_t f_sy)
{
  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  constexpr int C = ProlTile<K, T>::C, NT = XYTile<K>::NT;
  constexpr int WI = C * K + 1;  // coarse inputs per direction
  constexpr int WO = 2 * K * C;  // fine outputs per direction
  __shared__ T sIn[WI * WI];
  __shared__ T sX[WI * WO];
  const int cx0 = blockIdx.x * C, cy0 = blockIdx.y * C;
  // The current fine values are loaded first, so that their latency overlaps
  // the coarse tile's load and the x stage: into registers where a thread has
  // at most one y-stage task (FP64 tiles), else by asynchronous copies into
  // shared memory, issued right after the coarse tile's (the registers of two
  // tasks cost more than the overlap gained).
  constexpr bool PREFETCH = WO * C <= NT;
  __shared__ T sCur[PREFETCH ? 1 : WO * WO];
  T cur[2 * K];
  if constexpr (PREFETCH) {
    const int t = threadIdx.x;
    const int xx = t % WO, c = t / WO;
    const int gx = 2 * K * cx0 + xx;
#pragma unroll
    for (int f = 0; f < 2 * K; ++f) {
      const int gy = 2 * K * (cy0 + c) + f;
      const bool interior = t < WO * C && gx > 0 && gx < N1f - 1 && gy > 0 && gy < N1f - 1;
      cur[f] = interior ? fine[gx + gy * f_sy] : T(0);
    }
  }
  {
    const uint32_t s_in = smem_u32(sIn);
    for (int e = threadIdx.x; e < WI * WI; e += NT) {
      const int lx = e % WI, ly = e / WI;
      const int gx = cx0 * K + lx, gy = cy0 * K + ly;
      const bool bnd = gx == 0 || gx == N1c - 1 || gy == 0 || gy == N1c - 1;
      const bool ok = gx < N1c && gy < N1c && !(MASK && bnd);
      cp_async_zfill_s<sizeof(T)>(s_in + static_cast<uint32_t>(sizeof(T) * e), ok ? coarse + gx + gy * c_sy : coarse,
                                  ok ? static_cast<uint32_t>(sizeof(T)) : 0u);
    }
    cp_async_commit();
  }
  if constexpr (!PREFETCH) {
    const uint32_t s_cur = smem_u32(sCur);
    for (int e = threadIdx.x; e < WO * WO; e += NT) {
      const int xx = e % WO, yy = e / WO;
      const int gx = 2 * K * cx0 + xx, gy = 2 * K * cy0 + yy;
      const bool ok = gx < N1f && gy < N1f;
      cp_async_zfill_s<sizeof(T)>(s_cur + static_cast<uint32_t>(sizeof(T) * e), ok ? fine + gx + gy * f_sy : fine,
                                  ok ? static_cast<uint32_t>(sizeof(T)) : 0u);
    }
    cp_async_commit();
    cp_async_wait_1();  // the coarse tile has landed; the fine one may be in flight
  } else {
    cp_async_wait_all();
  }
  __syncthreads();
  for (int t = threadIdx.x; t < WI * C; t += NT) {
    const int c = t % C, y = t / C;
    T v[K + 1], o[2 * K];
#pragma unroll
    for (int b = 0; b <= K; ++b) v[b] = sIn[y * WI + c * K + b];
    prol_cell<K, T>(v, o);
#pragma unroll
    for (int f = 0; f < 2 * K; ++f) sX[y * WO + c * 2 * K + f] = o[f];
  }
  if constexpr (!PREFETCH) cp_async_wait_all();  // this thread's share of the fine tile
  __syncthreads();
  for (int t = threadIdx.x; t < WO * C; t += NT) {
    const int xx = t % WO, c = t / WO;
    T v[K + 1], o[2 * K];
#pragma unroll
    for (int b = 0; b <= K; ++b) v[b] = sX[(c * K + b) * WO + xx];
    prol_cell<K, T>(v, o);
    const int gx = 2 * K * cx0 + xx;
    if (gx == 0 || gx >= N1f - 1) continue;
#pragma unroll
    for (int f = 0; f < 2 * K; ++f) {
      const int gy = 2 * K * (cy0 + c) + f;
      if (gy == 0 || gy >= N1f - 1) continue;
      fine[gx + gy * f_sy] = (PREFETCH ? cur[f] : sCur[(2 * K * c + f) * WO + xx]) + o[f];
    }
  }
}

// xy pass, restriction: fine plane -> coarse plane.  Fine boundary entries
// are read as zero (weight 0 on Dirichlet DoFs).  zero_plane != 0 writes
// zeros instead (fine z-boundary planes).  zero (may be null, SetInterior): a
// vector of the coarse layout whose interior is zeroed with the same stores.
template <int K, typename T, XYOut OUT>
__global__ void __launch_bounds__(XYTile<K>::NT)
    restrict_xy_kernel(T *__restrict__ out, const T *__restrict__ in, int N1c, int N1f,
                       int64_t in_sy, int64_t in_plane, int64_t out_sy, int64_t out_plane,
                       int plane0, int n_planes_total, T *__restrict__ zero)
{
  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  constexpr int C = XYTile<K>::C, NT = XYTile<K>::NT;
  constexpr int WI = 2 * K * (C + 1) + 1;  // fine inputs per direction
  constexpr int WO = C * K;                // coarse outputs per direction
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T *sIn = reinterpret_cast<T *>(smem_raw);
  T *sX = sIn + WI * WI;
  const int plane = plane0 + blockIdx.z;
  const bool zero_plane = n_planes_total > 1 && (plane == 0 || plane == n_planes_total - 1);
  const T *inp = in + plane * in_plane;
  T *outp = out + plane * out_plane;
  const int cx0 = blockIdx.x * C, cy0 = blockIdx.y * C;
  const int fx0 = 2 * K * (cx0 - 1), fy0 = 2 * K * (cy0 - 1);
  // the fine tile (with its halo) by asynchronous copies, all in flight at
  // once; a loop of plain loads waited on each (measured at 3D 64^3, us per
  // restriction, plain / asynchronous: Q4 FP32 69.9 / 56.9, Q4 FP64 112.8 /
  // 92.3, Q3 FP64 37.7 / 33.1; Q7 32^3 FP64 101.5 / 65.9, FP32 51.3 / 56.0);
  // entries outside the interior are zero-filled
  const uint32_t s_in = smem_u32(sIn);
  for (int e = threadIdx.x; e < WI * WI; e += NT) {
    const int lx = e % WI, ly = e / WI;
    const int gx = fx0 + lx, gy = fy0 + ly;
    const bool ok = !zero_plane && gx > 0 && gx < N1f - 1 && gy > 0 && gy < N1f - 1;
    cp_async_zfill_s<sizeof(T)>(s_in + static_cast<uint32_t>(sizeof(T) * e), ok ? inp + gx + gy * in_sy : inp,
                                ok ? static_cast<uint32_t>(sizeof(T)) : 0u);
  }
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  for (int t = threadIdx.x; t < WI * C; t += NT) {
    const int c = t % C, y = t / C;
    T v[4 * K + 1], o[K];
#pragma unroll
    for (int j = 0; j <= 4 * K; ++j) v[j] = sIn[y * WI + c * 2 * K + j];
    restr_cell<K, T>(v, o);
#pragma unroll
    for (int b = 0; b < K; ++b) sX[y * WO + c * K + b] = o[b];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < WO * C; t += NT) {
    const int xx = t % WO, c = t / WO;
    T v[4 * K + 1], o[K];
#pragma unroll
    for (int j = 0; j <= 4 * K; ++j) v[j] = sX[(c * 2 * K + j) * WO + xx];
    restr_cell<K, T>(v, o);
    const int gx = K * cx0 + xx;
    if (gx >= N1c) continue;
#pragma unroll
    for (int b = 0; b < K; ++b) {
      const int gy = K * (cy0 + c) + b;
      if (gy >= N1c) continue;
      const int64_t gi = gx + gy * out_sy;
      const bool interior = gx > 0 && gx < N1c - 1 && gy > 0 && gy < N1c - 1;
      if constexpr (OUT == XYOut::AddInterior) {
        if (interior) outp[gi] += o[b];
      } else if constexpr (OUT == XYOut::SetInterior) {
        if (interior) {
          outp[gi] = o[b];
          if (zero) zero[gi] = T(0);
        }
      } else {
        outp[gi] = o[b];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// 3D prolongation in one pass: fine interior += P coarse for the fine nodes of a
// tile of TX x TY coarse cells in one cell layer.  The tile's coarse box is
// contracted in z, x and y through shared memory (the order of the passes over
// whole levels that it replaces, so the same rounding), while the current fine
// values of the thread's (z, x) columns are already on their way.  Coarse
// boundary entries read as zero (MASK) or as they are (the FMG prolongation of
// the solution).
//
// What bounds it: instruction issue (74 % busy at Q4 64^3 FP32, where DRAM is 25 %
// busy) in three short stages; the coarse box is
// read about 1.5 times (L2), the intermediate fine-z level (a quarter of the
// fine one, written and read) is gone, and so is one launch.  Measured, us per
// prolongate-and-add, two passes / now: Q4 64^3 FP64 82 / 72, FP32 53 / 40; Q7 32^3
// FP64 129 / 39, FP32 94 / 27; Q5 32^3 FP64 45 / 17; Q2 96^3 FP64 41 / 21; Q4 8^3
// 18 / 14.
template <int K, typename T>
struct Prol3 {
  static constexpr int TX = K == 1 ? 16 : K == 2 ? 8 : K == 3 ? 5 : K == 4 ? 4 : K == 5 ? 3 : 2;
  static constexpr int TY = K == 1 ? 8 : K == 2 ? 4 : K <= 4 ? 2 : 1;
  static constexpr int NT = 256;
  static constexpr int CX = TX * K + 1, CY = TY * K + 1, F = 2 * K, WX = F * TX;
  static constexpr int CB = (K + 1) * CY * CX, ZB = F * CY * CX, XB = F * CY * WX;
  static constexpr int YTASKS = F * TY * WX, YPT = (YTASKS + NT - 1) / NT;
  // the x-contracted lines take the place of the coarse box
  static constexpr int R0 = CB > XB ? CB : XB;
  static constexpr size_t BYTES = sizeof(T) * (R0 + ZB);
};

template <int K, typename T, bool MASK>
__global__ void __launch_bounds__(Prol3<K, T>::NT)
    prolong3d_kernel(T *__restrict__ fine, const T *__restrict__ coarse, int N1c, int N1f, int64_t c_sy, int64_t c_sz,
                     int64_t f_sy, int64_t f_sz)
{
  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  using S = Prol3<K, T>;
  constexpr int NT = S::NT, F = S::F, CX = S::CX, CY = S::CY, WX = S::WX;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T *sC = reinterpret_cast<T *>(smem_raw), *sX = sC, *sZ = sC + S::R0;
  const int gx0 = blockIdx.x * S::TX * K, gy0 = blockIdx.y * S::TY * K, gz0 = blockIdx.z * K;
  const uint32_t s_c = smem_u32(sC);
  for (int e = threadIdx.x; e < S::CB; e += NT) {
    const int r = e / CX, lx = e - r * CX, lz = r / CY, ly = r - lz * CY;
    const int gx = gx0 + lx, gy = gy0 + ly, gz = gz0 + lz;
    const bool in = gx < N1c && gy < N1c &&
                    (!MASK || (gx > 0 && gx < N1c - 1 && gy > 0 && gy < N1c - 1 && gz > 0 && gz < N1c - 1));
    cp_async_zfill_s<sizeof(T)>(s_c + static_cast<uint32_t>(sizeof(T) * e),
                                in ? coarse + gx + gy * c_sy + gz * c_sz : coarse,
                                in ? static_cast<uint32_t>(sizeof(T)) : 0u);
  }
  cp_async_commit();
  // y task: fine plane, coarse cell in y, fine column; its 2k current values
  T cur[S::YPT][F];
#pragma unroll
  for (int u = 0; u < S::YPT; ++u) {
    const int t = threadIdx.x + u * NT, r = t / WX, xx = t - r * WX, pz = r / S::TY, c = r - pz * S::TY;
    const int gx = 2 * gx0 + xx, gz = 2 * gz0 + pz, gy1 = 2 * gy0 + c * F;
    const bool col = t < S::YTASKS && gx > 0 && gx < N1f - 1 && gz > 0 && gz < N1f - 1;
    const T *q = fine + gx + gz * f_sz + gy1 * f_sy;
#pragma unroll
    for (int f = 0; f < F; ++f) {
      const int gy = gy1 + f;
      cur[u][f] = col && gy > 0 && gy < N1f - 1 ? q[f * f_sy] : T(0);
    }
  }
  cp_async_wait_all();
  __syncthreads();
  for (int t = threadIdx.x; t < CX * CY; t += NT) {
    T v[K + 1], o[F];
#pragma unroll
    for (int b = 0; b <= K; ++b) v[b] = sC[b * CX * CY + t];
    prol_cell<K, T>(v, o);
#pragma unroll
    for (int f = 0; f < F; ++f) sZ[f * CX * CY + t] = o[f];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < F * CY * S::TX; t += NT) {
    const int r = t / S::TX, c = t - r * S::TX;  // r: (fine plane, coarse row)
    T v[K + 1], o[F];
#pragma unroll
    for (int b = 0; b <= K; ++b) v[b] = sZ[r * CX + c * K + b];
    prol_cell<K, T>(v, o);
#pragma unroll
    for (int f = 0; f < F; ++f) sX[r * WX + c * F + f] = o[f];
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < S::YPT; ++u) {
    const int t = threadIdx.x + u * NT, r = t / WX, xx = t - r * WX, pz = r / S::TY, c = r - pz * S::TY;
    const int gx = 2 * gx0 + xx, gz = 2 * gz0 + pz, gy1 = 2 * gy0 + c * F;
    if (t < S::YTASKS && gx > 0 && gx < N1f - 1 && gz > 0 && gz < N1f - 1) {
      T v[K + 1], o[F];
#pragma unroll
      for (int b = 0; b <= K; ++b) v[b] = sX[(pz * CY + c * K + b) * WX + xx];
      prol_cell<K, T>(v, o);
      T *q = fine + gx + gz * f_sz + gy1 * f_sy;
#pragma unroll
      for (int f = 0; f < F; ++f) {
        const int gy = gy1 + f;
        if (gy > 0 && gy < N1f - 1) q[f * f_sy] = cur[u][f] + o[f];
      }
    }
  }
}

// z pass, restriction: tmp (N1f planes of P = N1c^2 entries) -> coarse.  zero
// (may be null): a vector of the same layout whose interior is zeroed with it
// (the V-cycle's next solution vector, without a fill of its own).
template <int K, typename T, bool ADD>
__global__ void restrict_z_kernel(T *__restrict__ coarse, const T *__restrict__ tmp, int N1c,
                                  int N1f, int64_t c_sy, int64_t c_sz, T *__restrict__ zero)
{
  griddep_wait();  // programmatic launch: the previous kernel's writes are visible
  const int64_t P = static_cast<int64_t>(N1c) * N1c;
  const int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int c = blockIdx.y;  // coarse cell along z: outputs c*k + b, b < k
  if (idx >= P) return;
  const int gy = static_cast<int>(idx) / N1c, gx = static_cast<int>(idx) - gy * N1c;  // idx < N1c^2 < 2^31
  if (gx == 0 || gx == N1c - 1 || gy == 0 || gy == N1c - 1) return;
  T v[4 * K + 1], o[K];
#pragma unroll
  for (int j = 0; j <= 4 * K; ++j) {
    const int fz = 2 * K * (c - 1) + j;
    v[j] = (fz <= 0 || fz >= N1f - 1) ? T(0) : __ldg(&tmp[fz * P + idx]);
  }
  restr_cell<K, T>(v, o);
#pragma unroll
  for (int b = 0; b < K; ++b) {
    const int gz = c * K + b;
    if (gz == 0 || gz >= N1c - 1) continue;
    const int64_t at = gz * c_sz + gy * c_sy + gx;
    if constexpr (ADD) {
      coarse[at] += o[b];
    } else {
      coarse[at] = o[b];
      if (zero) zero[at] = T(0);
    }
  }
}

}  // namespace tps
