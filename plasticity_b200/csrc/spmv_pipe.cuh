// spmv_pipe.cuh -- block-CSR SpMV with the matrix streamed through shared memory.
//
// What bounds it: the matrix is read once (HBM, or L2 when it fits).  Read straight
// into registers, a lane's 36-byte block is nine loads whose 32 addresses lie 36
// bytes apart, each of them touching every 128-byte line of the warp's kilobyte, and
// the gathered vector entries cost another line per neighbour: the kernel then runs
// at the L1's rate of lines, 4.6 TB/s from HBM and no faster from L2 (3.65 TB/s at
// 40^3).  Here every warp copies its tile of rows (contiguous in the value, column
// and row-pointer arrays) with cp.async.bulk into shared memory of its own, so the
// bytes in flight cost no registers and no warp waits for another one.
//
// 3 x 3 blocks: eight rows per tile, four lanes per row.  A lane takes every fourth
// block of its row; the lanes of a warp read shared memory at the rows' stride (27
// blocks = 243 words, odd: few bank conflicts), and in a node-ordered mesh the rows'
// k-th neighbours are consecutive nodes, so the gathers of x fall into a few lines.
// Each component has four partial sums of two blocks each, added as a tree: the register
// kernel's two blocks per lane and four shuffles in the same order, so that a product is
// the same number whichever kernel makes it (seven sums of one block took the same time).
// 6 x 6 blocks: half a warp per row, lane k takes blocks k and k + 16, 16-byte reads
// at a stride of 36 words (no conflicts).
#pragma once
#include <cstdint>

#include "bulk_copy.cuh"
#include "linalg.cuh"

namespace pfem {

// What an SpMV works on, and what it does with a row's sum v = (A x), by mode:
//   0: y = v   1: y = b - v   2: y -= Dinv v, xo += x   3: xo = c2 x + c1 (y - Dinv v)
//   4: as 3, added to xo      5: y = Dinv (b - v), xo = y / th      6: y = Dinv v, x scaled
//   7: z = b - v, y = Dinv z, xo = y / th
// 2 is a Chebyshev step on x = d; 3 and 4 the degree-2 smoother in one pass (x = d0,
// y = r0); 5 its start on a residual, 7 the same with the residual kept; 6 a step of
// the power iteration, on x / |x|.  1 / th, c1 and c2 are the level's scalars co.  Vectors that
// earlier kernels of a programmatic launch chain write are not __restrict__ const: such
// a load could be served by the read-only path while they are still being written.
template <typename T>
struct SpmvVec {
  const T* x = nullptr;
  T* y = nullptr;
  const T* b = nullptr;
  const T* dinv = nullptr;
  T* xo = nullptr;
  const T* co = nullptr;
  T* z = nullptr;
  T* part = nullptr;  // partials of x.y (mode 0) or b.xo (mode 4), one per CTA (FP64)
};

// LANES lanes per row and ROWS rows per tile; a CTA is one warp with one tile in shared
// memory (8 rows of 27 blocks: 8 KB float, 16 KB double; 4 rows of 6 x 6: 15 KB), so
// that 13 to 24 of them share an SM and the copies of some overlap the arithmetic of
// the others.  Measured at 64^3, FP32, per pass over 281 MB: 42.6 us (6.6 TB/s; the
// register kernel 59.8); one warp with two stages 49.2, two warps with two stages
// 50.5, a producer lane feeding eight half-warp-per-row warps through four stages
// 51.4.  FP64 79.0 us (103.1).  Two lanes per row: the same at 64^3, 14 % slower at
// 40^3 (16.5 against 14.4 us).  The cycle in its graph: 431 -> 342 us at 64^3.
template <typename T, int BS>
struct PipeShape {
  static constexpr int LANES = BS == 3 ? 4 : 16;
  static constexpr int ROWS = BS == 3 ? 32 / LANES : 4;
  static_assert(ROWS % 4 == 0, "a tile's row pointers start on 16 bytes");
};

// Byte layout of a tile: values, column ids, row pointers; each region starts on 16
// bytes and has room for the slack of copies whose ends are rounded out to 16 bytes.
struct PipeLay {
  int cols, rows, bytes;
};
template <typename T, int BS>
__host__ __device__ constexpr PipeLay pipe_lay(int max_row, bool c16) {
  constexpr int R = PipeShape<T, BS>::ROWS;
  PipeLay l = {};
  l.cols = (R * max_row * BS * BS * (int)sizeof(T) + 32 + 15) & ~15;
  l.rows = l.cols + ((R * max_row * (c16 ? 2 : 4) + 32 + 15) & ~15);
  l.bytes = l.rows + R * 4 + 16;
  return l;
}
constexpr int kPipeHead = 16;  // the barrier, in front of the tile
constexpr int kPipeMaxRow = 32;  // blocks of a row that two passes of 16 lanes take
template <typename T, int BS>
constexpr int pipe_smem_bytes(int max_row, bool c16) {
  return kPipeHead + pipe_lay<T, BS>(max_row, c16).bytes;
}
// Without cudaFuncAttributeMaxDynamicSharedMemorySize, which is the process's and not the
// launch's: a context that set it for its rows would take it from another one's launch.
static_assert(pipe_smem_bytes<double, 6>(kPipeMaxRow, false) <= 48 * 1024 &&
                  pipe_smem_bytes<double, 3>(kPipeMaxRow, false) <= 48 * 1024, "a tile needs no attribute");

// Start the copies of tile t (rows t R .., blocks s0 .. s1); one lane.
template <typename T, int BS, bool C16>
__device__ __forceinline__ void pipe_issue(unsigned char* stage, const PipeLay& lay, uint32_t bar, int t, int nbrow, int s0,
                                           int s1, const int* rowptr, const int* col, const int16_t* col16, const T* val) {
  constexpr int R = PipeShape<T, BS>::ROWS, VB = BS * BS * (int)sizeof(T), CB = C16 ? 2 : 4;
  const int r0 = t * R, rows = min(R, nbrow - r0);
  const long long va = ((long long)s0 * VB) & ~15ll, ca = ((long long)s0 * CB) & ~15ll;
  const uint32_t vb = (uint32_t)((((long long)s1 * VB + 15) & ~15ll) - va);
  const uint32_t cb = (uint32_t)((((long long)s1 * CB + 15) & ~15ll) - ca);
  const uint32_t rb = (uint32_t)(((rows + 1) * 4 + 15) & ~15);
  const uint32_t dst = bulk_smem(stage);
  bulk_expect(bar, vb + cb + rb);
  bulk_copy(dst + lay.rows, rowptr + r0, rb, bar);
  if (cb) bulk_copy(dst + lay.cols, (C16 ? (const char*)col16 : (const char*)col) + ca, cb, bar);
  if (vb) bulk_copy_first(dst, (const char*)val + va, vb, bar);
}

template <typename T, int BS, int MODE, bool C16, bool DOT>
__global__ void __launch_bounds__(32)
bsr_spmv_pipe_kernel(int nbrow, int ntiles, int max_row, const int* __restrict__ rowptr, const int* __restrict__ col,
                     const int16_t* __restrict__ col16, const T* __restrict__ val, SpmvVec<T> a, int* err) {
  using SH = PipeShape<T, BS>;
  constexpr int R = SH::ROWS, BB = BS * BS;
  extern __shared__ __align__(128) unsigned char psm[];
  const PipeLay lay = pipe_lay<T, BS>(max_row, C16);
  const int lane = threadIdx.x;
  pdl_go();
  unsigned char* const st = psm + kPipeHead;
  const uint32_t bar = bulk_smem(psm);
  int n0 = 0, n1 = 0;  // block range of the next tile to copy (lane 0)
  if (lane == 0) {
    bulk_bar_init(bar, 1);
    bulk_init_fence();
    const int t = blockIdx.x, tn = t + gridDim.x;
    const int s0 = rowptr[t * R], s1 = rowptr[min(t * R + R, nbrow)];
    if (tn < ntiles) {
      n0 = rowptr[tn * R];
      n1 = rowptr[min(tn * R + R, nbrow)];
    }
    pipe_issue<T, BS, C16>(st, lay, bar, t, nbrow, s0, s1, rowptr, col, col16, val);
  }
  __syncwarp();
  uint32_t phase = 0;
  const T c1 = MODE == 3 || MODE == 4 ? a.co[CO_C1] : MODE == 5 || MODE == 7 ? a.co[CO_ITH] : T(0);
  const T c2 = MODE == 3 || MODE == 4 ? a.co[CO_C2] : MODE == 6 ? a.co[CO_INV] : T(0);
  double dot = 0.0;
  pdl_wait();  // the first tile is on its way
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x, phase ^= 1u) {
    // a lane's row(s) of the tile and the epilogue's operands, in flight while the tile arrives
    if constexpr (BS == 3) {
      constexpr int LN = SH::LANES;  // par: which of the row's lanes this one is
      const int rl = lane & (R - 1), par = lane / R;
      const int row = t * R + rl;
      const bool ok = row < nbrow, own = ok && par == 0;
      const long long at = (long long)row * 3;
      T bi[3], yi[3], xi[3], oi[3], D[9];
      if (own) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          if (MODE == 1 || MODE == 5 || MODE == 7 || (DOT && MODE == 4)) bi[i] = a.b[at + i];
          if (MODE == 2 || MODE == 3 || MODE == 4) yi[i] = a.y[at + i];
          if (MODE == 2 || MODE == 3 || MODE == 4 || (DOT && MODE == 0)) xi[i] = a.x[at + i];
          if (MODE == 2 || MODE == 4) oi[i] = a.xo[at + i];
        }
        if (MODE >= 2) {
#pragma unroll
          for (int i = 0; i < 9; ++i) D[i] = a.dinv[(long long)row * 9 + i];
        }
      }
      if (!__all_sync(0xffffffffu, bulk_bar_wait(bar, phase, err))) return;
      const int* rp = reinterpret_cast<const int*>(st + lay.rows);
      const int s0 = rp[0];
      const int b0 = ok ? rp[rl] - s0 : 0, len = ok ? rp[rl + 1] - s0 - b0 : 0;
      const T* vs = reinterpret_cast<const T*>(st + (((long long)s0 * (9 * (int)sizeof(T))) & 15)) + (long long)b0 * 9;
      const int* cs = reinterpret_cast<const int*>(st + lay.cols + (((long long)s0 * 4) & 15)) + b0;
      const int16_t* cs16 = reinterpret_cast<const int16_t*>(st + lay.cols + (((long long)s0 * 2) & 15)) + b0;
      // four partial sums per component, as the register kernel's lanes par + 4 m have them:
      // block q = par + 4 m, then block q + 16
      constexpr int NP = 16 / LN;
      T acc[NP][3];
#pragma unroll
      for (int m = 0; m < NP; ++m) acc[m][0] = acc[m][1] = acc[m][2] = T(0);
      T xv[2 * NP][3];
#pragma unroll
      for (int m = 0; m < 2 * NP; ++m) {
        const int q = par + LN * m;
        const bool in = q < len;
        const long long c = in ? (C16 ? row + (int)cs16[q] : cs[q]) : 0;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          xv[m][j] = in ? a.x[c * 3 + j] : T(0);
          if (MODE == 6) xv[m][j] *= c2;
        }
      }
#pragma unroll
      for (int m = 0; m < 2 * NP; ++m) {
        const int q = par + LN * m;
        if (q < len) {
          const T* B = vs + q * 9;
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) acc[m % NP][i] += B[i * 3 + j] * xv[m][j];
        }
      }
      __syncwarp();
      if (lane == 0 && t + (int)gridDim.x < ntiles) {
        const int tn = t + gridDim.x, tf = tn + gridDim.x;
        pipe_issue<T, BS, C16>(st, lay, bar, tn, nbrow, n0, n1, rowptr, col, col16, val);
        n0 = tf < ntiles ? rowptr[tf * R] : 0;
        n1 = tf < ntiles ? rowptr[min(tf * R + R, nbrow)] : 0;
      }
      T v[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        v[i] = (acc[0][i] + acc[2][i]) + (acc[1][i] + acc[3][i]);
#pragma unroll
        for (int o = 16; o >= R; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
      }
      if (own) {
        if (MODE == 0) {
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            a.y[at + i] = v[i];
            if (DOT) dot += (double)xi[i] * (double)v[i];
          }
        } else if (MODE == 1) {
#pragma unroll
          for (int i = 0; i < 3; ++i) a.y[at + i] = bi[i] - v[i];
        } else {
          if (MODE == 5 || MODE == 7) {
#pragma unroll
            for (int i = 0; i < 3; ++i) v[i] = bi[i] - v[i];
          }
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            T w = T(0);
#pragma unroll
            for (int j = 0; j < 3; ++j) w += D[i * 3 + j] * v[j];
            if (MODE == 2) {
              a.y[at + i] = yi[i] - w;
              a.xo[at + i] = oi[i] + xi[i];
            } else if (MODE == 5 || MODE == 7) {
              if (MODE == 7) a.z[at + i] = v[i];
              a.y[at + i] = w;
              a.xo[at + i] = c1 * w;
            } else if (MODE == 6) {
              a.y[at + i] = w;
            } else {
              T upd = c2 * xi[i] + c1 * (yi[i] - w);
              if (MODE == 4) upd = oi[i] + upd;
              a.xo[at + i] = upd;
              if (DOT) dot += (double)bi[i] * (double)upd;
            }
          }
        }
      }
    } else {
      const int hl = lane & 15;
      bool waited = false;
#pragma unroll 1
      for (int r2 = 0; r2 < R / 2; ++r2) {
        const int rl = 2 * r2 + (lane >> 4);
        const int row = t * R + rl;
        const bool ok = row < nbrow, own = ok && hl < BS;
        const long long at = (long long)row * BS + hl;
        T bi = T(0), yi = T(0), xi = T(0), oi = T(0), D[BS];
#pragma unroll
        for (int j = 0; j < BS; ++j) D[j] = T(0);
        if (own) {
          if (MODE == 1 || MODE == 5 || MODE == 7) bi = a.b[at];
          if (MODE == 2 || MODE == 3 || MODE == 4) { yi = a.y[at]; xi = a.x[at]; }
          if (MODE == 2 || MODE == 4) oi = a.xo[at];
          if (MODE >= 2) {
#pragma unroll
            for (int j = 0; j < BS; ++j) D[j] = a.dinv[(long long)row * BB + hl * BS + j];
          }
        }
        if (!waited) {
          waited = __all_sync(0xffffffffu, bulk_bar_wait(bar, phase, err));
          if (!waited) break;
        }
        const int* rp = reinterpret_cast<const int*>(st + lay.rows);
        const int s0 = rp[0];
        const int b0 = ok ? rp[rl] - s0 : 0, b1 = ok ? rp[rl + 1] - s0 : 0;
        const T* vs = reinterpret_cast<const T*>(st);
        const int* cs = reinterpret_cast<const int*>(st + lay.cols + (((long long)s0 * 4) & 15));
        T xv[2][BS];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int q = b0 + hl + 16 * h;
          const bool in = q < b1;
          const long long c = in ? cs[q] : 0;
#pragma unroll
          for (int j = 0; j < BS; ++j) {
            xv[h][j] = in ? a.x[c * BS + j] : T(0);
            if (MODE == 6) xv[h][j] *= c2;
          }
        }
        T acc[BS];
#pragma unroll
        for (int i = 0; i < BS; ++i) acc[i] = T(0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int q = b0 + hl + 16 * h;
          if (q < b1) {
            using V = typename std::conditional<std::is_same<T, float>::value, float4, double2>::type;
            constexpr int PER = 16 / (int)sizeof(T);
            const V* B4 = reinterpret_cast<const V*>(vs + (long long)q * BB);
            T bv[BB];
#pragma unroll
            for (int m = 0; m < BB / PER; ++m) {
              const V u = B4[m];
              const T* ut = reinterpret_cast<const T*>(&u);
#pragma unroll
              for (int j = 0; j < PER; ++j) bv[m * PER + j] = ut[j];
            }
#pragma unroll
            for (int i = 0; i < BS; ++i)
#pragma unroll
              for (int j = 0; j < BS; ++j) acc[i] += bv[i * BS + j] * xv[h][j];
          }
        }
#pragma unroll
        for (int i = 0; i < BS; ++i) {
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
        }
        T v = acc[0];
#pragma unroll
        for (int i = 1; i < BS; ++i)
          if (hl == i) v = acc[i];
        T w = T(0);
        if (MODE >= 2) {
          if (MODE == 5 || MODE == 7) v = bi - v;
#pragma unroll
          for (int j = 0; j < BS; ++j) w += D[j] * __shfl_sync(0xffffffffu, v, (lane & 16) + j);
        }
        if (!own) continue;
        if (MODE == 0) {
          a.y[at] = v;
        } else if (MODE == 1) {
          a.y[at] = bi - v;
        } else if (MODE == 2) {
          a.y[at] = yi - w;
          a.xo[at] = oi + xi;
        } else if (MODE == 5 || MODE == 7) {
          if (MODE == 7) a.z[at] = v;
          a.y[at] = w;
          a.xo[at] = c1 * w;
        } else if (MODE == 6) {
          a.y[at] = w;
        } else {
          const T upd = c2 * xi + c1 * (yi - w);
          a.xo[at] = MODE == 3 ? upd : oi + upd;
        }
      }
      if (!waited) return;
      __syncwarp();
      if (lane == 0 && t + (int)gridDim.x < ntiles) {
        const int tn = t + gridDim.x, tf = tn + gridDim.x;
        pipe_issue<T, BS, C16>(st, lay, bar, tn, nbrow, n0, n1, rowptr, col, col16, val);
        n0 = tf < ntiles ? rowptr[tf * R] : 0;
        n1 = tf < ntiles ? rowptr[min(tf * R + R, nbrow)] : 0;
      }
    }
  }
  if constexpr (DOT) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (lane == 0) a.part[blockIdx.x] = dot;
  }
}

}  // namespace pfem
