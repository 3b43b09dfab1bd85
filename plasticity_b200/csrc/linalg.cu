// linalg.cu -- block-CSR SpMV, smoother / Krylov vector kernels, reductions,
// Dirichlet imposition and AMG transfer kernels.  All are HBM-bound; each is
// written so that one pass over the matrix does all the work the caller needs
// from that pass (SpMV + residual, SpMV + block-Jacobi Chebyshev update).
#include <cstdint>
#include <type_traits>

#include "linalg.cuh"
#include "spmv_pipe.cuh"

namespace pfem {

// ------------------------------------------------------------------ reductions
// Deterministic two-pass dot product: per-block partials, then one block.
constexpr int RED_THREADS = 256;
constexpr int RED_BLOCKS = 1184;  // 148 SMs x 8

template <typename T>
__device__ __forceinline__ T block_sum(T v, T* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  v = (threadIdx.x < (blockDim.x >> 5)) ? sh[threadIdx.x] : T(0);
  if (w == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  }
  return v;
}

// Partials of a.b (count returned): the first pass of dot, also inside a launch chain.
template <typename T>
__global__ void dot_partial_kernel(long long n, const T* a, const T* b, T* part) {
  __shared__ T sh[32];
  pdl_go();
  pdl_wait();
  T v = T(0);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    v += a[i] * b[i];
  v = block_sum(v, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = v;
}
template <typename T>
int dot_partials(long long n, const T* a, const T* b, T* part, const Queue& q) {
  const int blocks = (int)std::min<long long>(std::max<long long>((n + RED_THREADS - 1) / RED_THREADS, 1), RED_BLOCKS);
  launch(q, dot_partial_kernel<T>, blocks, RED_THREADS, 0, n, a, b, part);
  return blocks;
}

// ------------------------------------------------------------------ SpMV
// Half a warp per block row; lane k holds block rowptr[i]+k (+16, ...), loads
// the whole bs x bs block and the matching bs entries of x, and the half-warp
// reduces the bs partial sums by a fixed xor tree.  The modes are SpmvVec's.  DOT: the
// row's share of x.y (mode 0) or b.xo (mode 4) is summed per CTA into part.
template <typename T, int BS, int MODE, bool VEC = false, int LANES = 16, bool C16 = false, bool DOT = false>
__global__ void __launch_bounds__(128) bsr_spmv_kernel(int nbrow, const int* __restrict__ rowptr,
                                                       const int* __restrict__ col,
                                                       const int16_t* __restrict__ col16,
                                                       const T* __restrict__ val, SpmvVec<T> a) {
  // LANES lanes per block row: half a warp for 3 x 3 blocks (a level-0 row has at
  // most 27 blocks: two per lane), a warp for 6 x 6 blocks (one 144-byte block
  // per lane); values and column ids are read once, through the streaming
  // (evict-first) path so they do not push the gathered x out of the caches.  The
  // first block and the block inverse are in flight before the wait for the vectors.
  static_assert(LANES == 16 || LANES == 32, "half or whole warps per row");
  pdl_go();
  const int row = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) / LANES);
  const int lane = threadIdx.x & (LANES - 1);
  const bool ok = row < nbrow, own = ok && lane < BS;
  const long long at = (long long)row * BS + lane;
  const int s = ok ? rowptr[row] : 0, e = ok ? rowptr[row + 1] : 0;
  T bv[BS * BS], D[BS];
  int c = 0;
  auto block = [&](int k) {
    c = C16 ? row + (int)__ldcs(col16 + k) : __ldcs(col + k);
    const T* B = val + (long long)k * (BS * BS);
    if constexpr (VEC) {
      // 16-byte streaming loads (a 6 x 6 block is 144 / 288 bytes; the launcher
      // checks that val is 16-byte aligned, so every block is)
      using V = typename std::conditional<std::is_same<T, float>::value, float4, double2>::type;
      constexpr int PER = 16 / (int)sizeof(T), NV = BS * BS / PER;
      static_assert(BS * BS % PER == 0, "vector loads need whole 16-byte groups");
      const V* B4 = reinterpret_cast<const V*>(B);
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        const V v = __ldcs(B4 + q);
        const T* vt = reinterpret_cast<const T*>(&v);
#pragma unroll
        for (int j = 0; j < PER; ++j) bv[q * PER + j] = vt[j];
      }
    } else {
#pragma unroll
      for (int q = 0; q < BS * BS; ++q) bv[q] = __ldcs(B + q);
    }
  };
  int k = s + lane;
  if (k < e) block(k);
#pragma unroll
  for (int j = 0; j < BS; ++j) D[j] = (MODE >= 2 && own) ? a.dinv[(long long)row * (BS * BS) + lane * BS + j] : T(0);
  const T c1 = MODE == 3 || MODE == 4 ? a.co[CO_C1] : MODE == 5 || MODE == 7 ? a.co[CO_ITH] : T(0);
  const T c2 = MODE == 3 || MODE == 4 ? a.co[CO_C2] : MODE == 6 ? a.co[CO_INV] : T(0);
  pdl_wait();
  T bi = T(0), yi = T(0), xi = T(0), oi = T(0);
  if (own) {
    if (MODE == 1 || MODE == 5 || MODE == 7 || (DOT && MODE == 4)) bi = a.b[at];
    if (MODE == 2 || MODE == 3 || MODE == 4) yi = a.y[at];
    if (MODE == 2 || MODE == 3 || MODE == 4 || (DOT && MODE == 0)) xi = a.x[at];
    if (MODE == 2 || MODE == 4) oi = a.xo[at];
  }
  T acc[BS];
#pragma unroll
  for (int i = 0; i < BS; ++i) acc[i] = T(0);
  while (k < e) {
    T xv[BS];
#pragma unroll
    for (int j = 0; j < BS; ++j) {
      xv[j] = a.x[(long long)c * BS + j];
      if (MODE == 6) xv[j] *= c2;
    }
#pragma unroll
    for (int i = 0; i < BS; ++i)
#pragma unroll
      for (int j = 0; j < BS; ++j) acc[i] += bv[i * BS + j] * xv[j];
    k += LANES;
    if (k < e) block(k);
  }
#pragma unroll
  for (int i = 0; i < BS; ++i) {
    T v = acc[i];
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    acc[i] = v;
  }
  T v = acc[0];
#pragma unroll
  for (int i = 1; i < BS; ++i)
    if (lane == i) v = acc[i];
  T w = T(0);
  if (MODE == 5 || MODE == 7) {
    v = bi - v;
#pragma unroll
    for (int j = 0; j < BS; ++j) w += D[j] * __shfl_sync(0xffffffffu, v, (threadIdx.x & 31 & ~(LANES - 1)) + j);
  } else if (MODE >= 2) {
#pragma unroll
    for (int j = 0; j < BS; ++j) w += D[j] * acc[j];
  }
  double dot = 0.0;
  if (own) {
    if (MODE == 0) {
      a.y[at] = v;
      if (DOT) dot = (double)xi * (double)v;
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
      // degree-2 Chebyshev in one pass: r1 = r0 - Dinv A d0,
      // x2 = x0 + c2 d0 + c1 r1 (c2 = 1 + rn rho, c1 = 2 rn / delta)
      T upd = c2 * xi + c1 * (yi - w);
      if (MODE == 4) upd = oi + upd;
      a.xo[at] = upd;
      if (DOT) dot = (double)bi * (double)upd;
    }
  }
  if constexpr (DOT) {
    __shared__ double sh[32];
    dot = block_sum(dot, sh);
    if (threadIdx.x == 0) a.part[blockIdx.x] = dot;
  }
}

template <typename T, int BS, int MODE, bool C16, bool DOT>
static int pipe_launch_t(const BsrMat<T>& A, const SpmvVec<T>& a, const Queue& qu) {
  auto* kern = bsr_spmv_pipe_kernel<T, BS, MODE, C16, DOT>;
  const int sm = pipe_smem_bytes<T, BS>(A.max_row, C16);  // at most 38 KB: no limit to raise
  int dev = 0, sms = 148, per = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, 32, sm);
  constexpr int R = PipeShape<T, BS>::ROWS;
  const int tiles = (A.nbrow + R - 1) / R;
  const int grid = std::min(std::min(tiles, sms * std::max(per, 1)), kMaxPartials);
  launch(qu, kern, grid, 32, sm, A.nbrow, tiles, A.max_row, A.rowptr, A.col, A.col16, A.val, a, A.err);
  return grid;
}
// The streamed kernel takes a matrix whose rows have at most 32 blocks and whose
// arrays start on 16 bytes, from as many rows on as keep most warps of the chip busy:
// below, one row per half-warp (or warp) has less latency per launch.  The cycle,
// register / streamed: 20.6 / 22.6 us at 8^3 (729 rows), 26.4 / 26.7 at 16^3 (4,913),
// 54 / 51 at 24^3 (15,625), 117 / 100 at 40^3.  6 x 6 levels, with the finest level
// streamed: 152 / 146 us at 48^3 (4,913 rows of 6 x 6), 647 / 603 at 80^3 (19,683).
constexpr int kPipeRows3 = 8192, kPipeRows6 = 4096;
template <typename T>
static bool spmv_streams(const BsrMat<T>& A) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(A.val) | reinterpret_cast<uintptr_t>(A.rowptr) |
                       (A.bs == 3 && A.col16 ? reinterpret_cast<uintptr_t>(A.col16) : reinterpret_cast<uintptr_t>(A.col));
  return A.nbrow >= (A.bs == 3 ? kPipeRows3 : kPipeRows6) && A.max_row >= 1 && A.max_row <= kPipeMaxRow && A.err && !(at & 15);
}

// DOT (3 x 3 blocks): returns the number of partials, 0 when there would be too many.
template <typename T, int MODE, bool DOT = false>
static int spmv_launch(const BsrMat<T>& A, const SpmvVec<T>& a, const Queue& qu) {
  if (spmv_streams(A)) {
    if (A.bs == 3 && A.col16) return pipe_launch_t<T, 3, MODE, true, DOT>(A, a, qu);
    if (A.bs == 3) return pipe_launch_t<T, 3, MODE, false, DOT>(A, a, qu);
    if constexpr (!DOT) return pipe_launch_t<T, 6, MODE, false, false>(A, a, qu);
  }
  // 6 x 6 levels of fewer than kWarpRowsBelow rows fill too few warp slots with half
  // a warp per row: give each row a whole warp there (measured at 64^3: level 2,
  // 512 rows, 7.4 -> 6.5 us per pass; level 1, 10,648 rows, 14.3 -> 18.2 us)
  constexpr int kWarpRowsBelow = 4096;
  const bool wide = A.bs == 6 && A.nbrow < kWarpRowsBelow;
  // 128-thread blocks: the whole cycle inside a CUDA graph measured 422.1 us against
  // 425.0 us with 256 at 64^3 (1.3667 vs 1.3679 ms at 100^3)
  constexpr int kThreads = 128;
  const long long threads = (long long)A.nbrow * (wide ? 32 : 16);
  const int blocks = (int)((threads + kThreads - 1) / kThreads);
  const bool aligned = (reinterpret_cast<uintptr_t>(A.val) & 15) == 0;
  if constexpr (DOT) {
    if (blocks > kMaxPartials) return 0;
    if (A.col16) launch(qu, bsr_spmv_kernel<T, 3, MODE, false, 16, true, true>, blocks, kThreads, 0, A.nbrow, A.rowptr, A.col, A.col16, A.val, a);
    else launch(qu, bsr_spmv_kernel<T, 3, MODE, false, 16, false, true>, blocks, kThreads, 0, A.nbrow, A.rowptr, A.col, A.col16, A.val, a);
    return blocks;
  } else {
    auto* kern = A.bs == 3 ? (A.col16 ? bsr_spmv_kernel<T, 3, MODE, false, 16, true> : bsr_spmv_kernel<T, 3, MODE>)
                 : aligned ? (wide ? bsr_spmv_kernel<T, 6, MODE, true, 32> : bsr_spmv_kernel<T, 6, MODE, true>)
                           : bsr_spmv_kernel<T, 6, MODE>;
    launch(qu, kern, blocks, kThreads, 0, A.nbrow, A.rowptr, A.col, A.col16, A.val, a);
    return 0;
  }
}

// The dot products of a CG iteration.  FP64: inside the products that hold their operands.
// FP32: in passes of their own, in dot's order and type; the solution of a slender box
// differs by hundreds of roundings with another order.  A mixed CG iteration so / with the
// sums inside: 27.1 / 26.0 us at 8^3, 112 / 115 at 49 x 37 x 29, 373 / 367 at 64^3.
template <typename T>
constexpr bool kDotsInside = std::is_same<T, double>::value;
template <typename T>
int bsr_spmv(const BsrMat<T>& A, const T* x, T* y, Queue q, T* part) {
  SpmvVec<T> a;
  a.x = x; a.y = y; a.part = part;
  int np = 0;
  if constexpr (kDotsInside<T>) {
    if (part) np = spmv_launch<T, 0, true>(A, a, q);
  }
  if (np > 0) return np;
  spmv_launch<T, 0>(A, a, q);
  return part ? dot_partials<T>((long long)A.nbrow * A.bs, x, y, part, q) : 0;
}
template <typename T>
void bsr_residual(const BsrMat<T>& A, const T* x, const T* b, T* r, Queue q) {
  SpmvVec<T> a;
  a.x = x; a.y = r; a.b = b;
  spmv_launch<T, 1>(A, a, q);
}
template <typename T>
void bsr_cheb_step(const BsrMat<T>& A, const T* dinv, const T* d, T* r, T* x, cudaStream_t st) {
  SpmvVec<T> a;
  a.x = d; a.y = r; a.dinv = dinv; a.xo = x;
  spmv_launch<T, 2>(A, a, st);
}
template <typename T>
int bsr_cheb2(const BsrMat<T>& A, const T* dinv, const T* d0, const T* r0, T* x, bool zero, const T* co, Queue q,
              const T* b, T* part) {
  SpmvVec<T> a;
  a.x = d0; a.y = const_cast<T*>(r0); a.dinv = dinv; a.xo = x; a.co = co; a.b = b; a.part = part;
  if (zero) return spmv_launch<T, 3>(A, a, q);
  int np = 0;
  if constexpr (kDotsInside<T>) {
    if (part) np = spmv_launch<T, 4, true>(A, a, q);
  }
  if (np > 0) return np;
  spmv_launch<T, 4>(A, a, q);
  return part ? dot_partials<T>((long long)A.nbrow * A.bs, b, x, part, q) : 0;
}
template <typename T>
void bsr_residual_precond(const BsrMat<T>& A, const T* dinv, const T* x, const T* b, T* r, T* d, const T* co, Queue q) {
  SpmvVec<T> a;
  a.x = x; a.y = r; a.b = b; a.dinv = dinv; a.xo = d; a.co = co;
  spmv_launch<T, 5>(A, a, q);
}
template <typename T>
void bsr_residual_start(const BsrMat<T>& A, const T* dinv, const T* x, const T* b, T* res, T* r, T* d, const T* co,
                        Queue q) {
  SpmvVec<T> a;
  a.x = x; a.y = r; a.b = b; a.dinv = dinv; a.xo = d; a.co = co; a.z = res;
  spmv_launch<T, 7>(A, a, q);
}
template <typename T>
void bsr_power_step(const BsrMat<T>& A, const T* dinv, const T* x, T* y, const T* co, cudaStream_t st) {
  SpmvVec<T> a;
  a.x = x; a.y = y; a.dinv = dinv; a.co = co;
  spmv_launch<T, 6>(A, a, st);
}

// ------------------------------------------------------------------ block diagonal
// r = Dinv * v per block row (one thread per scalar row), d = *scale r.
template <typename T, int BS>
__global__ void blockdiag_apply_kernel(int nbrow, const T* __restrict__ dinv, const T* v, T* r,
                                       const T* __restrict__ scale, T* d) {
  pdl_go();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const bool in = i < (long long)nbrow * BS;
  const long long row = i / BS;
  const int li = (int)(i - row * BS);
  T D[BS];
#pragma unroll
  for (int j = 0; j < BS; ++j) D[j] = in ? dinv[row * (BS * BS) + li * BS + j] : T(0);
  const T s = *scale;
  pdl_wait();
  if (!in) return;
  const T* vv = v + row * BS;
  T t = T(0);
#pragma unroll
  for (int j = 0; j < BS; ++j) t += D[j] * vv[j];
  r[i] = t;
  d[i] = s * t;
}
template <typename T>
void blockdiag_apply(int nbrow, int bs, const T* dinv, const T* v, T* r, const T* scale, T* d, Queue q) {
  const long long n = (long long)nbrow * bs;
  launch(q, bs == 3 ? blockdiag_apply_kernel<T, 3> : blockdiag_apply_kernel<T, 6>, (int)((n + 255) / 256), 256, 0, nbrow,
         dinv, v, r, scale, d);
}

// Invert the diagonal blocks (Gauss-Jordan with partial pivoting in double).
// A singular block (a Dirichlet-free rigid aggregate, say) gets the inverse of
// its diagonal instead, with zero diagonal entries mapped to 1.
template <typename T, int BS>
__global__ void blockdiag_invert_kernel(int nbrow, const int* __restrict__ rowptr, const int* __restrict__ col,
                                        const T* __restrict__ val, T* __restrict__ dinv) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= nbrow) return;
  double a[BS][2 * BS];
  int kd = -1;
  for (int k = rowptr[row]; k < rowptr[row + 1]; ++k)
    if (col[k] == row) { kd = k; break; }
  for (int i = 0; i < BS; ++i)
    for (int j = 0; j < BS; ++j) {
      a[i][j] = kd >= 0 ? (double)val[(long long)kd * BS * BS + i * BS + j] : 0.0;
      a[i][BS + j] = (i == j) ? 1.0 : 0.0;
    }
  bool ok = true;
  double scl = 0.0;
  for (int i = 0; i < BS; ++i) scl = fmax(scl, fabs(a[i][i]));
  for (int c = 0; c < BS && ok; ++c) {
    int piv = c;
    double best = fabs(a[c][c]);
    for (int r = c + 1; r < BS; ++r)
      if (fabs(a[r][c]) > best) { best = fabs(a[r][c]); piv = r; }
    if (!(best > 1e-13 * scl) || !(best > 0.0)) { ok = false; break; }
    if (piv != c)
      for (int j = 0; j < 2 * BS; ++j) { double t = a[c][j]; a[c][j] = a[piv][j]; a[piv][j] = t; }
    const double ip = 1.0 / a[c][c];
    for (int j = 0; j < 2 * BS; ++j) a[c][j] *= ip;
    for (int r = 0; r < BS; ++r)
      if (r != c) {
        const double f = a[r][c];
        if (f != 0.0)
          for (int j = 0; j < 2 * BS; ++j) a[r][j] -= f * a[c][j];
      }
  }
  T* D = dinv + (long long)row * BS * BS;
  if (ok) {
    for (int i = 0; i < BS; ++i)
      for (int j = 0; j < BS; ++j) D[i * BS + j] = (T)a[i][BS + j];
  } else {
    for (int i = 0; i < BS; ++i)
      for (int j = 0; j < BS; ++j) {
        double dv = kd >= 0 ? (double)val[(long long)kd * BS * BS + i * BS + i] : 0.0;
        D[i * BS + j] = (i == j) ? (T)(dv != 0.0 ? 1.0 / dv : 1.0) : T(0);
      }
  }
}
template <typename T>
void blockdiag_invert(const BsrMat<T>& A, T* dinv, cudaStream_t st) {
  const int blocks = (A.nbrow + 127) / 128;
  if (A.bs == 3) { pfem::count_launch(); blockdiag_invert_kernel<T, 3><<<blocks, 128, 0, st>>>(A.nbrow, A.rowptr, A.col, A.val, dinv); }
  else { pfem::count_launch(); blockdiag_invert_kernel<T, 6><<<blocks, 128, 0, st>>>(A.nbrow, A.rowptr, A.col, A.val, dinv); }
}

// ------------------------------------------------------------------ dot products
template <typename T>
__global__ void sum_final_kernel(int np, const T* __restrict__ part, T* __restrict__ out, int sqrt_out) {
  __shared__ T sh[32];
  T v = T(0);
  for (int i = threadIdx.x; i < np; i += blockDim.x) v += part[i];
  v = block_sum(v, sh);
  if (threadIdx.x == 0) *out = sqrt_out ? sqrt(v) : v;
}
template <typename T>
void dot(long long n, const T* a, const T* b, T* out, T* part, cudaStream_t st, bool take_sqrt) {
  const int blocks = dot_partials<T>(n, a, b, part, st);
  pfem::count_launch(); sum_final_kernel<T><<<1, 1024, 0, st>>>(blocks, part, out, take_sqrt ? 1 : 0);
}

// ------------------------------------------------------------------ vector ops
template <typename T>
__global__ void fill_kernel(long long n, T* x, T v) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    x[i] = v;
}
template <typename T>
void fill(long long n, T* x, T v, cudaStream_t st) {
  const int blocks = (int)std::min<long long>((n + 255) / 256, 4096);
  if (n > 0) { pfem::count_launch(); fill_kernel<T><<<blocks > 0 ? blocks : 1, 256, 0, st>>>(n, x, v); }
}
// y = a*x + b*y with host scalars
template <typename T>
__global__ void axpby_kernel(long long n, T a, const T* __restrict__ x, T b, T* __restrict__ y) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = a * x[i] + b * y[i];
}
template <typename T>
void axpby(long long n, T a, const T* x, T b, T* y, cudaStream_t st) {
  const int blocks = (int)std::min<long long>((n + 255) / 256, 4096);
  if (n > 0) { pfem::count_launch(); axpby_kernel<T><<<blocks, 256, 0, st>>>(n, a, x, b, y); }
}
static int fused_update_blocks(long long n) {
  const long long nb = (n + RED_THREADS - 1) / RED_THREADS;
  return (int)(nb < RED_BLOCKS ? (nb > 0 ? nb : 1) : RED_BLOCKS);
}
// ---- PCG updates with the final reduction fused in ----
// Every CTA sums the same np partials in the same order (a strided pass and a
// fixed tree), so all CTAs see the same scalar and the result is deterministic.
template <typename T>
__device__ __forceinline__ T all_sum_partials(const T* part, int np, T* sh) {
  T v = T(0);
  for (int i = threadIdx.x; i < np; i += blockDim.x) v += part[i];
  v = block_sum(v, sh);
  __syncthreads();
  if (threadIdx.x == 0) sh[32] = v;
  __syncthreads();
  return sh[32];
}
// rz = sum(part_rz);  p = z + (rz / sc[0]) p;  sc[2] = rz
template <typename T>
__global__ void cg_p_fused_kernel(long long n, const T* part, int np, T* sc, const T* z, T* p) {
  __shared__ T sh[33];
  pdl_go();
  pdl_wait();
  const T rz = all_sum_partials(part, np, sh);
  const T be = rz / sc[0];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    p[i] = z[i] + be * p[i];
  if (blockIdx.x == 0 && threadIdx.x == 0) sc[2] = rz;
}
// pq = sum(part_pq);  alpha = sc[2] / pq;  x += alpha p;  r -= alpha q;  the smoother's
// start on the new r;  sc[0] = sc[2] (r.z of the next beta).  A thread per node.  The
// CTA that finishes last adds the CTAs' shares of r.r in their order and sets the
// loop's condition.
template <typename T>
__global__ void __launch_bounds__(256) cg_xr_fused_kernel(int nbrow, const T* part_pq, int np, T* sc, const T* p,
                                                          const T* q, T* x, T* r, const T* __restrict__ dinv,
                                                          const T* __restrict__ co, T* sr, T* sd, double* part_rr,
                                                          CgLoop loop) {
  __shared__ T sht[33];
  __shared__ double sh[33];
  __shared__ bool last;
  pdl_go();
  const T ith = co[CO_ITH];
  pdl_wait();
  const T pq = all_sum_partials(part_pq, np, sht);
  const T al = sc[2] / pq;
  double acc = 0.0;
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nbrow; n += gridDim.x * blockDim.x) {
    const long long at = (long long)n * 3;
    T ri[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      x[at + j] += al * p[at + j];
      ri[j] = r[at + j] - al * q[at + j];
      r[at + j] = ri[j];
      acc += (double)ri[j] * (double)ri[j];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      T t = T(0);
#pragma unroll
      for (int j = 0; j < 3; ++j) t += dinv[(long long)n * 9 + i * 3 + j] * ri[j];
      sr[at + i] = t;
      sd[at + i] = ith * t;
    }
  }
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) {
    part_rr[blockIdx.x] = acc;
    __threadfence();
    last = atomicInc(loop.ticket, gridDim.x - 1) == gridDim.x - 1;  // wraps to zero
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const double rr = all_sum_partials(part_rr, (int)gridDim.x, sh);
  if (threadIdx.x != 0) return;
  sc[0] = sc[2];
  const double rn = sqrt(rr);
  const int it = loop.state[0] + 1;
  const bool conv = rn <= loop.ctl[2];
  loop.state[0] = it;
  loop.state[1] = conv ? 1 : 0;
  cudaGraphSetConditional(loop.h, (!conv && isfinite(rn) && it < (int)loop.ctl[1]) ? 1u : 0u);
}
template <typename T>
void cg_p_fused(long long n, const T* part, int np, T* sc, const T* z, T* p, Queue q) {
  launch(q, cg_p_fused_kernel<T>, fused_update_blocks(n), RED_THREADS, 0, n, part, np, sc, z, p);
}
template <typename T>
void cg_xr_fused(int nbrow, const T* part_pq, int np, T* sc, const T* p, const T* q, T* x, T* r, const T* dinv,
                 const T* co, T* sr, T* sd, double* part_rr, const CgLoop& loop, Queue qu) {
  launch(qu, cg_xr_fused_kernel<T>, fused_update_blocks(nbrow), RED_THREADS, 0, nbrow, part_pq, np, sc, p, q, x, r, dinv,
         co, sr, sd, part_rr, loop);
}

// The sum of np partials (at most 2048) in the order in which sum_final_kernel adds them,
// by a CTA of 256 threads, each for four of that one's: to every thread.
template <typename T>
__device__ __forceinline__ T sum_as_final(const T* part, int np, T* sh) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    T v = T(0);
    for (int i = threadIdx.x + q * RED_THREADS; i < np; i += 1024) v += part[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (l == 0) sh[w + 8 * q] = v;
  }
  __syncthreads();
  T v = sh[l];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();  // sh may be written again
  return v;
}
// ---- power iteration.  The norm of an iterate in the matrix's type, in dot's order; its
// reciprocal goes to co[CO_INV], where the next step's product reads it: the scaled
// iterate is never stored, and a step is two launches.  FP32 coarse levels see the last
// bit of the estimate through the prolongator, so the order is kept. ----
template <typename T>
__global__ void __launch_bounds__(RED_THREADS) power_norm_kernel(long long n, const T* __restrict__ v, T* part,
                                                                 unsigned* ticket, bool finish, T* co) {
  __shared__ T sh[32];
  __shared__ bool last;
  T s = T(0);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    s += v[i] * v[i];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = s;
    __threadfence();
    last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;  // wraps to zero
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const T norm = sqrt(sum_as_final(part, (int)gridDim.x, sh));
  if (threadIdx.x != 0) return;
  co[CO_INV] = T(1) / norm;
  if (!finish) return;
  const double lm = (double)norm;
  const T lmax = (T)(1.1 * lm);
  const double lmx = (double)lmax, lmn = lmx / 30.0;
  const double th = 0.5 * (lmx + lmn), de = 0.5 * (lmx - lmn);
  const double sg = th / de, rho = 1.0 / sg;
  const double rn = 1.0 / (2.0 * sg - rho);
  co[CO_LMAX] = lmax;
  co[CO_ITH] = T(1.0 / th);
  co[CO_C1] = T(2.0 * rn / de);
  co[CO_C2] = T(1.0 + rn * rho);
  co[CO_OMEGA] = T(4.0 / (3.0 * lm));
}
template <typename T>
void power_norm(long long n, const T* v, T* part, unsigned* ticket, bool finish, T* co, cudaStream_t st) {
  pfem::count_launch();
  power_norm_kernel<T><<<fused_update_blocks(n), RED_THREADS, 0, st>>>(n, v, part, ticket, finish, co);
}
// ---- BiCGStab updates.  Scalars: sc[0] rho = rh.r, sc[1] rho of the iteration before,
// sc[2] alpha, sc[3] omega.  A thread per node, as cg_xr_fused; the dot products come as
// dot's partials and are added in its order.  An iteration used to be 44 plain launches
// from the host with a read-back of |r|, bound by the launches below about 40^3; in the
// graph with the smoother's starts in its own updates it takes 410 us at 40^3 FP64, 550
// before.
template <typename T>
__device__ __forceinline__ void smoother_start(const T* __restrict__ dinv, T ith, long long n, const T v[3], T* sr,
                                               T* sd) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    T t = T(0);
#pragma unroll
    for (int j = 0; j < 3; ++j) t += dinv[n * 9 + i * 3 + j] * v[j];
    sr[n * 3 + i] = t;
    sd[n * 3 + i] = ith * t;
  }
}
// beta = (rho / rho_old) (alpha / omega);  p = r + beta (p - omega v)
template <typename T>
__global__ void __launch_bounds__(256) bicg_p_kernel(int nbrow, const T* sc, const T* r, const T* v, T* p,
                                                     const T* __restrict__ dinv, const T* __restrict__ co, T* sr,
                                                     T* sd) {
  pdl_go();
  const T ith = co[CO_ITH];
  pdl_wait();
  const T beta = (sc[0] / sc[1]) * (sc[2] / sc[3]);
  const T om = sc[3];
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nbrow; n += gridDim.x * blockDim.x) {
    T e[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const long long i = (long long)n * 3 + j;
      e[j] = r[i] + beta * (p[i] - om * v[i]);
      p[i] = e[j];
    }
    smoother_start(dinv, ith, n, e, sr, sd);
  }
}
// alpha = rho / sum(part);  s = r - alpha v
template <typename T>
__global__ void __launch_bounds__(256) bicg_s_kernel(int nbrow, const T* part, int np, T* sc, const T* r,
                                                     const T* v, T* s, const T* __restrict__ dinv,
                                                     const T* __restrict__ co, T* sr, T* sd) {
  __shared__ T sh[32];
  pdl_go();
  const T ith = co[CO_ITH];
  pdl_wait();
  const T al = sc[0] / sum_as_final(part, np, sh);
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nbrow; n += gridDim.x * blockDim.x) {
    T e[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const long long i = (long long)n * 3 + j;
      e[j] = r[i] - al * v[i];
      s[i] = e[j];
    }
    smoother_start(dinv, ith, n, e, sr, sd);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) sc[2] = al;
}
// Partials of t.s and of t.t.
template <typename T>
__global__ void __launch_bounds__(256) bicg_dots_kernel(long long n, const T* t, const T* s, T* part_ts,
                                                        T* part_tt) {
  __shared__ T sh[32];
  pdl_go();
  pdl_wait();
  T a = T(0), b = T(0);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const T ti = t[i];
    a += ti * s[i];
    b += ti * ti;
  }
  a = block_sum(a, sh);
  __syncthreads();
  b = block_sum(b, sh);
  if (threadIdx.x == 0) {
    part_ts[blockIdx.x] = a;
    part_tt[blockIdx.x] = b;
  }
}
// omega = sum(part_ts) / sum(part_tt);  x += alpha ph + omega sh;  r = s - omega t.  The
// CTA that finishes last adds the shares of r.r and rh.r in their order, leaves the next
// iteration's scalars and sets the loop's condition.
template <typename T>
__global__ void __launch_bounds__(256) bicg_xr_kernel(long long n, const T* part_ts, const T* part_tt,
                                                      int np, T* sc, const T* ph, const T* sh_, const T* s, const T* t,
                                                      const T* rh, T* x, T* r, T* part_rr, T* part_rho,
                                                      CgLoop loop) {
  __shared__ T sh[32];
  __shared__ bool last;
  pdl_go();
  pdl_wait();
  const T al = sc[2];
  const T ts = sum_as_final(part_ts, np, sh);
  const T om = ts / sum_as_final(part_tt, np, sh);
  T rr = T(0), rho = T(0);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    x[i] += al * ph[i] + om * sh_[i];
    const T e = s[i] - om * t[i];
    r[i] = e;
    rr += e * e;
    rho += rh[i] * e;
  }
  rr = block_sum(rr, sh);
  __syncthreads();
  rho = block_sum(rho, sh);
  if (threadIdx.x == 0) {
    part_rr[blockIdx.x] = rr;
    part_rho[blockIdx.x] = rho;
    __threadfence();
    last = atomicInc(loop.ticket, gridDim.x - 1) == gridDim.x - 1;  // wraps to zero
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  rr = sum_as_final(part_rr, (int)gridDim.x, sh);
  rho = sum_as_final(part_rho, (int)gridDim.x, sh);
  if (threadIdx.x != 0) return;
  sc[1] = sc[0];
  sc[0] = rho;
  sc[3] = om;
  const double rn = (double)sqrt(rr);
  const int it = loop.state[0] + 1;
  const bool conv = rn <= loop.ctl[2];
  loop.state[0] = it;
  loop.state[1] = conv ? 1 : 0;
  cudaGraphSetConditional(loop.h, (!conv && isfinite(rn) && it < (int)loop.ctl[1]) ? 1u : 0u);
}
template <typename T>
void bicg_p(int nbrow, const T* sc, const T* r, const T* v, T* p, const T* dinv, const T* co, T* sr, T* sd, Queue q) {
  launch(q, bicg_p_kernel<T>, fused_update_blocks(nbrow), RED_THREADS, 0, nbrow, sc, r, v, p, dinv, co, sr, sd);
}
template <typename T>
void bicg_s(int nbrow, const T* part, int np, T* sc, const T* r, const T* v, T* s, const T* dinv, const T* co,
            T* sr, T* sd, Queue q) {
  launch(q, bicg_s_kernel<T>, fused_update_blocks(nbrow), RED_THREADS, 0, nbrow, part, np, sc, r, v, s, dinv, co, sr,
         sd);
}
template <typename T>
void bicg_xr(long long n, T* sc, const T* ph, const T* sh, const T* s, const T* t, const T* rh, T* x, T* r,
             T* part, const CgLoop& loop, Queue q) {
  const int blocks = fused_update_blocks(n);
  T* const part_ts = part, * const part_tt = part + kMaxPartials;
  launch(q, bicg_dots_kernel<T>, blocks, RED_THREADS, 0, n, t, s, part_ts, part_tt);
  launch(q, bicg_xr_kernel<T>, blocks, RED_THREADS, 0, n, part_ts, part_tt, blocks, sc, ph, sh, s, t, rh, x, r,
         part + 2 * kMaxPartials, part + 3 * kMaxPartials, loop);
}

// precision conversion
template <typename A, typename B>
__global__ void convert_kernel(long long n, const A* __restrict__ a, B* __restrict__ b, double s) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    b[i] = (B)(s * (double)a[i]);
}
template <typename A, typename B>
void convert(long long n, const A* a, B* b, double s, cudaStream_t st) {
  const int blocks = (int)std::min<long long>((n + 255) / 256, 4096);
  pfem::count_launch(); convert_kernel<A, B><<<blocks, 256, 0, st>>>(n, a, b, s);
}
// U += (double) x
template <typename T>
__global__ void add_to_double_kernel(long long n, const T* __restrict__ x, double* __restrict__ U) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    U[i] += (double)x[i];
}
template <typename T>
void add_to_double(long long n, const T* x, double* U, cudaStream_t st) {
  const int blocks = (int)std::min<long long>((n + 255) / 256, 4096);
  pfem::count_launch(); add_to_double_kernel<T><<<blocks, 256, 0, st>>>(n, x, U);
}

// ------------------------------------------------------------------ Dirichlet (K3)
// With dg = g(lambda) - U on constrained dofs (impose_dirichlet!, BoundaryConditions.jl):
//   free rows touching constrained columns: R[row] += sum_k K[row, col_k] dg[col_k] and
//   these entries become 0 (248-256); eight lanes per row, CTAs [0, nb_rows);
//   the other entries of constrained rows: 0, 1 on the diagonal (259-266);
//   constrained dofs: R[d] = -dg[d] (269-272).
// No entry of K or R belongs to two of the three, so they are one launch.  What bounds
// it is the row's chain of loads: 14.6 us at 57 x 43 x 31 FP64 (34.7 with one entry per
// lane at a time), where a thread per row took 16.3 us and four more launches the rest.  With
// load_norm_kernel two launches in place of seven: a residual there 575 -> 552 us.
template <typename KT>
__global__ void __launch_bounds__(256) bc_impose_kernel(BcDev bc, int nb_rows, int nb_zero, double lam,
                                                        const double* __restrict__ U, KT* __restrict__ K,
                                                        double* __restrict__ R) {
  auto dg = [&](int k) {
    const double v = bc.vals[k];
    return (bc.ramp[k] ? lam * v : v) - U[bc.dofs[k]];
  };
  int b = (int)blockIdx.x;
  if (b < nb_rows) {
    const int i = b * 32 + ((int)threadIdx.x >> 3), sub = threadIdx.x & 7;
    const bool in = i < bc.nrows;
    double s = 0.0;
    const int e = in ? bc.rptr[i + 1] : 0;
    // four entries per lane at a time, their loads in flight together
    for (int k0 = in ? bc.rptr[i] + sub : 0; k0 < e; k0 += 32) {
      long long pos[4];
      int c[4];
      double kv[4], g[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool have = k0 + 8 * u < e;
        pos[u] = have ? bc.rpos[k0 + 8 * u] : -1;
        c[u] = have ? bc.rbc[k0 + 8 * u] : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        kv[u] = pos[u] >= 0 ? (double)K[pos[u]] : 0.0;
        g[u] = dg(c[u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (pos[u] < 0) continue;
        s += kv[u] * g[u];
        K[pos[u]] = KT(0);
      }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (in && sub == 0) R[bc.rows[i]] += s;
    return;
  }
  b -= nb_rows;
  if (b < nb_zero) {
    for (long long i = b * 256ll + threadIdx.x; i < bc.nzero; i += nb_zero * 256ll) K[bc.zpos[i]] = bc.zone[i] ? KT(1) : KT(0);
    return;
  }
  const int k = (b - nb_zero) * 256 + (int)threadIdx.x;
  if (k < bc.nbc) R[bc.dofs[k]] = -dg(k);
}
// R -= lambda Fn (Fn is 0 on constrained dofs), and out = |R|: the CTA that finishes last
// adds the CTAs' shares in their order.
__global__ void __launch_bounds__(RED_THREADS) load_norm_kernel(long long n, double lam, const double* __restrict__ fn,
                                                                double* __restrict__ R, double* part,
                                                                unsigned* ticket, double* out) {
  __shared__ double sh[33];
  __shared__ bool last;
  double s = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double r = R[i] - lam * fn[i];
    R[i] = r;
    s += r * r;
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = s;
    __threadfence();
    last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;  // wraps to zero
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  s = all_sum_partials(part, (int)gridDim.x, sh);
  if (threadIdx.x == 0) *out = sqrt(s);
}
template <typename KT>
void impose_dirichlet(const BcDev& bc, long long ndof, double lam, const double* U, KT* K, double* R, double* part,
                      unsigned* ticket, double* rnorm, cudaStream_t st) {
  if (bc.nbc > 0) {
    const int nb_rows = (bc.nrows + 31) / 32;  // none when every dof is constrained
    const int nb_zero = (int)std::min<long long>((bc.nzero + 255) / 256, 4096);
    pfem::count_launch();
    bc_impose_kernel<KT><<<nb_rows + nb_zero + (bc.nbc + 255) / 256, 256, 0, st>>>(bc, nb_rows, nb_zero, lam, U, K, R);
  }
  pfem::count_launch();
  load_norm_kernel<<<fused_update_blocks(ndof), RED_THREADS, 0, st>>>(ndof, lam, bc.fn, R, part, ticket, rnorm);
}
// Set U[d] = g(lambda) on constrained dofs (predictors honour the BCs).
__global__ void bc_apply_kernel(int nbc, const int* __restrict__ dofs, const double* __restrict__ vals,
                                const uint8_t* __restrict__ ramp, double lam, double* __restrict__ U) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nbc) return;
  U[dofs[i]] = ramp[i] ? lam * vals[i] : vals[i];
}
void bc_apply(const BcDev& bc, double lam, double* U, cudaStream_t st) {
  if (bc.nbc > 0) { pfem::count_launch(); bc_apply_kernel<<<(bc.nbc + 255) / 256, 256, 0, st>>>(bc.nbc, bc.dofs, bc.vals, bc.ramp, lam, U); }
}

// ------------------------------------------------------------------ coarse solve
// Dense coarse solve y = Ainv b (one warp per row; the row's first entries are in
// flight before the wait for b).
template <typename T>
__global__ void dense_mv_kernel(int n, const T* __restrict__ M, const T* b, T* y) {
  pdl_go();
  const int row = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  constexpr int AHEAD = 6;
  const T* m = M + (long long)row * n;
  T a[AHEAD];
#pragma unroll
  for (int u = 0; u < AHEAD; ++u) a[u] = (row < n && lane + 32 * u < n) ? m[lane + 32 * u] : T(0);
  pdl_wait();
  if (row >= n) return;
  T s = T(0);
#pragma unroll
  for (int u = 0; u < AHEAD; ++u)
    if (lane + 32 * u < n) s += a[u] * b[lane + 32 * u];
  for (int j = lane + 32 * AHEAD; j < n; j += 32) s += m[j] * b[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) y[row] = s;
}
template <typename T>
void dense_mv(int n, const T* M, const T* b, T* y, Queue q) {
  launch(q, dense_mv_kernel<T>, (int)(((long long)n * 32 + 255) / 256), 256, 0, n, M, b, y);
}

// ------------------------------------------------------------------ smoothed aggregation
// Six consecutive values from an address that is 8-byte aligned (float) or
// 16-byte aligned (double), as three 8- or 16-byte loads: every 6-value row of a
// bs x 6 transfer block and every 6-vector of a coarse level is.
template <typename T, bool STREAM>
__device__ __forceinline__ void load6(const T* p, T* v) {
  using V2 = typename std::conditional<std::is_same<T, float>::value, float2, double2>::type;
  const V2* q = reinterpret_cast<const V2*>(p);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const V2 w = STREAM ? __ldcs(q + k) : q[k];
    v[2 * k] = w.x;
    v[2 * k + 1] = w.y;
  }
}

// P = (I - w D^-1 A) T with the tentative T (one bs x 6 block per fine row).
// One thread per P block p (row n, aggregate J):
//   P_p = [J == agg(n)] T_n - w Dinv_n sum_{k in row n, agg(col k) == J} A_k T_col(k)
// pslot[k] names the P block that A block k feeds.
template <typename T, int BS>
__global__ void sa_prolongator_kernel(int nnzP, const int* __restrict__ p_row, const int* __restrict__ p_cl,
                                      const int* __restrict__ rowptr, const int* __restrict__ col,
                                      const T* __restrict__ val, const int* __restrict__ pslot,
                                      const int* __restrict__ agg, const T* __restrict__ Tb,
                                      const T* __restrict__ dinv, const T* __restrict__ omega,
                                      T* __restrict__ pval) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nnzP) return;
  const int n = p_row[p];
  T acc[BS][6];
#pragma unroll
  for (int i = 0; i < BS; ++i)
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[i][c] = T(0);
  for (int k = rowptr[n]; k < rowptr[n + 1]; ++k) {
    if (pslot[k] != p) continue;
    const T* A = val + (long long)k * BS * BS;
    const T* Tm = Tb + (long long)col[k] * BS * 6;
#pragma unroll
    for (int j = 0; j < BS; ++j) {
      T tv[6];
      load6<T, false>(Tm + j * 6, tv);
#pragma unroll
      for (int i = 0; i < BS; ++i) {
        const T a = A[i * BS + j];
#pragma unroll
        for (int c = 0; c < 6; ++c) acc[i][c] += a * tv[c];
      }
    }
  }
  const T* D = dinv + (long long)n * BS * BS;
  const bool own = p_cl[p] == agg[n];
  const T* Tn = Tb + (long long)n * BS * 6;
  T* P = pval + (long long)p * BS * 6;
  const T w = *omega;
#pragma unroll
  for (int i = 0; i < BS; ++i)
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      T s = T(0);
#pragma unroll
      for (int j = 0; j < BS; ++j) s += D[i * BS + j] * acc[j][c];
      P[i * 6 + c] = (own ? Tn[i * 6 + c] : T(0)) - w * s;
    }
}

__device__ __forceinline__ int find_sorted(const int* __restrict__ a, int lo, int hi, int key) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    const int v = a[mid];
    if (v == key) return mid;
    if (v < key) lo = mid + 1; else hi = mid;
  }
  return -1;
}

// AP block q (row n, coarse column J) = sum_{k in row n} A_k P[col k, J].
template <typename T, int BS>
__global__ void sa_ap_kernel(int nnzAP, const int* __restrict__ ap_row, const int* __restrict__ ap_cl,
                             const int* __restrict__ rowptr, const int* __restrict__ col,
                             const T* __restrict__ val, const int* __restrict__ p_rp,
                             const int* __restrict__ p_cl, const T* __restrict__ pval, T* __restrict__ apval) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nnzAP) return;
  const int n = ap_row[q], J = ap_cl[q];
  T acc[BS][6];
#pragma unroll
  for (int i = 0; i < BS; ++i)
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[i][c] = T(0);
  for (int k = rowptr[n]; k < rowptr[n + 1]; ++k) {
    const int m = col[k];
    const int p = find_sorted(p_cl, p_rp[m], p_rp[m + 1], J);
    if (p < 0) continue;
    const T* A = val + (long long)k * BS * BS;
    const T* P = pval + (long long)p * BS * 6;
#pragma unroll
    for (int j = 0; j < BS; ++j) {
      T pv[6];
      load6<T, false>(P + j * 6, pv);
#pragma unroll
      for (int i = 0; i < BS; ++i) {
        const T a = A[i * BS + j];
#pragma unroll
        for (int c = 0; c < 6; ++c) acc[i][c] += a * pv[c];
      }
    }
  }
  T* O = apval + (long long)q * BS * 6;
#pragma unroll
  for (int i = 0; i < BS; ++i)
#pragma unroll
    for (int c = 0; c < 6; ++c) O[i * 6 + c] = acc[i][c];
}

// Coarse block c (I, J) = sum_{p in P^T row I} P_p^T AP[row(p), J]   (6 x 6).  LN lanes
// per block stride over the P^T row (its copy ptval: consecutive lanes read
// consecutive blocks), each searching its row of AP for J, and add their 36 partial
// sums by a fixed xor tree.  One thread per block walked the whole row, about 115
// blocks at level 0: 770 us there at 64^3 and 403 us at level 1, 320 us for the whole of a
// 23x9x7 mesh; so 634, 58 and 45 us (FP32).
template <typename T, int BS, int LN>
__global__ void __launch_bounds__(128) sa_rap_kernel(int nnzC, const int* __restrict__ c_row, const int* __restrict__ c_cl,
                              const int* __restrict__ pt_rp, const int* __restrict__ pt_row,
                              const T* __restrict__ ptval,
                              const int* __restrict__ ap_rp, const int* __restrict__ ap_cl,
                              const T* __restrict__ apval, T* __restrict__ cval) {
  const long long th = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int c = (int)(th / LN), lane = (int)(th % LN);
  const bool in = c < nnzC;
  const int I = in ? c_row[c] : 0, J = in ? c_cl[c] : 0;
  T acc[6][6];
#pragma unroll
  for (int r = 0; r < 6; ++r)
#pragma unroll
    for (int q = 0; q < 6; ++q) acc[r][q] = T(0);
  const int t1 = in ? pt_rp[I + 1] : 0;
  for (int t = in ? pt_rp[I] + lane : 0; t < t1; t += LN) {
    const int n = pt_row[t];
    const int q = find_sorted(ap_cl, ap_rp[n], ap_rp[n + 1], J);
    if (q < 0) continue;
    const T* P = ptval + (long long)t * BS * 6;
    const T* AP = apval + (long long)q * BS * 6;
#pragma unroll
    for (int i = 0; i < BS; ++i) {
      T pv[6], av[6];
      load6<T, false>(P + i * 6, pv);
      load6<T, false>(AP + i * 6, av);
#pragma unroll
      for (int r = 0; r < 6; ++r)
#pragma unroll
        for (int q2 = 0; q2 < 6; ++q2) acc[r][q2] += pv[r] * av[q2];
    }
  }
#pragma unroll
  for (int r = 0; r < 6; ++r)
#pragma unroll
    for (int q = 0; q < 6; ++q) {
#pragma unroll
      for (int o = LN / 2; o > 0; o >>= 1) acc[r][q] += __shfl_xor_sync(0xffffffffu, acc[r][q], o);
    }
  if (!in) return;
  T* O = cval + (long long)c * 36;
#pragma unroll
  for (int r = 0; r < 6; ++r)
#pragma unroll
    for (int q = 0; q < 6; ++q)
      if ((r * 6 + q) % LN == lane) O[r * 6 + q] = acc[r][q];
}

// The same for FP32 in the order of the P^T row, as one thread per block adds it: the
// coarse operator's small eigenvalues are what is left of terms hundreds of times larger,
// so in FP32 another order is another operator, and the solution of a slender box moves
// with it.  What the LN lanes of a block find is taken in turn, lane r with the six entries
// of row r.  Set-up with this / with the kernel above, FP32: 0.40 / 0.40 ms at 8^3, 1.01 /
// 1.03 at 80 x 16 x 16, 1.57 / 1.54 at 40^3; one at a time 0.45, 1.13 and 1.58; 16 lanes
// 0.39, 1.04 and 1.63.  (FP64 2.23 / 2.07 ms at 40^3.)
template <typename T, int BS, int LN>
__global__ void __launch_bounds__(128) sa_rap_ordered_kernel(int nnzC, const int* __restrict__ c_row, const int* __restrict__ c_cl,
                              const int* __restrict__ pt_rp, const int* __restrict__ pt_row,
                              const T* __restrict__ ptval,
                              const int* __restrict__ ap_rp, const int* __restrict__ ap_cl,
                              const T* __restrict__ apval, T* __restrict__ cval) {
  static_assert(LN >= 6 && 32 % LN == 0, "a lane per row of the block");
  constexpr int AT = BS == 3 ? 4 : 2;
  const long long th = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int c = (int)(th / LN), lane = threadIdx.x % LN, base = (threadIdx.x & 31) - lane;
  const bool in = c < nnzC;
  const int I = in ? c_row[c] : 0, J = in ? c_cl[c] : 0;
  const int r = min(lane, 5);
  T acc[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) acc[q] = T(0);
  const int t1 = in ? pt_rp[I + 1] : 0;
  int t = in ? pt_rp[I] + lane : 0;
  while (__any_sync(0xffffffffu, t - lane < t1)) {  // whole warps, for the shuffles
    int q = -1;
    if (t < t1) {
      const int n = pt_row[t];
      q = find_sorted(ap_cl, ap_rp[n], ap_rp[n + 1], J);
    }
    unsigned m = (__ballot_sync(0xffffffffu, q >= 0) >> base) & ((1u << (LN - 1)) * 2u - 1u);
    while (__any_sync(0xffffffffu, m != 0u)) {
      // AT of them at a time, their loads in flight together
      T p[AT][BS], av[AT][BS][6];
      bool have[AT];
#pragma unroll
      for (int e = 0; e < AT; ++e) {
        have[e] = m != 0u;
        const int u = m ? __ffs(m) - 1 : 0;
        m &= m - 1u;
        const int qu = __shfl_sync(0xffffffffu, q, base + u);
        if (have[e]) {
          const T* P = ptval + (long long)(t - lane + u) * BS * 6 + r;
          const T* AP = apval + (long long)qu * BS * 6;
#pragma unroll
          for (int i = 0; i < BS; ++i) {
            p[e][i] = P[i * 6];
            load6<T, false>(AP + i * 6, av[e][i]);
          }
        }
      }
#pragma unroll
      for (int e = 0; e < AT; ++e)
        if (have[e]) {
#pragma unroll
          for (int i = 0; i < BS; ++i)
#pragma unroll
            for (int k = 0; k < 6; ++k) acc[k] += p[e][i] * av[e][i][k];
        }
    }
    t += LN;
  }
  if (!in || lane >= 6) return;
  T* O = cval + (long long)c * 36 + r * 6;
#pragma unroll
  for (int k = 0; k < 6; ++k) O[k] = acc[k];
}

// P^T copy: block t of the aggregate-ordered list is P block pt_blk[t].
template <typename T, int BS>
__global__ void sa_transpose_copy_kernel(int nnzP, const int* __restrict__ pt_blk, const T* __restrict__ pval,
                                         T* __restrict__ ptval) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)nnzP * BS * 6) return;
  const long long t = e / (BS * 6);
  const int q = (int)(e - t * (BS * 6));
  ptval[e] = pval[(long long)pt_blk[t] * (BS * 6) + q];
}

// Restriction bc = P^T r, WPA warps per aggregate: the lanes stride over the
// aggregate's P blocks in the P^T-ordered copy (consecutive lanes read
// consecutive blocks), each warp combines its six partial sums by a fixed xor
// tree and the WPA warp sums are added in warp order, so the result is
// deterministic.  Coarse levels have few aggregates of many blocks each; there
// WPA = 4 spreads an aggregate over 128 lanes.
// START: the smoother's start on bc at the next level (block size 6) as well, sr =
// Dinv bc and sd = co[CO_ITH] sr, from the six sums that the last warp holds.
template <typename T, int BS, int WPA, bool START>
__global__ void __launch_bounds__(256) sa_restrict_kernel(int nagg, const int* __restrict__ pt_rp,
                                                          const int* __restrict__ pt_row,
                                                          const T* __restrict__ ptval, const T* r, T* bc,
                                                          const T* __restrict__ dinv, const T* __restrict__ co, T* sr,
                                                          T* sd) {
  __shared__ T part[8][6];
  pdl_go();
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int I = blockIdx.x * (8 / WPA) + wid / WPA;
  const int w = wid % WPA;
  T s[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
  const bool in = I < nagg;
  const int t1 = in ? pt_rp[I + 1] : 0;
  int t = in ? pt_rp[I] + w * 32 + lane : 0;
  // the first block of each lane is in flight before the wait for r
  T pv[BS][6];
  long long n = 0;
  auto block = [&]() {
    const T* P = ptval + (long long)t * BS * 6;
    n = pt_row[t];
#pragma unroll
    for (int j = 0; j < BS; ++j) load6<T, false>(P + j * 6, pv[j]);
  };
  if (t < t1) block();
  T D[6], ith = T(0);
  const bool own = in && w == 0 && lane < 6;
  if constexpr (START) {
#pragma unroll
    for (int j = 0; j < 6; ++j) D[j] = own ? dinv[(long long)I * 36 + lane * 6 + j] : T(0);
    ith = co[CO_ITH];
  }
  pdl_wait();
  while (t < t1) {
    const T* rv = r + n * BS;
#pragma unroll
    for (int j = 0; j < BS; ++j) {
      const T rj = rv[j];
#pragma unroll
      for (int c = 0; c < 6; ++c) s[c] += pv[j][c] * rj;
    }
    t += 32 * WPA;
    if (t < t1) block();
  }
#pragma unroll
  for (int c = 0; c < 6; ++c)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
  T out = s[0];
#pragma unroll
  for (int c = 1; c < 6; ++c)
    if (lane == c) out = s[c];
  if constexpr (WPA > 1) {
    if (lane < 6) part[wid][lane] = out;
    __syncthreads();
    if (w == 0 && lane < 6) {
#pragma unroll
      for (int q = 1; q < WPA; ++q) out += part[wid + q][lane];
    }
  }
  if constexpr (START) {
    T v = T(0);
#pragma unroll
    for (int j = 0; j < 6; ++j) v += D[j] * __shfl_sync(0xffffffffu, out, j);
    if (own) {
      sr[(long long)I * 6 + lane] = v;
      sd[(long long)I * 6 + lane] = ith * v;
    }
  }
  if (own) bc[(long long)I * 6 + lane] = out;
}
// Prolongation x[n*BS+j] += sum_{p in P row n} (P_p xc[col(p)])_j
// (TWO: x += P (xc + xc2), the two corrections of a W-cycle visit).
template <typename T, int BS, bool TWO = false>
__global__ void sa_prolong_kernel(int nbrow, const int* __restrict__ p_rp, const int* __restrict__ p_cl,
                                  const T* __restrict__ pval, const T* xc, const T* xc2, T* x) {
  pdl_go();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const bool in = i < (long long)nbrow * BS;
  const int n = (int)(i / BS), j = (int)(i % BS);
  int p = in ? p_rp[n] : 0;
  const int p1 = in ? p_rp[n + 1] : 0;
  // the first block's row is in flight before the wait for the corrections
  T pv[6];
  long long a = 0;
  auto block = [&]() {
    load6<T, true>(pval + (long long)p * BS * 6 + j * 6, pv);
    a = (long long)p_cl[p] * 6;
  };
  if (p < p1) block();
  pdl_wait();
  T s = T(0);
  while (p < p1) {
    T xv[6];
    load6<T, false>(xc + a, xv);
    if (TWO) {
      T x2v[6];
      load6<T, false>(xc2 + a, x2v);
#pragma unroll
      for (int c = 0; c < 6; ++c) xv[c] += x2v[c];
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) s += pv[c] * xv[c];
    if (++p < p1) block();
  }
  if (in) x[i] += s;
}

template <typename T, int BS>
static void setup_level_t(const AmgLevel<T>& v, T* cval, int nnzC, cudaStream_t st) {
  launch(st, sa_prolongator_kernel<T, BS>, (v.nnzP + 127) / 128, 128, 0, v.nnzP, v.p_row, v.p_cl, v.A.rowptr, v.A.col, v.A.val,
         v.pslot, v.agg, v.T, v.dinv, v.co + CO_OMEGA, v.p_val);
  launch(st, sa_transpose_copy_kernel<T, BS>, (int)(((long long)v.nnzP * BS * 6 + 255) / 256), 256, 0, v.nnzP, v.pt_blk,
         v.p_val, v.pt_val);
  launch(st, sa_ap_kernel<T, BS>, (v.nnzAP + 127) / 128, 128, 0, v.nnzAP, v.ap_row, v.ap_cl, v.A.rowptr, v.A.col, v.A.val,
         v.p_rp, v.p_cl, v.p_val, v.ap_val);
  // FP32: a thread per block where those fill the chip (set-up with one / with eight lanes
  // per block: 0.61 / 0.39 ms at 8^3, 1.67 / 1.60 at 40^3, 2.82 / 2.85 at 52^3 with 140,608
  // blocks, 3.54 / 3.94 at 64^3 with 262,144); both add in the order of the P^T row.
  constexpr int kRapOneThread = 150000;
  const bool one = std::is_same<T, float>::value && nnzC >= kRapOneThread;
  constexpr int LN = 8;
  auto* rap = [one] {
    if constexpr (std::is_same<T, float>::value) return one ? &sa_rap_kernel<T, BS, 1> : &sa_rap_ordered_kernel<T, BS, LN>;
    else return &sa_rap_kernel<T, BS, LN>;
  }();
  launch(st, rap, (int)(((long long)nnzC * (one ? 1 : LN) + 127) / 128), 128, 0, nnzC, v.c_row, v.c_cl, v.pt_rp,
         v.pt_row, v.pt_val, v.ap_rp, v.ap_cl, v.ap_val, cval);
}
template <typename T>
void sa_setup_level(const AmgLevel<T>& v, T* cval, int nnzC, cudaStream_t st) {
  if (v.A.bs == 3) setup_level_t<T, 3>(v, cval, nnzC, st);
  else setup_level_t<T, 6>(v, cval, nnzC, st);
}
// ---- transfers of the finest level with the blocks streamed through shared memory ----
// Read straight into registers a lane's 72-byte block costs the L1 a line per lane and
// load, as the matrix does (spmv_pipe.cuh).  Bytes of a tile's copies: the barrier, the
// ids, the blocks, each with room for ends rounded out to 16 bytes.
template <typename T>
__host__ __device__ inline int stream_vals(int blocks) { return 16 + ((blocks * 4 + 32 + 15) & ~15); }
template <typename T>
inline int stream_bytes(int blocks) { return stream_vals<T>(blocks) + blocks * 18 * (int)sizeof(T) + 32; }
// Blocks t0 .. t1 and their ids; one thread.
template <typename T>
__device__ __forceinline__ void stream_issue(unsigned char* sm, int cap, int t0, int t1, const int* ids, const T* vals) {
  constexpr int VB = 18 * (int)sizeof(T);
  const uint32_t bar = bulk_smem(sm);
  const long long ia = ((long long)t0 * 4) & ~15ll, va = ((long long)t0 * VB) & ~15ll;
  const uint32_t ib = (uint32_t)((((long long)t1 * 4 + 15) & ~15ll) - ia);
  const uint32_t vb = (uint32_t)((((long long)t1 * VB + 15) & ~15ll) - va);
  bulk_bar_init(bar, 1);
  bulk_init_fence();
  if (t0 == t1) {
    bulk_expect(bar, 0);
    return;
  }
  bulk_expect(bar, ib + vb);
  bulk_copy(bar + 16, (const char*)ids + ia, ib, bar);
  bulk_copy_first(bar + (uint32_t)stream_vals<T>(cap), (const char*)vals + va, vb, bar);
}
// sa_restrict_kernel<T, 3, 1, START> with a one-warp CTA per aggregate, its P^T row in
// shared memory; the sums are added in the same order.
template <typename T, bool START>
__global__ void __launch_bounds__(32)
sa_restrict_stream_kernel(int cap, const int* __restrict__ pt_rp, const int* __restrict__ pt_row,
                          const T* __restrict__ ptval, const T* r, T* bc, const T* __restrict__ dinv,
                          const T* __restrict__ co, T* sr, T* sd, int* err) {
  extern __shared__ __align__(128) unsigned char tsm[];
  pdl_go();
  const int I = blockIdx.x, lane = threadIdx.x;
  const int t0 = pt_rp[I], t1 = pt_rp[I + 1];
  if (lane == 0) stream_issue<T>(tsm, cap, t0, t1, pt_row, ptval);
  __syncwarp();
  T D[6], ith = T(0);
  if constexpr (START) {
#pragma unroll
    for (int j = 0; j < 6; ++j) D[j] = lane < 6 ? dinv[(long long)I * 36 + lane * 6 + j] : T(0);
    ith = co[CO_ITH];
  }
  pdl_wait();
  if (!__all_sync(0xffffffffu, bulk_bar_wait(bulk_smem(tsm), 0, err))) return;
  const int* ids = reinterpret_cast<const int*>(tsm + 16 + (((long long)t0 * 4) & 15));
  const T* vals = reinterpret_cast<const T*>(tsm + stream_vals<T>(cap) + (((long long)t0 * 18 * (int)sizeof(T)) & 15));
  T s[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
#pragma unroll 4
  for (int t = lane; t < t1 - t0; t += 32) {
    const T* rv = r + (long long)ids[t] * 3;
    const T* P = vals + t * 18;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const T rj = rv[j];
      T pv[6];
      load6<T, false>(P + j * 6, pv);
#pragma unroll
      for (int c = 0; c < 6; ++c) s[c] += pv[c] * rj;
    }
  }
#pragma unroll
  for (int c = 0; c < 6; ++c)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
  if (lane >= 6) return;
  T out = s[0];
#pragma unroll
  for (int c = 1; c < 6; ++c)
    if (lane == c) out = s[c];
  bc[(long long)I * 6 + lane] = out;
  if constexpr (START) {
    T w = T(0);
#pragma unroll
    for (int j = 0; j < 6; ++j) w += D[j] * s[j];
    sr[(long long)I * 6 + lane] = w;
    sd[(long long)I * 6 + lane] = ith * w;
  }
}
// sa_prolong_kernel<T, 3> with the P rows of a CTA's 32 nodes in shared memory, a thread
// per entry; the same sums.
template <typename T>
__global__ void __launch_bounds__(3 * kProlongTile)
sa_prolong_stream_kernel(int nbrow, int cap, const int* __restrict__ p_rp, const int* __restrict__ p_cl,
                         const T* __restrict__ pval, const T* xc, T* x, int* err) {
  extern __shared__ __align__(128) unsigned char tsm[];
  pdl_go();
  const int n0 = blockIdx.x * kProlongTile, n1 = min(nbrow, n0 + kProlongTile);
  const int n = n0 + (int)threadIdx.x / 3, j = (int)threadIdx.x % 3;
  const bool in = n < n1;
  const int t0 = p_rp[n0];
  if (threadIdx.x == 0) stream_issue<T>(tsm, cap, t0, p_rp[n1], p_cl, pval);
  const int p0 = in ? p_rp[n] - t0 : 0, p1 = in ? p_rp[n + 1] - t0 : 0;
  __syncthreads();
  pdl_wait();
  const long long i = (long long)n * 3 + j;
  const T xi = in ? x[i] : T(0);
  if (!bulk_bar_wait(bulk_smem(tsm), 0, err)) return;
  const int* ids = reinterpret_cast<const int*>(tsm + 16 + (((long long)t0 * 4) & 15));
  const T* vals = reinterpret_cast<const T*>(tsm + stream_vals<T>(cap) + (((long long)t0 * 18 * (int)sizeof(T)) & 15));
  T s = T(0);
#pragma unroll 4
  for (int p = p0; p < p1; ++p) {
    T xv[6], pv[6];
    load6<T, false>(xc + (long long)ids[p] * 6, xv);
    load6<T, false>(vals + p * 18 + j * 6, pv);
#pragma unroll
    for (int c = 0; c < 6; ++c) s += pv[c] * xv[c];
  }
  if (in) x[i] = xi + s;
}
// The prolongation streams from as many rows on as the matrix does (kPipeRows3; at 16^3,
// 4,913 rows, the cycle takes 22.7 us either way).  The restriction streams where the
// matrix alone fills L2 (126 MB): there it is the early eviction of the streamed blocks,
// more than the shorter kernel, that counts, as it leaves L2 to the vectors; below, it
// evicts what would have stayed.  CG iteration, neither / prolongation / both streamed:
// 139.7 / 137.8 / 140.9 us at 32^3 FP64 (66 MB of matrix), 184 / 184 / 188 at
// 49 x 37 x 29 FP64 (105 MB), 224.9 / 225.0 / 213.2 at 40^3 FP64 (128 MB), 249 / 245 / 230
// at 56 x 50 x 48 FP32 (133 MB), 392 / 385 / 377 at 64^3 FP32 (259 MB); both without
// early eviction 230.9 at 40^3 FP64 and 384 at 64^3.
constexpr int kStreamSmem = 48 * 1024;  // a tile's most, so that four or more CTAs share an SM
constexpr long long kMatrixFillsL2 = 120000000;
template <typename T>
static bool transfer_streams(const AmgLevel<T>& v, int blocks) {
  return v.A.bs == 3 && v.A.nbrow >= kPipeRows3 && v.A.err && blocks > 0 && stream_bytes<T>(blocks) <= kStreamSmem;
}
template <typename T>
static bool matrix_fills_l2(const AmgLevel<T>& v) {
  return v.A.nnzb * 9 * (long long)sizeof(T) > kMatrixFillsL2;
}

// Aggregates below this count get four warps each in the restriction.
constexpr int kRestrictWideBelow = 4096;

template <typename T>
void sa_restrict(const AmgLevel<T>& v, const T* r, T* bc, const AmgLevel<T>* next, Queue q) {
  if (transfer_streams(v, v.pt_max) && matrix_fills_l2(v)) {
    auto* kern = next ? sa_restrict_stream_kernel<T, true> : sa_restrict_stream_kernel<T, false>;
    launch(q, kern, v.nagg, 32, stream_bytes<T>(v.pt_max), v.pt_max, v.pt_rp, v.pt_row, v.pt_val, r, bc,
           next ? next->dinv : nullptr, next ? next->co : nullptr, next ? next->r : nullptr, next ? next->d : nullptr,
           v.A.err);
    return;
  }
  const bool wide = v.nagg < kRestrictWideBelow;
  const long long warps = (long long)v.nagg * (wide ? 4 : 1);
  const int blocks = (int)((warps + 7) / 8);
  auto* kern = v.A.bs == 3 ? (wide ? (next ? sa_restrict_kernel<T, 3, 4, true> : sa_restrict_kernel<T, 3, 4, false>)
                                   : (next ? sa_restrict_kernel<T, 3, 1, true> : sa_restrict_kernel<T, 3, 1, false>))
                           : (wide ? (next ? sa_restrict_kernel<T, 6, 4, true> : sa_restrict_kernel<T, 6, 4, false>)
                                   : (next ? sa_restrict_kernel<T, 6, 1, true> : sa_restrict_kernel<T, 6, 1, false>));
  launch(q, kern, blocks, 256, 0, v.nagg, v.pt_rp, v.pt_row, v.pt_val, r, bc, next ? next->dinv : nullptr,
         next ? next->co : nullptr, next ? next->r : nullptr, next ? next->d : nullptr);
}
template <typename T>
static void prolong_launch(const AmgLevel<T>& v, const T* xc, const T* xc2, T* x, const Queue& q) {
  const long long n = (long long)v.A.nbrow * v.A.bs;
  auto* kern = v.A.bs == 3 ? (xc2 ? sa_prolong_kernel<T, 3, true> : sa_prolong_kernel<T, 3>)
                           : (xc2 ? sa_prolong_kernel<T, 6, true> : sa_prolong_kernel<T, 6>);
  launch(q, kern, (int)((n + 255) / 256), 256, 0, v.A.nbrow, v.p_rp, v.p_cl, v.p_val, xc, xc2, x);
}
template <typename T>
void sa_prolong(const AmgLevel<T>& v, const T* xc, T* x, Queue q) {
  if (transfer_streams(v, v.p_tile)) {
    launch(q, sa_prolong_stream_kernel<T>, (v.A.nbrow + kProlongTile - 1) / kProlongTile, 3 * kProlongTile,
           stream_bytes<T>(v.p_tile), v.A.nbrow, v.p_tile, v.p_rp, v.p_cl, v.p_val, xc, x, v.A.err);
    return;
  }
  prolong_launch<T>(v, xc, nullptr, x, q);
}
template <typename T>
void sa_prolong2(const AmgLevel<T>& v, const T* xc, const T* xc2, T* x, Queue q) {
  prolong_launch<T>(v, xc, xc2, x, q);
}

// ------------------------------------------------------------------ instantiations
#define PFEM_INST(T)                                                                               \
  template int bsr_spmv<T>(const BsrMat<T>&, const T*, T*, Queue, T*);                             \
  template void bsr_residual<T>(const BsrMat<T>&, const T*, const T*, T*, Queue);                  \
  template void bsr_cheb_step<T>(const BsrMat<T>&, const T*, const T*, T*, T*, cudaStream_t);      \
  template int bsr_cheb2<T>(const BsrMat<T>&, const T*, const T*, const T*, T*, bool, const T*, Queue, const T*, \
                            T*);                                                                   \
  template void bsr_residual_precond<T>(const BsrMat<T>&, const T*, const T*, const T*, T*, T*, const T*, Queue); \
  template void bsr_residual_start<T>(const BsrMat<T>&, const T*, const T*, const T*, T*, T*, T*, const T*, Queue); \
  template void bsr_power_step<T>(const BsrMat<T>&, const T*, const T*, T*, const T*, cudaStream_t); \
  template void power_norm<T>(long long, const T*, T*, unsigned*, bool, T*, cudaStream_t);         \
  template void blockdiag_apply<T>(int, int, const T*, const T*, T*, const T*, T*, Queue);         \
  template void blockdiag_invert<T>(const BsrMat<T>&, T*, cudaStream_t);                           \
  template void dot<T>(long long, const T*, const T*, T*, T*, cudaStream_t, bool);                 \
  template void fill<T>(long long, T*, T, cudaStream_t);                                           \
  template void axpby<T>(long long, T, const T*, T, T*, cudaStream_t);                             \
  template void bicg_p<T>(int, const T*, const T*, const T*, T*, const T*, const T*, T*, T*,       \
                          Queue);                                                                  \
  template void bicg_s<T>(int, const T*, int, T*, const T*, const T*, T*, const T*, const T*,      \
                          T*, T*, Queue);                                                          \
  template void bicg_xr<T>(long long, T*, const T*, const T*, const T*, const T*, const T*, T*,    \
                           T*, T*, const CgLoop&, Queue);                                          \
  template int dot_partials<T>(long long, const T*, const T*, T*, const Queue&);                   \
  template void cg_p_fused<T>(long long, const T*, int, T*, const T*, T*, Queue);                  \
  template void cg_xr_fused<T>(int, const T*, int, T*, const T*, const T*, T*, T*, const T*, const T*, T*, T*, \
                               double*, const CgLoop&, Queue);                                     \
  template void add_to_double<T>(long long, const T*, double*, cudaStream_t);                      \
  template void impose_dirichlet<T>(const BcDev&, long long, double, const double*, T*, double*,   \
                                      double*, unsigned*, double*, cudaStream_t);                  \
  template void dense_mv<T>(int, const T*, const T*, T*, Queue);                            \
  template void sa_setup_level<T>(const AmgLevel<T>&, T*, int, cudaStream_t);                   \
  template void sa_restrict<T>(const AmgLevel<T>&, const T*, T*, const AmgLevel<T>*, Queue);       \
  template void sa_prolong<T>(const AmgLevel<T>&, const T*, T*, Queue);                     \
  template void sa_prolong2<T>(const AmgLevel<T>&, const T*, const T*, T*, Queue);
PFEM_INST(float)
PFEM_INST(double)
template void convert<double, float>(long long, const double*, float*, double, cudaStream_t);
template void convert<float, double>(long long, const float*, double*, double, cudaStream_t);
template void convert<double, double>(long long, const double*, double*, double, cudaStream_t);

}  // namespace pfem
