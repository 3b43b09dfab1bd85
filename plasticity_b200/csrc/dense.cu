// dense.cu -- dense inverse of the coarsest AMG operator, on the device.
//
// The smoothed-aggregation hierarchy ends in a dense solve (the reference's
// AlgebraicMultigrid.jl ends its hierarchy in a direct coarse solve as well,
// Solver.jl:136-154).  The coarsest operator (6 x 6 blocks, a few thousand
// unknowns) is expanded to a dense FP64 matrix and inverted in place by blocked
// Gauss-Jordan elimination; the cycle then applies the inverse as one dense
// matrix-vector product.  One kernel per panel of NB columns K, over NB x NB tiles; it
// gets copies of the panel's rows R = A[K, :] and columns C = A[:, K] and the inverse
// Dg = A[K,K]^{-1}, all made by the kernel before, so a CTA reads from A only the tiles
// that it writes itself:
//   P = Dg R[:, j] for its columns j (Dg itself in the panel's own columns),
//   A[i, j] <- A[i, j] - C[i, :] P outside the panel's rows (0 - C Dg in its columns),
//   A[K, j] <- P,
// and it copies what belongs to the next panel.  The CTA with the next diagonal block
// inverts that before its other tiles: 64 serial steps, which the other CTAs' work hides.
// No row exchanges: the Galerkin operator of the (Dirichlet-imposed) tangent of a
// large mesh is close to symmetric positive definite; a pivot below 1e-14 of the
// largest diagonal entry is replaced by that floor.  Coarsest levels of up to
// kPivotMax unknowns take pivot_inverse_kernel, which chooses its pivots.
#include <cstdint>

#include "linalg.cuh"

namespace pfem {
namespace {

constexpr int NB = 64;      // panel width
constexpr int PITCH = 68;   // of a tile in shared memory: a half-warp's fragment falls on 16 bank pairs
constexpr int GTHREADS = 256;

// Dense row-major n x n FP64 matrix from the coarsest level's 6 x 6 blocks.
template <typename T>
__global__ void bsr6_to_dense_kernel(int nbrow, const int* __restrict__ rp, const int* __restrict__ cl,
                                     const T* __restrict__ val, int n, double* __restrict__ A) {
  const long long nnzb = rp[nbrow];
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nnzb * 36;
       t += (long long)gridDim.x * blockDim.x) {
    const long long k = t / 36;
    const int e = (int)(t % 36), r = e / 6, c = e % 6;
    // block row of k: binary search in rp
    int lo = 0, hi = nbrow;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (rp[mid] <= k) lo = mid; else hi = mid;
    }
    A[(long long)(lo * 6 + r) * n + cl[k] * 6 + c] = (double)val[t];
  }
}

// Rows with no entry (rigid modes absent from an aggregate) get a unit
// diagonal; one warp per row.
__global__ void dense_fix_rows_kernel(int n, double* __restrict__ A) {
  const int i = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= n) return;  // whole warps
  bool nz = false;
  for (int j = lane; j < n; j += 32) nz |= A[(long long)i * n + j] != 0.0;
  nz = __any_sync(0xffffffffu, nz);
  if (!nz && lane == 0) A[(long long)i * n + i] = 1.0;
}

// scl[0] = the largest |diagonal entry| (the pivot floor's scale), one CTA.
__global__ void dense_diag_max_kernel(int n, const double* __restrict__ A, double* __restrict__ scl) {
  __shared__ double sh[32];
  double mx = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) mx = fmax(mx, fabs(A[(long long)i * n + i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) m = fmax(m, sh[k]);
    scl[0] = m;
  }
}

// Dg = inverse of the NB x NB block at src: in-place Gauss-Jordan by one CTA of
// eight warps with the block in registers: warp w holds the columns w, w + 8, ..., lane
// l the rows l and l + 32.  What bounds it is the chain of 64 steps, so each has one
// __syncthreads: the column's warp publishes it as the multipliers, every warp takes the
// pivot from there.  As in pivot_inverse_kernel a row is divided by its pivot at the
// end.  19.7 us as a kernel of its own; with the block in shared memory and five
// barriers per step 60 us.
__device__ __forceinline__ void gj_invert(const double* src, int ld, double (*F)[NB], const double* scl, double* Dg) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double a[8][2];
#pragma unroll
  for (int m = 0; m < 8; ++m)
#pragma unroll
    for (int r = 0; r < 2; ++r) a[m][r] = src[(long long)(lane + 32 * r) * ld + w + 8 * m];
  const double floor_abs = 1e-14 * fmax(scl[0], 1e-300);
  double ips[2] = {1.0, 1.0};  // 1 / pivot of the lane's rows
#pragma unroll
  for (int m0 = 0; m0 < 8; ++m0) {
#pragma unroll 1
    for (int q = 0; q < 8; ++q) {
      const int k = 8 * m0 + q, kl = k & 31;
      constexpr int HALF = 4;  // k < 32 exactly when m0 < HALF
      const int kr = m0 < HALF ? 0 : 1;
      double* const f = F[k & 1];
      if (w == q) {
        f[lane] = a[m0][0];
        f[lane + 32] = a[m0][1];
      }
      __syncthreads();
      double pv = f[k];
      double f0 = f[lane], f1 = f[lane + 32];
      double e[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) e[m] = __shfl_sync(0xffffffffu, a[m][kr], kl);
      if (fabs(pv) < floor_abs) pv = pv >= 0.0 ? floor_abs : -floor_abs;
      const double ip = 1.0 / pv;
      if (lane == kl) {
        ips[kr] = ip;
        if (kr == 0) f0 = 0.0; else f1 = 0.0;
      }
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const double x = e[m] * ip;
        a[m][0] = fma(-f0, x, a[m][0]);
        a[m][1] = fma(-f1, x, a[m][1]);
      }
      if (w == q) {  // the column becomes the inverse's
        a[m0][0] = -f0 * ip;
        a[m0][1] = -f1 * ip;
        if (lane == kl) a[m0][kr] = 1.0;
      }
    }
  }
#pragma unroll
  for (int m = 0; m < 8; ++m)
#pragma unroll
    for (int r = 0; r < 2; ++r) Dg[(lane + 32 * r) * NB + w + 8 * m] = a[m][r] * ips[r];
}

// A 64 x 64 tile to shared memory, 16 bytes at a time.
__device__ __forceinline__ void gj_load(double* dst, const double* src, long long ld) {
  const uint32_t d0 = (uint32_t)__cvta_generic_to_shared(dst);
#pragma unroll
  for (int u = 0; u < NB * NB / 2 / GTHREADS; ++u) {
    const int e = threadIdx.x + u * GTHREADS, r = e / (NB / 2), c = e % (NB / 2) * 2;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d0 + (uint32_t)(r * PITCH + c) * 8u),
                 "l"(src + r * ld + c) : "memory");
  }
}
__device__ __forceinline__ void gj_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}
// acc = X Y of two tiles in shared memory on the FP64 matrix pipe: warp w takes the rows
// 32 (w % 2) .. and the columns 16 (w / 2) .., as 4 x 2 fragments of 8 x 8.
__device__ __forceinline__ void gj_mul(const double* X, const double* Y, double (&acc)[4][2][2]) {
  const int w = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
  const double* x = X + (32 * (w & 1) + g) * PITCH + q;
  const double* y = Y + q * PITCH + 16 * (w >> 1) + g;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll 4
  for (int s = 0; s < NB; s += 4) {
    double xa[4], yb[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) xa[i] = x[8 * i * PITCH + s];
#pragma unroll
    for (int j = 0; j < 2; ++j) yb[j] = y[s * PITCH + 8 * j];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                     : "+d"(acc[i][j][0]), "+d"(acc[i][j][1])
                     : "d"(xa[i]), "d"(yb[j]));
  }
}
// Row and column within the tile of fragment (i, j)'s first of two entries.
__device__ __forceinline__ int gj_row(int i) { return 32 * ((threadIdx.x >> 5) & 1) + 8 * i + ((threadIdx.x & 31) >> 2); }
__device__ __forceinline__ int gj_col(int j) { return 16 * (threadIdx.x >> 6) + 8 * j + 2 * (threadIdx.x & 3); }

// Copies and the inverse for the first panel; CTA b copies tile b of each.
__global__ void __launch_bounds__(GTHREADS) gj_start_kernel(int np, const double* __restrict__ A, double* __restrict__ C,
                                                            double* __restrict__ R, double* __restrict__ Dg,
                                                            const double* __restrict__ scl) {
  __shared__ double F[2][NB];
  const long long t0 = (long long)blockIdx.x * NB;
  for (int e = threadIdx.x; e < NB * NB; e += GTHREADS) {
    const int r = e / NB, c = e % NB;
    R[(long long)r * np + t0 + c] = A[(long long)r * np + t0 + c];
    C[t0 * NB + e] = A[(t0 + r) * np + c];
  }
  if (blockIdx.x == 0) gj_invert(A, np, F, scl, Dg);
}

// Step k (the comment at the top).  CTA (j, y): column tile j and every gridDim.y-th row
// tile, from k + 1 on.  Two CTAs on an SM; the grid is at most that many.  What bounds it
// is the chain copies -> P -> update -> inverse of one CTA.  A panel at 1440 unknowns
// takes 32 us; as three kernels (diagonal 20 us, panel rows 22, update 43 with its loads
// and stores of A one after another) 85 us.  The set-up at 21 x 17 x 13 with it 1.3 ms,
// 2.0 before; at 40^3 (750 unknowns) 0.75 ms less.
__global__ void __launch_bounds__(GTHREADS, 2) gj_step_kernel(int np, int k, double* A, const double* C, const double* R,
                                                              const double* Dg, double* C1, double* R1, double* Dg1,
                                                              const double* scl) {
  extern __shared__ __align__(16) double gsm[];
  __shared__ double F[2][NB];
  double* const D = gsm;
  double* const V = gsm + NB * PITCH;
  double* const Cs = gsm + 2 * NB * PITCH;
  const int nt = np / NB, jt = (int)blockIdx.x;
  const long long j0 = (long long)jt * NB;
  pdl_go();
  pdl_wait();
  auto row_tile = [&](int i) { return (k + 1 + i) % nt; };
  gj_load(D, Dg, NB);
  if (jt != k) gj_load(V, R + j0, np);
  const int first = row_tile((int)blockIdx.y);
  if (first != k) gj_load(Cs, C + (long long)first * NB * NB, NB);
  gj_wait();
  double acc[4][2][2];
  if (jt != k) {
    gj_mul(D, V, acc);
    __syncthreads();  // V has been read
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
        *reinterpret_cast<double2*>(V + gj_row(i) * PITCH + gj_col(j)) = make_double2(acc[i][j][0], acc[i][j][1]);
    __syncthreads();
  }
  const double* const P = jt != k ? V : D;
  for (int it = (int)blockIdx.y; it < nt; it += (int)gridDim.y) {
    const int rt = row_tile(it);
    const long long i0 = (long long)rt * NB;
    double2 v[4][2];
    if (rt == k) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) v[i][j] = *reinterpret_cast<const double2*>(P + gj_row(i) * PITCH + gj_col(j));
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          v[i][j] = jt == k ? make_double2(0.0, 0.0)
                            : *reinterpret_cast<const double2*>(A + (i0 + gj_row(i)) * np + j0 + gj_col(j));
      if (it != (int)blockIdx.y) {
        __syncthreads();  // Cs has been read
        gj_load(Cs, C + i0 * NB, NB);
        gj_wait();
      }
      gj_mul(Cs, P, acc);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          v[i][j].x -= acc[i][j][0];
          v[i][j].y -= acc[i][j][1];
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int r = gj_row(i), c = gj_col(j);
        *reinterpret_cast<double2*>(A + (i0 + r) * np + j0 + c) = v[i][j];
        if (jt == k + 1) *reinterpret_cast<double2*>(C1 + (i0 + r) * NB + c) = v[i][j];
        if (rt == k + 1) *reinterpret_cast<double2*>(R1 + (long long)r * np + j0 + c) = v[i][j];
      }
    if (rt == k + 1 && jt == k + 1) {  // the next diagonal block
      __syncthreads();  // Cs has been read
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) *reinterpret_cast<double2*>(Cs + gj_row(i) * PITCH + gj_col(j)) = v[i][j];
      __syncthreads();
      gj_invert(Cs, PITCH, F, scl, Dg1);
    }
  }
}

// Inverse with partial pivoting of up to kPivotMax unknowns, in one launch: a cluster
// of eight CTAs holds the matrix in registers, CTA k a panel of columns, a warp up to
// CPW of them, lane l the rows l, l + 32, ...
//
// In-place Gauss-Jordan: column c of the identity is never stored.  Rows are not
// exchanged: step c takes the unused row with the largest |a[., c]| (to 11 bits, the
// lowest such row when equal) and remembers it, and the inverse is written through that
// permutation.  A pivot row is not divided by its pivot until the end (its later
// updates are linear in it), so an update is one fused multiply-add per entry, with a
// multiplier of 0 in the pivot row.  What bounds it is the chain of n steps and their
// instructions.  A pivot search needs one column only, so the CTA that owns a panel
// runs the panel's steps by itself (one __syncthreads each), keeping the multipliers
// of every step in shared memory; one cluster barrier later the other CTAs copy them
// (through global memory, W: seven CTAs reading one's shared memory at once took five
// times as long) and apply the whole panel to their own columns without any barrier.  Measured at
// 162 unknowns (the coarsest level at 8^3 and 64^3): 173 us; with a barrier of
// the cluster per step 551 us, dividing at once and selecting the pivot row in every
// update 286 us, the copies from the owner's shared memory 224 us; the host's inverse with its two copies took 600-750 us.
constexpr int PC = 8, PT = 256;  // CTAs of the cluster, threads of a CTA

inline int pivot_cols(int n) { return (n + PC - 1) / PC; }
inline size_t pivot_smem(int n) { return (size_t)2 * pivot_cols(n) * n * sizeof(double); }

template <typename T, int RR, int CPW>
__global__ void __cluster_dims__(PC, 1, 1) __launch_bounds__(PT)
pivot_inverse_kernel(int cp, int nnzb, const int* __restrict__ br, const int* __restrict__ cl, const T* __restrict__ val,
                     int n, double* W, T* __restrict__ inv) {
  constexpr int NW = PT / 32, CMAX = NW * CPW;
  extern __shared__ __align__(16) double pvm[];
  __shared__ double ipv[2][CMAX];  // 1 / pivot of the own panel's steps, of a copied panel's
  __shared__ int prow[2][CMAX];    // and their rows
  __shared__ double wmax[NW];      // largest diagonal entry that a warp has seen
  __shared__ double rowip[32 * RR];  // 1 / pivot of each row
  __shared__ int perm[32 * RR], pos[32 * RR];
  const int rank = (int)(blockIdx.x % PC), t = threadIdx.x, w = t >> 5, lane = t & 31;
  double* const F = pvm;                   // multipliers of the own panel, [step][row]
  double* const G = pvm + (size_t)cp * n;  // a copied panel's
  const int j0 = rank * cp, ncol = max(0, min(cp, n - j0));
  auto barrier = []() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  };
  auto remote = [](const void* p, int cta) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(cta));
    return r;
  };
  // ordered with the barriers (both volatile), free to be in flight together
  auto get = [](uint32_t a) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
  };
  // ---- own columns from the 6 x 6 blocks (br, cl: row and column of each), through
  // shared memory; a row with no entry gets a unit diagonal ----
  for (int e = t; e < ncol * n; e += PT) F[e] = 0.0;
  for (int i = t; i < n; i += PT) pos[i] = 0;  // until the elimination: whether row i has an entry
  __syncthreads();
  double dm = 0.0;
#pragma unroll 4
  for (int e = t; e < nnzb * 36; e += PT) {
    const int k = e / 36, rc = e - 36 * k, i = br[k] * 6 + rc / 6, j = cl[k] * 6 + rc % 6;
    const double v = (double)val[e];
    if (v != 0.0) pos[i] = 1;
    if (j == i) dm = fmax(dm, fabs(v));
    if (j >= j0 && j < j0 + ncol) F[(size_t)(j - j0) * n + i] = v;
  }
  __syncthreads();
  for (int i = t; i < n; i += PT)
    if (!pos[i]) {
      dm = fmax(dm, 1.0);
      if (i >= j0 && i < j0 + ncol) F[(size_t)(i - j0) * n + i] = 1.0;
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dm = fmax(dm, __shfl_xor_sync(0xffffffffu, dm, o));
  if (lane == 0) wmax[w] = dm;
  __syncthreads();
  double a[CPW][RR];
#pragma unroll
  for (int m = 0; m < CPW; ++m)
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      const int q = w + NW * m, i = lane + 32 * r;
      a[m][r] = (q < ncol && i < n) ? F[(size_t)q * n + i] : 0.0;
    }
  double scl = 0.0;
  for (int q = 0; q < NW; ++q) scl = fmax(scl, wmax[q]);
  const double floor_abs = 1e-14 * fmax(scl, 1e-300);
  unsigned used = 0;  // of this lane's rows, bit r
  // Step with multipliers f (the pivot row's entry counts as 0), pivot row p, 1 / pivot ip
  // on the warp's columns but `skip`, which becomes the inverse's.
  auto apply = [&](const double* f, int p, double ip, int skip) {
    const int pr = p >> 5, pl = p & 31;
    double fr[RR], x[CPW];
#pragma unroll
    for (int m = 0; m < CPW; ++m) {
      double e = a[m][0];
#pragma unroll
      for (int r = 1; r < RR; ++r) e = pr == r ? a[m][r] : e;
      x[m] = __shfl_sync(0xffffffffu, e, pl) * ip;
    }
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      fr[r] = lane + 32 * r < n ? f[lane + 32 * r] : 0.0;
      if (lane + 32 * r == p) fr[r] = 0.0;
    }
#pragma unroll
    for (int m = 0; m < CPW; ++m) {
      if (m == skip) {
#pragma unroll
        for (int r = 0; r < RR; ++r) a[m][r] = lane + 32 * r == p ? 1.0 : -fr[r] * ip;
      } else {
#pragma unroll
        for (int r = 0; r < RR; ++r) a[m][r] = fma(-fr[r], x[m], a[m][r]);
      }
    }
    if (lane == pl) used |= 1u << pr;
  };
  // The warp that holds step s's column publishes it and its choice of the pivot: the
  // largest |v| by the upper 23 bits of the number (sign aside: 2^-11 of it; a NaN is
  // above all) and among equals the lowest row, in one 32-bit maximum.
  auto publish = [&](const double (&v)[RR], int s) {
    unsigned key = 0u;
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      const int i = lane + 32 * r;
      const unsigned h = ((unsigned)__double2hiint(v[r]) & 0x7ffffe00u) | (unsigned)(511 - i);
      if (i < n && !((used >> r) & 1u)) key = max(key, h);
      if (i < n) {
        F[(size_t)s * n + i] = v[r];
        W[(size_t)(j0 + s) * n + i] = v[r];
      }
    }
    key = __reduce_max_sync(0xffffffffu, key);
    if (lane == 0) prow[0][s] = 511 - (int)(key & 511u);
  };
  __syncthreads();  // F and pos have been read
  for (int k = 0; k < PC; ++k) {
    const int steps = max(0, min(cp, n - k * cp));
    if (k == rank) {
      for (int s = 0; s < steps; ++s) {
        int skip = -1;
        if (w == s % NW) {
          skip = s / NW;
#pragma unroll
          for (int m = 0; m < CPW; ++m)
            if (m == skip) publish(a[m], s);
        }
        __syncthreads();
        const int p = prow[0][s];
        double pv = F[(size_t)s * n + p];
        if (fabs(pv) < floor_abs) pv = (pv >= 0 ? 1.0 : -1.0) * floor_abs;
        const double ip = 1.0 / pv;
        if (threadIdx.x == 0) ipv[0][s] = ip;
        apply(F + (size_t)s * n, p, ip, skip);
      }
    }
    barrier();  // the panel's steps are in its CTA's shared memory
    if (k != rank) {
      const uint32_t ip = remote(ipv[0], k), pr = remote(prow[0], k);
      const double* f = W + (size_t)k * cp * n;
      for (int e0 = t; e0 < steps * n; e0 += 8 * PT) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (e0 + u * PT < steps * n) v[u] = __ldcg(f + e0 + u * PT);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (e0 + u * PT < steps * n) G[e0 + u * PT] = v[u];
      }
      if (t < steps) {
        ipv[1][t] = get(ip + 8u * (uint32_t)t);
        int v;
        asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(pr + 4u * (uint32_t)t));
        prow[1][t] = v;
      }
      __syncthreads();
      for (int s = 0; s < steps; ++s) apply(G + (size_t)s * n, prow[1][s], ipv[1][s], -1);
    }
    if (t < steps) {
      const int o = k == rank ? 0 : 1, p = prow[o][t];
      perm[k * cp + t] = p;
      pos[p] = k * cp + t;
      rowip[p] = ipv[o][t];
    }
    __syncthreads();  // G and prow[1] may be overwritten
  }
#pragma unroll
  for (int m = 0; m < CPW; ++m)
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      const int q = w + NW * m, i = lane + 32 * r;
      if (q < ncol && i < n) inv[(long long)pos[i] * n + perm[j0 + q]] = (T)(a[m][r] * rowip[i]);
    }
  barrier();  // no CTA leaves while another may read its shared memory
}

// out (n x n, stride n) = the leading n x n block of A (stride np), in precision T.
template <typename T>
__global__ void dense_out_kernel(int n, int np, const double* __restrict__ A, T* __restrict__ out) {
  const long long nn = (long long)n * n;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nn; e += (long long)gridDim.x * blockDim.x)
    out[e] = (T)A[(e / n) * np + e % n];
}

}  // namespace

long long dense_inverse_work_doubles(int n) {
  const int np = (n + NB - 1) / NB * NB;
  return (long long)np * np + 4 * (long long)np * NB + 2 * NB * NB + 8;
}

// inv (n x n, row-major, precision T) = inverse of the coarsest operator given by
// its 6 x 6 block pattern (rp, cl: device) and values.  work holds
// dense_inverse_work_doubles(n) doubles.  The matrix is padded to a multiple of
// NB with identity rows, which leaves the inverse of the leading block unchanged.
template <typename T>
void dense_coarse_inverse(int nbrow, const int* rp, const int* cl, const T* val, int n, double* work, T* inv,
                          cudaStream_t st) {
  const int np = (n + NB - 1) / NB * NB;
  double* A = work;
  const long long slab = (long long)np * NB;
  double* const C = work + (long long)np * np;  // two each, taken in turn
  double* const R = C + 2 * slab;
  double* const Dg = R + 2 * slab;
  double* const scl = Dg + 2 * NB * NB;
  const int step_sm = 3 * NB * PITCH * (int)sizeof(double), nt = np / NB;
  cudaFuncSetAttribute(gj_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, step_sm);
  cudaMemsetAsync(A, 0, (size_t)np * np * sizeof(double), st);
  count_launch();
  bsr6_to_dense_kernel<T><<<1024, 256, 0, st>>>(nbrow, rp, cl, val, np, A);
  count_launch();
  dense_fix_rows_kernel<<<(np + 7) / 8, 256, 0, st>>>(np, A);
  count_launch();
  dense_diag_max_kernel<<<1, 1024, 0, st>>>(np, A, scl);
  count_launch();
  gj_start_kernel<<<nt, GTHREADS, 0, st>>>(np, A, C, R, Dg, scl);
  // all CTAs run at once, two on an SM, so that the one with the next diagonal block
  // does not wait for a place
  const dim3 grid(nt, std::max(1, std::min(nt, 2 * 148 / nt)));
  int chain = 0;
  for (int k = 0; k < nt; ++k) {
    const int a = k & 1, b = a ^ 1;
    launch(Queue(st, &chain), gj_step_kernel, grid, GTHREADS, step_sm, np, k, A, C + a * slab, R + a * slab,
           Dg + a * NB * NB, C + b * slab, R + b * slab, Dg + b * NB * NB, scl);
  }
  count_launch();
  dense_out_kernel<T><<<2048, 256, 0, st>>>(n, np, A, inv);
}

// NMAX: the largest size of the instantiation, whose shared memory is the kernel's limit
// for every launch of it (the limit is the process's: with a launch's own size in it, another
// context's launch in between could meet a smaller one).
template <typename T, int RR, int CPW, int NMAX>
static cudaError_t pivot_launch(int nnzb, const int* br, const int* cl, const T* val, int n, double* work, T* inv, cudaStream_t st) {
  auto* kern = pivot_inverse_kernel<T, RR, CPW>;
  static_assert(NMAX <= 32 * RR && (NMAX + PC - 1) / PC <= CPW * (PT / 32), "rows and columns fit");
  const cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pivot_smem(NMAX));
  if (e != cudaSuccess) return e;
  count_launch();
  kern<<<PC, PT, pivot_smem(n), st>>>(pivot_cols(n), nnzb, br, cl, val, n, work, inv);
  return cudaGetLastError();
}
// Rows per lane and columns per warp: six and three up to 192 unknowns, seven and four up
// to 224, ten and five up to kPivotMax (set-up with 216 unknowns 0.55 ms; 0.71 ms with ten
// and five).
template <typename T>
cudaError_t pivot_inverse(int nnzb, const int* br, const int* cl, const T* val, int n, double* work, T* inv,
                          cudaStream_t st) {
  if (n <= 192) return pivot_launch<T, 6, 3, 192>(nnzb, br, cl, val, n, work, inv, st);
  if (n <= 224) return pivot_launch<T, 7, 4, 224>(nnzb, br, cl, val, n, work, inv, st);
  return pivot_launch<T, 10, 5, kPivotMax>(nnzb, br, cl, val, n, work, inv, st);
}
template cudaError_t pivot_inverse<float>(int, const int*, const int*, const float*, int, double*, float*, cudaStream_t);
template cudaError_t pivot_inverse<double>(int, const int*, const int*, const double*, int, double*, double*,
                                           cudaStream_t);

template void dense_coarse_inverse<float>(int, const int*, const int*, const float*, int, double*, float*,
                                          cudaStream_t);
template void dense_coarse_inverse<double>(int, const int*, const int*, const double*, int, double*, double*,
                                           cudaStream_t);

}  // namespace pfem
