// dense.cu -- dense inverse of the coarsest AMG operator, on the device.
//
// The smoothed-aggregation hierarchy ends in a dense solve (the reference's
// AlgebraicMultigrid.jl ends its hierarchy in a direct coarse solve as well,
// Solver.jl:136-154).  The coarsest operator (6 x 6 blocks, a few thousand
// unknowns) is expanded to a dense FP64 matrix and inverted in place by blocked
// Gauss-Jordan elimination; the cycle then applies the inverse as one dense
// matrix-vector product.  Per panel of NB columns K:
//   1. diagonal kernel (one CTA): Dg = A[K,K]^{-1} by Gauss-Jordan in shared memory;
//   2. panel kernel: the panel rows outside the diagonal block, A[K,j] <- Dg A[K,j],
//      and a copy C = A[i,K] of the panel columns of the other rows;
//   3. update kernel: A[i, j] -= C[i, :] P[:, j] for every row i outside the panel
//      (P the scaled panel rows, Dg in the panel's own columns), with the panel's
//      own columns starting from 0, which turns them into -C Dg; the tile that
//      holds the diagonal block writes Dg there.
// Every kernel reads only what the previous one finished writing, and A[K,K] is
// read only by the diagonal kernel, so no CTA sees a block half replaced.
// No row exchanges: the Galerkin operator of the (Dirichlet-imposed) tangent of a
// large mesh is close to symmetric positive definite; a pivot below 1e-14 of the
// largest diagonal entry is replaced by that floor.  Coarsest levels of up to
// kPivotMax unknowns take pivot_inverse_kernel, which chooses its pivots.
#include <cstdint>

#include "linalg.cuh"

namespace pfem {
namespace {

constexpr int NB = 64;      // panel width
constexpr int TR_ = 128;    // update tile rows
constexpr int TC_ = 64;     // update tile columns

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

// Dg = A[K,K]^{-1}: in-place Gauss-Jordan on the NB x NB diagonal block, one CTA of
// eight warps with the block in registers: warp w holds the columns w, w + 8, ..., lane
// l the rows l and l + 32.  What bounds it is the chain of 64 steps, so each has one
// __syncthreads: the column's warp publishes it as the multipliers, every warp takes the
// pivot from there.  As in pivot_inverse_kernel a row is divided by its pivot at the
// end.  19.7 us; with the block in shared memory and five barriers per step 60 us.
__global__ void __launch_bounds__(256) gj_diag_kernel(int n, int kb, const double* __restrict__ A,
                                                      double* __restrict__ Dg, const double* __restrict__ scl) {
  __shared__ double F[2][NB];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double a[8][2];
#pragma unroll
  for (int m = 0; m < 8; ++m)
#pragma unroll
    for (int r = 0; r < 2; ++r) a[m][r] = A[(long long)(kb + lane + 32 * r) * n + kb + w + 8 * m];
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

// Panel step kb.  CTAs [0, ncb): 64 panel-row columns each, A[K, j] <- Dg A[K, j]
// for j outside K (the 64 x 64 slab staged in shared memory; a thread computes four
// rows of four columns, 16 apart: eight reads for 16 multiply-adds).  CTAs [ncb, ...): C[i, :] = A[i, K] for rows i
// outside K, a warp per row.
__global__ void __launch_bounds__(256) gj_panel_kernel(int n, int kb, int ncb, double* __restrict__ A,
                                                       double* __restrict__ C, const double* __restrict__ Dg) {
  extern __shared__ __align__(16) double psm[];
  const int t = threadIdx.x;
  if ((int)blockIdx.x >= ncb) {
    const int w = t >> 5, lane = t & 31;
    const int i = ((int)blockIdx.x - ncb) * 8 + w;
    if (i < n && (i < kb || i >= kb + NB)) {
      C[(long long)i * NB + lane] = A[(long long)i * n + kb + lane];
      C[(long long)i * NB + 32 + lane] = A[(long long)i * n + kb + 32 + lane];
    }
    return;
  }
  const int j0 = (int)blockIdx.x * 64;
  if (j0 == kb) return;  // the diagonal block's columns: Dg, written by the update kernel
  double(*D)[NB + 1] = reinterpret_cast<double(*)[NB + 1]>(psm);
  double(*V)[65] = reinterpret_cast<double(*)[65]>(psm + NB * (NB + 1));
  for (int e = t; e < NB * NB; e += 256) D[e / NB][e % NB] = Dg[e];
  for (int e = t; e < NB * 64; e += 256) {
    const int r = e / 64, c = e % 64, j = j0 + c;
    V[r][c] = j < n ? A[(long long)(kb + r) * n + j] : 0.0;
  }
  __syncthreads();
  const int c = t & 15, q = t >> 4;
  double out[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int u = 0; u < 4; ++u) out[r][u] = 0.0;
#pragma unroll 8
  for (int s = 0; s < NB; ++s) {
    double d[4], v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) d[r] = D[q * 4 + r][s];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = V[s][c + 16 * u];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int u = 0; u < 4; ++u) out[r][u] += d[r] * v[u];
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = j0 + c + 16 * u;
      if (j < n) A[(long long)(kb + q * 4 + r) * n + j] = out[r][u];
    }
}

// Trailing update of step kb over TR_ x TC_ tiles; rows of the panel are final.
// Thread (rg, cg) holds rows rg*8 .. +7 and columns cg + 16 b, b < 4.
__global__ void __launch_bounds__(256, 2) gj_update_kernel(int n, int kb, double* __restrict__ A,
                                                           const double* __restrict__ C,
                                                           const double* __restrict__ Dg) {
  extern __shared__ __align__(16) double usm[];
  double(*Cs)[NB + 1] = reinterpret_cast<double(*)[NB + 1]>(usm);              // TR_ x NB
  double(*Ps)[TC_ + 1] = reinterpret_cast<double(*)[TC_ + 1]>(usm + TR_ * (NB + 1));  // NB x TC_
  const int i0 = (int)blockIdx.y * TR_, j0 = (int)blockIdx.x * TC_;
  const int t = threadIdx.x;
  for (int e = t; e < TR_ * NB; e += 256) {
    const int r = e / NB, s = e % NB, i = i0 + r;
    Cs[r][s] = (i < n && (i < kb || i >= kb + NB)) ? C[(long long)i * NB + s] : 0.0;
  }
  const bool diag_cols = j0 == kb;  // TC_ == NB and both are multiples of NB: the panel is one column tile
  for (int e = t; e < NB * TC_; e += 256) {
    const int s = e / TC_, c = e % TC_, j = j0 + c;
    Ps[s][c] = j >= n ? 0.0 : diag_cols ? Dg[s * NB + c] : A[(long long)(kb + s) * n + j];
  }
  // the tile holding the diagonal block writes it (no other CTA reads it from A)
  if (diag_cols && kb >= i0 && kb < i0 + TR_)
    for (int e = t; e < NB * NB; e += 256) A[(long long)(kb + e / NB) * n + kb + e % NB] = Dg[e];
  __syncthreads();
  const int rg = t / 16, cg = t % 16;
  double acc[8][4];
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
#pragma unroll 4
  for (int s = 0; s < NB; ++s) {
    double cv[8], pv[4];
#pragma unroll
    for (int a = 0; a < 8; ++a) cv[a] = Cs[rg * 8 + a][s];
#pragma unroll
    for (int b = 0; b < 4; ++b) pv[b] = Ps[s][cg + 16 * b];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] += cv[a] * pv[b];
  }
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const int i = i0 + rg * 8 + a;
    if (i >= n || (i >= kb && i < kb + NB)) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int j = j0 + cg + 16 * b;
      if (j >= n) continue;
      double* p = A + (long long)i * n + j;
      const double old = diag_cols ? 0.0 : *p;
      *p = old - acc[a][b];
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
  return (long long)np * np + (long long)np * NB + NB * NB + 8;
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
  double* C = work + (long long)np * np;
  double* Dg = C + (long long)np * NB;
  double* scl = Dg + NB * NB;
  const size_t panel_sm = (size_t)(NB * (NB + 1) + NB * 65) * sizeof(double);
  const size_t update_sm = (size_t)(TR_ * (NB + 1) + NB * (TC_ + 1)) * sizeof(double);
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(gj_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)panel_sm);
    cudaFuncSetAttribute(gj_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)update_sm);
    attr = true;
  }
  cudaMemsetAsync(A, 0, (size_t)np * np * sizeof(double), st);
  count_launch();
  bsr6_to_dense_kernel<T><<<1024, 256, 0, st>>>(nbrow, rp, cl, val, np, A);
  count_launch();
  dense_fix_rows_kernel<<<(np + 7) / 8, 256, 0, st>>>(np, A);
  count_launch();
  dense_diag_max_kernel<<<1, 1024, 0, st>>>(np, A, scl);
  const int ncb = np / 64, nrb = (np + 7) / 8;
  const dim3 ug((np + TC_ - 1) / TC_, (np + TR_ - 1) / TR_);
  for (int kb = 0; kb < np; kb += NB) {
    count_launch();
    gj_diag_kernel<<<1, 256, 0, st>>>(np, kb, A, Dg, scl);
    count_launch();
    gj_panel_kernel<<<ncb + nrb, 256, panel_sm, st>>>(np, kb, ncb, A, C, Dg);
    count_launch();
    gj_update_kernel<<<ug, 256, update_sm, st>>>(np, kb, A, C, Dg);
  }
  count_launch();
  dense_out_kernel<T><<<2048, 256, 0, st>>>(n, np, A, inv);
}

template <typename T, int RR, int CPW>
static cudaError_t pivot_launch(int nnzb, const int* br, const int* cl, const T* val, int n, double* work, T* inv, cudaStream_t st) {
  auto* kern = pivot_inverse_kernel<T, RR, CPW>;
  const size_t sm = pivot_smem(n);
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  count_launch();
  kern<<<PC, PT, sm, st>>>(pivot_cols(n), nnzb, br, cl, val, n, work, inv);
  return cudaGetLastError();
}
// Rows per lane and columns per warp: six and three up to 192 unknowns, seven and four up
// to 224, ten and five up to kPivotMax.
template <typename T>
cudaError_t pivot_inverse(int nnzb, const int* br, const int* cl, const T* val, int n, double* work, T* inv,
                          cudaStream_t st) {
  static_assert(kPivotMax <= 32 * 10 && (kPivotMax + PC - 1) / PC <= 5 * (PT / 32), "rows and columns fit");
  if (n <= 192) return pivot_launch<T, 6, 3>(nnzb, br, cl, val, n, work, inv, st);
  if (n <= 224) return pivot_launch<T, 7, 4>(nnzb, br, cl, val, n, work, inv, st);
  return pivot_launch<T, 10, 5>(nnzb, br, cl, val, n, work, inv, st);
}
template cudaError_t pivot_inverse<float>(int, const int*, const int*, const float*, int, double*, float*, cudaStream_t);
template cudaError_t pivot_inverse<double>(int, const int*, const int*, const double*, int, double*, double*,
                                           cudaStream_t);

template void dense_coarse_inverse<float>(int, const int*, const int*, const float*, int, double*, float*,
                                          cudaStream_t);
template void dense_coarse_inverse<double>(int, const int*, const int*, const double*, int, double*, double*,
                                           cudaStream_t);

}  // namespace pfem
