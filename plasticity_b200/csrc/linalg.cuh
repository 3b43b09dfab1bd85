// linalg.cuh -- declarations of the solver-side kernels (linalg.cu).
#pragma once
#include <algorithm>
#include "pfem_internal.h"

namespace pfem {

// Where a kernel of the solver's cycle goes.  chain (when not null): the kernels after
// the first are launched before their predecessor on the stream has finished
// (programmatic dependent launch); *chain counts them.  Only
// kernels that call pdl_wait() before they touch anything a predecessor writes take
// it, and only where matrices, prolongators and block inverses are not being written:
// they are read ahead of that wait.  Grids of more than four CTAs per SM (kChainGrid)
// are launched the plain way: their CTAs would take the slots of the running kernel's
// last ones and wait there.  The cycle in its graph, plain / all chained / this rule:
// 18.6 / 16.5 / 15.6 us at 8^3, 68 / 72 / 64 at 32^3, 104 / 109 / 100 at 40^3,
// 337 / 356 / 325 at 64^3 (before the transfers there were streamed: 293 since).
constexpr int kChainGrid = 4 * 148;
struct Queue {
  cudaStream_t st = nullptr;
  int* chain = nullptr;
  Queue(cudaStream_t s) : st(s) {}
  Queue(cudaStream_t s, int* c) : st(s), chain(c) {}
};
template <typename... K, typename... A>
inline void launch(const Queue& q, void (*kern)(K...), dim3 grid, int block, size_t smem, A... args) {
  count_launch();
  if (!q.chain || (*q.chain)++ == 0 || grid.x * grid.y > (unsigned)kChainGrid) {
    kern<<<grid, block, smem, q.st>>>(static_cast<K>(args)...);
    return;
  }
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = q.st;
  cudaLaunchAttribute a[1];
  a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = a;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kern, static_cast<K>(args)...);
}
// Let the next kernel of the stream start its part before pdl_wait(); wait for the
// previous ones' results.  Neither does anything in a kernel launched the plain way.
__device__ __forceinline__ void pdl_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Device copy of the frozen boundary conditions plus the precomputed list of
// tangent entries that Dirichlet imposition reads and overwrites.
struct BcDev {
  int nbc = 0;                 // constrained dofs (deduplicated)
  int* dofs = nullptr;         // 0-based dof
  double* vals = nullptr;
  uint8_t* ramp = nullptr;
  double* fn = nullptr;        // ndof nodal forces at lambda = 1, 0 on constrained dofs
  int nrows = 0;               // free rows with entries in constrained columns
  int* rows = nullptr;
  int* rptr = nullptr;         // nrows+1
  long long* rpos = nullptr;   // scalar value index into the block-CSR value array
  int* rbc = nullptr;          // constrained column (index into dofs)
  long long nzero = 0;         // entries in constrained rows
  long long* zpos = nullptr;
  uint8_t* zone = nullptr;     // 1 on the diagonal of a constrained row
};

// y = A x; with part, also the partials of x.y (their count is returned).
template <typename T> int bsr_spmv(const BsrMat<T>& A, const T* x, T* y, Queue q, T* part = nullptr);
template <typename T> void bsr_residual(const BsrMat<T>& A, const T* x, const T* b, T* r, Queue q);
template <typename T> void bsr_cheb_step(const BsrMat<T>& A, const T* dinv, const T* d, T* r, T* x, cudaStream_t st);
// Degree-2 Chebyshev in one pass: x (=, or += unless zero) c2 d0 + c1 (r0 - Dinv A d0);
// co holds the level's scalars on the device.  With part (not zero): also the partials
// of b.x (count returned).
template <typename T> int bsr_cheb2(const BsrMat<T>& A, const T* dinv, const T* d0, const T* r0, T* x, bool zero,
                                    const T* co, Queue q, const T* b = nullptr, T* part = nullptr);
// r = Dinv (b - A x), d = co[CO_ITH] r.
template <typename T> void bsr_residual_precond(const BsrMat<T>& A, const T* dinv, const T* x, const T* b, T* r,
                                                T* d, const T* co, Queue q);
// res = b - A x, r = Dinv res, d = co[CO_ITH] r: a residual and the smoother's start on it.
template <typename T> void bsr_residual_start(const BsrMat<T>& A, const T* dinv, const T* x, const T* b, T* res, T* r,
                                              T* d, const T* co, Queue q);
// Power iteration: y = Dinv A (co[CO_INV] x); co[CO_INV] = 1 / |v|, with finish also the
// level's other scalars from |v|.  part: 2048; ticket: zero between launches.
template <typename T> void bsr_power_step(const BsrMat<T>& A, const T* dinv, const T* x, T* y, const T* co,
                                          cudaStream_t st);
template <typename T> void power_norm(long long n, const T* v, T* part, unsigned* ticket, bool finish, T* co,
                                      cudaStream_t st);
// r = Dinv v, d = *scale r (scale on the device).
template <typename T> void blockdiag_apply(int nbrow, int bs, const T* dinv, const T* v, T* r, const T* scale, T* d, Queue q);
template <typename T> void blockdiag_invert(const BsrMat<T>& A, T* dinv, cudaStream_t st);
template <typename T> void dot(long long n, const T* a, const T* b, T* out, T* part, cudaStream_t st, bool take_sqrt);
template <typename T> void fill(long long n, T* x, T v, cudaStream_t st);
template <typename T> void axpby(long long n, T a, const T* x, T b, T* y, cudaStream_t st);
// PCG updates with the dot products' final sums inside (deterministic):
// cg_p_fused: rz = sum(part), p = z + (rz / sc[0]) p, sc[2] = rz;
// cg_xr_fused: alpha = sc[2] / sum(part_pq), x += alpha p, r -= alpha q, sr = Dinv r,
// sd = co[CO_ITH] sr (the smoother's start on the next residual), sc[0] = sc[2], and
// from the last CTA |r| and the loop condition (CgLoop).
constexpr int kMaxPartials = 4096;
struct CgLoop {
  cudaGraphConditionalHandle h;
  const double* ctl;    // [1] iteration cap, [2] absolute threshold
  int* state;           // [0] iterations, [1] converged
  unsigned* ticket;     // zero between launches
};
// Partials of a.b in dot's order (count returned).
template <typename T> int dot_partials(long long n, const T* a, const T* b, T* part, const Queue& q);
template <typename T> void cg_p_fused(long long n, const T* part, int np, T* sc, const T* z, T* p, Queue q);
template <typename T> void cg_xr_fused(int nbrow, const T* part_pq, int np, T* sc, const T* p, const T* q, T* x,
                                       T* r, const T* dinv, const T* co, T* sr, T* sd, double* part_rr,
                                       const CgLoop& loop, Queue qu);
// BiCGStab updates, with the smoother's start on p and on s (sr, sd as above):
// bicg_p: p = r + beta (p - omega v); bicg_s: alpha = sc[0] / sum(part), s = r - alpha v;
// bicg_xr: omega from the dot products of t with s and itself, x += alpha ph + omega sh,
// r = s - omega t, the next rho and the loop condition (part: four of kMaxPartials).  The
// dot products are dot's.
template <typename T> void bicg_p(int nbrow, const T* sc, const T* r, const T* v, T* p, const T* dinv, const T* co,
                                  T* sr, T* sd, Queue q);
template <typename T> void bicg_s(int nbrow, const T* part, int np, T* sc, const T* r, const T* v, T* s,
                                  const T* dinv, const T* co, T* sr, T* sd, Queue q);
template <typename T> void bicg_xr(long long n, T* sc, const T* ph, const T* sh, const T* s, const T* t, const T* rh,
                                   T* x, T* r, T* part, const CgLoop& loop, Queue q);
template <typename A, typename B> void convert(long long n, const A* a, B* b, double s, cudaStream_t st);
template <typename T> void add_to_double(long long n, const T* x, double* U, cudaStream_t st);
// Impose the constraints on K and R at lambda, subtract the load, *rnorm = |R| (device).
// part: 2048 doubles; ticket: zero between launches.
template <typename KT> void impose_dirichlet(const BcDev& bc, long long ndof, double lam, const double* U, KT* K,
                                             double* R, double* part, unsigned* ticket, double* rnorm, cudaStream_t st);
void bc_apply(const BcDev& bc, double lam, double* U, cudaStream_t st);
template <typename T> void dense_mv(int n, const T* M, const T* b, T* y, Queue q);
template <typename T> void sa_setup_level(const AmgLevel<T>& v, T* cval, int nnzC, cudaStream_t st);
// bc = P^T r; with next, also the smoother's start on bc there (next->r, next->d).
template <typename T> void sa_restrict(const AmgLevel<T>& v, const T* r, T* bc, const AmgLevel<T>* next, Queue q);
template <typename T> void sa_prolong(const AmgLevel<T>& v, const T* xc, T* x, Queue q);
template <typename T> void sa_prolong2(const AmgLevel<T>& v, const T* xc, const T* xc2, T* x, Queue q);
// Dense inverse of the coarsest operator (dense.cu): its 6 x 6 block pattern
// (device rp, cl) and values in, the n x n row-major inverse in precision T out;
// work holds dense_inverse_work_doubles(n) doubles.
// Up to kPivotMax unknowns pivot_inverse takes its place: the same with partial
// pivoting; work holds dense_inverse_work_doubles(n) doubles as well.
constexpr int kPivotMax = 300;
// br, cl: block row and column of each of the nnzb blocks.
template <typename T> cudaError_t pivot_inverse(int nnzb, const int* br, const int* cl, const T* val, int n,
                                                double* work, T* inv, cudaStream_t st);
long long dense_inverse_work_doubles(int n);
template <typename T> void dense_coarse_inverse(int nbrow, const int* rp, const int* cl, const T* val, int n,
                                                double* work, T* inv, cudaStream_t st);

}  // namespace pfem
