// Parameters of the persistent coarse-grid V-cycle kernel (kernels_coarse.cu).
#pragma once

#include "tpo_internal.h"

namespace tpo {

constexpr int kMaxChebDegree = 8;
constexpr int kMaxCoarseLevels = 8;
// levels with at most this many nodes run inside the persistent kernel
constexpr int64_t kPersistentMaxNodes = 65536;

// Every vector below holds `nb` columns (CoarseCycle::nb), component by
// component: component c of node n of column j at (3 j + c) * nn + n; A and
// dinv are shared by the columns.  CTA s of the grid owns the nodes s * npc
// .. (s + 1) * npc - 1.
template <typename T>
struct CoarseLevel {
  int dims[3];
  int nn;
  int npc, npcp;   // nodes per CTA, rounded up to a multiple of 4
  int gres;        // neighbour rows (of 9) whose blocks stay in shared memory
  int smem;        // byte offset of those in the kernel's shared memory
  // the Galerkin stencil by CTA: block nb, entry rs of node s * npc + i at
  // A[(s * 243 + nb * 9 + rs) * npcp + i]
  const T *A;
  const T *dinv;   // 1 / (lambda diag), 3 n + c
  T *b;            // right-hand side (restricted residual of the parent)
  T *xpre;         // pre-smoothed iterate, then + P x_child
  T *xout;         // post-smoothed result (read by the parent)
  T *r, *d0, *d1;  // Chebyshev residual and ping-pong directions; d0 holds
                   // inv_theta D^-1 b on entry (written with b)
  T *res;          // b - A xpre
  T inv_theta;
  T c1[kMaxChebDegree], c2[kMaxChebDegree];
  int deg;
};

// one phase of the cycle
struct CoarseOp {
  int8_t kind;    // CoarseKind
  int8_t level;
  int8_t k;       // Chebyshev step (its c1, c2)
  int8_t flip;    // kOpFirst, kOpStep: the direction goes from d1 to d0
};
enum CoarseKind : int8_t {
  kOpFirst,     // from x = d0: the first Chebyshev step
  kOpStart,     // degree 1: x = d0
  kOpStep,      // a further step on xpre
  kOpRes,       // res = b - A xpre
  kOpRestrict,  // b of the next level = P^T res, and its d0
  kOpDense,     // the coarsest solve
  kOpProlong,   // xpre += P x of the next level
  kOpPost,      // post-smoothing from xpre: d0, xout
  kOpPostStep   // a further step on xout
};
constexpr int kMaxCoarseOps = kMaxCoarseLevels * (2 * kMaxChebDegree + 4) + 1;

template <typename T>
struct CoarseCycle {
  int nlev;                          // stencil levels handled in the kernel
  int nb;                            // columns (1, 2, 4 or 8)
  int chunk;                         // nodes whose partial sums are held at
                                     // once (a multiple of 32; set by the launch)
  CoarseLevel<T> lev[kMaxCoarseLevels];
  int nop;                           // the phases, in order (set by the launch)
  CoarseOp op[kMaxCoarseOps];
  const double *Ainv;                // dense inverse of the coarsest operator
  int64_t nc;                        // coarsest dof count
  int cdims[3];                      // coarsest nodes per dimension
  T *bc, *xc;                        // coarsest right-hand side / solution,
                                     // dof order (column stride nc)
  unsigned int *bar;                 // grid-barrier counter (zero between
                                     // launches)
  double *fault;                     // set to 1 when a wait runs out
};

template <typename T>
cudaError_t launch_coarse_cycle(CoarseCycle<T> P, cudaStream_t s);

}  // namespace tpo
