// Dense inverse of the coarsest-level operator by blocked symmetric sweeps
// (Gauss-Jordan elimination without pivoting) in a cyclic-reduction order.
//
// The coarsest operator is symmetric positive definite (the Galerkin
// product of the clamped fine operator; the reference factorises it with a
// direct solver, FEAnalysis.cpp:555-573), so every pivot block -- a Schur
// complement -- is SPD and no pivoting is needed.  The V-cycle applies the
// explicit inverse as one bandwidth-parallel matrix-vector product.
//
// The sweep of a pivot block K (P = A_KK^-1, F = the column block A_{.K},
// G = F P):
//   A_KK <- -P;  A_iK <- G_i;  A_Kj <- G_j^T;  A_ij <- A_ij - G_i F_j^T
// keeps the matrix symmetric; after every block has been swept it is -A^-1.
//
// Order.  What bounds the inversion is the chain of pivot blocks (a few
// microseconds of dependent arithmetic each), not its n^3 operations.  The
// operator is a 27-point stencil, so with the unknowns grouped by the planes
// normal to the longest dimension it is block tridiagonal, and every other
// plane can be swept at the same time: pivot blocks that are not coupled
// have a block-diagonal pivot matrix.  What is left is again a chain, of
// half the length.  A 13 x 7 x 7 level (1,911 unknowns) takes 4 rounds of 3
// blocks of 49, 12 dependent steps, where the natural order takes 30 steps
// of 64; tiles that no pivot of a step couples are skipped (the structure is
// worked out once per context on the host, coarse_inverse_plan).
//
// A step is two launches over task lists: F and G of every coupled (row
// block, pivot) pair (k_ci_fg), and the updates of the lower tiles by
// FP64 tensor-core MMAs (k_ci_update), where the tiles that are the next
// step's pivots come first and are inverted in registers as soon as they
// are updated (invert_tile), so the inversions overlap the other updates.
// The matrix is kept as T x T tiles in plane order (T = 24 .. 64, the block
// size rounded up, padded with the identity), each contiguous: every operand
// is one run of 16-byte copies.
//
// Measured at 1,911 unknowns (serialised kernel time of one inversion): the
// natural order in 64-blocks took 1,480 us, 36 us a step for the update
// with the scalar inversion of the next block (22 us of it) and 12 us for F
// and G; this form takes 356 us (12 x (6.4 + 19.7), fill 5, first pivots 13,
// final pass 25), 3% more since the updates' sums are kept apart.  The launches
// of the chain are programmatic dependent ones, released when a block's
// arithmetic is done (released at its start, the waiting blocks kept those of
// the side streams out): FEAssemble of a 48 x 24 x 24 mesh 0.67 -> 0.60 ms, of
// 12 x 6 x 6 0.247 -> 0.227.
#include <algorithm>
#include <cmath>
#include <new>
#include <vector>

#include <sys/mman.h>

#include "pdl.cuh"
#include "tpo_internal.h"

namespace tpo {

namespace {

constexpr int kMaxTile = 64;

// D (8 x 8) += A (8 x 4) B (4 x 8) in FP64 on the tensor cores.  Fragments
// (PTX ISA, mma.m8n8k4 .f64): lane = 4 g + q holds A[g][q], B[q][g] and
// D[g][2q], D[g][2q + 1].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async16(double *dst, const double *src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

__host__ __device__ constexpr int64_t tile_index(int I, int J) {   // I >= J
  return (int64_t)I * (I + 1) / 2 + J;
}

// rows of T doubles are staged at a stride of T + 4: T is a multiple of 8,
// so four consecutive rows start 8 banks apart and the fragment reads (8
// consecutive doubles of 4 rows) are free of conflicts
template <int T>
struct Tile {
  static constexpr int kLd = T + 4;
  static constexpr int kWarps = T / 8;        // one 8-row strip per warp
  static constexpr int kThreads = 32 * kWarps;
  static constexpr int kElems = T * T;
  static constexpr size_t kSmem = 2 * sizeof(double) * T * kLd;
};

template <int T>
__device__ __forceinline__ void stage_tile(double *dst, const double *src) {
  for (int e = threadIdx.x; e < T * T / 2; e += Tile<T>::kThreads) {
    const int r = e / (T / 2), c = 2 * (e % (T / 2));
    cp_async16(dst + r * Tile<T>::kLd + c, src + r * T + c);
  }
}

// the D-fragment pair (d[g][2q], d[g][2q+1]) of an 8 x 8 block as the two
// A fragments (d[g][q], d[g][4 + q])
__device__ __forceinline__ void d_to_a(double d0, double d1, int lane, double &a0, double &a1) {
  const int q = lane & 3, s = (lane & ~3) + (q >> 1);
  const double x0 = __shfl_sync(0xffffffffu, d0, s), x1 = __shfl_sync(0xffffffffu, d1, s);
  const double y0 = __shfl_sync(0xffffffffu, d0, s + 2), y1 = __shfl_sync(0xffffffffu, d1, s + 2);
  a0 = (q & 1) ? x1 : x0;
  a1 = (q & 1) ? y1 : y0;
}

// -M^-1 of the symmetric T x T tile whose 8-row strip w each warp holds in
// acc (D fragments of T / 8 blocks), by sweeps of 8 x 8 pivots: the block
// column of the pivot goes to shared memory, every warp inverts the pivot
// block for itself (one barrier per pivot) and updates its strip with
// tensor-core MMAs.  The pivot block is factorised by shuffles, M = L D L^T, L^-1
// taking the place of L, and its inverse formed as L^-T D^-1 L^-1: by
// Gauss-Jordan steps in place the inverse loses its symmetry to rounding, and the
// soft modes of a slender beam with it (300 x 1 x 1 elements: relative error of
// K^-1 r in the energy norm 0.2, now 1e-6).  A pivot that is not positive records its
// dof + 1 in *info (the first one wins).
// Fs: 2 x T x 12 doubles.
template <int T>
__device__ __forceinline__ void invert_tile(double (&acc)[T / 8][2], double *Fs, const int *dof,
                                            int *info) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int kb = 0; kb < T / 8; ++kb) {
    double *F = Fs + (kb & 1) * T * 12;
    *reinterpret_cast<double2 *>(F + (8 * w + g) * 12 + 2 * q) =
        make_double2(acc[kb][0], acc[kb][1]);
    __syncthreads();
    const double2 m = *reinterpret_cast<const double2 *>(F + (8 * kb + g) * 12 + 2 * q);
    double m0 = m.x, m1 = m.y, ipa = 0.0, ipb = 0.0;   // 1 / D of rows q and 4 + q
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const double ms = (k & 1) ? m1 : m0;
      const double p = __shfl_sync(0xffffffffu, ms, 4 * k + (k >> 1));
      const double rk0 = __shfl_sync(0xffffffffu, m0, 4 * k + q);
      const double rk1 = __shfl_sync(0xffffffffu, m1, 4 * k + q);
      const double ck = __shfl_sync(0xffffffffu, ms, 4 * g + (k >> 1));
      const bool ok = p > 0.0 && p < INFINITY;
      if (!ok && threadIdx.x == 0) atomicCAS(info, 0, dof[8 * kb + k] + 1);
      const double ip = ok ? 1.0 / p : 0.0;
      if (q == (k & 3)) (k < 4 ? ipa : ipb) = ip;
      if (g > k) {   // rows below: of M right of the pivot, of L^-1 left of it
        const double l = ck * ip;
        m0 = 2 * q == k ? -l : fma(-l, rk0, m0);
        m1 = 2 * q + 1 == k ? -l : fma(-l, rk1, m1);
      }
    }
    // L^-1[q][g], L^-1[4 + q][g]: B fragments of L^-1 and A fragments of L^-T
    double l0, l1;
    {
      const int s = 4 * q + (g >> 1);
      const double x0 = __shfl_sync(0xffffffffu, m0, s), x1 = __shfl_sync(0xffffffffu, m1, s);
      const double y0 = __shfl_sync(0xffffffffu, m0, s + 16);
      const double y1 = __shfl_sync(0xffffffffu, m1, s + 16);
      l0 = g < q ? ((g & 1) ? x1 : x0) : (g == q ? 1.0 : 0.0);
      l1 = g < 4 + q ? ((g & 1) ? y1 : y0) : (g == 4 + q ? 1.0 : 0.0);
    }
    double pd[2] = {0.0, 0.0};
    dmma(pd, l0 * ipa, l0);
    dmma(pd, l1 * ipb, l1);
    m0 = pd[0];
    m1 = pd[1];
    // P8 = (m0, m1); it is symmetric, so its A fragments are its B
    // fragments too
    double p0, p1;
    d_to_a(m0, m1, lane, p0, p1);
    double gd[2] = {0.0, 0.0}, a0, a1;
    dmma(gd, F[(8 * w + g) * 12 + q], p0);
    dmma(gd, F[(8 * w + g) * 12 + 4 + q], p1);
    d_to_a(-gd[0], -gd[1], lane, a0, a1);
    const bool own = w == kb;   // the pivot's strip becomes P8 F_j^T
    if (own) {
      a0 = p0;
      a1 = p1;
    }
#pragma unroll
    for (int j = 0; j < T / 8; ++j) {
      if (j == kb) continue;
      double sum[2] = {0.0, 0.0};
      dmma(sum, a0, F[(8 * j + g) * 12 + q]);
      dmma(sum, a1, F[(8 * j + g) * 12 + 4 + q]);
      acc[j][0] = own ? sum[0] : acc[j][0] + sum[0];
      acc[j][1] = own ? sum[1] : acc[j][1] + sum[1];
    }
    acc[kb][0] = own ? -m0 : gd[0];
    acc[kb][1] = own ? -m1 : gd[1];
  }
}

// element (8w + g, 8j + 2q + h) of a column-major tile
template <int T>
__device__ __forceinline__ void load_strip(double (&acc)[T / 8][2], const double *tile) {
  const int lane = threadIdx.x & 31, r = 8 * (threadIdx.x >> 5) + (lane >> 2), q = lane & 3;
#pragma unroll
  for (int j = 0; j < T / 8; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) acc[j][h] = tile[(8 * j + 2 * q + h) * T + r];
}
template <int T>
__device__ __forceinline__ void store_strip(const double (&acc)[T / 8][2], double *tile,
                                            double s) {
  const int lane = threadIdx.x & 31, r = 8 * (threadIdx.x >> 5) + (lane >> 2), q = lane & 3;
#pragma unroll
  for (int j = 0; j < T / 8; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) tile[(8 * j + 2 * q + h) * T + r] = s * acc[j][h];
}

// inverts the pivot tile held in acc: P to the workspace, -P to the matrix
template <int T>
__device__ __forceinline__ void pivot_out(double (&acc)[T / 8][2], double *smem, int I,
                                          double *W, double *P, const int *dofs, int *info) {
  __syncthreads();   // the shared buffers are free
  invert_tile<T>(acc, smem, dofs + I * T, info);
  pdl_launch_dependents();   // late: blocks that wait keep the side streams' out
  store_strip<T>(acc, W + tile_index(I, I) * T * T, 1.0);
  store_strip<T>(acc, P, -1.0);
}

// the first step's pivots
template <int T>
__global__ void __launch_bounds__(Tile<T>::kThreads)
    k_ci_pivots(const int *__restrict__ piv, double *W, double *P, const int *__restrict__ dofs,
                int *info) {
  extern __shared__ __align__(16) double smem[];
  const int I = piv[blockIdx.x];
  pdl_wait();   // the task lists are constant: they are read before it
  double acc[T / 8][2];
  load_strip<T>(acc, W + tile_index(I, I) * T * T);
  pivot_out<T>(acc, smem, I, W, P + (size_t)blockIdx.x * T * T, dofs, info);
}

// task (I, K, pivot slot): F_I = A_IK (the transposed tile (K, I) above the
// diagonal) and G_I = F_I P; both to the workspace, [k][i], and G_I to the
// matrix
template <int T>
__global__ void __launch_bounds__(Tile<T>::kThreads)
    k_ci_fg(const int4 *__restrict__ tasks, double *W, const double *P, double *F,
            double *G) {
  extern __shared__ __align__(16) double smem[];
  constexpr int ld = Tile<T>::kLd;
  double *Xs = smem, *Ps = smem + T * ld;
  const int4 t = tasks[blockIdx.x];
  const int I = t.x, K = t.y;
  const bool below = I > K;
  pdl_wait();
  double *a = W + (below ? tile_index(I, K) : tile_index(K, I)) * T * T;
  stage_tile<T>(Xs, a);
  stage_tile<T>(Ps, P + (size_t)t.z * T * T);
  cp_async_wait_all();
  __syncthreads();
  const int lane = threadIdx.x & 31, r0 = 8 * (threadIdx.x >> 5), g = lane >> 2, q = lane & 3;
  double acc[T / 8][2];
#pragma unroll
  for (int j = 0; j < T / 8; ++j) acc[j][0] = acc[j][1] = 0.0;
#pragma unroll 2
  for (int k0 = 0; k0 < T; k0 += 4) {
    const double av = below ? Xs[(k0 + q) * ld + r0 + g] : Xs[(r0 + g) * ld + k0 + q];
#pragma unroll
    for (int j = 0; j < T / 8; ++j) dmma(acc[j], av, Ps[(k0 + q) * ld + 8 * j + g]);
  }
  pdl_launch_dependents();
  double *f = F + (size_t)blockIdx.x * T * T, *gw = G + (size_t)blockIdx.x * T * T;
  for (int e = threadIdx.x; e < T * T; e += Tile<T>::kThreads) {
    const int k = e / T, i = e % T;
    f[e] = below ? Xs[k * ld + i] : Xs[i * ld + k];
  }
  store_strip<T>(acc, gw, 1.0);
  if (below) {
    store_strip<T>(acc, a, 1.0);
  } else {
#pragma unroll
    for (int j = 0; j < T / 8; ++j)   // element (k = 8j + 2q + h, i) of tile (K, I)
      *reinterpret_cast<double2 *>(a + (r0 + g) * T + 8 * j + 2 * q) =
          make_double2(acc[j][0], acc[j][1]);
  }
}

// task (tile I | J << 16, first pair, pairs, pivot slot of the next step or
// -1): A_IJ -= sum over the pairs (G index, F index) of G_I F_J^T
template <int T>
__global__ void __launch_bounds__(Tile<T>::kThreads)
    k_ci_update(const int4 *__restrict__ tasks, const int2 *__restrict__ pairs, double *W,
                const double *F, const double *G, double *P,
                const int *__restrict__ dofs, int *info) {
  extern __shared__ __align__(16) double smem[];
  constexpr int ld = Tile<T>::kLd;
  double *Gs = smem, *Fs = smem + T * ld;
  const int4 t = tasks[blockIdx.x];
  const int I = t.x & 0xffff, J = t.x >> 16;
  double *a = W + tile_index(I, J) * T * T;
  const int lane = threadIdx.x & 31, r0 = 8 * (threadIdx.x >> 5), g = lane >> 2, q = lane & 3;
  // the products are summed by themselves and added to the tile once: summed
  // onto it, each step of four rounds to the tile's magnitude
  // (a tile of 64 is read after them: beside them it takes 124 registers for
  // 104, and one level of 14x14x14 elements 9.60 ms to assemble for 9.39)
  constexpr bool kLate = T == 64;
  double acc[T / 8][2], sum[T / 8][2];
#pragma unroll
  for (int j = 0; j < T / 8; ++j) sum[j][0] = sum[j][1] = 0.0;
  int2 pr = t.z > 0 ? pairs[t.y] : make_int2(0, 0);
  pdl_wait();
  for (int p = 0; p < t.z; ++p) {
    if (p) {
      pr = pairs[t.y + p];
      __syncthreads();
    }
    stage_tile<T>(Gs, G + (size_t)pr.x * T * T);
    stage_tile<T>(Fs, F + (size_t)pr.y * T * T);
    if (p == 0 && !kLate) load_strip<T>(acc, a);   // while the copies are in flight
    cp_async_wait_all();
    __syncthreads();
#pragma unroll 2
    for (int k0 = 0; k0 < T; k0 += 4) {
      const double av = -Gs[(k0 + q) * ld + r0 + g];
#pragma unroll
      for (int j = 0; j < T / 8; ++j) dmma(sum[j], av, Fs[(k0 + q) * ld + 8 * j + g]);
    }
  }
  if (t.z == 0 || kLate) load_strip<T>(acc, a);
#pragma unroll
  for (int j = 0; j < T / 8; ++j) {
    acc[j][0] += sum[j][0];
    acc[j][1] += sum[j][1];
  }
  if (t.w >= 0) {
    pivot_out<T>(acc, smem, I, W, P + (size_t)t.w * T * T, dofs, info);
  } else {
    pdl_launch_dependents();
    store_strip<T>(acc, a, 1.0);
  }
}

// the stencil's entries on or below the diagonal to their tiles (zeroed
// before), the identity on the padding
__global__ void k_ci_fill(int nx, int ny, int nz, const double *__restrict__ S,
                          const int *__restrict__ pos, const int *__restrict__ dofs, int nb,
                          int T, double *__restrict__ W) {
  const int64_t nn = (int64_t)nx * ny * nz, total = nn * 243;
  const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t st = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = t0; t < total; t += st) {
    const int q = (int)(t / nn);
    const int64_t n = t - (int64_t)q * nn;
    const int b = q / 9, r = (q % 9) / 3, s = q % 3;
    const int mi = (int)(n % nx) + b % 3 - 1, mj = (int)((n / nx) % ny) + (b / 3) % 3 - 1,
              mk = (int)(n / ((int64_t)nx * ny)) + b / 9 - 1;
    if (mi < 0 || mi >= nx || mj < 0 || mj >= ny || mk < 0 || mk >= nz) continue;
    const int64_t m = ((int64_t)mk * ny + mj) * nx + mi;
    const int pi = pos[3 * n + r], pj = pos[3 * m + s];
    const int I = pi / T, J = pj / T;
    if (I < J) continue;
    W[tile_index(I, J) * T * T + (pj % T) * T + pi % T] = S[t];
  }
  for (int64_t t = t0; t < (int64_t)nb * T; t += st)
    if (dofs[t] < 0) {
      const int I = (int)(t / T), o = (int)(t % T);
      W[tile_index(I, I) * T * T + o * T + o] = 1.0;
    }
}

// Ainv (n x n, dof order) = -W, one CTA per tile on or below the diagonal
__global__ void k_ci_final(int n, int T, const int *__restrict__ dofs,
                           const double *W, double *__restrict__ Ainv) {
  extern __shared__ __align__(16) double smem[];
  const int I = blockIdx.x, J = blockIdx.y;
  pdl_wait();
  pdl_launch_dependents();
  if (J > I) return;
  const double *a = W + tile_index(I, J) * T * T;
  for (int e = threadIdx.x; e < T * T; e += blockDim.x)
    smem[(e / T) * (T + 1) + e % T] = -a[e];   // [column][row]
  __syncthreads();
  for (int e = threadIdx.x; e < T * T; e += blockDim.x) {
    const int u = e / T, v = e % T;
    const int di = dofs[I * T + u], dj = dofs[J * T + v];
    if (di >= 0 && dj >= 0) Ainv[(int64_t)di * n + dj] = smem[v * (T + 1) + u];
    if (I != J) {
      const int dr = dofs[J * T + u], dc = dofs[I * T + v];
      if (dr >= 0 && dc >= 0) Ainv[(int64_t)dr * n + dc] = smem[u * (T + 1) + v];
    }
  }
}

template <int T>
void run_steps(const CoarseInvPlan &pl, double *work, int *info, cudaStream_t s) {
  double *W = work, *P = W + tile_index(pl.nb, 0) * T * T;
  double *F = P + (size_t)pl.max_pivots * T * T, *G = F + (size_t)pl.max_fg * T * T;
  const int4 *fg = reinterpret_cast<const int4 *>(pl.dev + pl.off_fg);
  const int4 *up = reinterpret_cast<const int4 *>(pl.dev + pl.off_up);
  const int2 *pairs = reinterpret_cast<const int2 *>(pl.dev + pl.off_pairs);
  const int *dofs = pl.dev + pl.off_dofs;
  const size_t sm = Tile<T>::kSmem;
  static unsigned long long attr_set = 0;   // bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!((attr_set >> (dev & 63)) & 1ull)) {
    cudaFuncSetAttribute(k_ci_pivots<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaFuncSetAttribute(k_ci_fg<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaFuncSetAttribute(k_ci_update<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    attr_set |= 1ull << (dev & 63);
  }
  constexpr int th = Tile<T>::kThreads;
  count_launch();
  launch_pdl(k_ci_pivots<T>, pl.first_pivots, th, sm, s, pl.dev + pl.off_piv, W, P, dofs, info);
  for (const CoarseInvPlan::Step &q : pl.steps) {
    if (q.nfg) {
      count_launch();
      launch_pdl(k_ci_fg<T>, q.nfg, th, sm, s, fg + q.fg, W, P, F, G);
    }
    if (q.nup) {
      count_launch();
      launch_pdl(k_ci_update<T>, q.nup, th, sm, s, up + q.up, pairs, W, F, G, P, dofs, info);
    }
  }
}

}  // namespace

template <typename E>
E *CoarseInvPlan::HugePages<E>::allocate(size_t n) {
  constexpr size_t kPage = 2u << 20;
  const size_t bytes = n * sizeof(E);
  void *p = nullptr;
  if (bytes < kPage) {
    p = std::malloc(bytes);
  } else if (posix_memalign(&p, kPage, (bytes + kPage - 1) / kPage * kPage) == 0) {
    madvise(p, (bytes + kPage - 1) / kPage * kPage, MADV_HUGEPAGE);   // a hint
  } else {
    p = nullptr;
  }
  if (!p) throw std::bad_alloc();
  return static_cast<E *>(p);
}

// The blocks, the elimination order and the task lists of a level of d[0] x
// d[1] x d[2] nodes (on the host; coarse_inverse_upload takes them to the
// device).
void coarse_inverse_plan(const int d[3], CoarseInvPlan &pl) {
  const int D = (d[0] >= d[1] && d[0] >= d[2]) ? 0 : (d[1] >= d[2] ? 1 : 2);
  const int planes = d[D];
  const int m = 3 * (d[0] * d[1] * d[2] / planes);   // unknowns of one plane
  // short planes are taken several at a time, long ones in several blocks
  const int grp = std::max(1, std::min(planes, kMaxTile / m));
  const int np = (planes + grp - 1) / grp, mp = grp * m;
  const int bpp = (mp + kMaxTile - 1) / kMaxTile;     // blocks per plane group
  const int bs = (mp + bpp - 1) / bpp;
  // a level has at least 2 nodes per dimension, so m >= 12 and the blocks
  // are of 24 (2 x 2 x 2 nodes) or 33 .. 64 unknowns
  const int T = bs <= 24 ? 24 : std::max(40, (bs + 7) / 8 * 8);
  const int nb = np * bpp;
  pl.T = T;
  pl.nb = nb;
  pl.n = 3LL * d[0] * d[1] * d[2];
  // position of each dof: plane group along D, then the nodes of its planes
  // in the level's own order, in blocks of bs
  std::vector<int> pos(pl.n), dofs((size_t)nb * T, -1);
  std::vector<int> fill(np, 0);
  for (int k = 0; k < d[2]; ++k)
    for (int j = 0; j < d[1]; ++j)
      for (int i = 0; i < d[0]; ++i) {
        const int c[3] = {i, j, k};
        const int g = c[D] / grp, n = (k * d[1] + j) * d[0] + i;
        for (int r = 0; r < 3; ++r) {
          const int o = fill[g]++;
          const int p = (g * bpp + o / bs) * T + o % bs;
          pos[3 * n + r] = p;
          dofs[p] = 3 * n + r;
        }
      }
  // coupled block pairs (a node's three unknowns are in one or two blocks)
  std::vector<uint8_t> nz((size_t)nb * nb, 0);
  const int nn = d[0] * d[1] * d[2];
  std::vector<int> lo(nn), hi(nn);
  for (int n = 0; n < nn; ++n) {
    lo[n] = pos[3 * n] / T;
    hi[n] = pos[3 * n + 2] / T;
  }
  for (int k = 0; k < d[2]; ++k)
    for (int j = 0; j < d[1]; ++j)
      for (int i = 0; i < d[0]; ++i) {
        const int n = (k * d[1] + j) * d[0] + i;
        for (int mk = std::max(k - 1, 0); mk <= std::min(k + 1, d[2] - 1); ++mk)
          for (int mj = std::max(j - 1, 0); mj <= std::min(j + 1, d[1] - 1); ++mj)
            for (int mi = std::max(i - 1, 0); mi <= std::min(i + 1, d[0] - 1); ++mi) {
              const int q = (mk * d[1] + mj) * d[0] + mi;
              for (int a : {lo[n], hi[n]})
                for (int b : {lo[q], hi[q]}) nz[(size_t)a * nb + b] = 1;
            }
      }
  // rounds of alternate plane groups; block b of every group of a round is
  // one step as long as the groups are uncoupled
  std::vector<std::vector<int>> steps;
  std::vector<int> chain(np);
  for (int g = 0; g < np; ++g) chain[g] = g;
  std::vector<uint8_t> st = nz;   // structure as the elimination proceeds
  auto coupled = [&](int a, int b) { return st[(size_t)a * nb + b] != 0; };
  std::vector<int> nzr;
  auto eliminate = [&](int k) {
    nzr.clear();
    for (int i = 0; i < nb; ++i)
      if (i != k && coupled(i, k)) nzr.push_back(i);
    for (int a : nzr)
      for (int b : nzr) st[(size_t)a * nb + b] = 1;
  };
  while (!chain.empty()) {
    std::vector<int> round, rest;
    for (size_t t = 0; t < chain.size(); ++t) (t % 2 ? rest : round).push_back(chain[t]);
    for (int b = 0; b < bpp; ++b) {
      std::vector<int> todo;
      for (int g : round) todo.push_back(g * bpp + b);
      while (!todo.empty()) {
        std::vector<int> now, later;
        for (int k : todo) {
          bool free = true;
          for (int o : now) free = free && !coupled(k, o);
          (free ? now : later).push_back(k);
        }
        steps.push_back(now);
        for (int k : now) eliminate(k);
        todo.swap(later);
      }
    }
    chain.swap(rest);
  }
  // task lists.  A step's F and G tiles are numbered row block by row block
  // within a pivot; row[I] lists those of row block I as (pivot, number), in the
  // order of the pivots, and a tile (I, J) is updated by the pivots that both
  // rows have (a merge: levels of 4,000 nodes have some 200,000 such pairs)
  using Pair = CoarseInvPlan::Pair;
  CoarseInvPlan::List<CoarseInvPlan::Task> fg, up;
  CoarseInvPlan::List<Pair> pairs;
  std::vector<std::vector<Pair>> row(nb);
  std::vector<int> rows;   // those that a pivot of the step couples
  std::vector<int> slot(nb);
  std::vector<uint8_t> is_piv(nb);
  st = nz;
  pl.max_pivots = 1;
  pl.max_fg = 1;
  pl.steps.clear();
  for (size_t q = 0; q < steps.size(); ++q) {
    const std::vector<int> &piv = steps[q];
    pl.max_pivots = std::max(pl.max_pivots, (int)piv.size());
    CoarseInvPlan::Step S{};
    S.fg = (int)fg.size();
    S.up = (int)up.size();
    std::fill(is_piv.begin(), is_piv.end(), 0);
    for (int k : piv) is_piv[k] = 1;
    for (auto &r : row) r.clear();
    int nfg = 0;
    for (size_t p = 0; p < piv.size(); ++p)
      for (int I = 0; I < nb; ++I)
        if (I != piv[p] && coupled(I, piv[p])) {
          row[I].push_back({(int)p, nfg++});
          fg.push_back({{I, piv[p], (int)p, 0}});
        }
    S.nfg = nfg;
    pl.max_fg = std::max(pl.max_fg, nfg);
    rows.clear();
    for (int I = 0; I < nb; ++I)
      if (!is_piv[I] && !row[I].empty()) rows.push_back(I);
    std::fill(slot.begin(), slot.end(), -1);
    if (q + 1 < steps.size())
      for (size_t p = 0; p < steps[q + 1].size(); ++p) slot[steps[q + 1][p]] = (int)p;
    auto task = [&](int I, int J) {
      const int next = I == J ? slot[I] : -1;
      const int first = (int)pairs.size();
      if (!is_piv[I] && !is_piv[J]) {
        const Pair *x = row[I].data(), *xe = x + row[I].size();
        const Pair *y = row[J].data(), *ye = y + row[J].size();
        while (x != xe && y != ye) {
          if (x->a == y->a) pairs.push_back({x->b, y->b});
          const bool nx = x->a <= y->a, ny = y->a <= x->a;
          x += nx;
          y += ny;
        }
      }
      const int cnt = (int)pairs.size() - first;
      if (cnt || next >= 0) up.push_back({{I | (J << 16), first, cnt, next}});
    };
    for (int I = 0; I < nb; ++I)   // the next step's pivots first
      if (slot[I] >= 0) task(I, I);
    for (int I : rows)
      for (int J : rows) {
        if (J > I) break;
        if (!(I == J && slot[I] >= 0)) task(I, J);
      }
    S.nup = (int)up.size() - S.up;
    pl.steps.push_back(S);
    for (int k : piv) eliminate(k);
  }
  pl.first_pivots = (int)steps[0].size();
  // one device array; the task lists (int4, int2) first, for their alignment
  pl.ints = 0;
  auto put = [&](size_t bytes) {
    const size_t o = pl.ints;
    pl.ints += (bytes + 15) / 16 * 4;
    return o;
  };
  pl.piv = steps[0];
  pl.fg.swap(fg);
  pl.up.swap(up);
  pl.pairs.swap(pairs);
  pl.dofs.swap(dofs);
  pl.pos.swap(pos);
  pl.off_fg = put(sizeof(pl.fg[0]) * pl.fg.size());
  pl.off_up = put(sizeof(pl.up[0]) * pl.up.size());
  pl.off_pairs = put(sizeof(pl.pairs[0]) * pl.pairs.size());
  pl.off_piv = put(sizeof(int) * pl.piv.size());
  pl.off_dofs = put(sizeof(int) * pl.dofs.size());
  pl.off_pos = put(sizeof(int) * pl.pos.size());
}

cudaError_t coarse_inverse_upload(CoarseInvPlan &pl, cudaStream_t s) {
  cudaError_t err = cudaSuccess;
  auto copy = [&](size_t off, const auto &v) {
    if (!v.empty() && err == cudaSuccess)
      err = cudaMemcpyAsync(pl.dev + off, v.data(), sizeof(v[0]) * v.size(),
                            cudaMemcpyHostToDevice, s);
  };
  copy(pl.off_fg, pl.fg);
  copy(pl.off_up, pl.up);
  copy(pl.off_pairs, pl.pairs);
  copy(pl.off_piv, pl.piv);
  copy(pl.off_dofs, pl.dofs);
  copy(pl.off_pos, pl.pos);
  if (err == cudaSuccess) err = cudaStreamSynchronize(s);
  pl.fg = pl.up = {};
  pl.pairs = {};
  pl.piv = pl.dofs = pl.pos = {};
  return err;
}

size_t coarse_inverse_work(const CoarseInvPlan &pl) {
  const size_t tile = (size_t)pl.T * pl.T;
  return tile * (tile_index(pl.nb, 0) + pl.max_pivots + 2 * (size_t)pl.max_fg);
}

void launch_coarse_inverse(const Level &v, const double *S, const CoarseInvPlan &pl,
                           double *Ainv, double *work, int *info, cudaStream_t s) {
  const int T = pl.T, nb = pl.nb;
  cudaMemsetAsync(info, 0, sizeof(int), s);
  cudaMemsetAsync(work, 0, sizeof(double) * tile_index(nb, 0) * T * T, s);
  count_launch(2);
  const int64_t g = std::min<int64_t>((v.nn * 243 + 255) / 256, 148 * 32);
  k_ci_fill<<<(int)g, 256, 0, s>>>(v.dims[0], v.dims[1], v.dims[2], S, pl.dev + pl.off_pos,
                                   pl.dev + pl.off_dofs, nb, T, work);
  switch (T) {
    case 24: run_steps<24>(pl, work, info, s); break;
    case 40: run_steps<40>(pl, work, info, s); break;
    case 48: run_steps<48>(pl, work, info, s); break;
    case 56: run_steps<56>(pl, work, info, s); break;
    default: run_steps<64>(pl, work, info, s); break;
  }
  launch_pdl(k_ci_final, dim3(nb, nb), 256, sizeof(double) * T * (T + 1), s, (int)pl.n, T,
             pl.dev + pl.off_dofs, work, Ainv);
}

}  // namespace tpo
