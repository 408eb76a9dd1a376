// Persistent coarse-grid V-cycle: every GMG level from `ps` down to the
// coarsest, and the dense coarsest solve, in ONE cooperative kernel.
//
// On the small levels (a few thousand to a few ten thousand nodes) each
// smoothing step, transfer or residual is a microseconds-long latency-bound
// launch; a launch per phase would cost more than the work.  Here one CTA per
// SM stays resident (a cooperative launch) and the phases are separated by
// grid-wide barriers (grid_barrier.cuh).
//
// What bounds a phase is the latency of its loads and, on the largest level,
// the bytes of the stencil: 243 values per node, read by each of the four
// stencil phases of a cycle.  So every CTA owns a contiguous range of each
// level's nodes (coarse.h) and keeps as much of their stencil as fits in
// shared memory for the whole cycle, copied there in bulk when the kernel
// starts (one mbarrier per neighbour row of the top level, so its first
// phase starts on the rows that have arrived); the rest is read from L2 in
// every phase.  192x96x96's level 2 (30,625 nodes, FP32) fits whole: 202 KB
// of each SM.
//
// A stencil phase: a warp takes 32 consecutive nodes and one of SPLIT groups
// of neighbour rows (dj, dk) -- 27 coefficients and 9 values of u a thread
// and column at SPLIT = 9, every load contiguous over the warp since vectors
// are stored component by component and neighbours are flat offsets -- and leaves its partial sums in shared
// memory; after a CTA barrier, one thread per (node, component, column) adds
// them in a fixed order and applies the Chebyshev update.  In a block of
// columns each coefficient serves all of them.
//
// Per level (Chebyshev degree m, Jacobi):
//   pre:  r = D^-1 b, d = r/theta, x = d;  m-1 x [r -= D^-1 A d;
//         d' = c1 d + c2 r; x += d']
//   res = b - A x;  b_c = P^T res;  (recurse);  x += P x_c
//   post: r = D^-1 (b - A x), d = r/theta, x' = x + d;  m-1 x [...]
// with the search direction ping-ponged so a Chebyshev step costs one
// barrier; the restriction also writes the child's first direction.
//
// Measured (us a cycle in a solve's launch list; before: a warp per node, 592
// CTAs, every phase from L2, 89 and 112 by itself at 192x96x96; and now):
// 192x96x96 FP32 91 -> 65, FP64 116 -> 85; 91x47x53 FP32 84 -> 57; 48x24x24
// FP64 36 -> 26; 128x64x64, 8 FP32 columns 128 -> 74; 75x41x34 FP64, 4 columns
// 139 -> 85, 1 column 77 -> 50; 96x48x48 FP64, 8 columns 341 -> 310, 4 columns
// 215 -> 167.  What is left at 192x96x96 (121 k cycles): 12 barriers of 2.7 k,
// the first phase's 30 MB of stencil from DRAM 17 k, the inverse (29 MB) 14 k,
// the other phases 2 - 9 k.
#include "coarse.h"
#include "grid_barrier.cuh"
#include "umma.cuh"

namespace tpo {

namespace {

template <typename T, int NB, int SPLIT>
struct Shape {
  static constexpr int kRows = 9 / SPLIT;   // neighbour rows of one unit
  static constexpr int kThreads = (sizeof(T) == 4 && NB <= 2) ? 1024 : 512;
  static constexpr int kWarps = kThreads / 32;
  // partial sums: values per node, and the shared memory they may take
  static constexpr int kPart = SPLIT * NB * 3;
  static constexpr size_t kPartCap = (NB <= 2 ? 48 : 128) * 1024;
  // finished units a thread has at most when it keeps their operands
  static constexpr int kPre = NB == 1 ? (kThreads == 1024 ? 1 : 2) : 0;
};

constexpr uint32_t kBulkPolls = 1u << 20;

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes,
                                          uint64_t *mbar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                   umma::smem_u32(mbar)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(umma::smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(umma::smem_u32(mbar))
      : "memory");
}

// one component, and one z plane k (0 .. 2) of the taps, of the sum over the
// fine nodes f around coarse node (ix,iy,iz) of P(f,I) r_f; r_f at stride 1
template <typename T>
__device__ __forceinline__ T restrict_plane(const int f[3], int ix, int iy, int iz, int k,
                                            const T *rf) {
  auto weight = [](int a, int x, int n) {
    return (x >= 0 && x < n) ? ((a == 1 || x + 1 > n - 1) ? T(1) : T(0.5)) : T(0);
  };
  const int z = 2 * iz + k - 1;
  const T wz = weight(k, z, f[2]);
  const T *p = rf + min(max(z, 0), f[2] - 1) * f[1] * f[0];
  T s = T(0);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int y = 2 * iy + j - 1;
    const T wy = wz * weight(j, y, f[1]);
    const T *q = p + min(max(y, 0), f[1] - 1) * f[0];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int x = 2 * ix + i - 1;
      s += (wy * weight(i, x, f[0])) * q[min(max(x, 0), f[0] - 1)];
    }
  }
  return s;
}

// one component of sum over the coarse nodes I around fine node (gx,gy,gz)
// of P(f,I) x_I; x_I at stride st
template <typename T>
__device__ __forceinline__ T prolong_one(const int F[3], const int C[3], int gx, int gy, int gz,
                                         const T *xc, int st) {
  const int g[3] = {gx, gy, gz};
  int c0[3], c1[3];
  T w0[3], w1[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const bool odd = g[d] & 1;
    c0[d] = g[d] >> 1;
    const bool has = odd && g[d] + 1 <= F[d] - 1;
    w0[d] = has ? T(0.5) : T(1);
    w1[d] = has ? T(0.5) : T(0);
    c1[d] = min(c0[d] + 1, C[d] - 1);
  }
  T s = T(0);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int ax = k & 1, ay = (k >> 1) & 1, az = k >> 2;
    const T w = (ax ? w1[0] : w0[0]) * (ay ? w1[1] : w0[1]) * (az ? w1[2] : w0[2]);
    const int I = ((az ? c1[2] : c0[2]) * C[1] + (ay ? c1[1] : c0[1])) * C[0] +
                  (ax ? c1[0] : c0[0]);
    s += w * xc[I * st];
  }
  return s;
}

// The stencil phases of one cycle differ in their update only:
//   kPhFirst  r = D^-1 b - D^-1 A u, d = c1 u + c2 r, x = u + d   (u = d0)
//   kPhStep   r -= D^-1 A u, d = c1 u + c2 r, x += d
//   kPhRes    res = b - A u
//   kPhPost   r = D^-1 (b - A u), d = r / theta, x = u + d
// with b = the rows' own u, c = b or r, d = x (kPhStep; else unused), dn =
// where d goes.  The kernel walks a
// list of phases so that each kind of work is in the code once: a phase whose
// code runs for the first time in a launch spends some 2 us on instruction
// fetches (with a copy per phase a level's post-smoothing took 7.2 k cycles
// where its residual, run before on another level, took 3.0 k).
enum { kPhFirst, kPhStep, kPhRes, kPhPost };
template <typename T>
struct Phase {
  int mode;
  const T *u, *b, *c, *d;
  T *dn, *x;
  T c1, c2;
};
template <typename T>
struct Ops4 {
  T a, b, c, d;
};

// v(node, component, column) = (A u) for the CTA's nodes of level L, and the
// update of those entries.  With one column, and few enough nodes, the
// operands of the update are loaded before the products so that their latency
// overlaps.
template <typename T, int NB, int SPLIT>
__device__ __forceinline__ void stencil_phase(const CoarseLevel<T> &L, const Phase<T> &ph,
                                           unsigned char *smem, T *part, int chunk,
                                           uint64_t *mbar, bool per_row, bool *failed) {
  using Sh = Shape<T, NB, SPLIT>;
  using Ops = Ops4<T>;
  const T *u = ph.u;
  const bool out = ph.mode != kPhRes;
  // the operands of entry i = (3 col + c) nn + n, all of them in every mode
  // (a load under a condition would be waited for at once)
  auto pre = [&](int i, int n, int c) {
    return Ops{L.dinv[3 * n + c], ph.b[i], ph.c[i], ph.d[i]};
  };
  auto f = [&](int i, T Au, const Ops &o) {
    if (!out) {
      L.res[i] = o.c - Au;
      return;
    }
    T r, d, x;
    if (ph.mode == kPhPost) {
      r = o.a * (o.c - Au);
      d = r * L.inv_theta;
      x = o.b;
    } else {
      r = (ph.mode == kPhFirst ? o.a * o.c : o.c) - o.a * Au;
      d = ph.c1 * o.b + ph.c2 * r;
      x = ph.mode == kPhFirst ? o.b : o.d;
    }
    L.r[i] = r;
    ph.dn[i] = d;
    ph.x[i] = x + d;
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nx = L.dims[0], nxy = nx * L.dims[1], nn = L.nn;
  const int n0 = blockIdx.x * L.npc, cnt = min(L.npc, nn - n0), ld = L.npcp;
  const T *slab = L.A + (int64_t)blockIdx.x * 243 * ld;
  const T *res = reinterpret_cast<const T *>(smem + L.smem);
  for (int c0 = 0; c0 < cnt; c0 += chunk) {
    const int ng = (min(chunk, cnt - c0) + 31) / 32;
    const bool ahead = NB * 3 * ng <= Sh::kPre * Sh::kWarps;
    Ops ops[Sh::kPre > 0 ? Sh::kPre : 1];
    if (ahead) {
#pragma unroll
      for (int q = 0; q < Sh::kPre; ++q) {
        // units past the last load some other unit's (no branch to wait in)
        const int w = min(warp + q * Sh::kWarps, NB * 3 * ng - 1), cr = w / ng;
        const int n = n0 + min(c0 + (w % ng) * 32 + lane, cnt - 1);
        ops[q] = pre(cr * nn + n, n, cr % 3);
      }
    }
    // the rows read from L2 (the last ones) first
    for (int w = warp; w < SPLIT * ng; w += Sh::kWarps) {
      const int s = SPLIT - 1 - w / ng, il = (w % ng) * 32 + lane;
      const bool valid = c0 + il < cnt;
      const int i = valid ? c0 + il : c0;
      T p[NB][3];
#pragma unroll
      for (int c = 0; c < NB; ++c) p[c][0] = p[c][1] = p[c][2] = T(0);
#pragma unroll 1
      for (int gg = 0; gg < Sh::kRows; ++gg) {
        const int g = s * Sh::kRows + gg;
        // neighbours by flat offsets: one outside the level has a zero block,
        // whatever node its offset lands on (clamped to stay in the vector)
        const int m = n0 + i + (g / 3 - 1) * nxy + (g % 3 - 1) * nx;
        const T *um[3] = {u + min(max(m - 1, 0), nn - 1), u + min(max(m, 0), nn - 1),
                          u + min(max(m + 1, 0), nn - 1)};
        // all of a row's values in flight together where registers allow
        constexpr bool kAll = NB * sizeof(T) <= 32;
        T v[kAll ? 3 : 1][NB][3];
        auto load = [&](int di, T (&o)[NB][3]) {
#pragma unroll
          for (int c = 0; c < NB; ++c)
#pragma unroll
            for (int r = 0; r < 3; ++r) o[c][r] = um[di][(3 * c + r) * nn];
        };
        if (kAll) {
#pragma unroll
          for (int di = 0; di < 3; ++di) load(di, v[kAll ? di : 0]);
        }
        auto row = [&](const T *a) {
#pragma unroll
          for (int di = 0; di < 3; ++di) {
            T k[9];
#pragma unroll
            for (int q = 0; q < 9; ++q) k[q] = a[(di * 9 + q) * ld];
            if (!kAll) load(di, v[0]);
#pragma unroll
            for (int c = 0; c < NB; ++c) {
              const T(&x)[3] = v[kAll ? di : 0][c];
              p[c][0] += k[0] * x[0] + k[1] * x[1] + k[2] * x[2];
              p[c][1] += k[3] * x[0] + k[4] * x[1] + k[5] * x[2];
              p[c][2] += k[6] * x[0] + k[7] * x[1] + k[8] * x[2];
            }
          }
        };
        if (g < L.gres) {
          if (!umma::mbar_wait(mbar + (per_row ? g : 0), 0, kBulkPolls)) *failed = true;
          row(res + g * 27 * ld + i);
        } else {
          row(slab + g * 27 * ld + i);
        }
      }
      if (valid) {
#pragma unroll
        for (int c = 0; c < NB; ++c)
#pragma unroll
          for (int r = 0; r < 3; ++r) part[((s * NB + c) * 3 + r) * chunk + il] = p[c][r];
      }
    }
    __syncthreads();
    auto sum = [&](int cr, int il) {
      T v = part[cr * chunk + il];
#pragma unroll
      for (int s = 1; s < SPLIT; ++s) v += part[(s * NB * 3 + cr) * chunk + il];
      return v;
    };
    if (ahead) {
#pragma unroll
      for (int q = 0; q < Sh::kPre; ++q) {
        const int w = warp + q * Sh::kWarps, cr = w / ng, il = (w % ng) * 32 + lane;
        if (w < NB * 3 * ng && c0 + il < cnt) f(cr * nn + n0 + c0 + il, sum(cr, il), ops[q]);
      }
    } else {
#pragma unroll 2
      for (int w = warp; w < NB * 3 * ng; w += Sh::kWarps) {
        const int cr = w / ng, il = (w % ng) * 32 + lane, n = n0 + c0 + il;
        if (c0 + il < cnt) {
          const Ops o = pre(cr * nn + n, n, cr % 3);
          f(cr * nn + n, sum(cr, il), o);
        }
      }
    }
    if (c0 + chunk < cnt) __syncthreads();
  }
}

template <typename T, int NB, int SPLIT>
__global__ void __launch_bounds__(Shape<T, NB, SPLIT>::kThreads, 1)
    k_coarse_cycle(const __grid_constant__ CoarseCycle<T> P) {
  using Sh = Shape<T, NB, SPLIT>;
  extern __shared__ __align__(128) unsigned char smem[];
  // mbarriers: rows 0 .. 8 of the top level, then one per further level
  __shared__ uint64_t mbar[9 + kMaxCoarseLevels];
  T *part = reinterpret_cast<T *>(smem);
  // the transfers' units, 32 at a time, spread evenly over the CTAs
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tid = (warp * (int)gridDim.x + (int)blockIdx.x) * 32 + lane;
  const int nthr = gridDim.x * Sh::kThreads;
  bool failed = false;
  unsigned int sense = grid_barrier_sense(P.bar);

  if (threadIdx.x == 0)
    for (int i = 0; i < 9 + P.nlev; ++i) umma::mbar_init(mbar + i, 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int l = 0; l < P.nlev; ++l) {
      const CoarseLevel<T> &L = P.lev[l];
      if ((int)blockIdx.x * L.npc >= L.nn) continue;   // no nodes here
      const T *slab = L.A + (int64_t)blockIdx.x * 243 * L.npcp;
      const uint32_t row = 27u * L.npcp * sizeof(T);
      if (l == 0) {
        for (int g = L.gres - 1; g >= 0; --g)   // in the order of their use
          bulk_load(smem + L.smem + g * row, slab + g * 27 * L.npcp, row, mbar + g);
      } else if (L.gres) {
        bulk_load(smem + L.smem, slab, L.gres * row, mbar + 8 + l);
      }
    }
  }
  // this CTA's rows of the dense inverse to L2, for the middle of the cycle
  auto prefetch_inverse = [&]() {
    if (threadIdx.x != 32) return;
    const int rows = Sh::kWarps / 2;
    for (int r0 = blockIdx.x * rows; r0 < P.nc; r0 += gridDim.x * rows) {
      const double *a = P.Ainv + (int64_t)r0 * P.nc;
      const int64_t n = (int64_t)min((int64_t)rows, P.nc - r0) * P.nc;
      const char *lo = reinterpret_cast<const char *>(
          reinterpret_cast<uintptr_t>(a) & ~(uintptr_t)15);
      const uint32_t bytes = (uint32_t)(reinterpret_cast<const char *>(a + n) - lo) & ~15u;
      if (bytes)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lo), "r"(bytes)
                     : "memory");
    }
  };
  // a CTA that leaves early waits for its own copies first
  auto drain = [&]() {
    if (threadIdx.x == 0) {
      *(volatile double *)P.fault = 1.0;
      for (int l = 0; l < P.nlev; ++l) {
        if ((int)blockIdx.x * P.lev[l].npc >= P.lev[l].nn) continue;
        for (int g = 0; g < (l == 0 ? P.lev[l].gres : (P.lev[l].gres ? 1 : 0)); ++g)
          umma::mbar_wait(mbar + (l == 0 ? g : 8 + l), 0, kBulkPolls);
      }
    }
    __syncthreads();
  };
  for (int t = 0; t < P.nop; ++t) {
    const CoarseOp op = P.op[t];
    const CoarseLevel<T> &L = P.lev[op.level];
    const int nn = L.nn;
    // the level below, or the dense solve's vectors in dof order
    const bool bottom = op.level + 1 == P.nlev;
    const CoarseLevel<T> &N = P.lev[bottom ? op.level : op.level + 1];
    const int *cd = bottom ? P.cdims : N.dims;
    const int nnc = cd[0] * cd[1] * cd[2];
    if (op.kind == kOpRestrict) {
      // four lane groups of eight: three planes of taps of eight outputs, so
      // that a thread's chain is 9 loads (27 in one thread took 3 us)
      for (int e0 = (tid >> 5) * 8; e0 < 3 * NB * nnc; e0 += (nthr >> 5) * 8) {
        const int e = min(e0 + (lane & 7), 3 * NB * nnc - 1), k = lane >> 3;
        const int cr = e / nnc, I = e - cr * nnc;
        const int ix = I % cd[0], iy = (I / cd[0]) % cd[1], iz = I / (cd[0] * cd[1]);
        const T di = bottom ? T(0) : N.dinv[3 * I + cr % 3];
        T v = k < 3 ? restrict_plane(L.dims, ix, iy, iz, k, L.res + cr * nn) : T(0);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (k == 0 && e0 + lane < 3 * NB * nnc) {
          if (bottom) {
            P.bc[(cr / 3) * P.nc + 3 * I + cr % 3] = v;
          } else {
            N.b[e] = v;
            N.d0[e] = N.inv_theta * (di * v);
          }
        }
      }
    } else if (op.kind == kOpDense) {
      // x = Ainv b in FP64, two warps a row
      const int nc = (int)P.nc, rows = Sh::kWarps / 2, half = (nc + 1) / 2;
      double *sum = reinterpret_cast<double *>(smem);   // [rows][2][NB]
      // the top level's partial sums are free here; its resident rows are not
      for (int r0 = blockIdx.x * rows; r0 < nc; r0 += gridDim.x * rows) {
        const int row = r0 + (warp >> 1);
        const int k0 = (warp & 1) * half, k1 = min(nc, k0 + half);
        double s[NB];
#pragma unroll
        for (int c = 0; c < NB; ++c) s[c] = 0.0;
        if (row < nc) {
          const double *a = P.Ainv + (int64_t)row * nc;
          // whole batches of loads in flight, the last one predicated
          constexpr int kU = NB == 1 ? 16 : (NB == 2 ? 8 : 4);
          for (int k = k0 + lane; k < k1; k += 32 * kU) {
            double av[kU];
            T bv[kU][NB];
#pragma unroll
            for (int q = 0; q < kU; ++q) {
              const bool in = k + 32 * q < k1;
              av[q] = in ? __ldg(a + k + 32 * q) : 0.0;
#pragma unroll
              for (int c = 0; c < NB; ++c) bv[q][c] = in ? P.bc[c * nc + k + 32 * q] : T(0);
            }
#pragma unroll
            for (int q = 0; q < kU; ++q)
#pragma unroll
              for (int c = 0; c < NB; ++c) s[c] += av[q] * static_cast<double>(bv[q][c]);
          }
        }
#pragma unroll
        for (int c = 0; c < NB; ++c) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
          if (lane == c) sum[warp * NB + c] = s[c];
        }
        __syncthreads();
        if (threadIdx.x < rows * NB) {
          const int q = threadIdx.x / NB, c = threadIdx.x % NB;
          if (r0 + q < nc)
            P.xc[c * nc + r0 + q] =
                static_cast<T>(sum[2 * q * NB + c] + sum[(2 * q + 1) * NB + c]);
        }
        __syncthreads();
      }
  
    } else if (op.kind == kOpProlong) {
      const int st = bottom ? 3 : 1;
      for (int e = tid; e < 3 * NB * nn; e += nthr) {
        const int cr = e / nn, n = e - cr * nn;
        const int gx = n % L.dims[0], gy = (n / L.dims[0]) % L.dims[1],
                  gz = n / (L.dims[0] * L.dims[1]);
        const T *xc = bottom ? P.xc + (cr / 3) * P.nc + cr % 3 : N.xout + cr * nnc;
        L.xpre[e] += prolong_one(L.dims, cd, gx, gy, gz, xc, st);
      }
    } else if (op.kind == kOpStart) {
      for (int e = tid; e < 3 * NB * nn; e += nthr) L.xpre[e] = L.d0[e];
    } else {
      T *dc = op.flip ? L.d1 : L.d0, *dn = op.flip ? L.d0 : L.d1;
      Phase<T> ph{kPhStep, dc, dc, L.r, L.xpre, dn, L.xpre, L.c1[op.k], L.c2[op.k]};
      if (op.kind == kOpFirst) {
        ph.mode = kPhFirst;
        ph.c = L.b;
      } else if (op.kind == kOpRes) {
        ph.mode = kPhRes;
        ph.u = ph.b = L.xpre;
        ph.c = L.b;
      } else if (op.kind == kOpPost) {
        ph.mode = kPhPost;
        ph.u = ph.b = L.xpre;
        ph.c = L.b;
        ph.dn = L.d0;
        ph.x = L.xout;
      } else if (op.kind == kOpPostStep) {
        ph.d = ph.x = L.xout;
      }
      stencil_phase<T, NB, SPLIT>(L, ph, smem, part, P.chunk,
                                  op.level == 0 ? mbar : mbar + 8 + op.level, op.level == 0,
                                  &failed);
    }
    if (t + 1 < P.nop && !grid_barrier_red(P.bar, P.fault, &sense)) {
      drain();
      return;
    }
    if (t == 0) prefetch_inverse();   // the stencil copies have gone before it
  }
  if (failed) *(volatile double *)P.fault = 1.0;
}

// shared memory per CTA, found and opted in to once per device
template <typename T, int NB, int SPLIT>
cudaError_t smem_limit(int dev, size_t *limit) {
  static size_t cached[64] = {0};
  size_t &c = cached[dev & 63];
  if (!c) {
    int opt = 0;
    cudaFuncAttributes fa{};
    cudaError_t err = cudaDeviceGetAttribute(&opt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (err == cudaSuccess)
      err = cudaFuncGetAttributes(&fa, (const void *)k_coarse_cycle<T, NB, SPLIT>);
    if (err != cudaSuccess) return err;
    const size_t lim = ((size_t)opt - fa.sharedSizeBytes) / 128 * 128;
    err = cudaFuncSetAttribute(k_coarse_cycle<T, NB, SPLIT>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lim);
    if (err != cudaSuccess) return err;
    c = lim;
  }
  *limit = c;
  return cudaSuccess;
}

template <typename T, int NB, int SPLIT>
cudaError_t launch_split(CoarseCycle<T> &P, cudaStream_t s) {
  using Sh = Shape<T, NB, SPLIT>;
  int dev = 0;
  cudaGetDevice(&dev);
  size_t lim = 0;
  if (cudaError_t err = smem_limit<T, NB, SPLIT>(dev, &lim); err != cudaSuccess) return err;
  // partial sums of up to kPartCap bytes, then the resident rows
  int npc = 32;
  for (int l = 0; l < P.nlev; ++l) npc = npc > P.lev[l].npc ? npc : P.lev[l].npc;
  const size_t per = Sh::kPart * sizeof(T);
  const int cap = (int)(Sh::kPartCap / per) / 32 * 32;
  P.chunk = (npc + 31) / 32 * 32 < cap ? (npc + 31) / 32 * 32 : cap;
  size_t used = per * P.chunk;
  const size_t dense = sizeof(double) * Sh::kWarps * NB;
  if (used < dense) used = dense;
  used = (used + 127) / 128 * 128;
  if (used > lim) return cudaErrorInvalidConfiguration;
  // the small levels whole first (their phases are pure latency), then what
  // fits of the top level
  for (int l = P.nlev - 1; l >= 0; --l) {
    CoarseLevel<T> &L = P.lev[l];
    const size_t row = (size_t)27 * L.npcp * sizeof(T);   // a multiple of 16
    const size_t fit = (lim - used) / row;
    L.gres = (int)(fit < 9 ? fit : 9);
    L.smem = (int)used;
    used += (L.gres * row + 127) / 128 * 128;   // lim is a multiple of 128
  }
  P.nop = 0;
  auto push = [&](CoarseKind kind, int l, int k = 1, int flip = 0) {
    P.op[P.nop++] = CoarseOp{kind, (int8_t)l, (int8_t)k, (int8_t)flip};
  };
  for (int l = 0; l < P.nlev; ++l) {
    push(P.lev[l].deg >= 2 ? kOpFirst : kOpStart, l);
    for (int k = 2; k < P.lev[l].deg; ++k) push(kOpStep, l, k, (k + 1) & 1);
    push(kOpRes, l);
    push(kOpRestrict, l);
  }
  push(kOpDense, 0);
  for (int l = P.nlev - 1; l >= 0; --l) {
    push(kOpProlong, l);
    push(kOpPost, l);
    for (int k = 1; k < P.lev[l].deg; ++k) push(kOpPostStep, l, k, (k + 1) & 1);
  }
  void *args[] = {&P};
  return cudaLaunchCooperativeKernel((const void *)k_coarse_cycle<T, NB, SPLIT>, coarse_ctas(dev),
                                     Sh::kThreads, args, used, s);
}

// Column blocks: nine units a node group where their partial sums fit at
// once, else three.  (8 FP32 columns of 33x17x17 nodes, 65 a CTA, are nine
// warps' work at three units; 8 FP64 columns of 49x25x25 would need 358 KB at
// nine.)
template <typename T, int NB>
cudaError_t launch_nb(CoarseCycle<T> &P, cudaStream_t s) {
  int npc = 0;
  for (int l = 0; l < P.nlev; ++l) npc = npc > P.lev[l].npc ? npc : P.lev[l].npc;
  const size_t need = (size_t)Shape<T, NB, 9>::kPart * sizeof(T) * ((npc + 31) / 32 * 32);
  if (need <= Shape<T, NB, 9>::kPartCap) return launch_split<T, NB, 9>(P, s);
  return launch_split<T, NB, 3>(P, s);
}

__global__ void k_coarse_slabs(int nn, int npc, int npcp, int ctas, const double *__restrict__ S,
                               double *__restrict__ A64, float *__restrict__ A32) {
  const int64_t total = (int64_t)ctas * 243 * npcp;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(t % npcp), q = (int)((t / npcp) % 243), s = (int)(t / (243 * (int64_t)npcp));
    const int n = s * npc + i;
    const double v = (i < npc && n < nn) ? S[(int64_t)q * nn + n] : 0.0;
    A64[t] = v;
    A32[t] = static_cast<float>(v);
  }
}

}  // namespace

int coarse_ctas(int dev) {
  static int cached[64] = {0};
  int &c = cached[dev & 63];
  if (!c) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1)
      n = 1;
    c = n;
  }
  return c;
}

void coarse_slab(int64_t nn, int ctas, int *npc, int *npcp) {
  *npc = (int)((nn + ctas - 1) / ctas);
  *npcp = (*npc + 3) / 4 * 4;
}

void launch_coarse_slabs(const Level &v, int ctas, const double *S, double *A64, float *A32,
                         cudaStream_t s) {
  int npc = 0, npcp = 0;
  coarse_slab(v.nn, ctas, &npc, &npcp);
  const int64_t total = (int64_t)ctas * 243 * npcp;
  const int64_t g = (total + 255) / 256;
  count_launch();
  k_coarse_slabs<<<(int)(g < 148 * 32 ? g : 148 * 32), 256, 0, s>>>((int)v.nn, npc, npcp, ctas, S,
                                                                    A64, A32);
}

template <typename T>
cudaError_t launch_coarse_cycle(CoarseCycle<T> P, cudaStream_t s) {
  count_launch();
  switch (P.nb) {
    case 1: return launch_split<T, 1, 9>(P, s);
    case 2: return launch_nb<T, 2>(P, s);
    case 4: return launch_nb<T, 4>(P, s);
    case 8: return launch_nb<T, 8>(P, s);
    default: return cudaErrorInvalidValue;
  }
}

template cudaError_t launch_coarse_cycle<double>(CoarseCycle<double>, cudaStream_t);
template cudaError_t launch_coarse_cycle<float>(CoarseCycle<float>, cudaStream_t);

}  // namespace tpo
