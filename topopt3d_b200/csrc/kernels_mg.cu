// Geometric multigrid kernels: Galerkin coarse operators, stencil operator
// on the coarse levels, trilinear transfers, Chebyshev/Jacobi smoother
// updates and the dense coarsest-level solve.
//
// Level layout (Interpolation.cpp:31-169): a coarse node sits on every even
// fine node index; level l+1 has (N_l + 1) / 2 nodes per dimension,
// numbered lexicographically.  The prolongation weight of coarse node c for
// fine node f is prod_d w_d with w_d = 1 (f_d = 2c_d) or 1/2 (|f_d - 2c_d| =
// 1), each row normalised to sum 1 (Interpolation.cpp:330-347).  The
// normalisation factorises per dimension, so weights are computed on the
// fly from the indices; no interpolation matrix is stored.
//
// Coarse operators are A_{l+1} = P^T A_l P (PCMG Galerkin,
// FEAnalysis.cpp:412), stored as 27-point 3x3-block stencils in SoA form
// S[(nb*9 + 3r + s) * nn + node].
#include <algorithm>

#include "tpo_internal.h"
#include "fused_out.cuh"
#include "pdl.cuh"

namespace tpo {

namespace {

int grid_for(int64_t n, int threads, int64_t cap = 148 * 32) {
  int64_t g = (n + threads - 1) / threads;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

// normalised 1-D prolongation weight of coarse index c for fine index f
// (fine extent Nf)
__device__ __forceinline__ double pw1(int f, int c, int Nf) {
  const int d = f - 2 * c;
  if (d < -1 || d > 1) return 0.0;
  if (d == 0) return 1.0;
  // odd f: neighbours (f-1)/2 always, (f+1)/2 if f+1 <= Nf-1
  return (f + 1 <= Nf - 1) ? 0.5 : 1.0;
}

// ---- level 1 straight from the element moduli ----------------------------
//
// A_1 = P^T A_0 P with A_0 = M (sum_e E_e K0_e) M + (I - M), M the mask of
// dofs without an identity row (idm).  Every fine element lies inside one
// level-1 coarse element (2x2x2 fine elements) and its 8 nodes interpolate
// from that coarse element's 8 nodes, so
//   A_1 = sum_E sum_{e in E} E_e Q_e^T (M K0 M) Q_e + P^T (I - M) P.
// For a fine element without identity dofs at offset i of a coarse element
// with all 8 corners, Q_e^T K0 Q_e is one of 8 fixed 24x24 matrices (GMi,
// element.cpp); the 3x3 block (ln, lm) of the coarse stencil is then
// sum_i E_{e_i} GMi[i][ln][lm].  Coarse elements whose closed fine box holds
// an identity dof, or that miss a corner (odd element counts), take the
// general path: masked K0 with the interpolation weights of pw1.

// slot[E] >= 0: level-1 coarse element E needs the general path (an
// identity dof in its closed fine box, or a missing corner); slots are
// handed out by an atomic counter (their order does not affect any value)
__global__ void k_coarse_elem_flags(int nelx, int nely, int nelz,
                                    const uint8_t *__restrict__ idm,
                                    int *__restrict__ slot,
                                    int *__restrict__ slot_elem,
                                    unsigned int *__restrict__ count) {
  const int fx = nelx + 1, fy = nely + 1, fz = nelz + 1;
  const int ncx = (nelx + 1) / 2, ncy = (nely + 1) / 2, ncz = (nelz + 1) / 2;
  const int64_t nce = (int64_t)ncx * ncy * ncz;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nce;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int ex = (int)(t % ncx), ey = (int)((t / ncx) % ncy), ez = (int)(t / ((int64_t)ncx * ncy));
    unsigned any = (2 * ex + 2 > fx - 1) || (2 * ey + 2 > fy - 1) || (2 * ez + 2 > fz - 1);
    for (int z = 2 * ez; z <= min(2 * ez + 2, fz - 1) && !any; ++z)
      for (int y = 2 * ey; y <= min(2 * ey + 2, fy - 1); ++y)
        for (int x = 2 * ex; x <= min(2 * ex + 2, fx - 1); ++x)
          any |= idm[((int64_t)z * fy + y) * fx + x];
    int sl = -1;
    if (any) {
      sl = (int)atomicAdd(count, 1u);
      slot_elem[sl] = (int)t;
    }
    slot[t] = sl;
  }
}

// general path: the 3x3 block (ln, lm) of a flagged coarse element,
// sum_{fine e in E} E_e sum_{p,q} w(p->ln) w(q->lm) (M K0 M)_pq with the
// interpolation weights of pw1 and the identity-dof masks.  A CTA takes one
// (ln, lm) of 32 elements, a warp one of their fine elements i, so that which
// of the 64 corner pairs have a weight is the same for a warp and the others
// are skipped (a thread per block, or lanes of different i, went through all:
// 184 and 241 us for the 2,304 elements of a 192x96x96 cantilever's face; now
// 121 us).  A fine element without identity dofs uses its fixed block.  The
// eight sums are added in order.
__global__ void __launch_bounds__(256)
    k_galerkin_general(int nelx, int nely, int nelz, int nslots, const double *__restrict__ E,
                       const uint8_t *__restrict__ idm, const int *__restrict__ slot_elem,
                       const double *__restrict__ K0lex, const double *__restrict__ GMi,
                       double *__restrict__ G) {
  __shared__ double K0[576];
  __shared__ double sum[8][9][32];
  for (int e = threadIdx.x; e < 576; e += 256) K0[e] = K0lex[e];
  __syncthreads();
  const int fx = nelx + 1, fy = nely + 1, fz = nelz + 1;
  const int ncx = (nelx + 1) / 2, ncy = (nely + 1) / 2;
  const int lane = threadIdx.x & 31, i = threadIdx.x >> 5;
  const int ln = blockIdx.y / 8, lm = blockIdx.y % 8;
  const int sl = blockIdx.x * 32 + lane;
  double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (sl < nslots) {
    const int ce = slot_elem[sl];
    const int EI = ce % ncx, EJ = (ce / ncx) % ncy, EK = ce / (ncx * ncy);
    const int ex = 2 * EI + (i & 1), ey = 2 * EJ + ((i >> 1) & 1), ez = 2 * EK + ((i >> 2) & 1);
    if (ex < nelx && ey < nely && ez < nelz) {
      const double Ee = E[((int64_t)ez * nely + ey) * nelx + ex];
      // 1-D weights of the two corners of the fine element per dimension
      // (zero where a far coarse corner does not exist)
      const int f0[3] = {ex, ey, ez}, C[3] = {EI, EJ, EK}, N[3] = {fx, fy, fz};
      double wn[3][2], wm[3][2];
#pragma unroll
      for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          wn[d][t] = pw1(f0[d] + t, C[d] + ((ln >> d) & 1), N[d]);
          wm[d][t] = pw1(f0[d] + t, C[d] + ((lm >> d) & 1), N[d]);
        }
      unsigned msk[8];
#pragma unroll
      for (int p = 0; p < 8; ++p)
        msk[p] = idm[((int64_t)(ez + (p >> 2)) * fy + ey + ((p >> 1) & 1)) * fx + ex + (p & 1)];
      // no identity dof here and all coarse corners there: the fixed block
      const bool plain = !(msk[0] | msk[1] | msk[2] | msk[3] | msk[4] | msk[5] | msk[6] | msk[7]) &&
                         2 * EI + 2 <= nelx && 2 * EJ + 2 <= nely && 2 * EK + 2 <= nelz;
      if (plain) {
        const double *m = GMi + ((i * 8 + ln) * 8 + lm) * 9;
#pragma unroll
        for (int q = 0; q < 9; ++q) acc[q] = Ee * m[q];
      }
      // corner p of fine element i lies at t = i + p per dimension from the
      // coarse element's origin: no weight on ln when |t - 2 ln| = 2
      auto off = [&](int p, int l) {
        bool z = false;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const int t = ((i >> d) & 1) + ((p >> d) & 1) - 2 * ((l >> d) & 1);
          z |= t == 2 || t == -2;
        }
        return z;
      };
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        if (plain || off(p, ln)) continue;
        const double wp = Ee * (wn[0][p & 1] * wn[1][(p >> 1) & 1] * wn[2][p >> 2]);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          if (off(q, lm)) continue;
          const double w = wp * (wm[0][q & 1] * wm[1][(q >> 1) & 1] * wm[2][q >> 2]);
          const double *k0 = K0 + 24 * (3 * p) + 3 * q;
#pragma unroll
          for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c)
              if (!(((msk[p] >> r) | (msk[q] >> c)) & 1u)) acc[3 * r + c] += w * k0[24 * r + c];
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 9; ++q) sum[i][q][lane] = acc[q];
  __syncthreads();
  for (int e = threadIdx.x; e < 288; e += 256) {
    const int s = e / 9, q = e % 9;
    if (blockIdx.x * 32 + s >= nslots) continue;
    double v = sum[0][q][s];
#pragma unroll
    for (int k = 1; k < 8; ++k) v += sum[k][q][s];
    G[((int64_t)(blockIdx.x * 32 + s) * 64 + blockIdx.y) * 9 + q] = v;
  }
}

// The FP32 copy of a half-stored stencil is grouped by tiles of 32 nodes:
// coefficient hq (0..125) of node n at ((n / 32) * 126 + hq) * 32 + n % 32,
// so the 126 x 32 values a warp reads for its 32 nodes are one contiguous
// 16,128-byte block that one bulk L2 prefetch covers.  The FP64 form is the
// second half of the full stencil itself, coefficient-major, hq * nn + n.
constexpr int kH32Tile = 32;
__host__ __device__ __forceinline__ int64_t h32_index(int hq, int64_t n) {
  return ((n / kH32Tile) * 126 + hq) * kH32Tile + n % kH32Tile;
}

// the level-1 stencil: per (coarse node, neighbour) block, the fast-path
// element sums, the general-path blocks of flagged elements and the
// P^T (I - M) P term of the identity dofs.  blockIdx.y = h: the centre block
// (h = 0) and the 13 forward ones, nb = 13 + h; the operator is symmetric, so
// the block goes, transposed, to the neighbour as well (26 - nb).  h fixes
// the elements a block sums over and their GMi blocks, so those are uniform
// over a CTA and come from shared memory, two at a time, for the two nodes
// of a thread.  (Every block summed by itself, GMi read through L1, took 416
// us at 192x96x96, and a second pass of 126 us split off the half stencil;
// this form takes 225 us; its 570 MB of writes would take 88 us and its FP64
// arithmetic 33 us.)  The FP32 half stencil and
// the inverse diagonal are written on the way.
constexpr int kGfThreads = 128, kGfNodes = 2;
__global__ void __launch_bounds__(kGfThreads)
    k_galerkin_fine(int nelx, int nely, int nelz, const double *__restrict__ E,
                    const uint8_t *__restrict__ idm, const int *__restrict__ slot,
                    const double *__restrict__ G, const double *__restrict__ GMi,
                    double *__restrict__ Sc, float *__restrict__ H32,
                    double *__restrict__ dinv64, float *__restrict__ dinv32) {
  // GMi blocks of this h: (element, i) x 9, padded to 10 for 16-byte reads
  __shared__ __align__(16) double Gs[8 * 8 * 10];
  const int fx = nelx + 1, fy = nely + 1, fz = nelz + 1;
  const int cx = (fx + 1) / 2, cy = (fy + 1) / 2, cz = (fz + 1) / 2;
  const int ncx = (nelx + 1) / 2, ncy = (nely + 1) / 2, ncz = (nelz + 1) / 2;
  const int nnc = cx * cy * cz;
  const int h = blockIdx.y, nb = 13 + h;
  const int dx = nb % 3 - 1, dy = (nb / 3) % 3 - 1, dz = nb / 9 - 1;
  // the elements holding both nodes: EI = ix - 1 + a with a in [a0, a1]
  const int a0 = dx > 0, a1 = dx >= 0, b0 = dy > 0, b1 = dy >= 0, c0 = dz > 0, c1 = dz >= 0;
  const int na = a1 - a0 + 1, nbb = b1 - b0 + 1, nel = na * nbb * (c1 - c0 + 1);
  for (int t = threadIdx.x; t < nel * 72; t += kGfThreads) {
    const int e = t / 72, i = (t / 9) % 8, q = t % 9;
    const int a = a0 + e % na, b = b0 + (e / na) % nbb, c = c0 + e / (na * nbb);
    const int ln = (1 - a) + 2 * (1 - b) + 4 * (1 - c);
    const int lm = (1 - a + dx) + 2 * (1 - b + dy) + 4 * (1 - c + dz);
    Gs[(e * 8 + i) * 10 + q] = GMi[((i * 8 + ln) * 8 + lm) * 9 + q];
  }
  __syncthreads();
  int I[kGfNodes], ix[kGfNodes], iy[kGfNodes], iz[kGfNodes];
  double acc[kGfNodes][9];
  bool anyflag[kGfNodes];
#pragma unroll
  for (int u = 0; u < kGfNodes; ++u) {
    I[u] = (blockIdx.x * kGfNodes + u) * kGfThreads + threadIdx.x;
    const int n = min(I[u], nnc - 1);
    ix[u] = n % cx;
    iy[u] = (n / cx) % cy;
    iz[u] = n / (cx * cy);
    anyflag[u] = false;
#pragma unroll
    for (int q = 0; q < 9; ++q) acc[u][q] = 0.0;
  }
  for (int e = 0; e < nel; ++e) {
    const int a = a0 + (e & (na - 1)), b = b0 + ((e >> (na - 1)) & (nbb - 1)),
              c = c0 + (e >> (na + nbb - 2));   // na, nbb are 1 or 2
    // slots and moduli together; a flagged element's moduli are then dropped
    double Ee[kGfNodes][8];
    int sl[kGfNodes];
#pragma unroll
    for (int u = 0; u < kGfNodes; ++u) {
      const int EI = ix[u] - 1 + a, EJ = iy[u] - 1 + b, EK = iz[u] - 1 + c;
      const bool in = EI >= 0 && EJ >= 0 && EK >= 0 && EI < ncx && EJ < ncy && EK < ncz;
      const int ei = min(max(EI, 0), ncx - 1), ej = min(max(EJ, 0), ncy - 1),
                ek = min(max(EK, 0), ncz - 1);
      const int s0 = slot[(ek * ncy + ej) * ncx + ei];
      sl[u] = in ? s0 : -1;
      // unconditional loads: an element outside is clamped and zeroed below;
      // a missing last fine element (odd counts) belongs to a flagged one
      const int ox = 2 * ei + 1 < nelx, oy = 2 * ej + 1 < nely ? nelx : 0,
                oz = 2 * ek + 1 < nelz ? nelx * nely : 0;
      const double *row = E + ((2 * ek * nely + 2 * ej) * nelx + 2 * ei);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        Ee[u][i] = row[((i & 1) ? ox : 0) + ((i & 2) ? oy : 0) + ((i & 4) ? oz : 0)];
      if (!in) {
#pragma unroll
        for (int i = 0; i < 8; ++i) Ee[u][i] = 0.0;
      }
    }
#pragma unroll
    for (int u = 0; u < kGfNodes; ++u)
      if (sl[u] >= 0) {   // the general path's block instead
        anyflag[u] = true;
        const int ln = (1 - a) + 2 * (1 - b) + 4 * (1 - c);
        const int lm = (1 - a + dx) + 2 * (1 - b + dy) + 4 * (1 - c + dz);
        const double *g = G + ((int64_t)sl[u] * 64 + ln * 8 + lm) * 9;
#pragma unroll
        for (int q = 0; q < 9; ++q) acc[u][q] += g[q];
#pragma unroll
        for (int i = 0; i < 8; ++i) Ee[u][i] = 0.0;
      }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const double2 *m2 = reinterpret_cast<const double2 *>(Gs + (e * 8 + i) * 10);
      const double2 p0 = m2[0], p1 = m2[1], p2 = m2[2], p3 = m2[3];
      const double m[9] = {p0.x, p0.y, p1.x, p1.y, p2.x, p2.y, p3.x, p3.y,
                           Gs[(e * 8 + i) * 10 + 8]};
#pragma unroll
      for (int u = 0; u < kGfNodes; ++u)
#pragma unroll
        for (int q = 0; q < 9; ++q) acc[u][q] = fma(Ee[u][i], m[q], acc[u][q]);
    }
  }
#pragma unroll
  for (int u = 0; u < kGfNodes; ++u) {
    if (I[u] >= nnc) continue;
    const int jx = ix[u] + dx, jy = iy[u] + dy, jz = iz[u] + dz;
    const bool inside = jx >= 0 && jx < cx && jy >= 0 && jy < cy && jz >= 0 && jz < cz;
    if (inside && anyflag[u]) {
      // P^T (I - M) P: identity dofs in the support of both N and M
      for (int gz = max(2 * iz[u], 2 * jz) - 1; gz <= min(2 * iz[u], 2 * jz) + 1; ++gz)
        for (int gy = max(2 * iy[u], 2 * jy) - 1; gy <= min(2 * iy[u], 2 * jy) + 1; ++gy)
          for (int gx = max(2 * ix[u], 2 * jx) - 1; gx <= min(2 * ix[u], 2 * jx) + 1; ++gx) {
            if (gx < 0 || gy < 0 || gz < 0 || gx >= fx || gy >= fy || gz >= fz) continue;
            const unsigned bits = idm[((int64_t)gz * fy + gy) * fx + gx];
            if (!bits) continue;
            const double w = pw1(gx, ix[u], fx) * pw1(gy, iy[u], fy) * pw1(gz, iz[u], fz) *
                             pw1(gx, jx, fx) * pw1(gy, jy, fy) * pw1(gz, jz, fz);
#pragma unroll
            for (int c = 0; c < 3; ++c)
              if ((bits >> c) & 1u) acc[u][4 * c] += w;
          }
    }
    const int J = I[u] + (dz * cy + dy) * cx + dx;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const double v = inside ? acc[u][q] : 0.0;
      Sc[(int64_t)(nb * 9 + q) * nnc + I[u]] = v;
      if (h > 0 && inside)
        Sc[(int64_t)((26 - nb) * 9 + 3 * (q % 3) + q / 3) * nnc + J] = v;
      if (H32) H32[h32_index(h * 9 + q, I[u])] = static_cast<float>(v);
    }
    // the backward block of a node without that neighbour
    const int kx = ix[u] - dx, ky = iy[u] - dy, kz = iz[u] - dz;
    if (!(kx >= 0 && kx < cx && ky >= 0 && ky < cy && kz >= 0 && kz < cz)) {
#pragma unroll
      for (int q = 0; q < 9; ++q) Sc[(int64_t)((26 - nb) * 9 + q) * nnc + I[u]] = 0.0;
    }
    if (h == 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        dinv64[3 * (int64_t)I[u] + c] = 1.0 / acc[u][4 * c];
        dinv32[3 * (int64_t)I[u] + c] = static_cast<float>(1.0 / acc[u][4 * c]);
      }
    }
  }
}

// One dimension of the Galerkin product: P = P_x (x) P_y (x) P_z, so
// P^T A P = P_z^T (P_y^T (P_x^T A P_x) P_y) P_z and each factor keeps a
// 27-point 3x3-block stencil.  Coarsening dimension D of a grid n[3]:
//   A'(O, O+Delta) = sum_{f_D} sum_{g_D = f_D + d_D} w(f_D -> O_D)
//                    w(g_D -> O_D + Delta_D) A(f, f + d),
// with f = O except f_D and d = Delta except d_D: at most 7 (Delta_D = 0)
// or 3 input blocks per output block, instead of up to 343 for the direct
// triple product.  w is the normalised 1-D weight pw1.
template <int D>
__global__ void k_galerkin_dim(int nx, int ny, int nz, const double *__restrict__ Sin,
                               double *__restrict__ Sout) {
  const int n[3] = {nx, ny, nz};
  int m[3] = {nx, ny, nz};
  m[D] = (n[D] + 1) / 2;
  const int64_t nin = (int64_t)nx * ny * nz, nout = (int64_t)m[0] * m[1] * m[2];
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < 27 * nout;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int nb = (int)(t / nout);
    const int64_t O = t - (int64_t)nb * nout;
    int o[3] = {(int)(O % m[0]), (int)((O / m[0]) % m[1]), (int)(O / ((int64_t)m[0] * m[1]))};
    const int dl[3] = {nb % 3 - 1, (nb / 3) % 3 - 1, nb / 9 - 1};
    double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    bool inside = true;
#pragma unroll
    for (int e = 0; e < 3; ++e) inside &= (o[e] + dl[e] >= 0 && o[e] + dl[e] < m[e]);
    if (inside) {
      const int I = o[D], J = o[D] + dl[D];
      for (int fd = 2 * I - 1; fd <= 2 * I + 1; ++fd) {
        if (fd < 0 || fd >= n[D]) continue;
        const double wi = pw1(fd, I, n[D]);
        if (wi == 0.0) continue;
        int f[3] = {o[0], o[1], o[2]};
        f[D] = fd;
        const int64_t fi = ((int64_t)f[2] * ny + f[1]) * nx + f[0];
        for (int dd = -1; dd <= 1; ++dd) {
          const int gd = fd + dd;
          if (gd < 0 || gd >= n[D]) continue;
          const double wj = pw1(gd, J, n[D]);
          if (wj == 0.0) continue;
          int d3[3] = {dl[0], dl[1], dl[2]};
          d3[D] = dd;
          const int fnb = (d3[2] + 1) * 9 + (d3[1] + 1) * 3 + (d3[0] + 1);
          const double w = wi * wj;
          const double *blk = Sin + (int64_t)fnb * 9 * nin + fi;
#pragma unroll
          for (int q = 0; q < 9; ++q) acc[q] += w * blk[q * nin];
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) Sout[(int64_t)(nb * 9 + q) * nout + O] = acc[q];
  }
}


// 32 nodes x 9 neighbour rows per CTA: thread (lane, g) takes node
// 32 * block + lane and the three neighbour blocks of row g = (dj, dk),
// i.e. 27 coefficient and 9 u loads, so the loads of a node are spread
// over 9 threads instead of one 324-load chain (the levels this kernel
// serves are small and latency-bound); the 9 partial sums are combined in
// shared memory in a fixed order.  Lanes span consecutive nodes, so each
// coefficient load is coalesced.
constexpr int kStencilRows = 9;
template <typename T, int OUT>
__global__ void __launch_bounds__(32 * kStencilRows)
    k_apply_stencil(int nx, int ny, int nz, const T *__restrict__ S,
                    const T *__restrict__ u, const T *__restrict__ b,
                    const T *__restrict__ dinv, T *__restrict__ y) {
  __shared__ T part[kStencilRows][3][32];
  const int64_t nn = (int64_t)nx * ny * nz;
  const int lane = threadIdx.x, g = threadIdx.y;
  const int dj = g % 3 - 1, dk = g / 3 - 1;
  for (int64_t n0 = (int64_t)blockIdx.x * 32; n0 < nn; n0 += (int64_t)gridDim.x * 32) {
    const int64_t n = n0 + lane;
    T a0 = 0, a1 = 0, a2 = 0;
    if (n < nn) {
      const int i = (int)(n % nx), j = (int)((n / nx) % ny), k = (int)(n / ((int64_t)nx * ny));
      const int mj = j + dj, mk = k + dk;
      if (mj >= 0 && mj < ny && mk >= 0 && mk < nz) {
#pragma unroll
        for (int di = -1; di <= 1; ++di) {
          const int mi = i + di;
          if (mi < 0 || mi >= nx) continue;
          const int nb = g * 3 + di + 1;
          const int64_t m = ((int64_t)mk * ny + mj) * nx + mi;
          const T u0 = u[3 * m], u1 = u[3 * m + 1], u2 = u[3 * m + 2];
          const T *s = S + (int64_t)nb * 9 * nn + n;
          a0 += s[0] * u0 + s[nn] * u1 + s[2 * nn] * u2;
          a1 += s[3 * nn] * u0 + s[4 * nn] * u1 + s[5 * nn] * u2;
          a2 += s[6 * nn] * u0 + s[7 * nn] * u1 + s[8 * nn] * u2;
        }
      }
    }
    part[g][0][lane] = a0;
    part[g][1][lane] = a1;
    part[g][2][lane] = a2;
    __syncthreads();
    if (g < 3 && n < nn) {
      T a = 0;
#pragma unroll
      for (int r = 0; r < kStencilRows; ++r) a += part[r][g][lane];
      if (OUT == OUT_RESID) a = b[3 * n + g] - a;
      if (OUT == OUT_SCALE) a *= dinv[3 * n + g];
      y[3 * n + g] = a;
    }
    __syncthreads();
  }
}

template <typename T>
__device__ __forceinline__ const T *hcoef(const T *H, int hq, int64_t n, int64_t nn);
template <>
__device__ __forceinline__ const double *hcoef(const double *H, int hq, int64_t n,
                                               int64_t nn) {
  return H + hq * nn + n;
}
template <>
__device__ __forceinline__ const float *hcoef(const float *H, int hq, int64_t n, int64_t) {
  return H + h32_index(hq, n);
}
// one bulk prefetch of a 32-node tile of the FP32 stencil into L2
__device__ __forceinline__ void prefetch_h32_tile(const float *H, int64_t n) {
  const float *p = H + (n / kH32Tile) * 126 * kH32Tile;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p),
               "r"(126 * kH32Tile * 4)
               : "memory");
}

// Symmetric half of a Galerkin stencil: A(n, n+d) = A(n+d, n)^T, so the
// apply needs only the centre block and the 13 forward offsets (nb =
// 13..26), H[(h*9 + 3r + s) * nn + n] with h = nb - 13: in FP64 the second
// half of the stencil in place, in FP32 a copy.  The apply reads the forward
// blocks of node n and, transposed, the forward blocks that its 13 backward
// neighbours store for it; those were read moments earlier by the
// neighbouring threads, so the second read hits L2 and DRAM traffic is the
// half-size array.
__global__ void k_stencil_to_half(int64_t nn, const double *__restrict__ H64,
                                  float *__restrict__ H32) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < 126 * nn;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t hq = t / nn, n = t - hq * nn;
    H32[h32_index((int)hq, n)] = static_cast<float>(H64[t]);
  }
}

// The kernel is bound by the latency of the coefficient loads.  The block
// loop is not unrolled, so a thread needs 32 registers and 16 blocks of 128
// fit on an SM: the 97x49x49 level 1 of 192x96x96 then runs in one wave at
// full occupancy.  Fully unrolled it took 64 registers, half the warps and
// 1.5 waves, and a solve was 1.4% (FP32) / 5.6% (FP64) slower.
template <typename T, int IN, int OUT>
__global__ void __launch_bounds__(128, 16)
    k_apply_stencil_sym1(int nx, int ny, int nz, const T *__restrict__ H,
                         const ApplyArgs<T> args) {
  const int nn = nx * ny * nz;
  // stride between the 9 coefficients of one block
  const int64_t qs = sizeof(T) == 4 ? kH32Tile : (int64_t)nn;
  const int stride = gridDim.x * blockDim.x;
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nn; n += stride) {
    // FP32: a warp's 32 nodes are one tile of the stencil; the tile this
    // warp takes next goes to L2 in one bulk prefetch
    if (sizeof(T) == 4 && (threadIdx.x & 31) == 0 && n + stride < nn)
      prefetch_h32_tile(reinterpret_cast<const float *>(H), n + stride);
    const int i = n % nx, j = (n / nx) % ny, k = n / (nx * ny);
    T a0 = 0, a1 = 0, a2 = 0;
#pragma unroll 1
    for (int h = 0; h < 14; ++h) {
      const int nb = 13 + h;
      const int di = nb % 3 - 1, dj = (nb / 3) % 3 - 1, dk = nb / 9 - 1;
      // forward block A(n, n+d): zero when n+d is outside, index clamped
      {
        const int mi = min(i + di, nx - 1), mj = min(max(j + dj, 0), ny - 1),
                  mk = min(k + dk, nz - 1);
        const int m = (mk * ny + mj) * nx + max(mi, 0);
        const T u0 = sym_in<T, IN>(args, 3 * m), u1 = sym_in<T, IN>(args, 3 * m + 1),
                u2 = sym_in<T, IN>(args, 3 * m + 2);
        const T *s = hcoef(H, h * 9, n, nn);
        a0 += s[0] * u0 + s[qs] * u1 + s[2 * qs] * u2;
        a1 += s[3 * qs] * u0 + s[4 * qs] * u1 + s[5 * qs] * u2;
        a2 += s[6 * qs] * u0 + s[7 * qs] * u1 + s[8 * qs] * u2;
      }
      // backward block A(n, n-d) = A(n-d, n)^T, stored by node n-d
      if (h > 0) {
        const int mi = i - di, mj = j - dj, mk = k - dk;
        const bool in = mi >= 0 && mi < nx && mj >= 0 && mj < ny && mk >= 0 && mk < nz;
        const int m = in ? (mk * ny + mj) * nx + mi : n;
        const T w = in ? T(1) : T(0);
        const T u0 = w * sym_in<T, IN>(args, 3 * m), u1 = w * sym_in<T, IN>(args, 3 * m + 1),
                u2 = w * sym_in<T, IN>(args, 3 * m + 2);
        const T *s = hcoef(H, h * 9, m, nn);
        a0 += s[0] * u0 + s[3 * qs] * u1 + s[6 * qs] * u2;
        a1 += s[qs] * u0 + s[4 * qs] * u1 + s[7 * qs] * u2;
        a2 += s[2 * qs] * u0 + s[5 * qs] * u1 + s[8 * qs] * u2;
      }
    }
    const bool need_u = OUT == OUT_CHEB2 || OUT == OUT_POST0 || OUT == OUT_POST1;
    const T Au[3] = {a0, a1, a2};
#pragma unroll
    for (int c = 0; c < 3; ++c)
      sym_out<T, OUT>(args, 3 * n + c, Au[c], need_u ? sym_in<T, IN>(args, 3 * n + c) : T(0));
  }
}

// NB columns (stride ld) share every coefficient load
template <typename T, bool RESID, int NB>
__global__ void k_apply_stencil_sym(int nx, int ny, int nz,
                                    const T *__restrict__ H,
                                    const T *__restrict__ u,
                                    const T *__restrict__ b, T *__restrict__ y,
                                    int64_t ld) {
  const int nn = nx * ny * nz;
  const int64_t qs = sizeof(T) == 4 ? kH32Tile : (int64_t)nn;
  const int stride = gridDim.x * blockDim.x;
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nn; n += stride) {
    if (sizeof(T) == 4 && (threadIdx.x & 31) == 0 && n + stride < nn)
      prefetch_h32_tile(reinterpret_cast<const float *>(H), n + stride);
    const int i = n % nx, j = (n / nx) % ny, k = n / (nx * ny);
    T a[NB][3];
#pragma unroll
    for (int col = 0; col < NB; ++col) a[col][0] = a[col][1] = a[col][2] = T(0);
#pragma unroll
    for (int h = 0; h < 14; ++h) {
      const int nb = 13 + h;
      const int di = nb % 3 - 1, dj = (nb / 3) % 3 - 1, dk = nb / 9 - 1;
      // forward block A(n, n+d): zero when n+d is outside, index clamped
      {
        const int mi = min(i + di, nx - 1), mj = min(max(j + dj, 0), ny - 1),
                  mk = min(k + dk, nz - 1);
        const int m = (mk * ny + mj) * nx + max(mi, 0);
        const T *sp = hcoef(H, h * 9, n, nn);
        T c[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) c[q] = sp[q * qs];
#pragma unroll
        for (int col = 0; col < NB; ++col) {
          const T *uc = u + col * ld;
          const T u0 = uc[3 * m], u1 = uc[3 * m + 1], u2 = uc[3 * m + 2];
          a[col][0] += c[0] * u0 + c[1] * u1 + c[2] * u2;
          a[col][1] += c[3] * u0 + c[4] * u1 + c[5] * u2;
          a[col][2] += c[6] * u0 + c[7] * u1 + c[8] * u2;
        }
      }
      // backward block A(n, n-d) = A(n-d, n)^T, stored by node n-d
      if (h > 0) {
        const int mi = i - di, mj = j - dj, mk = k - dk;
        const bool in = mi >= 0 && mi < nx && mj >= 0 && mj < ny && mk >= 0 && mk < nz;
        const int m = in ? (mk * ny + mj) * nx + mi : n;
        const T w = in ? T(1) : T(0);
        const T *sp = hcoef(H, h * 9, m, nn);
        T c[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) c[q] = sp[q * qs];
#pragma unroll
        for (int col = 0; col < NB; ++col) {
          const T *uc = u + col * ld;
          const T u0 = w * uc[3 * m], u1 = w * uc[3 * m + 1], u2 = w * uc[3 * m + 2];
          a[col][0] += c[0] * u0 + c[3] * u1 + c[6] * u2;
          a[col][1] += c[1] * u0 + c[4] * u1 + c[7] * u2;
          a[col][2] += c[2] * u0 + c[5] * u1 + c[8] * u2;
        }
      }
    }
#pragma unroll
    for (int col = 0; col < NB; ++col) {
      T *yc = y + col * ld;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        T v = a[col][q];
        if (RESID) v = b[col * ld + 3 * n + q] - v;
        yc[3 * n + q] = v;
      }
    }
  }
}

__global__ void k_stencil_diag(int64_t nn, const double *__restrict__ S,
                               double *dinv64, float *dinv32) {
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < nn;
       n += (int64_t)gridDim.x * blockDim.x) {
    for (int c = 0; c < 3; ++c) {
      const double d = S[(int64_t)(13 * 9 + 4 * c) * nn + n];
      dinv64[3 * n + c] = 1.0 / d;
      dinv32[3 * n + c] = static_cast<float>(1.0 / d);
    }
  }
}

// The transfers are separable, P = Px (x) Py (x) Pz, and both kernels give a
// thread one coarse index along x for one coarse (restriction) or fine
// (prolongation) y and z: consecutive lanes are consecutive coarse nodes, each
// value is loaded once per (y, z) pair that needs it, and the x direction takes
// the neighbouring lane's value (the lane at a warp's edge loads it).  One
// thread per output node with all of its 27 or 8 taps took, at 192x96x96 in
// FP32, 17 us for the restriction and 29 us for the prolongation (8 and 10 us
// on level 1); these take 10 and 17 us (6 and 6 us); 8 columns of 128x64x64,
// 37 and 44 us before, 19 and 35 us now.  A copy of the bytes takes 4 and 7
// us; both are bound by their instructions.

// weights of the three fine indices 2 c - 1, 2 c, 2 c + 1 around coarse c
template <typename T>
__device__ __forceinline__ void tap_weights(int c, int N, T (&w)[3]) {
  const int f = 2 * c;
  w[0] = f - 1 >= 0 ? T(0.5) : T(0);
  w[1] = T(1);
  w[2] = f + 1 < N ? (f + 2 < N ? T(0.5) : T(1)) : T(0);
}

// b_c = P^T r_f for nb columns (fine stride 3 nnf, coarse stride 3 nnc);
// COMP: b_c component by component, with the first Chebyshev direction.
// blockIdx.z = column; a thread per coarse node
template <typename T, bool COMP>
__global__ void __launch_bounds__(128)
    k_restrict(int fx, int fy, int fz, int cx, int cy, int cz, const T *rf, T *__restrict__ bc,
               const CompLevel<T> comp) {
  const int lane = threadIdx.x & 31;
  const int nnc = cx * cy * cz, t = (int)blockIdx.x * 128 + threadIdx.x;
  const int I = min(t, nnc - 1);
  const int ix = I % cx, iy = (I / cx) % cy, iz = I / (cx * cy);
  const int col = blockIdx.z;
  rf += col * 3 * ((int64_t)fx * fy * fz);
  T wx[3], wy[3], wz[3];
  tap_weights(ix, fx, wx);
  tap_weights(iy, fy, wy);
  tap_weights(iz, fz, wz);
  pdl_wait();
  const bool first = lane == 0 && ix > 0;   // loads its own left neighbour
  T s[3] = {T(0), T(0), T(0)};
  const int dl = ix > 0 ? -3 : 0, d1 = 2 * ix + 1 < fx ? 3 : 0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int z = min(max(2 * iz + c - 1, 0), fz - 1);
    T a0[3][3], a1[3][3], am[3][3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int y = min(max(2 * iy + b - 1, 0), fy - 1);
      const T *p = rf + 3 * ((z * fy + y) * fx + 2 * ix);   // 32-bit: 3 nn < 2^31
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        a0[b][q] = load_ro(p + q);
        a1[b][q] = load_ro(p + d1 + q);
        am[b][q] = first ? load_ro(p + dl + q) : T(0);
      }
    }
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const T wyz = wy[b] * wz[c];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        T left = __shfl_up_sync(0xffffffffu, a1[b][q], 1);
        if (lane == 0 || ix == 0) left = am[b][q];
        s[q] += wyz * (wx[0] * left + a0[b][q] + wx[2] * a1[b][q]);
      }
    }
  }
  if (t >= nnc) return;
  T *o = bc + col * 3 * (int64_t)nnc;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (COMP) {
      o[q * (int64_t)nnc + I] = s[q];
      comp.d0[(3 * col + q) * (int64_t)nnc + I] = comp.inv_theta * (comp.dinv[3 * I + q] * s[q]);
    } else {
      o[3 * I + q] = s[q];
    }
  }
  pdl_launch_dependents();
}

// x_f += P x_c for nb columns; COMP: x_c component by component.
// blockIdx.z = column; a thread per (coarse ix, fine gy, gz), writing the fine
// nodes 2 ix and 2 ix + 1
template <typename T, bool COMP>
__global__ void __launch_bounds__(128)
    k_prolong_add(int fx, int fy, int fz, int cx, int cy, int cz, const T *xc, T *__restrict__ xf) {
  const int lane = threadIdx.x & 31;
  const int total = cx * fy * fz, t = (int)blockIdx.x * 128 + threadIdx.x;
  const int i = min(t, total - 1);
  const int ix = i % cx, gy = (i / cx) % fy, gz = i / (cx * fy);
  const int nnc = cx * cy * cz;
  xc += (int64_t)blockIdx.z * 3 * nnc;
  xf += (int64_t)blockIdx.z * 3 * ((int64_t)fx * fy * fz);
  // within a column 32-bit offsets reach (3 nn < 2^31): the kernel is bound
  // by its instructions
  const int sn = COMP ? 1 : 3, sc = COMP ? nnc : 1;
  // one or two coarse rows in y and in z
  const bool ty = (gy & 1) && gy + 1 < fy, tz = (gz & 1) && gz + 1 < fz;
  const T wyz = (ty ? T(0.5) : T(1)) * (tz ? T(0.5) : T(1));
  pdl_wait();
  const int o00 = (((gz >> 1) * cy + (gy >> 1)) * cx + ix) * sn;
  const int dy = cx * sn, dz = cx * cy * sn, dr = ix + 1 < cx ? sn : 0;
  const bool last = lane == 31;   // loads its own right neighbour
  T v[3] = {T(0), T(0), T(0)}, r[3] = {T(0), T(0), T(0)};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (((k & 1) && !ty) || ((k >> 1) && !tz)) continue;
    const T *p = xc + (o00 + ((k & 1) ? dy : 0) + ((k >> 1) ? dz : 0));
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      v[q] += load_ro(p + q * sc);
      if (last) r[q] += load_ro(p + dr + q * sc);
    }
  }
  // the warp's 32 x 6 corrections through shared memory, so that the fine
  // vector is read and written by consecutive lanes (each lane its own 24
  // bytes took 20 us of partial-sector writes)
  __shared__ T vals[4][192];
  __shared__ int base[4][32];   // first dof of the lane's pair
  const int wp = threadIdx.x >> 5;
  const bool odd = 2 * ix + 1 < fx, tx = 2 * ix + 2 < fx;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    v[q] *= wyz;
    T right = __shfl_down_sync(0xffffffffu, v[q], 1);
    if (last) right = r[q] * wyz;
    vals[wp][6 * lane + q] = v[q];
    vals[wp][6 * lane + 3 + q] = tx ? T(0.5) * v[q] + T(0.5) * right : v[q];
  }
  // nodes of the pair: 2, 1 (odd last node missing) or 0 (past the end), as
  // one ballot each
  base[wp][lane] = 3 * ((gz * fy + gy) * fx + 2 * ix);
  const unsigned has0 = __ballot_sync(0xffffffffu, t < total);
  const unsigned has1 = __ballot_sync(0xffffffffu, t < total && odd);
  __syncwarp();
  T f[6];
  int at[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const unsigned e = lane + 32 * k, o = e / 6u, c = e - 6 * o;
    const bool in = ((c < 3 ? has0 : has1) >> o) & 1u;
    at[k] = in ? base[wp][o] + (int)c : -1;
    f[k] = in ? xf[at[k]] : T(0);
  }
#pragma unroll
  for (int k = 0; k < 6; ++k)
    if (at[k] >= 0) xf[at[k]] = f[k] + vals[wp][lane + 32 * k];
  pdl_launch_dependents();
}

// one row of x = Ainv b by one warp: four independent partial sums so the
// loads of consecutive chunks overlap; result valid in every lane
template <typename T>
__device__ __forceinline__ double gemv_row(const double *a, const T *b, int64_t n, int lane) {
  double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
  int64_t k = lane;
  for (; k + 96 < n; k += 128) {
    s0 += a[k] * static_cast<double>(b[k]);
    s1 += a[k + 32] * static_cast<double>(b[k + 32]);
    s2 += a[k + 64] * static_cast<double>(b[k + 64]);
    s3 += a[k + 96] * static_cast<double>(b[k + 96]);
  }
  for (; k < n; k += 32) s0 += a[k] * static_cast<double>(b[k]);
  double s = (s0 + s1) + (s2 + s3);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// x = Ainv b, one warp per row, FP64 accumulation
template <typename T>
__global__ void k_coarse_gemv(int64_t n, const double *A, const T *b, T *__restrict__ x) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  pdl_wait();
  for (int64_t row = warp; row < n; row += nwarps) {
    const double s = gemv_row(A + row * n, b, n, lane);
    if (lane == 0) x[row] = static_cast<T>(s);
  }
  pdl_launch_dependents();
}

// Chebyshev start: r = D^-1 (b or the residual already in r), d = r/theta,
// x (+)= d; column blockIdx.y (stride n), D^-1 shared
template <typename T>
__global__ void k_cheb_init(int64_t n, const T *__restrict__ dinv,
                            const T *__restrict__ b, T *__restrict__ r,
                            T *__restrict__ d, T *__restrict__ x, T inv_theta,
                            bool zero_guess) {
  const int64_t o = blockIdx.y * n;
  if (zero_guess) b += o;
  r += o;
  d += o;
  x += o;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const T ri = dinv[i] * (zero_guess ? b[i] : r[i]);
    const T di = ri * inv_theta;
    r[i] = ri;
    d[i] = di;
    x[i] = zero_guess ? di : x[i] + di;
  }
}

// r -= D^-1 A d ; d = c1 d + c2 r ; x += d; column blockIdx.y
template <typename T>
__global__ void k_cheb_step(int64_t n, const T *__restrict__ dinv,
                            const T *__restrict__ Ad, T *__restrict__ r,
                            T *__restrict__ d, T *__restrict__ x, T c1, T c2) {
  const int64_t o = blockIdx.y * n;
  Ad += o;
  r += o;
  d += o;
  x += o;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const T ri = r[i] - dinv[i] * Ad[i];
    const T di = c1 * d[i] + c2 * ri;
    r[i] = ri;
    d[i] = di;
    x[i] += di;
  }
}

}  // namespace

template <typename T>
void launch_apply_stencil(const Level &v, const T *S, const T *u, const T *b,
                          T *y, cudaStream_t s, const T *scale) {
  count_launch();
  const int g = grid_for(v.nn, 32);
  const dim3 blk(32, kStencilRows);
  const int nx = v.dims[0], ny = v.dims[1], nz = v.dims[2];
  if (scale)
    k_apply_stencil<T, OUT_SCALE><<<g, blk, 0, s>>>(nx, ny, nz, S, u, nullptr, scale, y);
  else if (b)
    k_apply_stencil<T, OUT_RESID><<<g, blk, 0, s>>>(nx, ny, nz, S, u, b, nullptr, y);
  else
    k_apply_stencil<T, OUT_Y><<<g, blk, 0, s>>>(nx, ny, nz, S, u, nullptr, nullptr, y);
}
template void launch_apply_stencil<double>(const Level &, const double *,
                                           const double *, const double *,
                                           double *, cudaStream_t, const double *);
template void launch_apply_stencil<float>(const Level &, const float *,
                                          const float *, const float *, float *,
                                          cudaStream_t, const float *);

template <typename T, bool RESID, int NB>
void sym_launch(const Level &v, const T *H, const T *u, const T *b, T *y,
                cudaStream_t s) {
  count_launch();
  const int g = grid_for(v.nn, 128);
  if (NB == 1) {
    ApplyArgs<T> a{};
    a.u = u;
    a.b = b;
    a.y = y;
    k_apply_stencil_sym1<T, IN_U, RESID ? OUT_RESID : OUT_Y><<<g, 128, 0, s>>>(
        v.dims[0], v.dims[1], v.dims[2], H, a);
  } else
    k_apply_stencil_sym<T, RESID, NB><<<g, 128, 0, s>>>(
        v.dims[0], v.dims[1], v.dims[2], H, u, b, y, 3 * v.nn);
}



template <typename T, bool RESID>
void sym_dispatch(const Level &v, const T *H, const T *u, const T *b, T *y,
                  cudaStream_t s, int nb) {
  const int64_t ld = 3 * v.nn;
  while (nb > 0) {
    const int w = nb >= 8 ? 8 : nb >= 4 ? 4 : nb >= 2 ? 2 : 1;
    if (w == 8) sym_launch<T, RESID, 8>(v, H, u, b, y, s);
    else if (w == 4) sym_launch<T, RESID, 4>(v, H, u, b, y, s);
    else if (w == 2) sym_launch<T, RESID, 2>(v, H, u, b, y, s);
    else sym_launch<T, RESID, 1>(v, H, u, b, y, s);
    u += w * ld;
    if (b) b += w * ld;
    y += w * ld;
    nb -= w;
  }
}

template <typename T>
void launch_apply_sym_fused(const Level &v, const T *H, int in, int out,
                            const ApplyArgs<T> &a, cudaStream_t s) {
  count_launch();
  const int g = grid_for(v.nn, 128);
  const int nx = v.dims[0], ny = v.dims[1], nz = v.dims[2];
  if (in == IN_CHEB && out == OUT_CHEB2)
    k_apply_stencil_sym1<T, IN_CHEB, OUT_CHEB2><<<g, 128, 0, s>>>(nx, ny, nz, H, a);
  else if (out == OUT_POST0)
    k_apply_stencil_sym1<T, IN_U, OUT_POST0><<<g, 128, 0, s>>>(nx, ny, nz, H, a);
  else if (out == OUT_POST1)
    k_apply_stencil_sym1<T, IN_U, OUT_POST1><<<g, 128, 0, s>>>(nx, ny, nz, H, a);
  else if (out == OUT_RESID)
    k_apply_stencil_sym1<T, IN_U, OUT_RESID><<<g, 128, 0, s>>>(nx, ny, nz, H, a);
  else if (out == OUT_SCALE)
    k_apply_stencil_sym1<T, IN_U, OUT_SCALE><<<g, 128, 0, s>>>(nx, ny, nz, H, a);
  else
    k_apply_stencil_sym1<T, IN_U, OUT_Y><<<g, 128, 0, s>>>(nx, ny, nz, H, a);
}
template void launch_apply_sym_fused<double>(const Level &, const double *, int, int,
                                             const ApplyArgs<double> &, cudaStream_t);
template void launch_apply_sym_fused<float>(const Level &, const float *, int, int,
                                            const ApplyArgs<float> &, cudaStream_t);

template <typename T>
void launch_apply_stencil_sym(const Level &v, const T *H, const T *u,
                              const T *b, T *y, cudaStream_t s, int nb) {
  if (b)
    sym_dispatch<T, true>(v, H, u, b, y, s, nb);
  else
    sym_dispatch<T, false>(v, H, u, b, y, s, nb);
}
template void launch_apply_stencil_sym<double>(const Level &, const double *,
                                               const double *, const double *,
                                               double *, cudaStream_t, int);
template void launch_apply_stencil_sym<float>(const Level &, const float *,
                                              const float *, const float *,
                                              float *, cudaStream_t, int);

void launch_stencil_to_half(int64_t nn, const double *H64, float *H32, cudaStream_t s) {
  count_launch();
  k_stencil_to_half<<<grid_for(126 * nn, 256), 256, 0, s>>>(nn, H64, H32);
}

int launch_galerkin_fine(Ctx &c, double *Sc, cudaStream_t s) {
  const int64_t nce = (int64_t)((c.nel[0] + 1) / 2) * ((c.nel[1] + 1) / 2) *
                      ((c.nel[2] + 1) / 2);
  count_launch(1);
  if (cudaMemsetAsync(c.gk_count, 0, sizeof(unsigned int), s) != cudaSuccess) return TPO_E_CUDA;
  k_coarse_elem_flags<<<grid_for(nce, 128), 128, 0, s>>>(c.nel[0], c.nel[1], c.nel[2],
                                                          c.idm, c.gk_slot, c.gk_elem,
                                                          c.gk_count);
  unsigned int nslots = 0;
  if (cudaMemcpyAsync(&nslots, c.gk_count, sizeof(unsigned int), cudaMemcpyDeviceToHost, s) !=
          cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return TPO_E_CUDA;
  if ((size_t)nslots * 576 > c.gk_cap) {
    if (c.gk_G) cudaFree(c.gk_G);
    c.gk_G = nullptr;
    c.gk_cap = 0;
    const size_t cap = std::max<size_t>((size_t)nslots * 576, 576);
    if (cudaMalloc(&c.gk_G, sizeof(double) * cap) != cudaSuccess) return TPO_E_CUDA;
    c.gk_cap = cap;
  }
  if (nslots) {
    count_launch();
    k_galerkin_general<<<dim3((nslots + 31) / 32, 64), 256, 0, s>>>(
        c.nel[0], c.nel[1], c.nel[2], (int)nslots, c.E64, c.idm, c.gk_elem, c.K0lex, c.GMi, c.gk_G);
  }
  count_launch();
  Level &v = c.lev[1];
  const dim3 grid((unsigned)((v.nn + kGfThreads * kGfNodes - 1) / (kGfThreads * kGfNodes)), 14);
  k_galerkin_fine<<<grid, kGfThreads, 0, s>>>(c.nel[0], c.nel[1], c.nel[2], c.E64, c.idm,
                                              c.gk_slot, c.gk_G, c.GMi, Sc, v.H32, v.dinv64,
                                              v.dinv32);
  c.gk_nslots = (int)nslots;
  return TPO_OK;
}

void launch_galerkin_dims(const Level &fine, const double *Sf, double *Sc,
                          double *tmp, cudaStream_t s) {
  const int fx = fine.dims[0], fy = fine.dims[1], fz = fine.dims[2];
  const int cx = (fx + 1) / 2, cy = (fy + 1) / 2;
  const int64_t n1 = (int64_t)cx * fy * fz, n2 = (int64_t)cx * cy * fz;
  double *t1 = tmp, *t2 = tmp + 243 * n1;
  count_launch(3);
  k_galerkin_dim<0><<<grid_for(27 * n1, 128, 1 << 20), 128, 0, s>>>(fx, fy, fz, Sf, t1);
  k_galerkin_dim<1><<<grid_for(27 * n2, 128, 1 << 20), 128, 0, s>>>(cx, fy, fz, t1, t2);
  const int64_t n3 = n2 / fz * ((fz + 1) / 2);
  k_galerkin_dim<2><<<grid_for(27 * n3, 128, 1 << 20), 128, 0, s>>>(cx, cy, fz, t2, Sc);
}

size_t galerkin_dims_scratch(const Level &fine) {
  const int fx = fine.dims[0], fy = fine.dims[1], fz = fine.dims[2];
  const int cx = (fx + 1) / 2, cy = (fy + 1) / 2;
  return 243 * ((size_t)cx * fy * fz + (size_t)cx * cy * fz);
}


void launch_stencil_diag(const Level &v, const double *S, double *dinv64,
                         float *dinv32, cudaStream_t s) {
  count_launch();
  k_stencil_diag<<<grid_for(v.nn, 256), 256, 0, s>>>(v.nn, S, dinv64, dinv32);
}

template <typename T>
void launch_restrict(const Level &fine, const Level &coarse, const T *rf, T *bc,
                     const CompLevel<T> *comp, cudaStream_t s, int nb) {
  count_launch();
  const int *f = fine.dims, *c = coarse.dims;
  const dim3 g((unsigned)((coarse.nn + 127) / 128), 1, nb);
  if (comp)
    launch_pdl(k_restrict<T, true>, g, 128, 0, s, f[0], f[1], f[2], c[0], c[1], c[2], rf, bc,
               *comp);
  else
    launch_pdl(k_restrict<T, false>, g, 128, 0, s, f[0], f[1], f[2], c[0], c[1], c[2], rf, bc,
               CompLevel<T>{});
}
template void launch_restrict<double>(const Level &, const Level &, const double *, double *,
                                      const CompLevel<double> *, cudaStream_t, int);
template void launch_restrict<float>(const Level &, const Level &, const float *, float *,
                                     const CompLevel<float> *, cudaStream_t, int);

template <typename T>
void launch_prolong_add(const Level &fine, const Level &coarse, const T *xc, T *xf, bool comp,
                        cudaStream_t s, int nb) {
  count_launch();
  const int *f = fine.dims, *c = coarse.dims;
  const dim3 g((unsigned)(((int64_t)c[0] * f[1] * f[2] + 127) / 128), 1, nb);
  if (comp)
    launch_pdl(k_prolong_add<T, true>, g, 128, 0, s, f[0], f[1], f[2], c[0], c[1], c[2], xc, xf);
  else
    launch_pdl(k_prolong_add<T, false>, g, 128, 0, s, f[0], f[1], f[2], c[0], c[1], c[2], xc, xf);
}
template void launch_prolong_add<double>(const Level &, const Level &, const double *, double *,
                                         bool, cudaStream_t, int);
template void launch_prolong_add<float>(const Level &, const Level &, const float *, float *,
                                        bool, cudaStream_t, int);

template <typename T>
void launch_coarse_gemv(int64_t n, const double *Ainv, const T *b, T *x,
                        cudaStream_t s, int nb) {
  const int64_t warps = n;
  const int threads = 256;
  int64_t blocks = (warps * 32 + threads - 1) / threads;
  if (blocks > 148 * 8) blocks = 148 * 8;
  for (int col = 0; col < nb; ++col) {
    count_launch();
    launch_pdl(k_coarse_gemv<T>, (int)blocks, threads, 0, s, n, Ainv, b + col * n, x + col * n);
  }
}
template void launch_coarse_gemv<double>(int64_t, const double *,
                                         const double *, double *,
                                         cudaStream_t, int);
template void launch_coarse_gemv<float>(int64_t, const double *, const float *,
                                        float *, cudaStream_t, int);

static dim3 col_grid(int64_t n, int nb) {
  int g = grid_for(n, 256);
  if (nb > 1) g = std::max(148, g / nb);
  return dim3(g, nb);
}

template <typename T>
void launch_cheb_init(int64_t n, const T *dinv, const T *b, T *r, T *d, T *x,
                      double inv_theta, bool zero_guess, cudaStream_t s,
                      int nb) {
  count_launch();
  k_cheb_init<T><<<col_grid(n, nb), 256, 0, s>>>(
      n, dinv, b, r, d, x, static_cast<T>(inv_theta), zero_guess);
}
template void launch_cheb_init<double>(int64_t, const double *, const double *,
                                       double *, double *, double *, double,
                                       bool, cudaStream_t, int);
template void launch_cheb_init<float>(int64_t, const float *, const float *,
                                      float *, float *, float *, double, bool,
                                      cudaStream_t, int);

template <typename T>
void launch_cheb_step(int64_t n, const T *dinv, const T *Ad, T *r, T *d, T *x,
                      double c1, double c2, cudaStream_t s, int nb) {
  count_launch();
  k_cheb_step<T><<<col_grid(n, nb), 256, 0, s>>>(
      n, dinv, Ad, r, d, x, static_cast<T>(c1), static_cast<T>(c2));
}
template void launch_cheb_step<double>(int64_t, const double *, const double *,
                                       double *, double *, double *, double,
                                       double, cudaStream_t, int);
template void launch_cheb_step<float>(int64_t, const float *, const float *,
                                      float *, float *, float *, double, double,
                                      cudaStream_t, int);

}  // namespace tpo
