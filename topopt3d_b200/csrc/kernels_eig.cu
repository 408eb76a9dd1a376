// Tall-skinny block kernels of the block eigensolver (eigen.cu): the Gram
// blocks of the Rayleigh-Ritz step, the recombination of the basis by the
// Ritz coefficients, and the residual block with its column norms.  The
// reference forms the same products with VecMDot/VecMAXPY over its search
// space (PRINVIT.cpp:319-330).
//
// Every kernel reads each n-row column it needs once per launch and both
// contractions run on the FP64 tensor-core MMAs, so all three are bound by
// the bytes of the basis; reductions over rows go through per-CTA partial
// sums that a second launch adds in a fixed order, so the results do not
// depend on scheduling.
//
// Measured at n = 698,691, m = 12 and three blocks (a 96x48x48 mesh), before
// (register tiles of DFMAs, operands loaded at their use) and now: Gram 955 ->
// 197 us (603 MB, 93 us at the copy rate; 4 GFLOP, 110 us at the FP64 rate
// these MMAs reach), recombination 518 -> 215 us (1.0 GB, 156 us), residual
// 77 -> 49 us (201 MB, 31 us), the two sums of partials 26 -> 6 and 31 -> 8 us.
#include "tpo_internal.h"

namespace tpo {

namespace {

// D (8 x 8) += A (8 x 4) B (4 x 8), lane = 4 g + q: A[g][q], B[q][g],
// D[g][2q], D[g][2q + 1] (PTX ISA, mma.m8n8k4 .f64)
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// 8-byte asynchronous copy (a column of an odd number of rows starts on an
// 8-byte boundary); bytes 0 writes zeros, the address must still be valid
__device__ __forceinline__ void cp_async8(double *dst, const double *src, int bytes) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes)
               : "memory");
}

// ---- Gram blocks ----------------------------------------------------------
//
// A CTA per SM takes every 148th chunk of 64 rows through a ring of three
// shared-memory stages (the copies of two chunks, 110 KB, are in flight
// while one is consumed) and holds a 40 x 72 block of outputs: four groups of
// three warps, a group taking 16 of the chunk's rows, a warp 5 x 3 tiles of
// 8 x 8 (8 fragment reads for 15 MMAs).  36 x 72 outputs -- a block of 12 and
// its two others -- are one block; larger ones are several, each reading its
// columns again.
constexpr int kGI = 40;   // left columns of a block
constexpr int kGJ = 72;   // right columns (A then B images)
constexpr int kGR = 64;   // rows of a chunk
constexpr int kGLd = kGR + 4;   // column stride: fragment reads free of conflicts
constexpr int kGStages = 3;
constexpr int kGGroups = 4, kGWarps = 3 * kGGroups, kGThreads = 32 * kGWarps;
constexpr int kGLoads = (2 * (kGI + kGJ) + kGWarps - 1) / kGWarps;   // half columns a warp copies
static_assert(kGLoads <= 20, "four parts of five");
constexpr int kGramParts = 148;
constexpr size_t kGStage = (size_t)(kGI + kGJ) * kGLd;
constexpr size_t kGSmem = kGStages * kGStage * sizeof(double);
static_assert((size_t)kGGroups * kGI * kGJ <= kGStages * kGStage, "group sums fit the stages");

__global__ void __launch_bounds__(kGThreads, 1)
    k_eig_gram(int64_t n, int m, int k, EigCols cols, double *part) {
  extern __shared__ __align__(16) double gs[];
  __shared__ const double *src[kGI + kGJ];
  const int nsi = (k + kGI - 1) / kGI;
  const int st = blockIdx.y;
  const int i0 = (st % nsi) * kGI, j0 = (st / nsi) * kGJ;
  const int nl = min(kGI, k - i0), nr = min(kGJ, 2 * k - j0);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, q = lane & 3;
  // the column of each shared-memory column, null where there is none
  // (it is not loaded, and what it holds reaches only outputs outside k)
  for (int c = t; c < kGI + kGJ; c += kGThreads) {
    const double *p = nullptr;
    if (c < nl) {
      p = cols.L[(i0 + c) / m] + (int64_t)((i0 + c) % m) * n;
    } else if (c >= kGI && c - kGI < nr) {
      const int j = j0 + c - kGI;
      p = j < k ? cols.A[j / m] + (int64_t)(j % m) * n
                : cols.B[(j - k) / m] + (int64_t)((j - k) % m) * n;
    }
    src[c] = p;
  }
  __syncthreads();
  const int64_t chunks = (n + kGR - 1) / kGR;
  // a warp copies half columns (32 rows): warp / 2 + 6 i, i = 0 .. 18, in four
  // parts so that a chunk's copies are issued between the products
  const int c0 = warp >> 1, rr = (warp & 1) * 32 + lane;
  auto load = [&](int64_t ch, int slot, int i0_, int i1_) {
    const int64_t row = ch * kGR + rr;
    const bool in = row < n;
    const int64_t off = in ? row : 0;
    const int bytes = in ? 8 : 0;
    double *d = gs + slot * kGStage + (size_t)c0 * kGLd + rr;
#pragma unroll
    for (int i = 0; i < kGLoads; ++i) {
      if (i < i0_ || i >= i1_) continue;
      if (c0 + 6 * i >= kGI + kGJ) continue;
      const double *p = src[c0 + 6 * i];
      if (p) cp_async8(d + (size_t)6 * i * kGLd, p + off, bytes);
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;\n" ::: "memory"); };
  double acc[5][3][2];
#pragma unroll
  for (int a = 0; a < 5; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  const int grp = warp / 3, wn = warp % 3;
  const int mt = (nl + 7) / 8, nt = min(3, max(0, (nr + 7) / 8 - 3 * wn));
  for (int c = 0; c < 2; ++c) {
    const int64_t ch = blockIdx.x + (int64_t)c * gridDim.x;
    if (ch < chunks) load(ch, c, 0, kGLoads);
    commit();
  }
  int slot = 0;
  for (int64_t ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();   // this chunk is here, and the slot refilled next is read
    const int64_t nch = ch + 2 * (int64_t)gridDim.x;
    const int nslot = slot == 0 ? 2 : slot - 1;
    const double *s = gs + slot * kGStage + 16 * grp + q;
    slot = slot == kGStages - 1 ? 0 : slot + 1;
#pragma unroll
    for (int k0 = 0; k0 < 16; k0 += 4) {
      double av[5], bv[3];
#pragma unroll
      for (int a = 0; a < 5; ++a) av[a] = s[(8 * a + g) * kGLd + k0];
#pragma unroll
      for (int b = 0; b < 3; ++b) bv[b] = s[(kGI + 8 * (3 * wn + b) + g) * kGLd + k0];
#pragma unroll
      for (int b = 0; b < 3; ++b)
        if (b < nt) {
#pragma unroll
          for (int a = 0; a < 5; ++a)
            if (a < mt) dmma(acc[a][b], av[a], bv[b]);
        }
      if (nch < chunks) load(nch, nslot, 5 * (k0 / 4), 5 * (k0 / 4) + 5);
    }
    commit();
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  // the groups' sums, added in order
#pragma unroll
  for (int a = 0; a < 5; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        gs[(grp * kGI + 8 * a + g) * kGJ + 8 * (3 * wn + b) + 2 * q + h] = acc[a][b][h];
  __syncthreads();
  double *p = part + ((size_t)st * gridDim.x + blockIdx.x) * (kGI * kGJ);
  for (int e = t; e < kGI * kGJ; e += kGThreads) {
    double v = gs[e];
#pragma unroll
    for (int c = 1; c < kGGroups; ++c) v += gs[c * kGI * kGJ + e];
    p[e] = v;
  }
}

// H (k x k) and G (k x k), column-major, from the partials: 32 outputs a CTA,
// 8 threads an output, their sums added in order
__global__ void __launch_bounds__(256)
    k_eig_gram_reduce(int k, int nsi, int nst, int nparts, const double *part, double *H,
                      double *G) {
  __shared__ double red[8][32];
  const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
  const int64_t total = (int64_t)nst * kGI * kGJ;
  const int64_t e = (int64_t)blockIdx.x * 32 + lane;
  double s = 0.0;
  if (e < total) {
    const int st = (int)(e / (kGI * kGJ)), w = (int)(e % (kGI * kGJ));
    const double *p = part + (size_t)st * nparts * (kGI * kGJ) + w;
#pragma unroll 4
    for (int c = sl; c < nparts; c += 8) s += p[(size_t)c * (kGI * kGJ)];
  }
  red[sl][lane] = s;
  __syncthreads();
  if (sl != 0 || e >= total) return;
#pragma unroll
  for (int c = 1; c < 8; ++c) s += red[c][lane];
  const int st = (int)(e / (kGI * kGJ)), w = (int)(e % (kGI * kGJ));
  const int i = (st % nsi) * kGI + w / kGJ, j = (st / nsi) * kGJ + w % kGJ;
  if (i >= k || j >= 2 * k) return;
  if (j < k)
    H[(size_t)j * k + i] = s;
  else
    G[(size_t)(j - k) * k + i] = s;
}

// ---- recombination --------------------------------------------------------
//
// out.X[g] = [V_0 .. V_nb-1] C and, with P, out.P[g] = [V_1 .. V_nb-1]
// C(m:, :), C (k x m) column-major, for the three image groups g: one product
// with the k x 2m matrix [C | C with its first m rows zero].  A warp takes
// 8 RG rows of one group: a fragment of the basis is 4 columns x 8 rows (64
// contiguous bytes of each) straight from memory, used once; the
// coefficients come from shared memory.  NT tiles of 8 output columns; the
// loads of KU steps of 4 columns are issued together (3 NT steps are a basis
// of three blocks).
constexpr int kCombThreads = 256;

template <int NT, int RG, int KU>
__global__ void __launch_bounds__(kCombThreads, 2)
    k_eig_combine(int64_t n, int m, int k, EigCols cols, const double *__restrict__ C,
                  EigOut out, int want_p) {
  constexpr int kLd = 8 * NT + 4;   // = 4 or 12 mod 16: reads free of conflicts
  extern __shared__ __align__(16) double Cs[];   // k4 x kLd
  __shared__ const double *src[3][3 * kMaxEigPairs];
  const int k4 = (k + 3) & ~3, nout = want_p ? 2 * m : m;
  for (int e = threadIdx.x; e < k4 * 8 * NT; e += kCombThreads) {
    const int i = e / (8 * NT), j = e % (8 * NT);
    double v = 0.0;
    if (i < k && j < nout && (j < m || i >= m)) v = C[(size_t)(j < m ? j : j - m) * k + i];
    Cs[i * kLd + j] = v;
  }
  for (int e = threadIdx.x; e < 3 * k4; e += kCombThreads) {
    const int g = e / k4, i = min(e % k4, k - 1), b = i / m;
    src[g][e % k4] = (g == 0 ? cols.L[b] : (g == 1 ? cols.A[b] : cols.B[b])) + (int64_t)(i % m) * n;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int64_t units = (n + 8 * RG - 1) / (8 * RG);
  const int64_t w0 = blockIdx.x * (int64_t)(kCombThreads / 32) + (threadIdx.x >> 5);
  const int64_t nw = (int64_t)gridDim.x * (kCombThreads / 32);
  for (int64_t u = w0; u < 3 * units; u += nw) {
    const int im = (int)(u / units);
    const int64_t r0 = (u - (int64_t)im * units) * (8 * RG) + g;
    double acc[RG][NT][2];
#pragma unroll
    for (int a = 0; a < RG; ++a)
#pragma unroll
      for (int b = 0; b < NT; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    // rows past the end read the last one; their results are not stored
    for (int kb = 0; kb < k4; kb += 4 * KU) {
      double av[KU][RG];   // all in flight together
#pragma unroll
      for (int i = 0; i < KU; ++i) {
        if (kb + 4 * i >= k4) break;
        const double *p = src[im][kb + 4 * i + q];
#pragma unroll
        for (int a = 0; a < RG; ++a) av[i][a] = p[min(r0 + 8 * a, n - 1)];
      }
#pragma unroll
      for (int i = 0; i < KU; ++i) {
        if (kb + 4 * i >= k4) break;
        double bv[NT];
#pragma unroll
        for (int b = 0; b < NT; ++b) bv[b] = Cs[(kb + 4 * i + q) * kLd + 8 * b + g];
#pragma unroll
        for (int a = 0; a < RG; ++a)
#pragma unroll
          for (int b = 0; b < NT; ++b) dmma(acc[a][b], av[i][a], bv[b]);
      }
    }
#pragma unroll
    for (int b = 0; b < NT; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = 8 * b + 2 * q + h;
        if (j >= nout) continue;
        double *o = j < m ? out.X[im] + (int64_t)j * n : out.P[im] + (int64_t)(j - m) * n;
#pragma unroll
        for (int a = 0; a < RG; ++a)
          if (r0 + 8 * a < n) o[r0 + 8 * a] = acc[a][b][h];
      }
  }
}

// ---- residuals ------------------------------------------------------------

// R[:, j] = AX[:, j] - theta_j BX[:, j], and per CTA the sums of R[:, j]^2
// (part[cta * 2m + j]) and BX[:, j]^2 (part[cta * 2m + m + j]); four rows a
// thread at a time, so that eight loads are in flight
constexpr int kNormThreads = 256;
constexpr int kNormParts = 592;
constexpr int kNormRows = 4;

__global__ void __launch_bounds__(kNormThreads)
    k_eig_resid_norms(int64_t n, int m, const double *__restrict__ AX,
                      const double *__restrict__ BX, EigTheta th, double *R, double *part) {
  __shared__ double red[kNormThreads / 32][2 * kMaxEigPairs];
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int64_t st = (int64_t)gridDim.x * kNormThreads;
  for (int j = 0; j < m; ++j) {
    const double *ax = AX + (int64_t)j * n, *bx = BX + (int64_t)j * n;
    double *r = R + (int64_t)j * n;
    double sr = 0.0, sb = 0.0;
    for (int64_t row = blockIdx.x * (int64_t)kNormThreads + threadIdx.x; row < n;
         row += kNormRows * st) {
      double a[kNormRows], b[kNormRows];
#pragma unroll
      for (int u = 0; u < kNormRows; ++u) {
        const bool in = row + u * st < n;
        a[u] = in ? ax[row + u * st] : 0.0;
        b[u] = in ? bx[row + u * st] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kNormRows; ++u) {
        const double v = a[u] - th.v[j] * b[u];
        if (row + u * st < n) r[row + u * st] = v;
        sr = fma(v, v, sr);
        sb = fma(b[u], b[u], sb);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sr += __shfl_down_sync(0xffffffffu, sr, o);
      sb += __shfl_down_sync(0xffffffffu, sb, o);
    }
    if (lane == 0) {
      red[warp][j] = sr;
      red[warp][m + j] = sb;
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < 2 * m; q += blockDim.x) {
    double s = 0.0;
    for (int w = 0; w < kNormThreads / 32; ++w) s += red[w][q];
    part[(size_t)blockIdx.x * 2 * m + q] = s;
  }
}

// nrm[q] = sqrt(sum over the CTAs of part[cta * 2m + q]), q < 2m: a warp
// per q, lanes in order of the CTAs, then a fixed tree
__global__ void __launch_bounds__(1024)
    k_eig_norms_reduce(int m, int nparts, const double *part, double *nrm) {
  const int lane = threadIdx.x & 31;
  for (int q = threadIdx.x >> 5; q < 2 * m; q += blockDim.x >> 5) {
    double s = 0.0;
#pragma unroll 4
    for (int c = lane; c < nparts; c += 32) s += part[(size_t)c * 2 * m + q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) nrm[q] = sqrt(s);
  }
}

template <int NT, int RG, int KU>
void combine(int64_t n, int m, int k, const EigCols &cols, const double *C, const EigOut &out,
             bool want_p, cudaStream_t s) {
  const int64_t warps = 3 * ((n + 8 * RG - 1) / (8 * RG));
  const int64_t g = (warps + kCombThreads / 32 - 1) / (kCombThreads / 32);
  // k <= 3 m and 8 NT output columns hold 2 m (or k = m: no P)
  const size_t smem = sizeof(double) * ((k + 3) & ~3) * (8 * NT + 4);
  if (NT == 8) {
    static unsigned long long attr_set = 0;   // bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (!((attr_set >> (dev & 63)) & 1ull)) {
      cudaFuncSetAttribute(k_eig_combine<NT, RG, KU>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(sizeof(double) * 3 * kMaxEigPairs * (8 * NT + 4)));
      attr_set |= 1ull << (dev & 63);
    }
  }
  k_eig_combine<NT, RG, KU><<<(int)(g < 148 * 4 ? g : 148 * 4), kCombThreads, smem, s>>>(
      n, m, k, cols, C, out, want_p);
}

}  // namespace

size_t eig_gram_scratch(int k) {
  const int nsi = (k + kGI - 1) / kGI, nsj = (2 * k + kGJ - 1) / kGJ;
  const size_t gram = (size_t)nsi * nsj * kGramParts * kGI * kGJ;
  const size_t norms = (size_t)kNormParts * 2 * kMaxEigPairs;
  return gram > norms ? gram : norms;
}

void launch_eig_gram(int64_t n, int m, int nblk, const EigCols &cols, double *part, double *H,
                     double *G, cudaStream_t s) {
  const int k = nblk * m;
  const int nsi = (k + kGI - 1) / kGI, nsj = (2 * k + kGJ - 1) / kGJ;
  static unsigned long long attr_set = 0;   // bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!((attr_set >> (dev & 63)) & 1ull)) {
    cudaFuncSetAttribute(k_eig_gram, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGSmem);
    attr_set |= 1ull << (dev & 63);
  }
  count_launch(2);
  k_eig_gram<<<dim3(kGramParts, nsi * nsj), kGThreads, kGSmem, s>>>(n, m, k, cols, part);
  k_eig_gram_reduce<<<(nsi * nsj * kGI * kGJ + 31) / 32, 256, 0, s>>>(k, nsi, nsi * nsj,
                                                                      kGramParts, part, H, G);
}

void launch_eig_combine(int64_t n, int m, int nblk, const EigCols &cols, const double *C,
                        const EigOut &out, bool want_p, cudaStream_t s) {
  const int k = nblk * m, nt = ((want_p ? 2 * m : m) + 7) / 8;
  count_launch();
  if (nt <= 1)
    combine<1, 4, 3>(n, m, k, cols, C, out, want_p, s);
  else if (nt == 2)
    combine<2, 2, 6>(n, m, k, cols, C, out, want_p, s);
  else if (nt == 3)
    combine<3, 2, 9>(n, m, k, cols, C, out, want_p, s);
  else if (nt == 4)
    combine<4, 2, 12>(n, m, k, cols, C, out, want_p, s);
  else
    combine<8, 2, 8>(n, m, k, cols, C, out, want_p, s);
}

void launch_eig_resid_norms(int64_t n, int m, const double *AX, const double *BX,
                            const EigTheta &th, double *R, double *part, double *nrm,
                            cudaStream_t s) {
  count_launch(2);
  k_eig_resid_norms<<<kNormParts, kNormThreads, 0, s>>>(n, m, AX, BX, th, R, part);
  k_eig_norms_reduce<<<1, 1024, 0, s>>>(m, kNormParts, part, nrm);
}

}  // namespace tpo
