// Fine-level matrix-free stiffness operator, staged form.
//
//   y = M K(rho) M u + (1 - M) u          (MODE 0)
//   y = b - [M K(rho) M u + (1 - M) u]    (MODE 1)
//
// K = sum_e E_e K0 (FEAnalysis.cpp:443-468), Dirichlet rows/columns replaced
// by identity (MatZeroRowsColumns, FEAnalysis.cpp:473); M masks the fixed
// components.  u, y, b are interleaved per node (dof 3n+c), E per element.
//
// The element matvec is y_e = T^T Kh T u_e in the 2x2x2 Hadamard basis
// (tpo_internal.h).  T factorises into an x, a y and a z butterfly, and on a
// structured grid the x butterfly of one x-edge is shared by the 4 elements
// around that edge and the y butterfly of one xy-face by the 2 elements
// above and below it.  So each stage is computed once per grid item:
//
//   node u  --x-->  x-edge (s, d)  --y-->  xy-face (4 modes)  --z-->  element
//   (7 modes) -> E Kh -> element --z^T--> face contributions, summed over the
//   two elements sharing the face --y^T--> edge contributions, summed over
//   the two faces sharing the edge --x^T--> node contributions, summed over
//   the two edges sharing the node.
//
// About 150 FP operations per element (the dense 24x24 product is 1152):
// x 6, y 12, z 21, Kh 45, and the z transpose with the modulus E_e and the
// sum over the two elements of a face folded into 42 multiply-adds.
//
// Thread (tx, ty) of a 32 x TY CTA owns the grid column (gx, gy) = tile
// origin + (tx, ty): its node, the x-edge to gx+1, the xy-face spanning
// (gx..gx+1, gy..gy+1) and the element column above that face; the CTA
// marches up z.  x-neighbours exchange values by warp shuffles (a warp is
// one tile row), y-neighbours through shared memory with one barrier per
// plane.  Lanes 0 and 31 and row 0 are the halo: the CTA writes the nodes of
// lanes 1..30 and rows 1..TY-1, so every lane's work is the same (lane 31
// only supplies its node to lane 30's edge); the last row (a warp-uniform
// role) also loads the row above the tile so every face of the tile is
// complete.  Node values of the next plane are prefetched into registers
// one plane ahead.  The pipeline: at step p the plane p is loaded into
// edges and faces, element layer p-1 is applied, the faces of plane p-1 are
// complete, and nodes of plane p-2 are written.
#include "fused_out.cuh"
#include "modal.cuh"
#include "pdl.cuh"
#include "reduce.cuh"

namespace tpo {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kLanesOut = 30;   // written nodes per tile row

// epilogue of dof i with Au_i = (M K M u + (1-M) u)_i and u_i the input; bi,
// di, y2i are b_i, dinv_i, y2_i where the form needs them (OutNeeds):
//   OUT_Y     y = Au
//   OUT_RESID y = b - Au
//   OUT_CHEB2 Chebyshev(2) from a zero guess, input d0 = invtheta dinv b:
//             r1 = dinv (b - Au); d1 = c1 d0 + c2 r1; y = d0 + d1
//   OUT_POST0 first Chebyshev step from x = u:  d0 = invtheta dinv (b - Au);
//             y = d0, y2 = u + d0
//   OUT_POST1 second step, input d0 = u (so r0 = theta d0):
//             d1 = c1 d0 + c2 (theta d0 - dinv Au); y = x1 + d1 (x1 = y2)
//   OUT_SCALE y = dinv Au
// (sym_out_v, fused_out.cuh)

// Operands that a thread reads for its own node only -- b, dinv, y2 of the
// epilogue, and b and dinv of the IN_CHEB input -- are copied to shared
// memory asynchronously one plane ahead.  A load at the point of use stalls
// the 16 warps of an SM for its latency in every plane, and there are no
// registers left to prefetch into.  At 192x96x96, before and after (us, FP32
// / FP64; the plain product takes 33 / 61): OUT_CHEB2 58 -> 40 / 130 -> 77,
// OUT_POST0 51 -> 41 / 109 -> 81, OUT_POST1 53 -> 40 / 121 -> 74, OUT_RESID
// 38 / 94 -> 70; 8 columns of 128x64x64 in FP32: 152 -> 104, 135 -> 107,
// 146 -> 104 and 123 -> 99.
__device__ __forceinline__ void copy_async(float *dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// staged arrays and planes: IN_CHEB keeps b and dinv of 4 planes (loaded
// ahead, input, and two planes later the epilogue) and the row above the
// tile; the other forms 2 planes of what their epilogue reads; the
// Chebyshev forms with IN_U, and the product whose dot with u is formed, also
// keep their input of 3 planes (4 slots)
template <int IN, int OUT, bool DOT>
struct Staged {
  static constexpr bool kIn = IN == IN_CHEB;
  static constexpr bool kB = OutNeeds<OUT>::b || (DOT && OUT == OUT_POST1), kD = OutNeeds<OUT>::dinv, kY = OutNeeds<OUT>::y2;
  static constexpr bool kU = !kIn && (OUT == OUT_CHEB2 || OUT == OUT_POST0 || OUT == OUT_POST1 ||
                                      (DOT && OUT == OUT_Y));
  static constexpr int kArrays = kIn ? 2 : int(kB) + int(kD) + int(kY);
  static constexpr int kSlots = kIn ? 4 : 2;
  static constexpr int kSlotB = 0, kSlotD = kIn ? 1 : int(kB), kSlotY = int(kB) + int(kD);
  static constexpr int planes() { return kArrays * kSlots + (kU ? 4 : 0); }
};

// six values per thread in shared memory with 16-byte accesses: FP32 as one
// float4 (v0, w0, v1, w1) and one float2 (v2, w2) per lane; FP64 as three
// double2 (v_c, w_c)
template <typename T>
struct Six;

template <>
struct Six<float> {
  float4 *a;   // [row][32]
  float2 *b;
  __device__ __forceinline__ void put(int row, int lane, const float (&v)[3],
                                      const float (&w)[3]) const {
    a[row * 32 + lane] = make_float4(v[0], w[0], v[1], w[1]);
    b[row * 32 + lane] = make_float2(v[2], w[2]);
  }
  __device__ __forceinline__ void get(int row, int lane, float (&v)[3],
                                      float (&w)[3]) const {
    const float4 p = a[row * 32 + lane];
    const float2 q = b[row * 32 + lane];
    v[0] = p.x; w[0] = p.y; v[1] = p.z; w[1] = p.w; v[2] = q.x; w[2] = q.y;
  }
  static constexpr size_t bytes_per_row() { return 32 * (16 + 8); }
  __device__ __forceinline__ void bind(unsigned char *base, int rows) {
    a = reinterpret_cast<float4 *>(base);
    b = reinterpret_cast<float2 *>(base + (size_t)rows * 32 * 16);
  }
};

template <>
struct Six<double> {
  double2 *a;   // [c][row][32]
  int stride;
  __device__ __forceinline__ void put(int row, int lane, const double (&v)[3],
                                      const double (&w)[3]) const {
#pragma unroll
    for (int c = 0; c < 3; ++c) a[c * stride + row * 32 + lane] = make_double2(v[c], w[c]);
  }
  __device__ __forceinline__ void get(int row, int lane, double (&v)[3],
                                      double (&w)[3]) const {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double2 p = a[c * stride + row * 32 + lane];
      v[c] = p.x;
      w[c] = p.y;
    }
  }
  static constexpr size_t bytes_per_row() { return 32 * 3 * 16; }
  __device__ __forceinline__ void bind(unsigned char *base, int rows) {
    a = reinterpret_cast<double2 *>(base);
    stride = rows * 32;
  }
};

// COLS: a block of columns, blockIdx.z = column * nchunk + z chunk, the
// column selecting u, b, y, y2 (stride ld).  The single-column
// instantiation reads the parameters in place.
//
// DOT: the epilogue also sums, in FP64, u.y (OUT_Y), y.y (OUT_RESID) or b.y
// (OUT_POST1): CG's p.q, r.r of a replaced residual and rho = r.z.  A pass of
// its own that reads both vectors again took 11 us in FP32 and 19 us in FP64 at
// 192x96x96 (6 us at 48x24x24); here p.q adds 4 and 6 us, rho 5 and 6.5 us (a
// third staged operand), r.r 4 us (FP64), most of it in FP32 the conversions.
template <typename T, int TY, int IN, int OUT, bool COLS, bool DOT>
__global__ void __launch_bounds__(32 * TY, sizeof(T) == 4 ? 2 : 1)
    k_apply_staged(int nelx, int nely, int nelz, int zchunk,
                   const T *E, const uint8_t *fix,
                   const ApplyArgs<T> args_in, const Kh<T> kh, const DotOut dot) {
  const int Nx = nelx + 1, Ny = nely + 1, Nz = nelz + 1;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int gx = (int)blockIdx.x * kLanesOut - 1 + tx;
  const int gy = (int)blockIdx.y * (TY - 1) - 1 + ty;
  int zs;
  ApplyArgs<T> args_col;
  if (COLS) {
    const int col = (int)blockIdx.z / args_in.nchunk;
    zs = ((int)blockIdx.z - col * args_in.nchunk) * zchunk;
    args_col = args_in;
    const int64_t o = col * args_in.ld;
    if (args_col.u) args_col.u += o;
    if (args_col.b) args_col.b += o;
    args_col.y += o;
    if (args_col.y2) args_col.y2 += o;
  } else {
    zs = (int)blockIdx.z * zchunk;
  }
  const ApplyArgs<T> &args = COLS ? args_col : args_in;
  const int ze = min(zs + zchunk, Nz);
  const bool lastrow = (ty == TY - 1);   // warp-uniform

  // plane-invariant per-thread offsets and predicates
  const bool xin = gx >= 0 && gx < Nx;
  const bool nin = xin && gy >= 0 && gy < Ny;
  const bool nin2 = lastrow && xin && gy + 1 < Ny;
  const bool exy = gx >= 0 && gx < nelx && gy >= 0 && gy < nely;
  const bool own = tx >= 1 && tx <= kLanesOut && ty >= 1 && nin;
  const int NP = Nx * Ny, EP = nelx * nely;
  const int nofs = nin ? gy * Nx + gx : 0;
  const int nofs2 = nin2 ? (gy + 1) * Nx + gx : 0;
  const int eofs = exy ? gy * nelx + gx : 0;

  // dynamic shared memory: se = x-edge (s, d) per row plus the row above
  // the tile, sc = edge contributions of the upper row of a face (row index
  // ty + 1 written by row ty), both double-buffered by plane parity
  // (rows buf * kRows + r of one array per buffer pair)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int kRows = TY + 1;
  Six<T> se, sc;
  se.bind(smem_raw, 2 * kRows);
  sc.bind(smem_raw + 2 * kRows * Six<T>::bytes_per_row(), 2 * kRows);

  // the staged operands, 3 values per thread: element (array, slot, row,
  // lane, component)
  using Sg = Staged<IN, OUT, DOT>;
  T *stage = reinterpret_cast<T *>(smem_raw + 4 * kRows * Six<T>::bytes_per_row());
  auto slot_at = [&](int arr, int z, int row) -> T * {
    return stage + ((arr * Sg::kSlots + (z & (Sg::kSlots - 1))) * kRows + row) * 96 + 3 * tx;
  };
  T *const ring_u = stage + Sg::kArrays * Sg::kSlots * kRows * 96;
  auto ring_at = [&](int z) -> T * { return ring_u + ((z & 3) * kRows + ty) * 96 + 3 * tx; };

  // prefetched next plane: own node, the row-above node (last row), the
  // fixed-component bits (all set where there is no node, so its value is
  // masked) and the modulus of the element layer below it
  T pu[3] = {T(0), T(0), T(0)}, pq[3] = {T(0), T(0), T(0)};
  unsigned pf = 7u, pf2 = 7u;
  T pE = T(0);
  auto fetch = [&](int z) {   // z is uniform over the CTA
    // fresh zeros every plane let the loads target renamed registers
    pf = pf2 = 7u;
    if (!Sg::kIn) {
#pragma unroll
      for (int c = 0; c < 3; ++c) pu[c] = pq[c] = T(0);
    }
    pE = T(0);
    if (z >= 0 && z < Nz) {
      const int n = nofs + z * NP;
      if (nin) {
        pf = load_ro(fix + n);
        if (Sg::kIn) {
          T *db = slot_at(Sg::kSlotB, z, ty), *dd = slot_at(Sg::kSlotD, z, ty);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            copy_async(db + c, args.b + 3 * (int64_t)n + c);
            copy_async(dd + c, args.dinv + 3 * (int64_t)n + c);
          }
        } else {
#pragma unroll
          for (int c = 0; c < 3; ++c) pu[c] = load_ro(args.u + 3 * (int64_t)n + c);
        }
      }
      if (nin2) {
        const int n2 = nofs2 + z * NP;
        pf2 = load_ro(fix + n2);
        if (Sg::kIn) {
          T *db = slot_at(Sg::kSlotB, z, TY), *dd = slot_at(Sg::kSlotD, z, TY);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            copy_async(db + c, args.b + 3 * (int64_t)n2 + c);
            copy_async(dd + c, args.dinv + 3 * (int64_t)n2 + c);
          }
        } else {
#pragma unroll
          for (int c = 0; c < 3; ++c) pq[c] = load_ro(args.u + 3 * (int64_t)n2 + c);
        }
      }
    }
    const int ez = z - 1;
    if (exy && ez >= 0 && ez < nelz) pE = load_ro(E + eofs + ez * EP);
  };
  // the epilogue operands of plane z
  auto fetch_out = [&](int z) {
    if (!Sg::kIn && Sg::kArrays > 0 && own && z >= zs && z < ze) {
      const int64_t i = 3 * ((int64_t)nofs + (int64_t)z * NP);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (Sg::kB) copy_async(slot_at(Sg::kSlotB, z, ty) + c, args.b + i + c);
        if (Sg::kD) copy_async(slot_at(Sg::kSlotD, z, ty) + c, args.dinv + i + c);
        if (Sg::kY) copy_async(slot_at(Sg::kSlotY, z, ty) + c, args.y2 + i + c);
      }
    }
  };

  T FA[4][3], FB[4][3], CA[4][3], CB[4][3], les[3], led[3];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int c = 0; c < 3; ++c) FA[m][c] = FB[m][c] = CA[m][c] = CB[m][c] = T(0);
#pragma unroll
  for (int c = 0; c < 3; ++c) les[c] = led[c] = T(0);
  double dsum = 0;       // this thread's share of the dot product
  unsigned fpipe = 0u;   // fixed bits of the last three planes, 8 bits each

  // one step of the z-march at plane p: Fprev = faces of plane p-1 (in),
  // Fp = faces of plane p (out), ctop = contributions of element layer p-2
  // to face p-1 (in), top = those of layer p-1 to face p (out)
  auto step = [&](int p, const T(&Fprev)[4][3], T(&Fp)[4][3], const T(&ctop)[4][3],
                  T(&top)[4][3]) {
    T cu[3], cq[3];
    const unsigned f = pf;
    if (Sg::kArrays > 0) copy_wait();   // issued one plane ago, by this thread for itself
    if (Sg::kIn) {
      const T *sb = slot_at(Sg::kSlotB, p, ty), *sd = slot_at(Sg::kSlotD, p, ty);
#pragma unroll
      for (int c = 0; c < 3; ++c) pu[c] = args.invtheta * (sd[c] * sb[c]);
      if (lastrow) {
        const T *qb = slot_at(Sg::kSlotB, p, TY), *qd = slot_at(Sg::kSlotD, p, TY);
#pragma unroll
        for (int c = 0; c < 3; ++c) pq[c] = args.invtheta * (qd[c] * qb[c]);
      }
    } else if (Sg::kU) {
      T *r = ring_at(p);
#pragma unroll
      for (int c = 0; c < 3; ++c) r[c] = pu[c];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      cu[c] = ((f >> c) & 1u) ? T(0) : pu[c];
      cq[c] = ((pf2 >> c) & 1u) ? T(0) : pq[c];
    }
    const T Ee = pE;
    fpipe = (fpipe << 8) | f;
    if (p + 1 <= ze) fetch(p + 1);
    fetch_out(p - 1);
    const int rb = (p & 1) * kRows, rb1 = kRows - rb;   // this / the other buffer

    // ---- x-edges of plane p (s = u(x+1) + u(x), d = u(x+1) - u(x)) and
    // the xy-faces: modes (1, x, y, xy)
    if (p <= ze) {
      T s0[3], d0[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const T r = __shfl_down_sync(kFull, cu[c], 1);
        s0[c] = r + cu[c];
        d0[c] = r - cu[c];
      }
      se.put(rb + ty, tx, s0, d0);
      if (lastrow) {
        T s2[3], d2[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const T r = __shfl_down_sync(kFull, cq[c], 1);
          s2[c] = r + cq[c];
          d2[c] = r - cq[c];
        }
        se.put(rb + TY, tx, s2, d2);
      }
      __syncthreads();
      T s1[3], d1[3];
      se.get(rb + ty + 1, tx, s1, d1);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        Fp[0][c] = s0[c] + s1[c];
        Fp[1][c] = d0[c] + d1[c];
        Fp[2][c] = s1[c] - s0[c];
        Fp[3][c] = d1[c] - d0[c];
      }
    } else {
      __syncthreads();
    }

    // ---- nodes of plane p-2: complete the edge (the face of row ty-1
    // left its part in sc row ty), transpose the x stage
    if (p - 2 >= zs && p - 2 < ze) {
      T gs[3], gd[3], val[3];
      sc.get(rb1 + ty, tx, gs, gd);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const T es = les[c] + gs[c], ed = led[c] + gd[c];
        const T right = es + ed;
        const T left = __shfl_up_sync(kFull, right, 1);
        val[c] = (es - ed) + left;
      }
      if (own) {
        const int64_t i = 3 * (nofs + (int64_t)(p - 2) * NP);
        const unsigned fo = (fpipe >> 16) & 0xffu;
        const T *sb = slot_at(Sg::kSlotB, p - 2, ty), *sd = slot_at(Sg::kSlotD, p - 2, ty),
                *sy = slot_at(Sg::kSlotY, p - 2, ty), *su = ring_at(p - 2);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const bool fixed = (fo >> c) & 1u;
          const T bi = Sg::kB ? sb[c] : T(0), di = Sg::kD ? sd[c] : T(0),
                  yi = Sg::kY ? sy[c] : T(0);
          // the input is needed on fixed dofs (identity rows) and by the
          // Chebyshev epilogues
          T uv = T(0);
          if (Sg::kIn)
            uv = args.invtheta * (di * bi);
          else if (Sg::kU)
            uv = su[c];
          else if (fixed)
            uv = load_ro(args.u + i + c);
          const T yv = sym_out_v<T, OUT>(args, i + c, fixed ? uv : val[c], uv, bi, di, yi);
          if (DOT)
            dsum += static_cast<double>(OUT == OUT_Y ? uv : OUT == OUT_RESID ? yv : bi) *
                    static_cast<double>(yv);
        }
      }
    }

    // ---- element layer p-1 between faces p-1 (Fprev) and p (Fp); the face
    // of plane p-1 is then complete: G = ctop + bottom contributions
    T G[4][3];
    if (p - 1 >= zs - 1 && p - 1 < ze) {
      T v[8][3], o[8][3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        v[0][c] = T(0);   // rigid translation: not coupled
#pragma unroll
        for (int m = 1; m < 4; ++m) v[m][c] = Fp[m][c] + Fprev[m][c];
#pragma unroll
        for (int m = 0; m < 4; ++m) v[m + 4][c] = Fp[m][c] - Fprev[m][c];
      }
      modal_couple(v, o, kh);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        top[0][c] = Ee * o[4][c];
        G[0][c] = fma(-Ee, o[4][c], ctop[0][c]);
#pragma unroll
        for (int m = 1; m < 4; ++m) {
          const T a = Ee * o[m][c];
          top[m][c] = fma(Ee, o[m + 4][c], a);
          G[m][c] = fma(-Ee, o[m + 4][c], ctop[m][c] + a);
        }
      }
    } else {
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          top[m][c] = T(0);
          G[m][c] = ctop[m][c];
        }
    }

    // ---- transpose the y stage of face p-1: the lower edge (own row) keeps
    // its part in registers, the upper edge's part goes to sc row ty + 1
    T gs[3], gd[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      les[c] = G[0][c] - G[2][c];
      led[c] = G[1][c] - G[3][c];
      gs[c] = G[0][c] + G[2][c];
      gd[c] = G[1][c] + G[3][c];
    }
    sc.put(rb + ty + 1, tx, gs, gd);
  };

  pdl_wait();
  fetch(zs - 1);
  // two steps per trip with the state arrays swapping roles, so nothing is
  // copied between planes
  for (int p = zs - 1; p <= ze + 1; p += 2) {
    step(p, FA, FB, CA, CB);
    if (p + 1 <= ze + 1) step(p + 1, FB, FA, CB, CA);
  }
  // after the stores (pdl.cuh); blocks that come earlier and wait are in the
  // way, too (91x47x53 mixed: 3.17 ms a solve for 3.07)
  pdl_launch_dependents();
  if (DOT) {
    // one partial per CTA of the column
    const int nchunk = args_in.nchunk, col = COLS ? (int)blockIdx.z / nchunk : 0;
    if (dot.skip && dot.skip[col * kColScal] != 0.0) return;
    const int per = gridDim.x * gridDim.y * nchunk;
    const int cta = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * (blockIdx.z - col * nchunk));
    finish_reduction(dsum, ty * 32 + tx, 32 * TY, cta, per, dot.part + (int64_t)col * per,
                     dot.ticket + col, dot.out + col * kColScal,
                     dot.shift ? dot.shift + col * kColScal : nullptr);
  }
}

constexpr int kTY = 8;

template <typename T, int IN, int OUT, bool DOT>
constexpr size_t staged_smem() {
  return (kTY + 1) * (4 * Six<T>::bytes_per_row() + Staged<IN, OUT, DOT>::planes() * 96 * sizeof(T));
}

// opts a kernel in to > 48 KB of dynamic shared memory (the FP64 tiles), at its
// first launch on a device (setting it loads the kernel)
template <typename T, int IN, int OUT, bool COLS, bool DOT>
void set_smem_attr(int dev) {
  static unsigned long long done = 0;   // bit per device
  if ((done >> (dev & 63)) & 1ull) return;
  cudaFuncSetAttribute(k_apply_staged<T, kTY, IN, OUT, COLS, DOT>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)staged_smem<T, IN, OUT, DOT>());
  done |= 1ull << (dev & 63);
}

// grid of the staged kernel: 30 x (kTY-1) owned node columns per CTA, and z
// chunks chosen by their time: a CTA takes its planes and about 2.3 more (the
// pipeline's fill, and the element layer a chunk computes again), 0.85 us
// (FP64) or 0.6 us (FP32) each, and the CTAs run in waves of what the SMs
// hold -- one an SM in FP64; two in FP32, which share it: the pair's planes
// take 1.55 times as long as one CTA's alone.  Against the best of all chunk
// counts, measured for ten meshes from 12x6x6 to 192x96x96 in FP32, FP64 and
// blocks of 5 and 8 columns, this choice is 0.3% slower in the mean, at most
// 9%.  Chunks of at least 8 planes in whole waves took, in us: 10.4 (now 5.5)
// for 12x6x6, 12.5 (6.4) for 48x24x24, 14.6 (14.6) for 91x47x53 and 29.9
// (27.0) for 128x64x64 in FP64; 12.6 (10.4) and 18.6 (16.6) for the last two
// in FP32.
template <typename T>
void staged_grid(const Ctx &c, int nb, dim3 &grid, int &zchunk) {
  const int Nx = c.nel[0] + 1, Ny = c.nel[1] + 1, Nz = c.nel[2] + 1;
  const int gx = (Nx + kLanesOut - 1) / kLanesOut, gy = (Ny + kTY - 2) / (kTY - 1);
  const int dev = c.device & 63;
  static unsigned long long attr_set = 0;   // bit per device
  static int slots_cache[64] = {0}, sms_cache[64] = {0};
  if (!((attr_set >> dev) & 1ull)) {
    set_smem_attr<T, IN_CHEB, OUT_CHEB2, true, false>(dev);
    int per_sm = 0, sms = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &per_sm, k_apply_staged<T, kTY, IN_CHEB, OUT_CHEB2, true, false>, 32 * kTY,
        staged_smem<T, IN_CHEB, OUT_CHEB2, false>());
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    sms_cache[dev] = std::max(1, sms);
    slots_cache[dev] = std::max(1, per_sm) * sms_cache[dev];
    attr_set |= 1ull << dev;
  }
  const int slots = slots_cache[dev], sms = sms_cache[dev], tiles = gx * gy * nb;
  double best = 0;
  int chunks = 1;
  // beyond eight waves more chunks only add planes
  for (int ch = 1; ch <= Nz && (ch == 1 || (int64_t)ch * tiles <= 8 * (int64_t)slots); ++ch) {
    const int zc = (Nz + ch - 1) / ch;
    const int64_t n = (int64_t)tiles * ((Nz + zc - 1) / zc), rest = n % slots;
    const double shared = slots > sms ? 1.55 : 1.0;
    const double waves = shared * (double)(n / slots) + (rest == 0 ? 0.0 : rest <= sms ? 1.0 : shared);
    const double t = waves * (zc + 2.3);
    if (ch == 1 || t < best) {
      best = t;
      chunks = ch;
    }
  }
  zchunk = (Nz + chunks - 1) / chunks;
  grid = dim3(gx, gy, nb * ((Nz + zchunk - 1) / zchunk));
}

template <typename T, int IN, int OUT, bool DOT = false>
void launch_mode(const Ctx &c, const T *E, const ApplyArgs<T> &args_in,
                 cudaStream_t s, int nb, DotOut dot = {}) {
  dim3 grid;
  int zchunk = 0;
  staged_grid<T>(c, nb, grid, zchunk);
  ApplyArgs<T> args = args_in;
  args.ld = 3 * c.nn;
  args.nchunk = (int)grid.z / nb;
  dot.part = c.apply_part;
  dot.ticket = c.ticket;
  const Kh<T> &kh = *reinterpret_cast<const Kh<T> *>(
      sizeof(T) == 8 ? (const void *)&c.kh64 : (const void *)&c.kh32);
  constexpr size_t smem = staged_smem<T, IN, OUT, DOT>();
  count_launch();
  if (nb == 1) {
    set_smem_attr<T, IN, OUT, false, DOT>(c.device);
    launch_pdl(k_apply_staged<T, kTY, IN, OUT, false, DOT>, grid, dim3(32, kTY), smem, s, c.nel[0],
               c.nel[1], c.nel[2], zchunk, E, c.idm, args, kh, dot);
  } else {
    set_smem_attr<T, IN, OUT, true, DOT>(c.device);
    launch_pdl(k_apply_staged<T, kTY, IN, OUT, true, DOT>, grid, dim3(32, kTY), smem, s, c.nel[0],
               c.nel[1], c.nel[2], zchunk, E, c.idm, args, kh, dot);
  }
}

}  // namespace

// staged_grid makes at most max(8 x resident CTAs, tiles x columns) CTAs
int64_t apply_dot_parts(const int *nel, int sms) {
  const int64_t gx = (nel[0] + 1 + kLanesOut - 1) / kLanesOut;
  const int64_t gy = (nel[1] + 1 + kTY - 2) / (kTY - 1);
  constexpr int kMaxPerSm = 2048 / (32 * kTY);
  return std::max<int64_t>(8 * kMaxPerSm * (int64_t)sms, gx * gy * kMaxBatch);
}

template <typename T>
void launch_apply_fine(const Ctx &c, const T *E, const T *u, const T *b, T *y,
                       cudaStream_t s, int nb, const DotOut *dot) {
  ApplyArgs<T> a{};
  a.u = u;
  a.b = b;
  a.y = y;
  if (b && dot)
    launch_mode<T, IN_U, OUT_RESID, true>(c, E, a, s, nb, *dot);
  else if (b)
    launch_mode<T, IN_U, OUT_RESID>(c, E, a, s, nb);
  else if (dot)
    launch_mode<T, IN_U, OUT_Y, true>(c, E, a, s, nb, *dot);
  else
    launch_mode<T, IN_U, OUT_Y>(c, E, a, s, nb);
}

template <typename T>
void launch_apply_fused(const Ctx &c, const T *E, int in, int out,
                        const ApplyArgs<T> &args, cudaStream_t s, int nb, const DotOut *dot) {
  if (in == IN_CHEB && out == OUT_CHEB2)
    launch_mode<T, IN_CHEB, OUT_CHEB2>(c, E, args, s, nb);
  else if (in == IN_U && out == OUT_POST0)
    launch_mode<T, IN_U, OUT_POST0>(c, E, args, s, nb);
  else if (in == IN_U && out == OUT_POST1 && dot)
    launch_mode<T, IN_U, OUT_POST1, true>(c, E, args, s, nb, *dot);
  else if (in == IN_U && out == OUT_POST1)
    launch_mode<T, IN_U, OUT_POST1>(c, E, args, s, nb);
  else if (in == IN_U && out == OUT_RESID)
    launch_mode<T, IN_U, OUT_RESID>(c, E, args, s, nb);
  else if (in == IN_U && out == OUT_SCALE)
    launch_mode<T, IN_U, OUT_SCALE>(c, E, args, s, nb);
  else
    launch_mode<T, IN_U, OUT_Y>(c, E, args, s, nb);
}

template void launch_apply_fine<double>(const Ctx &, const double *,
                                        const double *, const double *,
                                        double *, cudaStream_t, int, const DotOut *);
template void launch_apply_fine<float>(const Ctx &, const float *,
                                       const float *, const float *, float *,
                                       cudaStream_t, int, const DotOut *);
template void launch_apply_fused<double>(const Ctx &, const double *, int, int,
                                         const ApplyArgs<double> &,
                                         cudaStream_t, int, const DotOut *);
template void launch_apply_fused<float>(const Ctx &, const float *, int, int,
                                        const ApplyArgs<float> &, cudaStream_t,
                                        int, const DotOut *);

}  // namespace tpo
