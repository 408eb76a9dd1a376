// Input and epilogue forms shared by the level-1 operator kernels (the
// half-stored stencil, kernels_mg.cu; the tensor-core form, kernels_l1tc.cu).
// They match the fine-level kernel's (kernels_apply_staged.cu):
// IN_U reads u, IN_CHEB forms the Chebyshev start invtheta D^-1 b on the
// fly; OUT_Y / OUT_RESID / OUT_CHEB2 / OUT_POST0 / OUT_POST1 write Au,
// b - Au or the fused Chebyshev(2) updates, OUT_SCALE D^-1 Au (a step of the
// power iteration).
#pragma once

#include "tpo_internal.h"

namespace tpo {

template <typename T, int IN>
__device__ __forceinline__ T sym_in(const ApplyArgs<T> &a, int i) {
  if (IN == IN_CHEB) return a.invtheta * (a.dinv[i] * a.b[i]);
  return a.u[i];
}

// the epilogue on values already loaded: bi = b[i], di = dinv[i],
// y2i = y2[i] (each read only by the forms that use it); returns y[i]
template <typename T, int OUT, typename I>
__device__ __forceinline__ T sym_out_v(const ApplyArgs<T> &a, I i, T Au, T u, T bi, T di, T y2i) {
  T y;
  if (OUT == OUT_Y) {
    y = Au;
  } else if (OUT == OUT_RESID) {
    y = bi - Au;
  } else if (OUT == OUT_CHEB2) {
    const T r1 = di * bi - di * Au;
    y = u + (a.c1 * u + a.c2 * r1);
  } else if (OUT == OUT_POST0) {
    y = a.invtheta * (di * (bi - Au));
    a.y2[i] = u + y;
  } else if (OUT == OUT_SCALE) {
    y = Au * di;
  } else {   // OUT_POST1
    const T r1 = a.theta * u - di * Au;
    y = y2i + (a.c1 * u + a.c2 * r1);
  }
  a.y[i] = y;
  return y;
}

template <int OUT>
struct OutNeeds {
  static constexpr bool b = OUT == OUT_RESID || OUT == OUT_CHEB2 || OUT == OUT_POST0;
  static constexpr bool dinv = OUT == OUT_CHEB2 || OUT == OUT_POST0 || OUT == OUT_POST1 ||
                               OUT == OUT_SCALE;
  static constexpr bool y2 = OUT == OUT_POST1;
};

template <typename T, int OUT>
__device__ __forceinline__ void sym_out(const ApplyArgs<T> &a, int i, T Au, T u) {
  sym_out_v<T, OUT>(a, i, Au, u, OutNeeds<OUT>::b ? a.b[i] : T(0),
                    OutNeeds<OUT>::dinv ? a.dinv[i] : T(0), OutNeeds<OUT>::y2 ? a.y2[i] : T(0));
}

}  // namespace tpo
