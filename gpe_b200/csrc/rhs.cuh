// rhs.cuh -- the right-hand side of one site, shared by the kernels that
// evaluate it (stage_kernel.cuh, pair_kernel.cuh): the same operations in the
// same order whichever kernel computes a site, so that a state does not
// depend on the launch form.  Every sum of products is written as an explicit
// fused multiply-add, which leaves the compiler nothing to contract
// differently from one kernel to the other.
#pragma once

#include "vec2.cuh"

namespace gpe {

// Right-hand-side forms of a recipe (see the top of stage_kernel.cuh).
enum : int { FORM_PLAIN = 0, FORM_TRAP = 1, FORM_FULL = 2 };

// The star of one site: itself and its neighbours at distance 1 and (order 4)
// 2 along each axis.
template <typename V>
struct Star {
  V f0, xm1, xp1, ym1, yp1, zm1, zp1, xm2, xp2, ym2, yp2, zm2, zp2;
};

// Laplacian: sum_axes c1*(f1+f-1) + c2*(f2+f-2), plus c0*f0.
template <int R, typename V, typename C>
__device__ __forceinline__ V star_laplacian(const Star<V>& s, const C& c) {
  V L = vmul(c.cx1, vadd(s.xp1, s.xm1));
  L = vfma(c.cy1, vadd(s.yp1, s.ym1), L);
  L = vfma(c.cz1, vadd(s.zp1, s.zm1), L);
  if (R == 2) {
    L = vfma(c.cx2, vadd(s.xp2, s.xm2), L);
    L = vfma(c.cy2, vadd(s.yp2, s.ym2), L);
    L = vfma(c.cz2, vadd(s.zp2, s.zm2), L);
  }
  return vfma(c.c0l, s.f0, L);
}

// Stencil coefficients of a run, one value in both lanes.
template <typename V>
struct LapCoef {
  V cx1, cx2, cy1, cy2, cz1, cz2, c0l;
};

// K without sponge, gradient or sphere terms: cL*L + (c0 + cV*Vs + cn|u|^2) u
// (FORM_PLAIN has no trap).
template <bool TRAP, typename V, typename TC>
__device__ __forceinline__ V rhs_plain(V L, V f0, TC Vs, TC c0, TC cV, TC cn, V cL) {
  const TC a2 = fma(f0.y, f0.y, f0.x * f0.x);
  const TC s = TRAP ? fma(cn, a2, fma(cV, Vs, c0)) : fma(cn, a2, c0);
  return vfma(vsplat(s), f0, vmul(cL, L));
}

// Terms of the full form (see RunDesc in stage_kernel.cuh).
template <typename TC>
struct FullTerms {
  TC c0, cV, cn, ar0, ard, ai, gx1, gx2;
};

// K with every term the equation may have: sponge D, gradient U (0 weight:
// not evaluated), sphere mask m (1: none).
template <int R, typename V, typename TC>
__device__ __forceinline__ V rhs_full(const Star<V>& s, V L, V cL, const FullTerms<TC>& t, TC Vs,
                                      bool use_D, TC D, bool use_grad, TC U) {
  const TC a2 = fma(s.f0.y, s.f0.y, s.f0.x * s.f0.x);
  const TC sc = fma(t.cn, a2, fma(t.cV, Vs, t.c0));
  const V B = vfma(vsplat(sc), s.f0, vmul(cL, L));
  const TC arr = use_D ? fma(t.ard, D, t.ar0) : t.ar0;
  V K = vfma(vsplat(arr), B, vmul(vpair(-t.ai, t.ai), vswap(B)));
  if (use_grad) {
    const V mone = vsplat(TC(-1));
    V gx = vmul(vsplat(t.gx1), vfma(s.xm1, mone, s.xp1));
    if (R == 2) gx = vfma(vsplat(t.gx2), vfma(s.xm2, mone, s.xp2), gx);
    K = vfma(vsplat(U), gx, K);
  }
  return K;
}

// The mask of equation 3's sphere at the point (X, Y, Z).
__device__ __forceinline__ double sphere_mask(double X, double Y, double Z) {
  return 0.5 * (1.0 + tanh(sqrt(fma(Z, Z, fma(Y, Y, X * X))) - 10.0 - 2.0));
}

}  // namespace gpe
