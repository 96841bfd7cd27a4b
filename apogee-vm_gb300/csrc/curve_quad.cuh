// XYZZ points held by four lanes: lane l of an aligned group of four (a quad)
// holds coordinate l of (X, Y, ZZ, ZZZ), and a group operation runs its
// products side by side on the lanes.
//
// The serial parts of an MSM (edge runs, bucket reduction, window Horner) are
// chains of dependent point operations with few chains to run, so a chain's
// latency is what they cost. One thread's addition is fourteen products after
// one another (at 847 clocks each, 5.8 us); over a quad it is four product
// steps and the shuffles between them (measured 2.3 us), a doubling three (1.7):
// the lanes that have no product in a step repeat one, so a quad spends sixteen
// products on an addition's fourteen, and holds 8 registers a point, not 32.
//
// Every function here is called by all 32 lanes of a warp together.
#pragma once
#include "curve.cuh"

namespace apg {

__device__ __forceinline__ Fq quad_get(const Fq& a, int lane) {  // the value of another lane of the warp
  Fq r;
#pragma unroll
  for (int w = 0; w < 8; ++w) r.v[w] = __shfl_sync(0xffffffffu, a.v[w], lane);
  return r;
}

__device__ __forceinline__ Fq quad_sel(bool c, const Fq& a, const Fq& b) {
  Fq r;
#pragma unroll
  for (int w = 0; w < 8; ++w) r.v[w] = c ? a.v[w] : b.v[w];
  return r;
}

// Whether the flag holds in lane k of this lane's quad.
__device__ __forceinline__ bool quad_flag(bool f, int lane, int k) {
  return (__ballot_sync(0xffffffffu, f) >> ((lane & 28) | k)) & 1u;
}

__device__ __forceinline__ bool quad_is_inf(const Fq& p, int lane) { return quad_flag(fe_is_zero(p), lane, 2); }

// dbl-2008-s-1: 2 p (infinity stays infinity: ZZ3 = V ZZ = 0).
static __device__ __noinline__ Fq quad_dbl(const Fq p) {
  const int lane = threadIdx.x & 31, l = lane & 3, g = lane & 28;
  const Fq a = quad_sel(l == 1, fe_dbl(p), p);  // X, U = 2 Y
  const Fq t = cmul(a, a);                      // X^2, V
  const Fq v = quad_get(t, g | 1), x = quad_get(p, g);
  const Fq m = fe_add(fe_dbl(t), t);  // lane 0: M = 3 X^2
  Fq f = quad_sel(l == 3, x, p);
  f = quad_sel(l == 0, m, f);
  f = quad_sel(l == 1, a, f);
  const Fq s = cmul(f, quad_sel(l == 0, m, v));  // M^2, W = U V, ZZ3 = V ZZ, S = X V
  const Fq S = quad_get(s, g | 3), W = quad_get(s, g | 1);
  const Fq x3 = fe_sub(fe_sub(s, S), S);  // lane 0
  const Fq h = cmul(quad_sel(l == 0, m, W), quad_sel(l == 0, fe_sub(S, x3), p));  // M (S - X3), W Y, -, ZZZ3
  const Fq y3 = fe_sub(quad_get(h, g), h);                                        // lane 1
  Fq r = quad_sel(l == 2, s, h);
  r = quad_sel(l == 0, x3, r);
  return quad_sel(l == 1, y3, r);
}

// add-2008-s: p + q, infinities, doublings and opposites included.
static __device__ __noinline__ Fq quad_add(const Fq p, const Fq q) {
  const int lane = threadIdx.x & 31, l = lane & 3, g = lane & 28;
  const bool pinf = quad_is_inf(p, lane), qinf = quad_is_inf(q, lane);
  const Fq m = cmul(p, quad_get(q, lane ^ 2));  // U1 = X1 ZZ2, S1 = Y1 ZZZ2, U2 = ZZ1 X2, S2 = ZZZ1 Y2
  const Fq o = quad_get(m, lane ^ 2);
  const Fq d = fe_sub(quad_sel(l < 2, o, m), quad_sel(l < 2, m, o));  // P, R, P, R
  const unsigned z = __ballot_sync(0xffffffffu, fe_is_zero(d));
  const bool same_x = (z >> g) & 1u, same_y = (z >> (g | 1)) & 1u;
  const Fq t = cmul(quad_sel(l < 2, d, p), quad_sel(l < 2, d, q));  // PP, R^2, ZZ1 ZZ2, ZZZ1 ZZZ2
  const Fq pp = quad_get(t, g), u1 = quad_get(m, g);
  Fq f = quad_sel(l == 0, d, t);
  f = quad_sel(l == 1, u1, f);
  const Fq s = cmul(f, pp);  // PPP, Q = U1 PP, ZZ3, -
  const Fq ppp = quad_get(s, g), Q = quad_get(s, g | 1);
  const Fq x3 = fe_sub(fe_sub(fe_sub(quad_get(t, g | 1), ppp), Q), Q);
  const Fq r1 = quad_get(d, g | 1);
  f = quad_sel(l == 0, r1, t);
  f = quad_sel(l == 1, m, f);
  const Fq w = cmul(f, quad_sel(l == 0, fe_sub(Q, x3), ppp));  // R (Q - X3), S1 PPP, -, ZZZ3
  const Fq y3 = fe_sub(quad_get(w, g), w);                     // lane 1
  Fq r = quad_sel(l == 2, s, w);
  r = quad_sel(l == 0, x3, r);
  r = quad_sel(l == 1, y3, r);
  const bool special = !pinf && !qinf && same_x;
  if (__any_sync(0xffffffffu, special)) {  // equal x: 2 p, or infinity for opposite points
    const Fq twice = quad_dbl(p);
    if (special) r = quad_sel(same_y, twice, fe_zero<FqConsts>());
  }
  r = quad_sel(qinf, p, r);
  return quad_sel(pinf, q, r);
}

// Coordinate l of a stored point.
__device__ __forceinline__ Fq quad_ld(const Xyzz* p, int l) { return ld_fe(reinterpret_cast<const Fq*>(p) + l); }
__device__ __forceinline__ void quad_st(Xyzz* p, int l, const Fq& a) { st_fe(reinterpret_cast<Fq*>(p) + l, a); }

// The whole point, in every lane of the quad.
__device__ __forceinline__ Xyzz quad_gather(const Fq& p, int lane) {
  const int g = lane & 28;
  Xyzz r;
  r.x = quad_get(p, g);
  r.y = quad_get(p, g | 1);
  r.zz = quad_get(p, g | 2);
  r.zzz = quad_get(p, g | 3);
  return r;
}

}  // namespace apg
