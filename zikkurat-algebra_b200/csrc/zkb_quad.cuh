// XYZZ point arithmetic by four lanes.
//
// The short serial chains of an MSM (merges of cut segments, running sums, window sums, whole MSMs
// of a few thousand points) are bound by the latency of one point operation: a lone thread runs an
// addition's 14 products one after the other (in pairs at best), each about 0.5 us. Here four
// neighbouring lanes hold one point, lane L of the quad its coordinate L (X, Y, ZZ, ZZZ), and the
// independent products of a formula run in one product call across the lanes: an addition is four
// product latencies (14 of the 16 lane products are needed), a doubling three. A lane keeps one
// coordinate, so these kernels need few registers and spill nothing, and a quad's loads and stores
// of a point are one contiguous run.
//
// All 32 lanes of a warp call these functions together; a quad with nothing to add passes the
// identity (ZZ = 0), which leaves the accumulator as it is. Formulas and special cases are those of
// zkb_curve.cuh (add-2008-s, dbl-2008-s-1).
#pragma once
#include "zkb_curve.cuh"

namespace zkb {

static constexpr unsigned FULL = 0xffffffffu;

template <class F>
__device__ __forceinline__ Fe<F> fe_shfl(const Fe<F>& a, int src) {
  Fe<F> r;
#pragma unroll
  for (int i = 0; i < F::N; i++) r.v[i] = __shfl_sync(FULL, a.v[i], src);
  return r;
}
template <class F>
__device__ __forceinline__ Fe<F> fe_shfl_xor(const Fe<F>& a, int mask) {
  Fe<F> r;
#pragma unroll
  for (int i = 0; i < F::N; i++) r.v[i] = __shfl_xor_sync(FULL, a.v[i], mask);
  return r;
}
template <class F>
__device__ __forceinline__ Fe<F> fe_sel(bool c, const Fe<F>& a, const Fe<F>& b) {
  Fe<F> r;
#pragma unroll
  for (int i = 0; i < F::N; i++) r.v[i] = c ? a.v[i] : b.v[i];
  return r;
}

__device__ __forceinline__ int quad_lane() { return threadIdx.x & 3; }
// whether the quad's point is the identity
template <class F>
__device__ __forceinline__ bool quad_is_inf(const Fe<F>& a) {
  return __shfl_sync(FULL, (int)fe_is_zero(a), ((threadIdx.x & 31) & ~3) | 2) != 0;
}

// acc = 2 acc (the identity stays: ZZ3 = V ZZ)
template <class F>
__device__ __noinline__ Fe<F> quad_dbl(const Fe<F> acc) {
  const int L = quad_lane(), b = (threadIdx.x & 31) & ~3;
  const Fe<F> in = fe_sel(L == 1, fe_dbl(acc), acc);           // lane 1: U = 2 Y
  const Fe<F> r1 = fe_mul(in, in);                             // X^2, V
  const Fe<F> V = fe_shfl(r1, b + 1);
  const Fe<F> M = fe_add(fe_dbl(r1), r1);                      // lane 0
  const Fe<F> X = fe_shfl(acc, b);
  const Fe<F> a2 = fe_sel(L == 0, M, fe_sel(L == 3, X, in));
  const Fe<F> r2 = fe_mul(a2, fe_sel(L == 0, M, V));           // M^2, W, ZZ3, S
  const Fe<F> S = fe_shfl(r2, b + 3), W = fe_shfl(r2, b + 1);
  const Fe<F> X3 = fe_sub(r2, fe_dbl(S));
  const Fe<F> r3 = fe_mul(fe_sel(L == 0, M, W), fe_sel(L == 0, fe_sub(S, X3), acc));   // M (S - X3), W Y, -, ZZZ3
  const Fe<F> Y3 = fe_sub(fe_shfl_xor(r3, 1), r3);
  return fe_sel(L == 0, X3, fe_sel(L == 1, Y3, fe_sel(L == 2, r2, r3)));
}

// acc + q
template <class F>
__device__ __noinline__ Fe<F> quad_add(const Fe<F> acc, const Fe<F> q) {
  const int L = quad_lane(), b = (threadIdx.x & 31) & ~3;
  const bool qi = quad_is_inf(q), ai = quad_is_inf(acc);
  if (!__any_sync(FULL, !qi && !ai)) return fe_sel(ai, q, acc);
  const Fe<F> r1 = fe_mul(acc, fe_shfl_xor(q, 2));             // U1, S1, U2, S2
  const Fe<F> t = fe_shfl_xor(r1, 2);
  const Fe<F> lo = fe_sel(L < 2, r1, t);                       // U1, S1, U1, S1
  const Fe<F> D = fe_sub(fe_sel(L < 2, t, r1), lo);            // P, R, P, R
  const bool dz = fe_is_zero_mod(D);
  const bool pz = __shfl_sync(FULL, (int)dz, b), rz = __shfl_sync(FULL, (int)dz, b + 1);
  const Fe<F> r2 = fe_mul(fe_sel(L < 2, D, acc), fe_sel(L < 2, D, q));   // PP, RR, ZZ1 ZZ2, ZZZ1 ZZZ2
  const Fe<F> PP = fe_shfl(r2, b);
  const Fe<F> s = fe_shfl_xor(lo, 1);                          // S1, U1, S1, U1
  const Fe<F> r3 = fe_mul(fe_sel(L == 0, D, fe_sel(L == 1, s, r2)), PP);   // PPP, Q, ZZ3, -
  const Fe<F> PPP = fe_shfl(r3, b);
  const Fe<F> X3 = fe_sub(fe_sub(r2, PPP), fe_dbl(r3));        // lane 1
  const Fe<F> r4 = fe_mul(fe_sel(L == 0, s, fe_sel(L == 1, D, r2)),
                          fe_sel(L == 1, fe_sub(r3, X3), PPP));   // S1 PPP, R (Q - X3), -, ZZZ3
  const Fe<F> e = fe_shfl_xor(fe_sel(L == 1, X3, r4), 1);
  Fe<F> r = fe_sel(L == 0, e, fe_sel(L == 1, fe_sub(r4, e), fe_sel(L == 2, r3, r4)));
  const bool special = pz && !qi && !ai;
  if (__any_sync(FULL, special)) {   // equal or opposite points in some quad
    const Fe<F> d = quad_dbl(acc);
    r = fe_sel(special, fe_sel(rz, d, fe_zero<F>()), r);
  }
  return fe_sel(qi, acc, fe_sel(ai, q, r));
}

// The sum of the warp's eight quads, in every quad
template <class F>
__device__ __forceinline__ Fe<F> quad_warp_sum(Fe<F> a) {
#pragma unroll 1
  for (int d = 4; d < 32; d <<= 1) a = quad_add(a, fe_shfl_xor(a, d));
  return a;
}

// this lane's coordinate of the point at p (XYZZ)
template <class F>
__device__ __forceinline__ Fe<F> quad_load(const uint32_t* __restrict__ p) { return fe_load<F>(p + quad_lane() * F::N); }
template <class F>
__device__ __forceinline__ void quad_store(uint32_t* __restrict__ p, const Fe<F>& a) { fe_store<F>(p + quad_lane() * F::N, a); }
// this lane's coordinate of an affine point; (0, 0) is the identity
template <class F>
__device__ __forceinline__ Fe<F> quad_from_affine(const uint32_t* __restrict__ p, bool neg) {
  const int L = quad_lane(), b = (threadIdx.x & 31) & ~3;
  Fe<F> a = fe_load_nc<F>(p + (L & 1) * F::N);
  const int z = fe_is_zero(a);
  const int zx = __shfl_sync(FULL, z, b), zy = __shfl_sync(FULL, z, b + 1);   // both by every lane
  const bool inf = zx & zy;
  if (L == 1 && neg) a = fe_neg(a);
  return fe_sel(L < 2, a, fe_sel(inf, fe_zero<F>(), fe_one<F>()));
}

}  // namespace zkb
