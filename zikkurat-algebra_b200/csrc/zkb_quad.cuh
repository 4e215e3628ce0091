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

// t + c x as an integer of N + 1 words
template <class F>
__device__ __forceinline__ void int_madd(uint32_t (&t)[F::N + 1], const Fe<F>& x, uint32_t c) {
  uint64_t a = 0;
#pragma unroll
  for (int k = 0; k < F::N; k++) {
    a += (uint64_t)c * x.v[k] + t[k];
    t[k] = (uint32_t)a;
    a >>= 32;
  }
  t[F::N] += (uint32_t)a;
}
// p - x (canonical x, or p for 0)
template <class F>
__device__ __forceinline__ Fe<F> int_neg(const Fe<F>& x) {
  Fe<F> r;
  r.v[0] = sub_cc(F::mod(0), x.v[0]);
#pragma unroll
  for (int k = 1; k < F::N; k++) r.v[k] = subc_cc(F::mod(k), x.v[k]);
  return r;
}

// 16 acc + q, a window of a scalar multiplication, in 12 product latencies instead of 16: on a point of
// y^2 = x^3 + b a doubling needs two. With B = Y^2 and V = 3 b Z^6, X^3 = B - V / 3 takes X out of the
// doubling's higher powers, and with Z' = Y Z
//     X' = X (B - 3V) / 4,   Y' = (B^2 + 6 B V - 3 V^2) / 8,   V' = B^2 (B V).
// Z itself is not needed in between: f, the product of the four Y, scales ZZ and ZZZ by f^2 and f^3,
// and the addition's products with them are made before the doublings end. B - 3V and Y stay unreduced
// integers below 4p and 2.5p: they only enter products, whose results are canonical all the same for
// R' = 2^260 ((ab + mp) / R' < 1.2p). The points must lie on the curve, whose group has odd order (no Y is
// 0). Group FFT of BN254, against four doublings and an addition: 2^9 points 4.30 -> 3.83 ms, 2^12 6.5 ->
// 5.60, 2^14 13.16 -> 11.82. (BLS12-381, whose integer-pipe products are shorter beside the twelve-word
// shuffles and selections, lost 8% in a first form of this and keeps the doublings.)
template <class F>
__device__ __noinline__ Fe<F> quad_window(const Fe<F> acc, const Fe<F> q) {
  static_assert(F::N == 8 && F::DPF && !lazy_v<F>, "BN254's base field, radix 2^260");
  const int L = quad_lane(), b = (threadIdx.x & 31) & ~3;
  const bool qi = quad_is_inf(q), ai = quad_is_inf(acc);
  const Fe<F> q1 = fe_sel(qi && L >= 2, fe_one<F>(), q);   // the identity: ZZ and ZZZ as of 16 acc
  const Fe<F> ZZ = fe_shfl(acc, b + 2), ZZZ = fe_shfl(acc, b + 3);
  const Fe<F> ZZ2 = fe_shfl(q1, b + 2), ZZZ2 = fe_shfl(q1, b + 3);
  Fe<F> r = fe_mul(acc, fe_sel(L == 2, fe_shfl(q1, b), acc));  // -, B, ZZ X2, ZZZ^2
  const Fe<F> x2z = r;                                         // lane 2
  Fe<F> B = fe_shfl(r, b + 1), V = fe_shfl(r, b + 3);
  V = fe_add(fe_dbl(fe_dbl(fe_dbl(V))), V);                    // 3 b ZZZ^2 = 9 ZZZ^2
  Fe<F> f = fe_shfl(acc, b + 1), XY = acc;                     // f in lane 3; X in lane 0, Y elsewhere
  Fe<F> pre[3];                                                // lane 0: Y2 ZZZ, ZZ ZZ2, ZZZ ZZZ2
#pragma unroll
  for (int i = 0; i < 4; i++) {
    uint32_t t[F::N + 1];
#pragma unroll
    for (int k = 0; k < F::N; k++) t[k] = B.v[k];
    t[F::N] = 0;
    Fe<F> u, c1, c2;
    int_madd<F>(t, i == 3 ? fe_sel(L == 0, int_neg<F>(V), V) : int_neg<F>(V), 3);   // B - 3V; lane 1 of the last: B + 3V
#pragma unroll
    for (int k = 0; k < F::N; k++) u.v[k] = t[k];
    if (i == 3) r = fe_mul(fe_sel(L == 0, XY, fe_sel(L == 1, u, fe_sel(L == 2, V, f))),
                           fe_sel(L < 2, u, fe_sel(L == 2, V, f)));   // X (B - 3V), (B + 3V)^2, V^2, f^2
    else r = fe_mul(fe_sel(L == 0, XY, fe_sel(L == 3, V, B)),
                    fe_sel(L == 0, u, fe_sel(L == 1, B, V)));         // X (B - 3V), B^2, B V, V^2
    c1 = fe_shfl(r, b + 1);
    c2 = fe_shfl(r, b + 2);
#pragma unroll
    for (int k = 0; k < F::N; k++) t[k] = c1.v[k];
    t[F::N] = 0;
    if (i == 3) {
      int_madd<F>(t, int_neg<F>(c2), 12);
    } else {
      int_madd<F>(t, c2, 6);
      int_madd<F>(t, int_neg<F>(fe_shfl(r, b + 3)), 3);
      B = c1;
      V = c2;
    }
#pragma unroll
    for (int k = 0; k < F::N; k++) t[k] = L == 0 ? r.v[k] : t[k];
    if (L == 0) t[F::N] = 0;
    const int sh = L == 0 ? 2 : 3;                             // / 4, / 8: + m p makes the low bits zero
    Fe<F> mod;
#pragma unroll
    for (int k = 0; k < F::N; k++) mod.v[k] = F::mod(k);
    int_madd<F>(t, mod, (t[0] * F::n0) & ((1u << sh) - 1));
#pragma unroll
    for (int k = 0; k < F::N; k++) XY.v[k] = __funnelshift_r(t[k], t[k + 1], sh);
    if (i == 3) break;
    const Fe<F> pa = i == 0 ? fe_shfl(q1, b + 1) : i == 1 ? ZZ : ZZZ, pb = i == 0 ? ZZZ : i == 1 ? ZZ2 : ZZZ2;
    r = fe_mul(fe_sel(L == 0, pa, fe_sel(L == 2, B, XY)), fe_sel(L == 0, pb, fe_sel(L == 1, XY, fe_sel(L == 2, V, f))));
    pre[i] = r;                                                // -, B', V', f'
    B = fe_shfl(r, b + 1);
    V = fe_shfl(r, b + 2);
    f = fe_sel(L == 3, r, f);
  }
  const Fe<F> f2 = fe_shfl(r, b + 3);
  r = fe_mul(fe_sel(L == 2, x2z, fe_sel(L == 3, f, XY)), fe_sel(L == 0, ZZ2, fe_sel(L == 1, ZZZ2, f2)));   // U1, S1, U2, f^3
  const Fe<F> U1 = fe_shfl(r, b), S1 = r, f3 = fe_shfl(r, b + 3);
  const Fe<F> P = fe_sub(fe_shfl(r, b + 2), U1);
  const Fe<F> y2z = fe_shfl(pre[0], b), zz = fe_shfl(pre[1], b), zzz = fe_shfl(pre[2], b);
  r = fe_mul(fe_sel(L == 0, P, fe_sel(L == 1, y2z, fe_sel(L == 2, zz, zzz))),
             fe_sel(L == 0, P, fe_sel(L == 2, f2, f3)));        // PP, S2, ZZ, ZZZ
  Fe<F> at16 = fe_sel(L < 2, reduce_once<F, false>(reduce_once<F, false>(XY.v, 0u).v, 0u), r);   // 16 acc, for q the identity
  const Fe<F> R = fe_sub(r, S1);                                // lane 1
  const bool dz = fe_is_zero_mod(fe_sel(L == 0, P, R));
  const bool pz = __shfl_sync(FULL, (int)dz, b), rz = __shfl_sync(FULL, (int)dz, b + 1);
  const Fe<F> PP = fe_shfl(r, b), zzz16 = r;
  r = fe_mul(fe_sel(L == 0, P, fe_sel(L == 1, R, fe_sel(L == 2, r, U1))), fe_sel(L == 1, R, PP));   // PPP, RR, ZZ3, Q
  const Fe<F> PPP = fe_shfl(r, b), Q = fe_shfl(r, b + 3), r3 = r;
  const Fe<F> X3 = fe_sub(fe_sub(r, PPP), fe_dbl(Q));           // lane 1
  r = fe_mul(fe_sel(L == 0, fe_shfl(S1, b + 1), fe_sel(L == 1, R, zzz16)),
             fe_sel(L == 1, fe_sub(Q, X3), PPP));               // S1 PPP, R (Q - X3), -, ZZZ3
  const Fe<F> e = fe_shfl_xor(fe_sel(L == 1, X3, r), 1);
  Fe<F> o = fe_sel(L == 0, e, fe_sel(L == 1, fe_sub(r, e), fe_sel(L == 2, r3, r)));
  const bool special = pz && !qi && !ai;
  if (__any_sync(FULL, special)) {   // 16 acc = q or -q in some quad
    const Fe<F> d = quad_dbl(q);
    o = fe_sel(special, fe_sel(rz, d, fe_zero<F>()), o);
  }
  return fe_sel(ai, q, fe_sel(qi, at16, o));
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
