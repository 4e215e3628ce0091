// G1 group FFT and binary MSMs on the device.
//
// Group FFT: the reference's *_G1_{proj,jac}_fft_forward / _fft_inverse
// (lib/cbits/curves/g1/proj/bn128_G1_proj.c:791-902, jac/bn128_G1_jac.c:840-950) are the NTT
// networks of poly_mont with points in place of field elements: a forward DIT whose butterfly
// is (u + [w]v, u - [w]v) and an inverse DIF with (u + v)/2, [w^-1](u - v)/2, where [w]P is a
// scalar multiplication by the standard integer of a Montgomery Fr element. The map from input
// points to output points is Fr-linear, so any evaluation order of the same network gives the
// same group elements. Here:
//   - points live in XYZZ coordinates in one device buffer; the input is written in
//     bit-reversed order for the DIT (natural for the DIF) and stages run in place, one launch
//     per stage, one thread per butterfly;
//   - stage s (block size 2^s) uses the twiddle gen^(j 2^(m-s)) for j < 2^(s-1) (the reference
//     squares the generator per recursion level and multiplies up the powers), read from one
//     table of gen^e, e < N/2, in standard form; j = 0 needs no multiplication;
//   - the inverse's per-level halving, (1/2)^m per output, is folded into the first DIF stage:
//     its sum takes [2^-m] and its difference [2^-m ginv^j];
//   - scalar multiplication uses signed 4-bit windows (digits -7..8, table 1P..8P, 4 doublings
//     per window); the results are converted to the reference's normalised form
//     (bn128_G1_proj.c:78-97; the Jacobian normalisation bn128_G1_jac.c:62-85 writes the same
//     bytes: (x, y, 1), infinity (0, 1, 0)).
//
// Binary MSMs: *_MSM_binary_coeff_* (bn128_G1_proj.c:684-698) sums the bases whose byte
// coefficient is non-zero; *_multi_MSM_binary_coeff_* (bn128_G1_proj.c:718-782) does that for
// each row of an nrows x npoints byte matrix, with the bases split into windows of c columns and
// all 2^c subset sums of a window precomputed, so a row adds one table entry per window. Here the
// rows are grouped instead and the columns go to buckets by their bits in a group (zkb_msm_bits.h):
// 64 rows of 2^18 columns are 17 M field products against 60 M by subset sums. Columns are processed
// in chunks (host coefficient rows and bases are gathered into pinned staging and copied while the
// previous chunk computes), many rows in batches; the chunks' sums add up in the rows' points. The order
// of additions differs; every result is the same group element, written in the drop-in's encoding.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "zkb_curve.cuh"
#include "zkb_dpf.cuh"
#include "zkb_host_ec.h"
#include "zkb_msm_bits.h"
#include "zkb_quad.cuh"
#include "zkb_runtime.h"

namespace zkb {

// ------------------------------------------------------------------------ device helpers
template <class F>
__device__ __noinline__ Xyzz<F> xyzz_sum(Xyzz<F> a, const Xyzz<F> b) {
  xyzz_add(a, b);
  return a;
}

template <class F>
__device__ __forceinline__ Xyzz<F> xyzz_negate(Xyzz<F> p) {
  p.Y = fe_neg(p.Y);
  return p;
}

// Output encodings of the drop-in entry points (the host twin is host::xyzz_write). With CONV, p
// is in the FP64 radix R' (zkb_dpf.cuh) and the coordinates go back to the reference's radix R
// with kout = R mod p, which is also the radix-R form of 1.
template <class F, bool CONV>
__device__ void xyzz_write_out(const Xyzz<F>& p, int kind, uint32_t* __restrict__ out, const Fe<F>& kout) {
  const Fe<F> one = CONV ? kout : fe_one<F>();
  if (xyzz_is_inf(p)) {
    if (kind == ZKG_OUT_AFFINE) {
      for (int i = 0; i < 2 * F::N; i++) out[i] = 0xffffffffu;
      return;
    }
    fe_store<F>(out, kind == ZKG_OUT_JAC ? one : fe_zero<F>());
    fe_store<F>(out + F::N, one);
    fe_store<F>(out + 2 * F::N, fe_zero<F>());
    return;
  }
  const Fe<F> d = fe_inv(fe_mul(p.ZZ, p.ZZZ));
  Fe<F> x = fe_mul(p.X, fe_mul(d, p.ZZZ)), y = fe_mul(p.Y, fe_mul(d, p.ZZ));
  if (CONV) {
    x = fe_mul(x, kout);
    y = fe_mul(y, kout);
  }
  fe_store<F>(out, x);
  fe_store<F>(out + F::N, y);
  if (kind != ZKG_OUT_AFFINE) fe_store<F>(out + 2 * F::N, one);
}
template <class F>
__device__ void xyzz_write_dev(const Xyzz<F>& p, int kind, uint32_t* __restrict__ out) {
  xyzz_write_out<F, false>(p, kind, out, fe_zero<F>());
}

// [k]P by the GLV endomorphism phi(x, y) = (beta x, y) = [lambda](x, y): k = k1 + k2 lambda
// mod r with |k1|, |k2| < 2^136, split on the host (glv_split). Record g: words 0-4 |k1|,
// words 5-9 |k2| (little-endian), word 10 bit 0 = (k1 < 0), bit 1 = (k2 < 0).
// Both halves use signed 4-bit windows (35 digits in -7..8, the top one the final carry) over
// one table 1P..8P; phi of an entry costs one product (beta X). 4 doublings per window.
__device__ __forceinline__ void glv_digits(const uint32_t* k, uint32_t (&dg)[5]) {   // 35 nibbles, d + 7
#pragma unroll
  for (int i = 0; i < 5; i++) dg[i] = 0;
  uint32_t carry = 0;
#pragma unroll
  for (int w = 0; w < 34; w++) {
    const uint32_t v = ((k[w >> 3] >> (4 * (w & 7))) & 15u) + carry;
    const int d = v > 8 ? (int)v - 16 : (int)v;
    carry = v > 8 ? 1u : 0u;
    dg[w >> 3] |= (uint32_t)(d + 7) << (4 * (w & 7));
  }
  dg[4] |= (carry + 7) << 8;   // window 34
}

template <class F>
__device__ Xyzz<F> xyzz_mul_glv(const uint32_t (&g)[12], const Xyzz<F>& P, const Fe<F>& beta) {
  uint32_t d1[5], d2[5];
  glv_digits(g, d1);
  glv_digits(g + 5, d2);
  const uint32_t s1 = g[10] & 1u, s2 = (g[10] >> 1) & 1u;
  Xyzz<F> T[8];
  T[0] = P;
  T[1] = xyzz_dbl(P);
  T[2] = xyzz_sum(T[1], T[0]);
  T[3] = xyzz_dbl(T[1]);
  T[4] = xyzz_sum(T[3], T[0]);
  T[5] = xyzz_dbl(T[2]);
  T[6] = xyzz_sum(T[5], T[0]);
  T[7] = xyzz_dbl(T[3]);
  Xyzz<F> acc = xyzz_inf<F>();
  bool started = false;
  for (int w = 34; w >= 0; w--) {
    if (started) {
      acc = xyzz_dbl(acc);
      acc = xyzz_dbl(acc);
      acc = xyzz_dbl(acc);
      acc = xyzz_dbl(acc);
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t* dg = h ? d2 : d1;
      const int d = (int)((dg[w >> 3] >> (4 * (w & 7))) & 15u) - 7;
      if (d != 0) {
        Xyzz<F> q = T[(d < 0 ? -d : d) - 1];
        if (h) q.X = fe_mul(q.X, beta);
        if ((d < 0) != ((h ? s2 : s1) != 0)) q.Y = fe_neg(q.Y);
        if (started) acc = xyzz_sum(acc, q);
        else { acc = q; started = true; }
      }
    }
  }
  return acc;
}

__device__ __forceinline__ void load_glv(const uint32_t* __restrict__ p, uint32_t (&g)[12]) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const uint4 x = __ldg(q + i);
    g[4 * i] = x.x; g[4 * i + 1] = x.y; g[4 * i + 2] = x.z; g[4 * i + 3] = x.w;
  }
}

__device__ __forceinline__ uint32_t bitrev_m(uint32_t i, int m) { return m == 0 ? 0u : (__brev(i) >> (32 - m)); }

// ------------------------------------------------------------------------ group FFT kernels
// Input point i (projective x = X/Z, y = Y/Z, or Jacobian x = X/Z^2, y = Y/Z^3; Z = 0 is the
// identity) to XYZZ at position bitrev(i) or i.
// (FP64 curve types: the coordinates are first brought into radix R' with kin = R'^2 / R.)
template <class C>
__global__ void k_g1fft_load(int m, int jac, int bitrev, const uint32_t* __restrict__ src, const Fe<typename C::Fp> kin,
                             uint32_t* __restrict__ a) {
  using F = typename C::Fp;
  const uint32_t n = 1u << m;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t* p = src + (size_t)i * 3 * F::N;
  Fe<F> X = fe_load<F>(p), Y = fe_load<F>(p + F::N), Z = fe_load<F>(p + 2 * F::N);
  if constexpr (F::DPF) {
    X = fe_mul(X, kin);
    Y = fe_mul(Y, kin);
    Z = fe_mul(Z, kin);
  }
  Xyzz<F> r;
  if (fe_is_zero(Z)) {
    r = xyzz_inf<F>();
  } else {
    const Fe<F> zz = fe_sqr(Z);
    r.ZZ = zz;
    r.ZZZ = fe_mul(zz, Z);
    if (jac) { r.X = X; r.Y = Y; }
    else { r.X = fe_mul(X, Z); r.Y = fe_mul(Y, zz); }
  }
  const uint32_t pos = bitrev ? bitrev_m(i, m) : i;
  xyzz_store<F>(a + (size_t)pos * 4 * F::N, r);
}

// One radix-2 stage over all N/2 butterflies. Forward (DIT): (u + [w]v, u - [w]v) with
// w = tw[j << (m - s)]. Inverse (DIF): (u + v, [w](u - v)) with w = tw[j << (m - s)]; at s = m
// with a scale table, (u + v) takes [scale] and (u - v) takes [top[j]]. Twiddles are GLV records
// (GLV_WORDS words each, see xyzz_mul_glv).
static constexpr int GLV_WORDS = 12;
template <class C, bool INV>
__global__ void k_g1fft_stage(int m, int s, const uint32_t* __restrict__ tw, const uint32_t* __restrict__ top,
                              const Fe<typename C::Fp> beta, uint32_t* __restrict__ a) {
  using F = typename C::Fp;
  constexpr int XW = 4 * F::N;
  const uint32_t nbf = 1u << (m - 1);
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nbf) return;
  const uint32_t h = 1u << (s - 1);
  const uint32_t j = t & (h - 1);
  const uint32_t i0 = ((t >> (s - 1)) << s) + j, i1 = i0 + h;
  const Xyzz<F> u = xyzz_load<F>(a + (size_t)i0 * XW);
  Xyzz<F> v = xyzz_load<F>(a + (size_t)i1 * XW);
  uint32_t k[GLV_WORDS];
  Xyzz<F> o0, o1;
  if (!INV) {
    if (j != 0) {
      load_glv(tw + (size_t)GLV_WORDS * (j << (m - s)), k);
      v = xyzz_mul_glv(k, v, beta);
    }
    o0 = xyzz_sum(u, v);
    o1 = xyzz_sum(u, xyzz_negate(v));
  } else {
    o0 = xyzz_sum(u, v);
    o1 = xyzz_sum(u, xyzz_negate(v));
    if (top != nullptr) {
      load_glv(top, k);                     // top[0] = 2^-m
      o0 = xyzz_mul_glv(k, o0, beta);
      load_glv(top + (size_t)GLV_WORDS * j, k);
      o1 = xyzz_mul_glv(k, o1, beta);
    } else if (j != 0) {
      load_glv(tw + (size_t)GLV_WORDS * (j << (m - s)), k);
      o1 = xyzz_mul_glv(k, o1, beta);
    }
  }
  xyzz_store<F>(a + (size_t)i0 * XW, o0);
  xyzz_store<F>(a + (size_t)i1 * XW, o1);
}

// The same stage by quads (zkb_quad.cuh), for transforms with too few butterflies to fill the GPU: a
// scalar multiplication is a chain of ~210 point operations, and at 2^14 points a thread a butterfly
// left one warp a scheduler (BN254 16.4 ms; this 11.8). A butterfly has HALVES quads: with 2, each
// multiplies by one half of the split scalar (quad 1 the image under phi) and the two results are
// added: the shortest chain, at 1.5 times the work; with 1, the quad takes both halves in one scan.
// The top stage of an inverse transform has two scalars and always two quads, one a scalar.
// Tables 1P..8P lie in shared memory, a column a thread (sm), with the images' X in one more (smb).
static constexpr int QUAD_T = 128;
template <class F>
__device__ __forceinline__ Fe<F> tab_ld(const uint32_t* sm, int e) {
  Fe<F> r;
#pragma unroll
  for (int i = 0; i < F::N; i++) r.v[i] = sm[(e * F::N + i) * QUAD_T + threadIdx.x];
  return r;
}
template <class F>
__device__ __forceinline__ void tab_st(uint32_t* sm, int e, const Fe<F>& a) {
#pragma unroll
  for (int i = 0; i < F::N; i++) sm[(e * F::N + i) * QUAD_T + threadIdx.x] = a.v[i];
}
// [k]P with the digits of `both` halves (dg, dg2), or of one half (dg); all lanes call it
template <class F>
__device__ __noinline__ Fe<F> quad_mul_glv(const Fe<F> P, const uint32_t (&k)[GLV_WORDS], bool both, int half,
                                           const Fe<F> beta, uint32_t* sm, uint32_t* smb) {
  const int L = quad_lane();
  uint32_t d1[5], d2[5];
  glv_digits(half ? k + 5 : k, d1);
  glv_digits(k + 5, d2);
  const uint32_t s1 = (k[10] >> half) & 1u, s2 = (k[10] >> 1) & 1u;
  Fe<F> t = P;
  tab_st(sm, 0, t);
#pragma unroll 1
  for (int e = 2; e <= 8; e++) {   // 2P by doubling, then + P
    t = e == 2 ? quad_dbl(t) : quad_add(t, P);
    tab_st(sm, e - 1, t);
  }
  if (__any_sync(FULL, both)) {
#pragma unroll 1
    for (int e = 0; e < 8; e++) {
      const Fe<F> b = fe_mul(tab_ld<F>(sm, e), beta);
      if (L == 0)
#pragma unroll
        for (int i = 0; i < F::N; i++) smb[(e * F::N + i) * (QUAD_T / 4) + (threadIdx.x >> 2)] = b.v[i];
    }
  }
  auto digit = [](const uint32_t (&dg)[5], int w) {
    uint32_t v = 0;
#pragma unroll
    for (int i = 0; i < 5; i++)
      if (i == (w >> 3)) v = dg[i];
    return (int)((v >> (4 * (w & 7))) & 15u) - 7;
  };
  Fe<F> acc = fe_zero<F>();
#pragma unroll 1
  for (int w = 34; w >= 0; w--) {
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
      if (h == 1 && !__any_sync(FULL, both)) break;
      const int d = h == 0 ? digit(d1, w) : both ? digit(d2, w) : 0;
      const int e = (d < 0 ? -d : d) - 1;
      Fe<F> q = fe_zero<F>();
      if (d != 0) {
        q = tab_ld<F>(sm, e);
        if (h == 1 && L == 0)
#pragma unroll
          for (int i = 0; i < F::N; i++) q.v[i] = smb[(e * F::N + i) * (QUAD_T / 4) + (threadIdx.x >> 2)];
        if (L == 1 && (d < 0) != ((h ? s2 : s1) != 0)) q = fe_neg(q);
      }
      if constexpr (F::DPF) {
        acc = h == 0 ? quad_window(acc, q) : quad_add(acc, q);   // the first window finds the identity
      } else {
        if (h == 0 && w != 34)
#pragma unroll 1
          for (int i = 0; i < 4; i++) acc = quad_dbl(acc);
        acc = quad_add(acc, q);
      }
    }
  }
  return acc;
}

template <class C, bool INV, int HALVES>
__global__ void __launch_bounds__(QUAD_T) k_g1fft_stage_quad(int m, int s, const uint32_t* __restrict__ tw,
                                                             const uint32_t* __restrict__ top,
                                                             const Fe<typename C::Fp> beta, uint32_t* __restrict__ a) {
  using F = typename C::Fp;
  constexpr int XW = 4 * F::N;
  extern __shared__ uint4 smem_u4[];
  uint32_t* sm = reinterpret_cast<uint32_t*>(smem_u4);
  uint32_t* smb = sm + 8 * F::N * QUAD_T;
  const uint32_t nbf = 1u << (m - 1);
  const uint32_t quad = (blockIdx.x * QUAD_T + threadIdx.x) >> 2;
  const uint32_t t = quad / HALVES, sub = quad % HALVES;
  const bool live = t < nbf;
  const int L = quad_lane();
  const uint32_t h = 1u << (s - 1), j = live ? t & (h - 1) : 0;
  const uint32_t i0 = ((t >> (s - 1)) << s) + j, i1 = i0 + h;
  Fe<F> u = fe_zero<F>(), v = fe_zero<F>();
  if (live) {
    u = quad_load<F>(a + (size_t)i0 * XW);
    v = quad_load<F>(a + (size_t)i1 * XW);
  }
  const bool two = INV && top != nullptr;   // two scalars: quad `sub` has its own
  uint32_t k[GLV_WORDS];
  load_glv(two ? top + (size_t)GLV_WORDS * (sub ? j : 0) : tw + (size_t)GLV_WORDS * (j << (m - s)), k);
  auto neg = [&](const Fe<F>& x) { return L == 1 ? fe_neg(x) : x; };
  // [k]x in every quad of the butterfly (its own scalar with `two`)
  auto mul = [&](const Fe<F>& x) {
    const bool mine = two || j != 0;
    if (!__any_sync(FULL, mine)) return x;
    if (HALVES == 1 || two) return fe_sel(mine, quad_mul_glv(x, k, true, 0, beta, sm, smb), x);
    const Fe<F> bx = fe_mul(x, beta);
    Fe<F> r = quad_mul_glv(fe_sel(sub == 1 && L == 0, bx, x), k, false, (int)sub, beta, sm, smb);
    r = quad_add(r, fe_shfl_xor(r, 4));
    return fe_sel(mine, r, x);
  };
  if (!INV) {
    const Fe<F> r = mul(v);
    if (HALVES == 2) {
      const Fe<F> o = quad_add(u, sub ? neg(r) : r);
      if (live) quad_store(a + (size_t)(sub ? i1 : i0) * XW, o);
    } else {
      const Fe<F> o0 = quad_add(u, r), o1 = quad_add(u, neg(r));
      if (live) {
        quad_store(a + (size_t)i0 * XW, o0);
        quad_store(a + (size_t)i1 * XW, o1);
      }
    }
  } else if (HALVES == 2) {
    Fe<F> o = quad_add(u, sub ? neg(v) : v);
    if (two) {
      o = mul(o);
    } else {
      const Fe<F> d = fe_shfl(o, (threadIdx.x & 31) | 4);   // u - v, for both quads
      const Fe<F> r = mul(d);
      if (sub) o = r;
    }
    if (live) quad_store(a + (size_t)(sub ? i1 : i0) * XW, o);
  } else {
    const Fe<F> o0 = quad_add(u, v), o1 = mul(quad_add(u, neg(v)));
    if (live) {
      quad_store(a + (size_t)i0 * XW, o0);
      quad_store(a + (size_t)i1 * XW, o1);
    }
  }
}

// out[i] = normalised a[bitrev(i)] (or a[i])
template <class C>
__global__ void k_g1fft_store(int m, int bitrev, const uint32_t* __restrict__ a, const Fe<typename C::Fp> kout,
                              uint32_t* __restrict__ out) {
  using F = typename C::Fp;
  const uint32_t n = 1u << m;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t pos = bitrev ? bitrev_m(i, m) : i;
  xyzz_write_out<F, F::DPF>(xyzz_load<F>(a + (size_t)pos * 4 * F::N), ZKG_OUT_PROJ, out + (size_t)i * 3 * F::N, kout);
}

// ------------------------------------------------------------------------ binary MSM kernels
template <class C>
__global__ void k_xyzz_write(int n, int kind, const uint32_t* __restrict__ in, uint32_t* __restrict__ out) {
  using F = typename C::Fp;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int ow = (kind == ZKG_OUT_AFFINE ? 2 : 3) * F::N;
  xyzz_write_dev<F>(xyzz_load<F>(in + (size_t)i * 4 * F::N), kind, out + (size_t)i * ow);
}

// ------------------------------------------------------------------------ group FFT host side
template <class F>
static Fe<F> fe_zero_host() {
  Fe<F> r;
  for (int i = 0; i < F::N; i++) r.v[i] = 0;
  return r;
}
static inline size_t rup256(size_t x) { return (x + 255) & ~size_t(255); }

// GLV decomposition for phi(x, y) = (beta x, y) = [lambda](x, y) on G1. Lattice basis
// v1 = (a1, b1), v2 = (a2, b2) with a + b lambda = 0 mod r (extended Euclid on (r, lambda),
// det = r), b1 < 0 stored as mb1 = -b1. For k < r: c1 = floor(k G1 / 2^384), c2 = floor(k G2 / 2^384)
// with G1 = round(2^384 b2 / r), G2 = round(2^384 (-b1) / r) approximate the rounded lattice
// coordinates; k1 = k - c1 a1 - c2 a2, k2 = c1 mb1 - c2 b2 satisfy k1 + k2 lambda = k (mod r)
// for any c1, c2, and with these c1, c2 |k1|, |k2| < 2^130. beta is the cube root of unity in
// Fp paired with lambda (checked against the generator when the constants were derived).
struct GlvConst {
  uint64_t a1[2], mb1[2], a2[2], b2[2], G1[5], G2[5];
  uint64_t beta_std[6];
};
static const GlvConst GLV_BN254 = {
    {0x8211bbeb7d4f1128ULL, 0x6f4d8248eeb859fcULL}, {0x89d3256894d213e3ULL, 0},
    {0x89d3256894d213e3ULL, 0}, {0x0be4e1541221250bULL, 0x6f4d8248eeb859fdULL},
    {0x163b4843cb4b9a5fULL, 0x149d540fd5e495ccULL, 0x5398fd0300ff6565ULL, 0x4ccef014a773d2d2ULL, 0x2ULL},
    {0x8fa7d32d2fafba64ULL, 0x6eb9c714773a6ef2ULL, 0xd91d232ec7e0b3d7ULL, 0x2ULL, 0},
    {0xe4bd44e5607cfd48ULL, 0xc28f069fbb966e3dULL, 0x5e6dd9e7e0acccb0ULL, 0x30644e72e131a029ULL, 0, 0}};
static const GlvConst GLV_BLS12_381 = {
    {0x1ULL, 0}, {0x00000000ffffffffULL, 0xac45a4010001a402ULL},
    {0x0000000100000000ULL, 0xac45a4010001a402ULL}, {0x1ULL, 0},
    {0x38b5dcb707e08ed3ULL, 0x355094edfede377cULL, 0x2ULL, 0, 0},
    {0xa1a872d6818be407ULL, 0x034eb4b927adc027ULL, 0x63f6e522f6cfee2eULL, 0x7c6becf1e01faaddULL, 0x1ULL},
    {0x2e01fffffffefffeULL, 0xde17d813620a0002ULL, 0xddb3a93be6f89688ULL, 0xba69c6076a0f77eaULL,
     0x5f19672fdf76ce51ULL, 0}};

// floor(k * G / 2^384) for k < 2^256 (4 limbs), G 5 limbs; the result has at most 2 limbs here
static void glv_coord(const uint64_t k[4], const uint64_t G[5], uint64_t c[2]) {
  uint64_t prod[9] = {0};
  for (int i = 0; i < 4; i++) {
    unsigned __int128 carry = 0;
    for (int j = 0; j < 5; j++) {
      const unsigned __int128 t = (unsigned __int128)k[i] * G[j] + prod[i + j] + carry;
      prod[i + j] = (uint64_t)t;
      carry = t >> 64;
    }
    prod[i + 5] = (uint64_t)carry;
  }
  c[0] = prod[6];
  c[1] = prod[7];
}
// (x * y) mod 2^192 for 2-limb x, y
static void mul_mod192(const uint64_t x[2], const uint64_t y[2], uint64_t r[3]) {
  const unsigned __int128 p00 = (unsigned __int128)x[0] * y[0];
  const unsigned __int128 p01 = (unsigned __int128)x[0] * y[1];
  const unsigned __int128 p10 = (unsigned __int128)x[1] * y[0];
  const unsigned __int128 p11 = (unsigned __int128)x[1] * y[1];
  r[0] = (uint64_t)p00;
  const unsigned __int128 mid = (p00 >> 64) + (uint64_t)p01 + (uint64_t)p10;
  r[1] = (uint64_t)mid;
  r[2] = (uint64_t)(mid >> 64) + (uint64_t)(p01 >> 64) + (uint64_t)(p10 >> 64) + (uint64_t)p11;
}
static void sub192(uint64_t a[3], const uint64_t b[3]) {
  unsigned __int128 borrow = 0;
  for (int i = 0; i < 3; i++) {
    const unsigned __int128 t = (unsigned __int128)a[i] - b[i] - borrow;
    a[i] = (uint64_t)t;
    borrow = (t >> 64) ? 1 : 0;
  }
}
// signed 192-bit value -> sign and magnitude; false if the magnitude needs more than 136 bits
static bool sign_mag(uint64_t v[3], uint32_t& neg) {
  neg = (uint32_t)(v[2] >> 63);
  if (neg) {
    uint64_t z[3] = {0, 0, 0};
    sub192(z, v);
    v[0] = z[0]; v[1] = z[1]; v[2] = z[2];
  }
  return v[2] < (1ULL << 8);
}
// k (standard integer < r, 4 limbs) -> GLV record (GLV_WORDS 32-bit words, see xyzz_mul_glv)
static bool glv_split(const GlvConst& G, const uint64_t k[4], uint32_t out[12]) {
  uint64_t c1[2], c2[2], t[3];
  glv_coord(k, G.G1, c1);
  glv_coord(k, G.G2, c2);
  uint64_t k1[3] = {k[0], k[1], k[2]};
  mul_mod192(c1, G.a1, t);
  sub192(k1, t);
  mul_mod192(c2, G.a2, t);
  sub192(k1, t);
  uint64_t k2[3];
  mul_mod192(c1, G.mb1, k2);
  mul_mod192(c2, G.b2, t);
  sub192(k2, t);
  uint32_t n1 = 0, n2 = 0;
  if (!sign_mag(k1, n1) || !sign_mag(k2, n2)) return false;
  for (int i = 0; i < 5; i++) {
    out[i] = (uint32_t)(k1[i >> 1] >> (32 * (i & 1)));
    out[5 + i] = (uint32_t)(k2[i >> 1] >> (32 * (i & 1)));
  }
  out[10] = n1 | (n2 << 1);
  out[11] = 0;
  return true;
}

// Largest transforms by quads, and with two quads a butterfly.
static constexpr int QUAD_MMAX = 14, QUAD_MHALVES = 13;
template <class CP, int HALVES>
static zkg_status launch_stage_quad(int inverse, int m, int s, const uint32_t* tw, const uint32_t* top,
                                    const Fe<typename CP::Fp>& beta, uint32_t* a, cudaStream_t st) {
  constexpr size_t smem = 8 * CP::Fp::N * (QUAD_T + QUAD_T / 4) * 4;
  const size_t quads = ((size_t)1 << (m - 1)) * HALVES;
  auto k = inverse ? k_g1fft_stage_quad<CP, true, HALVES> : k_g1fft_stage_quad<CP, false, HALVES>;
  return launch("g1fft_stage", k, dim3((unsigned)((quads * 4 + QUAD_T - 1) / QUAD_T)), dim3(QUAD_T), smem, st, m, s, tw,
                top, beta, a);
}

// CP: the curve type the point arithmetic runs on (C, or its FP64-product twin, zkb_dpf.cuh)
template <class CP, class C, int NL>
static zkg_status g1_fft_run(Context& cx, int jac, int m, const uint64_t* gen, const uint32_t* d_src,
                             uint32_t* d_out, int inverse, cudaStream_t st) {
  const host::Field<4>& Fr = (C::ID == 0) ? host::BN_FR : host::BLS_FR;
  const size_t n = (size_t)1 << m, half = n >> 1;
  const size_t xb = 4 * NL * 8;
  // twiddles (standard form): tw[e] = g^e for e < N/2, g = gen (forward) or gen^-1 (inverse);
  // top[j] = 2^-m gen^-j (inverse only)
  using host::El;
  El<4> g, one_std = host::zero<4>();
  one_std.v[0] = 1;
  std::memcpy(g.v, gen, 32);
  if (inverse) g = host::inv(Fr, g);
  El<4> two_std = host::zero<4>();
  two_std.v[0] = 2;
  El<4> sc = host::one(Fr);
  if (inverse) {
    const El<4> ihalf = host::inv(Fr, host::from_std(Fr, two_std));
    for (int i = 0; i < m; i++) sc = host::mul(Fr, sc, ihalf);
  }
  const size_t ntw = std::max<size_t>(half, 1);
  const GlvConst& GC = (C::ID == 0) ? GLV_BN254 : GLV_BLS12_381;
  std::vector<uint32_t> tw((size_t)GLV_WORDS * ntw * (inverse ? 2 : 1), 0);
  El<4> pw = host::one(Fr);
  for (size_t e = 0; e < half; e++) {
    const El<4> s0 = host::mul(Fr, pw, one_std);
    if (!glv_split(GC, s0.v, &tw[(size_t)GLV_WORDS * e])) return set_status(ZKG_ERR_ARG, "g1_fft", "GLV split");
    if (inverse) {
      const El<4> s1 = host::mul(Fr, host::mul(Fr, pw, sc), one_std);
      if (!glv_split(GC, s1.v, &tw[(size_t)GLV_WORDS * (ntw + e)])) return set_status(ZKG_ERR_ARG, "g1_fft", "GLV split");
    }
    pw = host::mul(Fr, pw, g);
  }
  // beta in the Montgomery radix of the point arithmetic (R, or R' for the FP64 types:
  // beta R' = mont(beta R, R' mod p))
  using F = typename CP::Fp;
  Fe<F> beta, kin = fe_zero_host<F>(), kout = fe_zero_host<F>();
  {
    const host::Field<NL>* fp;
    if constexpr (NL == 4) fp = &host::BN_FP;
    else fp = &host::BLS_FP;
    const host::Field<NL>& Fp = *fp;
    El<NL> b;
    std::memcpy(b.v, GC.beta_std, 8 * NL);
    El<NL> bm = host::from_std(Fp, b);
    if constexpr (F::DPF) {
      El<NL> rp = host::zero<NL>();
      for (int w = 0; w < F::N; w++) rp.v[w >> 1] |= (uint64_t)F::one(w) << (32 * (w & 1));
      bm = host::mul(Fp, bm, rp);
      dpf_consts_for<CP>(kin, kout);
    }
    for (int w = 0; w < F::N; w++) beta.v[w] = (uint32_t)(bm.v[w >> 1] >> (32 * (w & 1)));
  }
  const size_t bytes = rup256(n * xb) + rup256(tw.size() * 4);
  ZKB_TRY(cx.arena.reserve(bytes));
  cx.arena.reset();
  uint32_t* a = static_cast<uint32_t*>(cx.arena.take(n * xb));
  uint32_t* d_tw = static_cast<uint32_t*>(cx.arena.take(tw.size() * 4));
  if (!a || !d_tw) return set_status(ZKG_ERR_NOMEM, "g1_fft", "arena");
  ZKB_CUDA(cudaMemcpyAsync(d_tw, tw.data(), tw.size() * 4, cudaMemcpyHostToDevice, st));
  const dim3 blk(128);
  const dim3 grid_n((unsigned)((n + 127) / 128));
  ZKB_TRY(launch("g1fft_load", k_g1fft_load<CP>, grid_n, blk, 0, st, m, jac, inverse ? 0 : 1, d_src, kin, a));
  const dim3 grid_h((unsigned)((half + 127) / 128));
  const uint32_t* d_top = d_tw + (size_t)GLV_WORDS * ntw;
  if (m >= 1 && m <= QUAD_MMAX) {
    for (int k = 0; k < m; k++) {
      const int s = inverse ? m - k : k + 1;
      const bool two = inverse && k == 0;
      if (m <= QUAD_MHALVES || two)
        ZKB_TRY((launch_stage_quad<CP, 2>(inverse, m, s, d_tw, two ? d_top : nullptr, beta, a, st)));
      else
        ZKB_TRY((launch_stage_quad<CP, 1>(inverse, m, s, d_tw, nullptr, beta, a, st)));
    }
  } else if (!inverse) {
    for (int s = 1; s <= m; s++)
      ZKB_TRY(launch("g1fft_stage", k_g1fft_stage<CP, false>, grid_h, blk, 0, st, m, s, (const uint32_t*)d_tw,
                     (const uint32_t*)nullptr, beta, a));
  } else {
    for (int s = m; s >= 1; s--)
      ZKB_TRY(launch("g1fft_stage", k_g1fft_stage<CP, true>, grid_h, blk, 0, st, m, s, (const uint32_t*)d_tw,
                     s == m ? d_top : (const uint32_t*)nullptr, beta, a));
  }
  ZKB_TRY(launch("g1fft_store", k_g1fft_store<CP>, grid_n, blk, 0, st, m, inverse ? 1 : 0, (const uint32_t*)a, kout,
                 d_out));
  return ZKG_OK;
}

// BN254 point arithmetic with FP64-pipe products unless ZKB_G1_DPF=0 (BLS12-381 stays on the
// integer pipes: its 8-limb FP64 product made these kernels slower, 55.0 vs 43.3 ms at 2^14)
static const bool g_g1_dpf = [] {
  const char* v = std::getenv("ZKB_G1_DPF");
  return v ? std::atoi(v) != 0 : true;
}();

template <class C, int NL>
static zkg_status g1_fft_launch(Context& cx, int jac, int m, const uint64_t* gen, const uint32_t* d_src,
                                uint32_t* d_out, int inverse, cudaStream_t st) {
  if constexpr (C::ID == 0) {
    if (g_g1_dpf) return g1_fft_run<typename DpfCurve<C>::type, C, NL>(cx, jac, m, gen, d_src, d_out, inverse, st);
  }
  return g1_fft_run<C, C, NL>(cx, jac, m, gen, d_src, d_out, inverse, st);
}

static zkg_status g1_fft_check(zkg_curve curve, int m, const void* gen, const void* src, const void* tgt) {
  if (curve != ZKG_BN254 && curve != ZKG_BLS12_381) return set_status(ZKG_ERR_ARG, "g1_fft", "unknown curve");
  if (m < 0 || m > 26) return set_status(ZKG_ERR_ARG, "g1_fft", "m out of range [0, 26]");
  if (!gen || !src || !tgt) return set_status(ZKG_ERR_ARG, "g1_fft", "null pointer");
  return ZKG_OK;
}

template <class C, int NL>
static zkg_status g1_fft_host(int jac, int m, const uint64_t* gen, const uint64_t* src, uint64_t* tgt, int inverse) {
  Context* cxp = nullptr;
  ZKB_TRY(get_context(&cxp));
  Context& cx = *cxp;
  std::lock_guard<std::mutex> lk(cx.mu);
  const size_t n = (size_t)1 << m, pb = 3 * NL * 8;
  uint32_t* d_io = nullptr;
  ZKB_CUDA(cudaMalloc(&d_io, n * pb));
  const cudaStream_t st = cx.compute();
  zkg_status rc = ZKG_OK;
  rc = copy_h2d(cx, d_io, src, n * pb, st);
  if (rc == ZKG_OK) rc = g1_fft_launch<C, NL>(cx, jac, m, gen, d_io, d_io, inverse, st);
  if (rc == ZKG_OK) rc = copy_d2h(cx, tgt, d_io, n * pb, st);
  if (rc == ZKG_OK && cudaStreamSynchronize(st) != cudaSuccess) rc = set_status(ZKG_ERR_CUDA, "g1_fft", "sync");
  cudaFree(d_io);
  return rc == ZKG_OK ? set_status(ZKG_OK, nullptr, nullptr) : rc;
}

template <class C, int NL>
static zkg_status g1_fft_dev(int jac, int m, const uint64_t* gen, const uint64_t* d_src, uint64_t* d_tgt, int inverse) {
  if ((reinterpret_cast<uintptr_t>(d_src) | reinterpret_cast<uintptr_t>(d_tgt)) & 15)
    return set_status(ZKG_ERR_ARG, "g1_fft_device", "device buffers must be 16-byte aligned");
  Context* cxp = nullptr;
  ZKB_TRY(get_context(&cxp));
  Context& cx = *cxp;
  std::lock_guard<std::mutex> lk(cx.mu);
  if (!cx.user_stream) ZKB_CUDA(cudaDeviceSynchronize());
  const cudaStream_t st = cx.compute();
  ZKB_TRY((g1_fft_launch<C, NL>(cx, jac, m, gen, reinterpret_cast<const uint32_t*>(d_src),
                                reinterpret_cast<uint32_t*>(d_tgt), inverse, st)));
  ZKB_CUDA(cudaStreamSynchronize(st));
  return set_status(ZKG_OK, nullptr, nullptr);
}

// ------------------------------------------------------------------------ binary MSM host side
struct BinPlan {
  int rho = 1;            // rows a group
  int batch = 0;          // rows a launch
  int cw = 0;             // columns a launch
  int nbatch = 0, nchunk = 0;
  size_t bits_bytes = 0;  // workspace of the launches: the largest any of them needs
  int rows(int r, int nrows) const { return std::min(batch, nrows - r * batch); }
  int cols(int q, int npoints) const { return std::min(cw, npoints - q * cw); }
};
static constexpr int BIN_ROWS_MIN = 1024, BIN_ROWS = 32768;   // rows a launch (grid dimensions)
static constexpr size_t BIN_ENTRIES = (size_t)1 << 26;        // entries a launch: a column has one a group of rows
static constexpr size_t BIN_STAGE = (size_t)32 << 20;         // staged coefficients, and bases, a launch

// A launch costs about 10 field products an entry and 8 2^rho a row, however few columns it has, so what
// is asked for is many columns first: rows go in batches such that a batch can have all the columns, if
// that leaves 1024 rows. (All rows at once left host calls 8192 columns a launch at 4096 rows, at a rho
// chosen for 2^20 of them: 5 times the products.) rho is chosen for the columns that a launch has.
static zkg_status bin_plan(int nrows, int npoints, int nl, bool host, BinPlan& P) {
  const zkg_curve curve = nl == 4 ? ZKG_BN254 : ZKG_BLS12_381;
  P.rho = msm_bits_group(nrows, npoints);
  size_t rows = BIN_ENTRIES * P.rho / npoints;
  if (host) rows = std::min(rows, BIN_STAGE / npoints);
  rows = std::min<size_t>(nrows, std::min<size_t>(std::max<size_t>(rows, BIN_ROWS_MIN), BIN_ROWS));
  P.nbatch = (int)((nrows + rows - 1) / rows);
  P.batch = (nrows + P.nbatch - 1) / P.nbatch;
  for (int round = 0; round < 4; round++) {
    size_t cw = std::min<size_t>(npoints, BIN_ENTRIES / ((P.batch + P.rho - 1) / P.rho));
    if (host) cw = std::min(cw, std::min(BIN_STAGE / P.batch, BIN_STAGE / (2 * (size_t)nl * 8)));
    P.nchunk = (int)((npoints + cw - 1) / cw);
    P.cw = (npoints + P.nchunk - 1) / P.nchunk;
    const int rho = msm_bits_group(P.batch, P.cw);
    if (rho == P.rho) break;
    P.rho = rho;
  }
  P.nbatch = (nrows + P.batch - 1) / P.batch;   // rounding up may have made the last ones empty
  P.nchunk = (npoints + P.cw - 1) / P.cw;
  // A launch's workspace does not grow steadily with its size (a little fewer entries can make shorter and
  // so more chunks), so the last rows and the last columns are asked for as well.
  P.bits_bytes = 0;
  for (const int r : {0, P.nbatch - 1})
    for (const int q : {0, P.nchunk - 1}) {
      size_t b = 0;
      ZKB_TRY(msm_bits_bytes(curve, P.rows(r, nrows), P.cols(q, npoints), P.rho, &b));
      P.bits_bytes = std::max(P.bits_bytes, b);
    }
  return ZKG_OK;
}

// Runs the launches: for each batch of rows the column chunks, whose sums add up in the rows' points.
// get_tile(t, row0, rows, col0, cols, &coeffs, &ld, &bases) makes launch t's coefficient rows (ld bytes
// apart) and bases available to the compute stream; done_tile(t) follows its kernels.
template <class C, int NL, class Get, class Done>
static zkg_status bin_run(Context& cx, const BinPlan& P, int nrows, int npoints, char* ws, cudaStream_t st,
                          Get get_tile, Done done_tile, int kind, uint32_t* d_out) {
  constexpr size_t XW = 4 * C::Fp::N;
  uint32_t* sums = reinterpret_cast<uint32_t*>(ws);
  char* work = ws + rup256((size_t)nrows * XW * 4);
  int t = 0;
  for (int r = 0; r < P.nbatch; r++)
    for (int q = 0; q < P.nchunk; q++, t++) {
      const int rows = P.rows(r, nrows), cols = P.cols(q, npoints), row0 = r * P.batch;
      const uint8_t* coeffs = nullptr;
      size_t ld = 0;
      const uint32_t* bases = nullptr;
      ZKB_TRY(get_tile(t, row0, rows, q * P.cw, cols, &coeffs, &ld, &bases));
      ZKB_TRY(msm_bits_launch(cx, C::ID == 0 ? ZKG_BN254 : ZKG_BLS12_381, rows, cols, P.rho, coeffs, ld, bases, work,
                              P.bits_bytes, sums + row0 * XW, q > 0, st));
      ZKB_TRY(done_tile(t));
    }
  return launch("xyzz_write", k_xyzz_write<C>, dim3((unsigned)((nrows + 31) / 32)), dim3(32), 0, st, nrows, kind,
                (const uint32_t*)sums, d_out);
}

template <int NL>
static size_t bin_ws_bytes(const BinPlan& P, int nrows) {
  return rup256((size_t)nrows * 4 * NL * 8) + rup256(P.bits_bytes);
}

static zkg_status bin_check(zkg_curve curve, int kind, int nrows, int npoints, const void* rows, const void* bases,
                            const void* out) {
  if (curve != ZKG_BN254 && curve != ZKG_BLS12_381) return set_status(ZKG_ERR_ARG, "msm_binary", "unknown curve");
  if (kind < ZKG_OUT_PROJ || kind > ZKG_OUT_AFFINE) return set_status(ZKG_ERR_ARG, "msm_binary", "bad output kind");
  if (nrows < 0 || npoints < 0) return set_status(ZKG_ERR_ARG, "msm_binary", "negative size");
  if (nrows > 0 && (!out || (npoints > 0 && (!rows || !bases))))
    return set_status(ZKG_ERR_ARG, "msm_binary", "null pointer");
  return ZKG_OK;
}

template <class C, int NL>
static zkg_status bin_host(const host::Field<NL>& Fp, int kind, int nrows, int npoints, const uint8_t* const* rows,
                           const uint64_t* grps, uint64_t* tgt) {
  const int ow = (kind == ZKG_OUT_AFFINE ? 2 : 3) * NL;
  if (nrows == 0) return set_status(ZKG_OK, nullptr, nullptr);
  if (npoints == 0) {
    for (int r = 0; r < nrows; r++) host::xyzz_write<NL>(Fp, host::xyzz_inf<NL>(), kind, tgt + (size_t)r * ow);
    return set_status(ZKG_OK, nullptr, nullptr);
  }
  for (int r = 0; r < nrows; r++)
    if (!rows[r]) return set_status(ZKG_ERR_ARG, "msm_binary", "null coefficient row");
  Context* cxp = nullptr;
  ZKB_TRY(get_context(&cxp));
  Context& cx = *cxp;
  std::lock_guard<std::mutex> lk(cx.mu);
  BinPlan P;
  ZKB_TRY(bin_plan(nrows, npoints, NL, true, P));
  const size_t bb = 2 * NL * 8;
  const size_t coef_chunk = rup256((size_t)P.batch * P.cw), base_chunk = rup256((size_t)P.cw * bb);
  const size_t out_bytes = rup256((size_t)nrows * ow * 8);
  const size_t stage = coef_chunk + base_chunk;   // one pinned / device staging slot
  const size_t bytes = 2 * stage + out_bytes + bin_ws_bytes<NL>(P, nrows);
  ZKB_TRY(cx.arena.reserve(bytes));
  cx.arena.reset();
  char* dstage = static_cast<char*>(cx.arena.take(2 * stage));
  uint32_t* d_out = static_cast<uint32_t*>(cx.arena.take(out_bytes));
  char* ws = static_cast<char*>(cx.arena.take(bytes - 2 * stage - out_bytes));
  if (!dstage || !d_out || !ws) return set_status(ZKG_ERR_NOMEM, "msm_binary", "arena");
  ZKB_TRY(pinned_reserve(cx, std::max(2 * stage, out_bytes)));
  char* pin = static_cast<char*>(cx.pinned);
  const cudaStream_t st = cx.compute();
  cudaEvent_t ev_copied[2] = {nullptr, nullptr}, ev_used[2] = {nullptr, nullptr};
  for (int b = 0; b < 2; b++) {
    ZKB_CUDA(cudaEventCreateWithFlags(&ev_copied[b], cudaEventDisableTiming));
    ZKB_CUDA(cudaEventCreateWithFlags(&ev_used[b], cudaEventDisableTiming));
  }
  // earlier work on the compute stream may still use the arena
  ZKB_CUDA(cudaEventRecord(ev_used[0], st));
  ZKB_CUDA(cudaEventRecord(ev_used[1], st));
  bool pending[2] = {false, false};
  auto get_tile = [&](int t, int row0, int rws, int col0, int cols, const uint8_t** coeffs, size_t* ld,
                      const uint32_t** bases) -> zkg_status {
    const int b = t & 1;
    char* hp = pin + b * stage;
    char* dp = dstage + b * stage;
    if (pending[b]) ZKB_CUDA(cudaEventSynchronize(ev_copied[b]));   // pinned slot b is free again
    for (int r = 0; r < rws; r++) std::memcpy(hp + (size_t)r * P.cw, rows[row0 + r] + col0, (size_t)cols);
    std::memcpy(hp + coef_chunk, grps + (size_t)col0 * 2 * NL, (size_t)cols * bb);
    ZKB_CUDA(cudaStreamWaitEvent(cx.copy_stream, ev_used[b], 0));
    ZKB_CUDA(cudaMemcpyAsync(dp, hp, coef_chunk + (size_t)cols * bb, cudaMemcpyHostToDevice, cx.copy_stream));
    ZKB_CUDA(cudaEventRecord(ev_copied[b], cx.copy_stream));
    pending[b] = true;
    ZKB_CUDA(cudaStreamWaitEvent(st, ev_copied[b], 0));
    *coeffs = reinterpret_cast<const uint8_t*>(dp);
    *ld = (size_t)P.cw;
    *bases = reinterpret_cast<const uint32_t*>(dp + coef_chunk);
    return ZKG_OK;
  };
  auto done_tile = [&](int t) -> zkg_status {   // launch t's inputs are consumed by the kernels just queued
    ZKB_CUDA(cudaEventRecord(ev_used[t & 1], st));
    return ZKG_OK;
  };
  zkg_status rc = bin_run<C, NL>(cx, P, nrows, npoints, ws, st, get_tile, done_tile, kind, d_out);
  if (rc == ZKG_OK) {
    // the pinned slots may still feed a copy; wait for all of them before reusing pinned memory
    if (cudaStreamSynchronize(cx.copy_stream) != cudaSuccess) rc = set_status(ZKG_ERR_CUDA, "msm_binary", "copy sync");
  }
  if (rc == ZKG_OK && cudaMemcpyAsync(pin, d_out, (size_t)nrows * ow * 8, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    rc = set_status(ZKG_ERR_CUDA, "msm_binary", "output copy");
  if (rc == ZKG_OK && cudaStreamSynchronize(st) != cudaSuccess) rc = set_status(ZKG_ERR_CUDA, "msm_binary", "sync");
  if (rc == ZKG_OK) rc = dev_check_report(cx, "msm_binary");
  if (rc == ZKG_OK) std::memcpy(tgt, pin, (size_t)nrows * ow * 8);
  if (rc != ZKG_OK) {
    cudaStreamSynchronize(cx.copy_stream);
    cudaStreamSynchronize(st);
  }
  for (int b = 0; b < 2; b++) {
    cudaEventDestroy(ev_copied[b]);
    cudaEventDestroy(ev_used[b]);
  }
  return rc == ZKG_OK ? set_status(ZKG_OK, nullptr, nullptr) : rc;
}

template <class C, int NL>
static zkg_status bin_dev(int kind, int nrows, int npoints, const uint8_t* d_coeffs, size_t ld, const uint64_t* d_bases,
                          uint64_t* d_out) {
  if (nrows == 0) return set_status(ZKG_OK, nullptr, nullptr);
  if (npoints > 0 && ld < (size_t)npoints) return set_status(ZKG_ERR_ARG, "msm_binary_device", "ld < npoints");
  if ((reinterpret_cast<uintptr_t>(d_bases) | reinterpret_cast<uintptr_t>(d_out)) & 15)
    return set_status(ZKG_ERR_ARG, "msm_binary_device", "device buffers must be 16-byte aligned");
  Context* cxp = nullptr;
  ZKB_TRY(get_context(&cxp));
  Context& cx = *cxp;
  std::lock_guard<std::mutex> lk(cx.mu);
  if (!cx.user_stream) ZKB_CUDA(cudaDeviceSynchronize());
  const cudaStream_t st = cx.compute();
  const dim3 blk(128);
  if (npoints == 0) {
    // every row is the identity: write it through the same conversion kernel
    const size_t xb = 4 * NL * 8;
    ZKB_TRY(cx.arena.reserve((size_t)nrows * xb));
    cx.arena.reset();
    uint32_t* z = static_cast<uint32_t*>(cx.arena.take((size_t)nrows * xb));
    if (!z) return set_status(ZKG_ERR_NOMEM, "msm_binary_device", "arena");
    ZKB_CUDA(cudaMemsetAsync(z, 0, (size_t)nrows * xb, st));
    ZKB_TRY(launch("xyzz_write", k_xyzz_write<C>, dim3((unsigned)((nrows + 127) / 128)), blk, 0, st, nrows, kind,
                   (const uint32_t*)z, reinterpret_cast<uint32_t*>(d_out)));
    ZKB_CUDA(cudaStreamSynchronize(st));
    return set_status(ZKG_OK, nullptr, nullptr);
  }
  BinPlan P;
  ZKB_TRY(bin_plan(nrows, npoints, NL, false, P));
  const size_t bytes = bin_ws_bytes<NL>(P, nrows);
  ZKB_TRY(cx.arena.reserve(bytes));
  cx.arena.reset();
  char* ws = static_cast<char*>(cx.arena.take(bytes));
  if (!ws) return set_status(ZKG_ERR_NOMEM, "msm_binary_device", "arena");
  auto get_tile = [&](int, int row0, int, int col0, int, const uint8_t** coeffs, size_t* pld,
                      const uint32_t** bases) -> zkg_status {
    *coeffs = d_coeffs + (size_t)row0 * ld + col0;
    *pld = ld;
    *bases = reinterpret_cast<const uint32_t*>(d_bases + (size_t)col0 * 2 * NL);
    return ZKG_OK;
  };
  auto done_tile = [](int) -> zkg_status { return ZKG_OK; };
  ZKB_TRY((bin_run<C, NL>(cx, P, nrows, npoints, ws, st, get_tile, done_tile, kind, reinterpret_cast<uint32_t*>(d_out))));
  ZKB_CUDA(cudaStreamSynchronize(st));
  ZKB_TRY(dev_check_report(cx, "msm_binary"));
  return set_status(ZKG_OK, nullptr, nullptr);
}

}  // namespace zkb

using namespace zkb;

extern "C" zkg_status zkg_g1_fft(zkg_curve curve, int jac, int m, const uint64_t* gen, const uint64_t* src,
                                 uint64_t* tgt, int inverse) {
  ZKB_TRY(g1_fft_check(curve, m, gen, src, tgt));
  if (curve == ZKG_BN254) return g1_fft_host<BN254, 4>(jac ? 1 : 0, m, gen, src, tgt, inverse ? 1 : 0);
  return g1_fft_host<BLS12_381, 6>(jac ? 1 : 0, m, gen, src, tgt, inverse ? 1 : 0);
}

extern "C" zkg_status zkg_g1_fft_device(zkg_curve curve, int jac, int m, const uint64_t* gen, const uint64_t* d_src,
                                        uint64_t* d_tgt, int inverse) {
  ZKB_TRY(g1_fft_check(curve, m, gen, d_src, d_tgt));
  if (curve == ZKG_BN254) return g1_fft_dev<BN254, 4>(jac ? 1 : 0, m, gen, d_src, d_tgt, inverse ? 1 : 0);
  return g1_fft_dev<BLS12_381, 6>(jac ? 1 : 0, m, gen, d_src, d_tgt, inverse ? 1 : 0);
}

extern "C" zkg_status zkg_msm_binary_plan(zkg_curve curve, int from_host, int nrows, int npoints, size_t info[3]) {
  if ((curve != ZKG_BN254 && curve != ZKG_BLS12_381) || nrows < 1 || npoints < 1 || !info)
    return set_status(ZKG_ERR_ARG, "msm_binary_plan", "bad argument");
  const int nl = curve == ZKG_BN254 ? 4 : 6;
  BinPlan P;
  ZKB_TRY(bin_plan(nrows, npoints, nl, from_host != 0, P));
  info[0] = P.bits_bytes;
  info[1] = 0;
  for (int r = 0; r < P.nbatch; r++)   // the launches of bin_run
    for (int q = 0; q < P.nchunk; q++) {
      size_t b = 0;
      ZKB_TRY(msm_bits_bytes(curve, P.rows(r, nrows), P.cols(q, npoints), P.rho, &b));
      info[1] = std::max(info[1], b);
    }
  info[2] = nl == 4 ? bin_ws_bytes<4>(P, nrows) : bin_ws_bytes<6>(P, nrows);
  return set_status(ZKG_OK, nullptr, nullptr);
}

extern "C" zkg_status zkg_msm_binary(zkg_curve curve, int out_kind, int nrows, int npoints,
                                     const uint8_t* const* rows, const uint64_t* bases, uint64_t* out) {
  ZKB_TRY(bin_check(curve, out_kind, nrows, npoints, rows, bases, out));
  if (curve == ZKG_BN254) return bin_host<BN254, 4>(host::BN_FP, out_kind, nrows, npoints, rows, bases, out);
  return bin_host<BLS12_381, 6>(host::BLS_FP, out_kind, nrows, npoints, rows, bases, out);
}

extern "C" zkg_status zkg_msm_binary_device(zkg_curve curve, int out_kind, int nrows, int npoints,
                                            const uint8_t* d_coeffs, size_t ld, const uint64_t* d_bases,
                                            uint64_t* d_out) {
  ZKB_TRY(bin_check(curve, out_kind, nrows, npoints, d_coeffs, d_bases, d_out));
  if (curve == ZKG_BN254) return bin_dev<BN254, 4>(out_kind, nrows, npoints, d_coeffs, ld, d_bases, d_out);
  return bin_dev<BLS12_381, 6>(out_kind, nrows, npoints, d_coeffs, ld, d_bases, d_out);
}
