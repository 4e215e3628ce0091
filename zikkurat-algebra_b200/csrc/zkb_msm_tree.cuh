// The first levels of the MSM bucket accumulation as a tree of affine additions.
//
// With T levels the sort pads every bucket segment to a multiple of 2^T entries (null entries, which
// add nothing), so a level is one list of pairs: slot q of level l + 1 is the sum of elements 2q and
// 2q + 1 of level l, and a segment's range is its first one shifted right by l. No slot needs to know
// its segment (walking segment boundaries with two cursors a thread, each step waiting for offsets,
// left the product pipes half idle: 6.1 ms for the first level at 2^22 points of BN254, now 5.0: forward
// 1.32 at 5.7 TB/s of DRAM, inversions 0.08, backward 3.63 bound by the products' issue), and threads take slots a block's width apart, so entries, running products and sums are read and
// written in full lines. An affine sum P0 + P1 needs one field inversion
// (lambda = (y1 - y0) / (x1 - x0), or 3 x0^2 / (2 y0) when P0 = P1); a whole level shares its
// inversions by Montgomery's simultaneous-inversion trick, so one addition costs six field
// products (one running product, two in the backward pass, lambda, lambda^2 and y3) against ten
// for the mixed XYZZ addition of the chunk accumulation (madd-2008-s). One level:
//   1. k_tree_fwd: each thread forms the denominators of its B slots and stores the running product
//      before each one; the thread's whole product goes to tt;
//   2. k_tree_inv: tt is inverted in place (simultaneous inversion again, one inversion per block);
//   3. k_tree_bwd: each thread walks its slots backwards, peeling one denominator inverse per slot
//      off the inverse of its product, and writes each slot's sum as canonical affine coordinates.
// The short segments left after the last level go through the XYZZ chunk accumulation, whose
// entries are then the identity map onto the last level's list. The identity is (0, 0) in the bases
// and in the last list, as in the reference's affine test (bn128_G1_affine.c:57-60), and a word
// pattern no coordinate has, all ones in x, in the lists between (so x alone tells it). A sum
// P + (-P) becomes the identity. The bases must be canonical (coordinates below p), as the
// reference's field operations assume: the equality tests compare words.
#pragma once
#include "zkb_batch_inv.cuh"
#include "zkb_msm_accum.cuh"
#include "zkb_msm_tail.cuh"

namespace zkb {

enum : uint32_t { TREE_COPY0 = 0, TREE_COPY1 = 1, TREE_INF = 2, TREE_ADD = 3, TREE_DBL = 4 };

// what the slot's sum is: a copy of one input (the other is the identity), the identity
// (both are, or P + (-P)), an addition or a doubling
template <class F>
__device__ __forceinline__ uint32_t tree_kind(const Fe<F>& x0, const Fe<F>& y0, const Fe<F>& x1, const Fe<F>& y1) {
  const bool inf0 = fe_is_zero(x0) && fe_is_zero(y0);
  const bool inf1 = fe_is_zero(x1) && fe_is_zero(y1);
  if (inf0) return inf1 ? TREE_INF : TREE_COPY1;
  if (inf1) return TREE_COPY0;
  if (!fe_eq(x0, x1)) return TREE_ADD;
  return fe_eq(y0, y1) ? TREE_DBL : TREE_INF;
}

// For the nseg segments of a slab: pads every segment of cnt[s] entries at off[s] with null entries up to its
// multiple of 2^T, writes the last list's offsets and adds the real entries up (*total, zeroed with the
// counts). cap: entries there is room for (device checks).
__global__ void __launch_bounds__(256) k_tree_pad(const uint32_t* __restrict__ cnt, const uint32_t* __restrict__ off,
                                                  uint32_t nseg, int T, uint32_t* __restrict__ entries,
                                                  uint32_t* __restrict__ last_off, uint32_t* __restrict__ total,
                                                  uint32_t* chk, uint32_t cap) {
  __shared__ uint32_t sum;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  const uint32_t s = blockIdx.x * 256 + threadIdx.x;
  uint32_t c = 0;
  if (s <= nseg) {
    const uint32_t lo = off[s];
    last_off[s] = (lo - off[0]) >> T;
    if (s < nseg) {
      c = cnt[s];
      const uint32_t m = (1u << T) - 1, end = (c + m) & ~m;
      for (uint32_t i = c; i < end; i++) {
        if (chk && lo + i >= cap) { atomicOr(chk, CHK_ENTRY); break; }
        entries[lo + i] = NULL_ENTRY;
      }
    }
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) atomicAdd(&sum, c);
  __syncthreads();
  if (threadIdx.x == 0) atomicAdd(total, sum);
}

// The two elements of slot q: level 0 gathers the bases of entries 2q and 2q + 1 (point index, negation
// in bit 31; a null entry reads the base 0), later levels read the list before. flags: bits 0, 1: null,
// bits 2, 3: negative.
template <class F, bool L0>
struct TreePair {
  const uint32_t *p0, *p1;
  uint32_t flags;
  __device__ __forceinline__ TreePair(uint2 e, const uint32_t* __restrict__ pts, uint32_t q, uint32_t npts, uint32_t* chk) {
    constexpr int AW = 2 * F::N;
    if constexpr (L0) {
      uint32_t a = e.x & 0x7fffffffu, b = e.y & 0x7fffffffu;
      flags = (a == NULL_ENTRY ? 1u : 0u) | (b == NULL_ENTRY ? 2u : 0u) | (e.x >> 31) << 2 | (e.y >> 31) << 3;
      if (flags & 1u) a = 0;
      if (flags & 2u) b = 0;
      if (chk && (a >= npts || b >= npts)) {
        atomicOr(chk, CHK_POINT);
        a = b = 0;
      }
      p0 = pts + (size_t)a * AW;
      p1 = pts + (size_t)b * AW;
    } else {
      p0 = pts + (size_t)(2 * (size_t)q) * AW;
      p1 = p0 + AW;
      flags = 0;
    }
  }
};
template <bool L0>
__device__ __forceinline__ uint2 tree_entries(const uint32_t* __restrict__ ent, uint32_t q, bool in) {
  if (L0 && in) return __ldg(reinterpret_cast<const uint2*>(ent) + q);
  return make_uint2(0, 0);
}
template <class F>
__device__ __forceinline__ bool tree_ident_x(const Fe<F>& x) {   // the lists' identity
  uint32_t o = x.v[0];
#pragma unroll
  for (int k = 1; k < F::N; k++) o &= x.v[k];
  return o == 0xffffffffu;
}
// y of an input, negated for a negative digit (canonically: p - y, and 0 stays 0)
template <class F>
__device__ __forceinline__ Fe<F> tree_y(const uint32_t* p, bool neg) {
  const Fe<F> y = fe_load_nc<F>(p + F::N);
  return neg ? fe_canon(fe_neg(y)) : y;
}

template <class F>
__device__ __forceinline__ Fe<F> fe_from_smem(const uint4* __restrict__ sm, int stride) {
  Fe<F> r;
#pragma unroll
  for (int k = 0; k < F::N / 4; k++) {
    const uint4 x = sm[k * stride];
    r.v[4 * k + 0] = x.x; r.v[4 * k + 1] = x.y; r.v[4 * k + 2] = x.z; r.v[4 * k + 3] = x.w;
  }
  return r;
}

// Shared memory of the tree passes: per thread and prefetch stage, the x coordinates of a slot's
// two inputs (forward pass), or both inputs and the slot's running product (backward pass), as
// 16-byte pieces; piece k of stage g of thread i at [(g * pieces + k) * NT + i].
template <class F>
constexpr int tree_fwd_pieces() { return 2 * (F::N / 4); }
template <class F>
constexpr int tree_bwd_pieces() { return 4 * (F::N / 4) + F::N / 4; }

// Slots a thread of a level of Q slots takes: about B, such that the blocks that have any make whole
// waves of the chip's `wave` resident threads (2^22 points of BN254 with B = 64 itself left the first
// level 9.3 waves and the second 4.7), and a list shorter than one wave still uses every SM.
__host__ __device__ inline uint32_t tree_waves(uint64_t Q, uint32_t wave, uint32_t B) {
  const uint64_t full = (uint64_t)wave * B, w = (Q + full / 2) / full;
  return w ? (uint32_t)w : 1u;
}
__host__ __device__ inline uint32_t tree_slots(uint32_t Q, uint32_t wave, uint32_t B) {
  const uint64_t t = (uint64_t)wave * tree_waves(Q, wave, B);
  return (uint32_t)((Q + t - 1) / t);
}

// What a level reads: the list of the level before, or the entries from the first one on, or those of a slab
// of windows further on, from off[0] (a form of its own: a pointer that is not a kernel argument cost
// BLS12-381's backward pass spills and 5%).
enum TreeSrc : int { SRC_LIST = 0, SRC_ENTRIES = 1, SRC_SLAB = 2 };
// The levels run over the entries [off[0], off[nseg]) of one slab of windows: level l has half of them >> l
// slots, numbered from 0.
__device__ __forceinline__ uint32_t tree_level_slots(const uint32_t* __restrict__ off, uint32_t nseg, int level) {
  return (__ldg(off + nseg) - __ldg(off)) >> (level + 1);
}

// Forward pass: thread i of block b has slots b NT B + k NT + i, k < B (B = tree_slots). pre[q] = product of the
// denominators of the thread's addition slots before q (stored for addition slots with k > 0);
// tt[thread] = product of all of them (1 when none). The inputs' x coordinates arrive through PF
// cp.async stages, PF - 1 slots ahead, their entries one slot earlier still.
template <class C, TreeSrc SRC, int NT, int PF>
__global__ void __launch_bounds__(NT) k_tree_fwd(const uint32_t* __restrict__ ent, const uint32_t* __restrict__ pts,
                                                 const uint32_t* __restrict__ off, uint32_t nseg, int level, uint32_t wave,
                                                 uint32_t tB, uint32_t* __restrict__ pre, uint32_t* __restrict__ tt,
                                                 uint32_t* chk, uint32_t npts) {
  using F = typename C::Fp;
  constexpr bool L0 = SRC != SRC_LIST;
  constexpr int FW = F::N, QF = F::N / 4, QS = tree_fwd_pieces<F>();
  extern __shared__ uint4 tsm[];
  const uint32_t Q = tree_level_slots(off, nseg, level), B = tree_slots(Q, wave, tB);
  if constexpr (SRC == SRC_SLAB) ent += __ldg(off);
  const uint32_t base = blockIdx.x * NT * B + threadIdx.x;
  const uint32_t n = base < Q ? min(B, (Q - base + NT - 1) / NT) : 0;   // slots of this thread
  Fe<F> acc = fe_one<F>();
  uint32_t fifo = 0;   // flags of the slots in flight, four bits each
  uint2 en = tree_entries<L0>(ent, base, n > 0);
  auto issue = [&](uint32_t k, int stage) {
    uint32_t fl = 0;
    if (k < n) {
      const TreePair<F, L0> pr(en, pts, base + k * NT, npts, chk);
      fl = pr.flags;
      const uint4 *p0 = reinterpret_cast<const uint4*>(pr.p0), *p1 = reinterpret_cast<const uint4*>(pr.p1);
#pragma unroll
      for (int c = 0; c < QF; c++) {
        cp_async16(&tsm[(stage * QS + c) * NT + threadIdx.x], p0 + c);
        cp_async16(&tsm[(stage * QS + QF + c) * NT + threadIdx.x], p1 + c);
      }
    }
    fifo = (fifo >> 4) | (fl << (4 * (PF - 1)));
    cp_async_commit();   // possibly empty: one group per slot keeps the wait count fixed
    en = tree_entries<L0>(ent, base + (k + 1) * NT, k + 1 < n);
  };
#pragma unroll
  for (int k = 0; k < PF - 1; k++) issue(k, k);
  for (uint32_t k = 0; k < n; k++) {
    issue(k + PF - 1, (int)((k + PF - 1) % PF));
    cp_async_wait<PF - 1>();   // this slot's group has landed
    const int stage = (int)(k % PF);
    const uint32_t q = base + k * NT;
    const Fe<F> x0 = fe_from_smem<F>(&tsm[(stage * QS) * NT + threadIdx.x], NT);
    const Fe<F> x1 = fe_from_smem<F>(&tsm[(stage * QS + QF) * NT + threadIdx.x], NT);
    const uint32_t fl = fifo & 15u;
    if (L0 ? (fl & 3u) != 0 : (tree_ident_x(x0) || tree_ident_x(x1))) continue;
    Fe<F> den;
    if (!fe_eq(x0, x1) && !fe_is_zero(x0) && !fe_is_zero(x1)) {   // the common case needs no y
      den = fe_sub(x1, x0);
    } else {
      const TreePair<F, L0> pr(tree_entries<L0>(ent, q, true), pts, q, npts, chk);
      const Fe<F> y0 = tree_y<F>(pr.p0, (fl >> 2) & 1u), y1 = tree_y<F>(pr.p1, (fl >> 3) & 1u);
      const uint32_t kind = tree_kind(x0, y0, x1, y1);
      if (kind == TREE_ADD) den = fe_sub(x1, x0);
      else if (kind == TREE_DBL) den = fe_add(y0, y0);
      else continue;
    }
    if (k > 0) fe_store<F>(pre + (size_t)q * FW, acc);
    acc = fe_mul(acc, den);
  }
  cp_async_wait<0>();
  fe_store<F>(tt + ((size_t)blockIdx.x * NT + threadIdx.x) * FW, acc);
}

// tt[0, n) <- their inverses (all non-zero mod p), by simultaneous inversion over each thread's
// strided subset (running products in scr) with one inversion per block of 256 threads
template <class F>
__global__ void __launch_bounds__(256) k_tree_inv(uint32_t n, uint32_t* __restrict__ tt, uint32_t* __restrict__ scr) {
  constexpr int FW = F::N;
  __shared__ Fe<F> sw[16];
  const size_t T = (size_t)gridDim.x * blockDim.x;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  Fe<F> acc = fe_one<F>();
  size_t last = t;
  for (size_t i = t; i < (size_t)n; i += T) {
    acc = fe_mul(acc, fe_load<F>(tt + i * FW));
    fe_store<F>(scr + i * FW, acc);
    last = i;
  }
  Fe<F> inv = block_inverse<F, 8>(acc, sw);
  if (t >= (size_t)n) return;
  for (size_t i = last;; i -= T) {
    const Fe<F> x = fe_load<F>(tt + i * FW);
    fe_store<F>(tt + i * FW, i >= t + T ? fe_mul(inv, fe_load<F>(scr + (i - T) * FW)) : inv);
    inv = fe_mul(inv, x);
    if (i < t + T) break;
  }
}

// Backward pass over the same slots from the last: acc is the inverse of the product of the
// denominators not yet peeled off, so a slot's inverse is acc * pre[q] and the next acc is
// acc * den. Every slot's sum is written, canonical, to out. A slot's inputs and running product
// arrive through PF cp.async stages, PF - 1 slots ahead.
template <class C, TreeSrc SRC, int NT, int PF>
__global__ void __launch_bounds__(NT, 1) k_tree_bwd(const uint32_t* __restrict__ ent, const uint32_t* __restrict__ pts,
                                                    const uint32_t* __restrict__ off, uint32_t nseg, int level, uint32_t wave,
                                                    uint32_t tB, const uint32_t* __restrict__ pre,
                                                    const uint32_t* __restrict__ tinv, uint32_t* __restrict__ out, int last,
                                                    uint32_t* chk, uint32_t npts) {
  using F = typename C::Fp;
  constexpr bool L0 = SRC != SRC_LIST;
  constexpr int FW = F::N, AW = 2 * F::N, QF = F::N / 4, QA = 2 * QF, QS = tree_bwd_pieces<F>();
  extern __shared__ uint4 tsm[];
  const uint32_t Q = tree_level_slots(off, nseg, level), B = tree_slots(Q, wave, tB);
  if constexpr (SRC == SRC_SLAB) ent += __ldg(off);
  const uint32_t base = blockIdx.x * NT * B + threadIdx.x;
  if (base >= Q) return;
  const int n = (int)min(B, (Q - base + NT - 1) / NT);
  Fe<F> acc = fe_load_nc<F>(tinv + ((size_t)blockIdx.x * NT + threadIdx.x) * FW);
  uint32_t fifo = 0;
  uint2 en = tree_entries<L0>(ent, base + (uint32_t)(n - 1) * NT, true);
  auto issue = [&](int k, int stage) {   // slot k, downwards
    uint32_t fl = 0;
    if (k >= 0) {
      const uint32_t q = base + (uint32_t)k * NT;
      const TreePair<F, L0> pr(en, pts, q, npts, chk);
      fl = pr.flags;
      const uint4 *p0 = reinterpret_cast<const uint4*>(pr.p0), *p1 = reinterpret_cast<const uint4*>(pr.p1);
#pragma unroll
      for (int c = 0; c < QA; c++) {
        cp_async16(&tsm[(stage * QS + c) * NT + threadIdx.x], p0 + c);
        cp_async16(&tsm[(stage * QS + QA + c) * NT + threadIdx.x], p1 + c);
      }
      if (k > 0) {
        const uint4* pp = reinterpret_cast<const uint4*>(pre + (size_t)q * FW);
#pragma unroll
        for (int c = 0; c < QF; c++) cp_async16(&tsm[(stage * QS + 2 * QA + c) * NT + threadIdx.x], pp + c);
      }
    }
    fifo = (fifo >> 4) | (fl << (4 * (PF - 1)));
    cp_async_commit();   // possibly empty: one group per slot keeps the wait count fixed
    en = tree_entries<L0>(ent, base + (uint32_t)(k - 1) * NT, k > 0);
  };
#pragma unroll
  for (int j = 0; j < PF - 1; j++) issue(n - 1 - j, j);
  for (int j = 0; j < n; j++) {
    const int k = n - 1 - j;
    issue(k - (PF - 1), (j + PF - 1) % PF);
    cp_async_wait<PF - 1>();   // this slot's group has landed
    const uint4* sa = &tsm[((j % PF) * QS) * NT + threadIdx.x];
    const uint32_t q = base + (uint32_t)k * NT, fl = fifo & 15u;
    Affine<F> a, b;
    a.x = fe_from_smem<F>(sa, NT);
    a.y = fe_from_smem<F>(sa + QF * NT, NT);
    b.x = fe_from_smem<F>(sa + QA * NT, NT);
    b.y = fe_from_smem<F>(sa + (QA + QF) * NT, NT);
    uint32_t kind;
    if constexpr (L0) {
      if (fl & 4u) a.y = fe_canon(fe_neg(a.y));
      if (fl & 8u) b.y = fe_canon(fe_neg(b.y));
      if (fl & 1u) { a.x = fe_zero<F>(); a.y = fe_zero<F>(); }
      if (fl & 2u) { b.x = fe_zero<F>(); b.y = fe_zero<F>(); }
      kind = tree_kind(a.x, a.y, b.x, b.y);
    } else {
      const bool i0 = tree_ident_x(a.x), i1 = tree_ident_x(b.x);
      kind = i0 ? (i1 ? TREE_INF : TREE_COPY1) : i1 ? TREE_COPY0
             : !fe_eq(a.x, b.x) ? TREE_ADD : fe_eq(a.y, b.y) ? TREE_DBL : TREE_INF;
    }
    Affine<F> r = kind == TREE_COPY1 ? b : a;
    if (kind >= TREE_ADD) {
      const Fe<F> den = kind == TREE_ADD ? fe_sub(b.x, a.x) : fe_add(a.y, a.y);
      Fe<F> inv;
      if (k > 0) {
        Fe<F> nacc;
        fe_mul2(inv, acc, fe_from_smem<F>(sa + 2 * QA * NT, NT), nacc, acc, den);
        acc = nacc;
      } else {
        inv = acc;
      }
      Fe<F> num;
      if (kind == TREE_ADD) {
        num = fe_sub(b.y, a.y);
      } else {
        const Fe<F> xx = fe_sqr(a.x);
        num = fe_add(fe_add(xx, xx), xx);
      }
      const Fe<F> lam = fe_mul(num, inv);
      const Fe<F> x3 = fe_sub(fe_sub(fe_sqr(lam), a.x), b.x);
      const Fe<F> y3 = fe_sub(fe_mul(lam, fe_sub(a.x, x3)), a.y);
      r.x = fe_canon(x3);
      r.y = fe_canon(y3);
    } else if (kind == TREE_INF) {
#pragma unroll
      for (int c = 0; c < F::N; c++) r.x.v[c] = r.y.v[c] = last ? 0u : 0xffffffffu;
    }
    fe_store<F>(out + (size_t)q * AW, r.x);
    fe_store<F>(out + (size_t)q * AW + FW, r.y);
  }
  cp_async_wait<0>();
}

}  // namespace zkb
