// From bucket partial sums to one point per window, by quads (zkb_quad.cuh).
//
//   k_sort_small     few points: digits, counts, offsets and entries of a window in one block
//   k_quad_accum     few entries: bucket accumulation with a quad a chunk
//   k_cut_merge      the partial sums of a segment cut by accumulation chunks
//   k_pieces         long segments, in pieces of 256 partial sums, a block a piece
//   k_bucket_rs      running sums T_g, R_g over groups of K buckets
//   k_window_bits    per window and bit k of g: 2^k K (sum of the T_g with that bit), and sum R_g; the
//                    sum of these is the window's value
//
// Everything here is a short chain of dependent additions with few points to work on, so what
// counts is the latency of one addition; measured before and after in the comments below.
#pragma once
#include "zkb_msm_accum.cuh"
#include "zkb_quad.cuh"

namespace zkb {

// The windows of a scalar: nwin of them over `bits` bits, widths differing by at most one, the wide
// ones lowest. (Equal windows of c bits leave a last window of a few bits, whose handful of buckets
// take every point: segments of hundreds to thousands of entries, which at 2^16 points cost 375 us
// of folding.)
struct WinShape {
  int base, extra;
  __host__ __device__ int width(int w) const { return base + (w < extra ? 1 : 0); }
  __host__ __device__ int start(int w) const { return w * base + (w < extra ? w : extra); }
  // buckets of a window (2^(width - 1)), and of all windows before it (= its first segment)
  __host__ __device__ uint32_t buckets(int w) const { return 1u << (width(w) - 1); }
  __host__ __device__ uint32_t seg(int w) const {
    return ((uint32_t)w << (base - 1)) + ((uint32_t)(w < extra ? w : extra) << (base - 1));
  }
};
__host__ __device__ inline WinShape win_shape(int bits, int nwin) { return {bits / nwin, bits % nwin}; }

// One MSM of the pipeline (a batch has many, in a table; a single MSM is passed by value).
struct MReq {
  const uint64_t* scal_in;   // a batch request's Montgomery scalars (device), 4 limbs each
  uint32_t pt_off;           // first point in the batch's concatenated standard scalars
  uint32_t n, nwin;          // points, windows
  WinShape win;
  uint32_t seg_base;         // first segment
  uint32_t K1, G, gbits;     // running-sum group size, groups of a wide window, log2 G
  uint32_t thr_off;          // first running-sum group (= first T/R entry)
  uint32_t blk_off;          // first (window, bit) block (= first U entry)
  uint32_t win_off;          // first window (= first V entry)
  uint32_t rank_base;        // first rank word (window-major per request: base + win n + point)
};

template <int FIELD>
__device__ __forceinline__ uint32_t mreq_key(const MReq& r) {
  return FIELD == 0 ? r.pt_off : FIELD == 1 ? r.thr_off : FIELD == 2 ? r.blk_off : r.win_off;
}
// largest r with key(r) <= x (keys ascending, key(0) = 0)
template <int FIELD>
__device__ __forceinline__ int mreq_find(const MReq* __restrict__ reqs, int nreq, uint32_t x) {
  int lo = 0, hi = nreq;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (mreq_key<FIELD>(reqs[mid]) <= x) lo = mid; else hi = mid;
  }
  return lo;
}
// The requests a kernel works on: a device table, or one by value.
struct MReqs {
  const MReq* tab;
  int n;
  MReq one;
};
template <int FIELD>
__device__ __forceinline__ MReq mreq_of(const MReqs& q, uint32_t x) {
  return q.tab ? q.tab[mreq_find<FIELD>(q.tab, q.n, x)] : q.one;
}

// ------------------------------------------------------------------------- long segments
// A piece is up to PIECE consecutive partial sums of one segment: index i of the segment is slot 2t + 1
// for i = 0 and 2 (t + i) after that.
static constexpr uint32_t PIECE = 256;
struct Piece {
  uint32_t s, t, i0, i1;      // segment, its first chunk, index range
  uint32_t first, n;          // the segment's pieces: first one's number, how many
};
struct PieceList {
  uint32_t* count;            // pieces listed (zeroed with the histogram)
  uint32_t cap;
  Piece* rec;
  uint32_t* done;             // finished pieces of the segment whose first piece this is
  uint32_t* pt;               // one point a piece
};
__device__ __forceinline__ void piece_push(const PieceList& L, uint32_t s, uint32_t t, uint32_t len) {
  const uint32_t n = (len + PIECE - 1) / PIECE, first = atomicAdd(L.count, n);
  for (uint32_t k = 0; k < n && first + k < L.cap; k++) {
    L.rec[first + k] = {s, t, k * PIECE, min(len, (k + 1) * PIECE), first, n};
    L.done[first + k] = 0;
  }
}

// Sum over the block's quads (128 threads), valid in every quad of warp 0.
template <class F>
__device__ __forceinline__ Fe<F> block_sum128(Fe<F> a, uint32_t* sm) {
  a = quad_warp_sum(a);
  if ((threadIdx.x & 31) < 4) quad_store(sm + (threadIdx.x >> 5) * 4 * F::N, a);
  __syncthreads();
  Fe<F> r = fe_zero<F>();
  if (threadIdx.x < 32) {
    r = quad_load<F>(sm + ((threadIdx.x >> 2) & 3) * 4 * F::N);
    r = quad_add(r, fe_shfl_xor(r, 4));
    r = quad_add(r, fe_shfl_xor(r, 8));
  }
  return r;
}

// The block that finishes a segment's last piece adds the pieces up.
template <class C>
__global__ void __launch_bounds__(128) k_pieces(const PieceList L, const uint32_t* __restrict__ spt,
                                                uint32_t* __restrict__ bsum) {
  using F = typename C::Fp;
  constexpr int XW = 4 * F::N;
  __shared__ __align__(16) uint32_t sm[4 * XW];
  __shared__ uint32_t s_last;
  const uint32_t count = min(*L.count, L.cap), quad = threadIdx.x >> 2;
  for (uint32_t p = blockIdx.x; p < count; p += gridDim.x) {
    const Piece pc = L.rec[p];
    Fe<F> a = fe_zero<F>();
    for (uint32_t i0 = pc.i0; i0 < pc.i1; i0 += 32) {
      const uint32_t i = i0 + quad;
      Fe<F> q = fe_zero<F>();
      if (i < pc.i1) q = quad_load<F>(spt + (size_t)(2 * (pc.t + i) + (i == 0 ? 1 : 0)) * XW);
      a = quad_add(a, q);
    }
    a = block_sum128(a, sm);
    if (pc.n == 1) {
      if (threadIdx.x < 4) quad_store(bsum + (size_t)pc.s * XW, a);
    } else {
      if (threadIdx.x < 4) {
        quad_store(L.pt + (size_t)p * XW, a);
        __threadfence();
      }
      __syncthreads();
      if (threadIdx.x == 0) s_last = atomicAdd(L.done + pc.first, 1u) + 1 == pc.n;
      __syncthreads();
      if (s_last) {
        __threadfence();
        a = fe_zero<F>();
        for (uint32_t k0 = 0; k0 < pc.n; k0 += 32) {
          Fe<F> q = fe_zero<F>();
          if (k0 + quad < pc.n) q = fe_load_cg<F>(L.pt + (size_t)(pc.first + k0 + quad) * XW + quad_lane() * F::N);
          a = quad_add(a, q);
        }
        a = block_sum128(a, sm);
        if (threadIdx.x < 4) quad_store(bsum + (size_t)pc.s * XW, a);
      }
    }
    __syncthreads();
  }
}

// -------------------------------------------------------------------- bucket accumulation
// The accumulation (accum_block, zkb_msm_accum.cuh) with one quad a chunk: chunk t is entries
// [tL, (t + 1)L). For MSMs of few entries, where a thread a chunk leaves most of the GPU idle and its
// chain of mixed additions is what takes the time (1000 points: 87 us for chunks of 8 in ten blocks).
// It does 16 lane products an addition against 10, so from QUAD_TOTAL entries on the thread form is
// the faster one. (One quad a segment instead of equal chunks took 66 us: a warp waits for the
// longest of its eight segments.)
static constexpr uint64_t QUAD_TOTAL = 250000;
static constexpr uint32_t NULL_ENTRY = 0x7fffffffu;   // an entry that adds nothing (k_sort_small)
template <class C>
__global__ void __launch_bounds__(128) k_quad_accum(const uint32_t* __restrict__ entries,
                                                    const uint32_t* __restrict__ off, uint32_t nseg, uint32_t nchunks,
                                                    uint32_t L, const uint32_t* __restrict__ bases,
                                                    uint32_t* __restrict__ bsum, uint32_t* __restrict__ skey,
                                                    uint32_t* __restrict__ spt, uint32_t* chk, uint32_t npts) {
  using F = typename C::Fp;
  constexpr int XW = 4 * F::N;
  const uint32_t t = (blockIdx.x * 128 + threadIdx.x) >> 2;
  const uint32_t total = __ldg(off + nseg);
  L = counted_len(total, nchunks, L);
  uint32_t pos = t * L, end = pos, s = 0, seg_hi = 0;
  bool cut = false;   // the run's segment began before the chunk
  if (t < nchunks && pos < total) {
    end = min(pos + L, total);
    s = find_seg(off, nseg, pos);
    cut = __ldg(off + s) < pos;
    seg_hi = __ldg(off + s + 1);
  }
  uint32_t keyA = INVALID, keyB = INVALID;
  // the next entry and its point are fetched while an addition runs
  auto point = [&](uint32_t at) {
    const uint32_t e = at < end ? __ldg(entries + at) : NULL_ENTRY;
    uint32_t i = e & 0x7fffffffu;
    const bool null = i == NULL_ENTRY;
    if (null) i = 0;
    if (chk && i >= npts) { atomicOr(chk, CHK_POINT); i = 0; }
    return fe_sel(null, fe_zero<F>(), quad_from_affine<F>(bases + (size_t)i * 2 * F::N, e >> 31));
  };
  Fe<F> a = fe_zero<F>(), q = point(pos);
  // the finished run of segment s: the whole segment to its bucket, a cut one to this chunk's slots
  auto flush = [&] {
    const bool after = seg_hi > end;
    if (cut) keyA = s; else if (after) keyB = s;
    quad_store(!cut && !after ? bsum + (size_t)s * XW : spt + (size_t)(2 * t + (cut ? 0 : 1)) * XW, a);
  };
  bool have = false;
#pragma unroll 1
  for (; __any_sync(FULL, pos < end); pos++) {
    const Fe<F> nx = point(pos + 1);
    if (pos < end) {
      while (pos >= seg_hi) {
        if (have) { flush(); a = fe_zero<F>(); }
        have = false;
        s++;
        cut = false;
        seg_hi = __ldg(off + s + 1);
      }
      have = true;
    }
    __syncwarp();
    a = quad_add(a, q);
    q = nx;
  }
  if (have) flush();
  if (t < nchunks && quad_lane() == 0) {
    skey[2 * (size_t)t] = keyA;
    skey[2 * (size_t)t + 1] = keyB;
  }
}

// Segments cut by chunk boundaries. A cut segment s starting in chunk t leaves its first partial sum
// in slot 2t + 1 and one in slot 2t' for every later chunk t' it reaches (a chunk inside s routes its
// whole sum there); it ends in chunk (off[s + 1] - 1) / L. One quad a segment, at most RUN_MAX + 1
// partial sums (with ~64-entry segments and ~128-entry chunks nearly every cut segment has two);
// longer ones go to k_pieces.
static constexpr uint32_t RUN_MAX = 8;
template <class C>
__global__ void __launch_bounds__(128) k_cut_merge(const uint32_t* __restrict__ off, uint32_t nchunks, uint32_t L,
                                                   const uint32_t* __restrict__ skey, const uint32_t* __restrict__ spt,
                                                   uint32_t* __restrict__ bsum, uint32_t* chk, uint32_t nseg,
                                                   const PieceList P) {
  using F = typename C::Fp;
  constexpr int XW = 4 * F::N;
  const uint32_t t = (blockIdx.x * 128 + threadIdx.x) >> 2;
  uint32_t s = INVALID, more = 0;   // partial sums after the first
  if (t + 1 < nchunks) {
    const uint32_t total = __ldg(off + nseg);
    s = __ldg(skey + 2 * (size_t)t + 1);
    if (chk && s != INVALID && s >= nseg) { atomicOr(chk, CHK_SEGMENT); s = INVALID; }
    if (s != INVALID) {
      const uint32_t last = __ldg(off + s + 1) - 1;   // on its way while the total is looked at
      more = last / counted_len(total, nchunks, L) - t;
      if (more > RUN_MAX) {
        if (quad_lane() == 0) piece_push(P, s, t, more + 1);
        s = INVALID;
        more = 0;
      }
    }
  }
  Fe<F> a = fe_zero<F>();
  if (s != INVALID) a = quad_load<F>(spt + (size_t)(2 * t + 1) * XW);
  for (uint32_t u = 1; __any_sync(FULL, u <= more); u++) {
    Fe<F> q = fe_zero<F>();
    if (u <= more) q = quad_load<F>(spt + (size_t)(2 * (t + u)) * XW);
    a = quad_add(a, q);
  }
  if (s != INVALID) quad_store(bsum + (size_t)s * XW, a);
}

// ------------------------------------------------------------------------ bucket reduction
// Group (w, g): buckets j = gK .. gK + K - 1 of window w (bucket number j + 1): T = sum S_j,
// R = sum (j - gK + 1) S_j, by running sums from the top. Two quads a group: one adds the buckets up
// (T), the other, one step behind, adds the T's up (R), so a step of both is one addition's latency.
// off == null: every bucket present. A narrow window has half the buckets; its missing groups are stored as
// the identity.
template <class C>
__global__ void __launch_bounds__(128) k_bucket_rs(const MReqs Q, uint32_t ngroups, const uint32_t* __restrict__ bsum,
                                                   const uint32_t* __restrict__ off, uint32_t* __restrict__ Tout,
                                                   uint32_t* __restrict__ Rout) {
  using F = typename C::Fp;
  constexpr int XW = 4 * F::N;
  const uint32_t t = (blockIdx.x * 128 + threadIdx.x) >> 3;
  const bool live = t < ngroups, upper = threadIdx.x & 4;   // lower quad: T, upper quad: R
  uint32_t K = 0;
  size_t s0 = 0;
  if (live) {
    const MReq q = mreq_of<1>(Q, t);
    const uint32_t tl = t - q.thr_off;
    const int w = tl / q.G;
    s0 = q.seg_base + q.win.seg(w) + (size_t)(tl % q.G) * q.K1;
    const uint32_t j0 = (tl % q.G) * q.K1, nb = q.win.buckets(w);
    if (j0 < nb) K = min(q.K1, nb - j0);   // a narrow window has half the buckets
  }
  auto bucket = [&](uint32_t i) {   // i-th from the top
    Fe<F> a = fe_zero<F>();
    if (i < K && !upper) {
      const size_t s = s0 + (K - 1 - i);
      if (!off || __ldg(off + s) != __ldg(off + s + 1)) a = quad_load<F>(bsum + s * XW);
    }
    return a;
  };
  Fe<F> a = fe_zero<F>(), q = bucket(0);
  for (uint32_t i = 0; __any_sync(FULL, i <= K && live); i++) {
    const Fe<F> prev = fe_shfl(a, (threadIdx.x & 31) & ~4);   // the lower quad's T
    const Fe<F> nx = bucket(i + 1);
    a = quad_add(a, upper ? fe_sel(i <= K, prev, fe_zero<F>()) : q);
    q = nx;
  }
  if (live) quad_store((upper ? Rout : Tout) + (size_t)t * XW, a);
}

// Block (w, k): k < gbits: 2^k K times the sum of the T_g with bit k of g set; k == gbits: sum R_g.
// The window's last block to finish adds its gbits + 1 terms up: the window's value, canonical. done:
// finished blocks a window (zeroed with the histogram). Block size: four rounds of its quads, up to
// eight warps (more warps wait for one another on the product pipes: 57 -> 45 us at 1000 points).
static inline unsigned window_bits_threads(uint32_t G) { return G >= 512 ? 256 : G >= 256 ? 128 : G >= 128 ? 64 : 32; }
template <class C>
__global__ void __launch_bounds__(256) k_window_bits(const MReqs Q, const uint32_t* __restrict__ Tin,
                                                     const uint32_t* __restrict__ Rin, uint32_t* __restrict__ U,
                                                     uint32_t* __restrict__ done, uint32_t* __restrict__ V) {
  using F = typename C::Fp;
  constexpr int XW = 4 * F::N;
  __shared__ __align__(16) uint32_t sm[8 * XW];
  const MReq q = mreq_of<2>(Q, blockIdx.x);
  const uint32_t terms = q.gbits + 1, bl = blockIdx.x - q.blk_off, w = bl / terms, k = bl % terms;
  const bool bit = k < q.gbits;
  const uint32_t cnt = bit ? q.G >> 1 : q.G, quad = threadIdx.x >> 2, quads = blockDim.x >> 2;
  const uint32_t* src = (bit ? Tin : Rin) + ((size_t)q.thr_off + (size_t)w * q.G) * XW;
  auto item = [&](uint32_t j) {   // j-th group of the block's
    const uint32_t g = bit ? ((j >> k) << (k + 1)) | (1u << k) | (j & ((1u << k) - 1)) : j;
    return j < cnt ? quad_load<F>(src + (size_t)g * XW) : fe_zero<F>();
  };
  Fe<F> a = fe_zero<F>(), nx = item(quad);
#pragma unroll 1
  for (uint32_t j0 = 0; j0 < cnt; j0 += quads) {
    const Fe<F> x = nx;
    nx = item(j0 + quads + quad);
    a = quad_add(a, x);
  }
  a = quad_warp_sum(a);
  if ((threadIdx.x & 31) < 4) quad_store(sm + (threadIdx.x >> 5) * XW, a);
  __syncthreads();
  if (threadIdx.x >= 32) return;
  if (quads > 8) {
    a = quad < quads >> 3 ? quad_load<F>(sm + quad * XW) : fe_zero<F>();
#pragma unroll 1
    for (uint32_t d = 4; d < quads >> 1; d <<= 1) a = quad_add(a, fe_shfl_xor(a, d));
  }
  const uint32_t dbls = bit ? k + 31 - __clz(q.K1) : 0;
#pragma unroll 1
  for (uint32_t i = 0; i < dbls; i++) a = quad_dbl(a);
  if (threadIdx.x < 4) {
    quad_store(U + (size_t)blockIdx.x * XW, a);
    __threadfence();
  }
  __syncwarp();
  uint32_t last = 0;
  if (threadIdx.x == 0) last = atomicAdd(done + q.win_off + w, 1u) + 1 == terms;
  if (!__shfl_sync(FULL, last, 0)) return;
  __threadfence();
  const uint32_t* u = U + ((size_t)q.blk_off + (size_t)w * terms) * XW;
  a = fe_zero<F>();
#pragma unroll 1
  for (uint32_t j0 = 0; j0 < terms; j0 += 8)
    a = quad_add(a, j0 + quad < terms ? fe_load_cg<F>(u + (size_t)(j0 + quad) * XW + quad_lane() * F::N) : fe_zero<F>());
  a = quad_warp_sum(a);
  if (threadIdx.x < 4) quad_store(V + (size_t)(q.win_off + w) * XW, fe_canon(a));
}

}  // namespace zkb
