// NTT passes as matrix products on the tensor cores (tcgen05, 8-bit integers).
//
// A pass of the transform (zkb_ntt_kernels.cuh) applies one fixed 2^k x 2^k matrix of field
// elements to many columns. Multiplication by a constant w is linear in the bytes of its operand:
//     w x = sum_j x_j (w 2^(8j) mod r)            (x_j: byte j of x, j < 32)
// so with the 32-byte rows (w 2^(8j) mod r) as a 32 x 32 matrix of bytes, the whole pass is ONE
// product of unsigned bytes with 32-bit sums: the rows of A are columns of the transform
// (2^k elements = 32 2^k bytes, exactly as they lie in memory), B holds the 2^k x 2^k byte blocks,
// and output element o of a row is the number sum_i D[32 o + i] 2^(8i), below 2^k 32 255 r < 2^17 r.
// Folding those 32 sums into 8 words and subtracting q r (q from the top bits) costs about 75
// instructions; a field product costs about 480, and the k stages of a radix-2 network take k / 2
// products an element. The data stay in the reference's Montgomery form: B's entries are plain
// integers, and sum (x R) w = (sum x w) R.
//
// Twiddles. Passes form groups of at most 12 bits. Inside a group the twiddle between two passes
// depends on the digits already transformed (u bits, kappa) and on the digit t of this pass, so it
// is part of the matrix: pass p has 2^u matrices, M_kappa[k1][t] = F[k1][t] g^((t kappa) << (S + M'))
// (S: bits before the group). Only between groups does every element take a product of its own,
// by a table in the order of the elements' positions (read as a stream). A 2^24 transform has one
// such product an element instead of 14; every exponent is the literal one of the reference's
// network, so the result is the same for any generator. 128 consecutive columns (one tile) share
// their kappa when S + M' >= 7, which holds from 2^14 elements on; below that every pass is its own group.
//
// One CTA per SM: warp 0 feeds A (128 columns x one element, 4 KB contiguous) into a ring and B (plain
// bulk copies) when the tile's matrix changes; warp 1 issues the MMAs (M = 128,
// K = 32: one transform element, N = 32 NOUT); 16 or 24 warps read the finished sums back from tensor
// memory while the next tile's MMAs fill the other half of it. Passes write what the next one reads
// as 4 KB runs, the 16-byte halves of every element already in the order of the 32-byte swizzle (only
// the first pass, on the caller's data, needs TMA boxes for that). For k = 4 a CTA holds B for 8 of
// the 16 outputs (128 KB) and another CTA has the other half, which reads the same A from L2.
//
// Measured (B200, BN254, kernel time, against the tile form's product-bound passes): 2^12 67 -> 21 us,
// 2^14 75 -> 23 us, 2^18 105 -> 50 us, 2^20 341 -> 141 us, 2^22 1.21 -> 0.48 ms, 2^24 5.03 -> 2.03 ms
// forward, 5.07 -> 2.05 ms inverse (2.05 to 2.37 over seven runs). At 2^24 a pass without twiddles takes 275 us: 1.6 GB through L2 (A is
// read by two CTAs) at 5.8 TB/s, the tensor pipe half busy, HBM's floor 164 us; the pass with the twiddle
// product 650 us, bound by its ~620 instructions an element at 96 registers and 16 warps. Ring slots of
// four elements (16 KB): one barrier an element took 0.69 ms at 2^22. Forward stores: keeping kappa in
// the low bits for M' < 7 instead scattered one pass's 32-byte stores over 2 MB strides (697 us).
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <algorithm>

#include "zkb_dpf.cuh"
#include "zkb_field.cuh"
#include "zkb_ntt.h"

namespace zkb {

// Epilogue warps: the fold alone runs in 72 registers, the twiddle product needs 96. (Plus four
// warps: copies, MMA issue, TMEM allocation, one idle.)
template <bool TW> constexpr int nm_epi() { return TW ? 16 : 24; }
template <bool TW> constexpr int nm_threads() { return 128 + 32 * nm_epi<TW>(); }
static constexpr uint32_t NM_ROWS = 4096;            // one element of 128 columns of A
static constexpr int NM_TS = 4;                      // elements per ring slot
static constexpr uint32_t NM_SLOT = NM_TS * NM_ROWS;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for the phase of the given parity, at most `limit` polls; false when the limit or another
// warp's failure (*stop) ended the wait.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t* stop, uint32_t limit) {
  for (uint32_t i = 0; i < limit; i++) {
    if (mbar_try(bar, parity)) return true;
    if (*stop) return false;
  }
  *stop = 1;
  return false;
}
// Waits for copies or MMAs of this thread's own that are in flight, before the block may leave: bounded
// like the others, but neither by the caller's limit nor by another warp's failure.
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < NTT_WAIT_LIMIT && !mbar_try(bar, parity); i++) {}
}

// Shared-memory matrix descriptor, K-major rows of 32 bytes with the 32-byte swizzle: 8-row groups
// 256 bytes apart.
__device__ __forceinline__ uint64_t nm_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3ffff) >> 4) | (1ull << 16) | ((uint64_t)(256 >> 4) << 32) | (1ull << 46) | (6ull << 61);
}

// The twiddle product: FP64 radix, result in [0, 2r) (it is less than 2^256, all the next pass needs)
struct BnFrDL : BnFrD {
  static constexpr bool LAZY = true;
};
struct BlsFrDL : BlsFrD {
  static constexpr bool LAZY = true;
};
template <class P> struct LazyDpfOf;
template <> struct LazyDpfOf<BnFr> { using type = BnFrDL; };
template <> struct LazyDpfOf<BlsFr> { using type = BlsFrDL; };

struct NttMatArgs {
  const uint8_t* mat;      // this pass's matrices (2^u images of (32 2^k)^2 bytes)
  uint32_t* out;
  const uint32_t* tw;      // group twiddles in position order (FP64 radix), or null
  uint32_t* fault;         // the execution's host-visible word, set when a wait ran out
  uint32_t wait_limit;     // polls of one barrier before the kernel gives up
  const uint8_t* in;
  int m, k, s, Mp, S, u;
  int inverse;             // load and store sides exchanged
  int first, last;         // first / last pass: plain order of an element's 16-byte halves
  int t_sh, r_bits;        // forward stores: (r >> r_bits) << t_sh | kappa' << r_bits | (r mod 2^r_bits)
  int tw_S;                // group twiddles: index ((kappa' >> tw_S) << bits left) | remaining position
  uint32_t ntiles, items;  // items = ntiles * (outputs / NOUT), output group outermost
};

// 2^240 / r rounded down to a float, less 2^-20 of itself: times the top 32 bits (weight 2^240) of a
// sum below 2^17 r it gives floor(sum / r) or one less
template <class P>
__device__ __forceinline__ float nm_qscale();
template <>
__device__ __forceinline__ float nm_qscale<BnFr>() { return 0x1.5291bcp-14f; }
template <>
__device__ __forceinline__ float nm_qscale<BlsFr>() { return 0x1.1aa838p-15f; }

// The 32 column sums of one output element -> its value mod r in [0, 2r) (in [0, r) with canon).
// Bounds: sums < 2^25, so four of them make a 64-bit word below 2^50; q < 2^18, and q times the
// words of 2^256 - r (adding q (2^256 - r) subtracts q r mod 2^256) stays below 2^51.
template <class P>
__device__ __forceinline__ Fe<P> nm_fold(const uint32_t (&c)[32], bool canon) {
  uint64_t w[8];
#pragma unroll
  for (int i = 0; i < 8; i++)
    w[i] = (uint64_t)c[4 * i] + (uint64_t)c[4 * i + 1] * 0x100u + (uint64_t)c[4 * i + 2] * 0x10000u +
           (uint64_t)c[4 * i + 3] * 0x1000000u;
  const uint32_t top = (uint32_t)(w[7] >> 16);
  const uint32_t q = __float2uint_rd(__uint2float_rd(top) * nm_qscale<P>());
  Fe<P> r;
  uint64_t v = 0, neg = 1;   // 2^256 - r, word by word: ~r + 1
#pragma unroll
  for (int i = 0; i < 8; i++) {
    neg += (uint32_t)~P::mod(i);
    v = w[i] + (uint64_t)q * (uint32_t)neg + (v >> 32);
    r.v[i] = (uint32_t)v;
    neg >>= 32;
  }
  if (canon) r = reduce_once<P, true>(r.v, 0u);
  return r;
}

__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&c)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7]), "=r"(c[8]),
        "=r"(c[9]), "=r"(c[10]), "=r"(c[11]), "=r"(c[12]), "=r"(c[13]), "=r"(c[14]), "=r"(c[15]), "=r"(c[16]),
        "=r"(c[17]), "=r"(c[18]), "=r"(c[19]), "=r"(c[20]), "=r"(c[21]), "=r"(c[22]), "=r"(c[23]), "=r"(c[24]),
        "=r"(c[25]), "=r"(c[26]), "=r"(c[27]), "=r"(c[28]), "=r"(c[29]), "=r"(c[30]), "=r"(c[31])
      : "r"(addr));
}

// Shared memory: B image (32 NOUT rows x 32 2^K bytes), NS ring slots of A, barriers.
template <int K, int NOUT>
struct NttMatShape {
  static constexpr int R = 1 << K;
  static constexpr int GROUPS = R / NOUT;              // CTAs that share a tile
  static constexpr uint32_t BSLICE = NOUT * 1024;      // one element's rows of B
  static constexpr uint32_t BBYTES = R * BSLICE;
  static constexpr int NS = BBYTES > 64 * 1024 ? 6 : 8;
  static constexpr uint32_t SMEM = BBYTES + NS * NM_SLOT + 1024 + 1024;   // + alignment, barriers
};

template <class P, int K, int NOUT, bool TW>
__global__ void __launch_bounds__(nm_threads<TW>(), 1) k_ntt_mat(const __grid_constant__ CUtensorMap amap, const NttMatArgs g) {
  using Sh = NttMatShape<K, NOUT>;
  using PL = typename LazyDpfOf<P>::type;
  constexpr int R = Sh::R, NS = Sh::NS;
  constexpr uint32_t TCOLS = 64 * NOUT;   // tensor-memory columns: two buffers of 32 NOUT
  extern __shared__ uint8_t nm_smem[];
  const uint32_t base = (smem_u32(nm_smem) + 1023u) & ~1023u;
  const uint32_t sB = base, sA = base + Sh::BBYTES, sBar = sA + NS * NM_SLOT;
  // barriers: full[NS], empty[NS], bfull, bfree, tfull[2], tempty[2]
  const uint32_t full = sBar, empty = sBar + 8 * NS, bfull = sBar + 16 * NS, bfree = bfull + 8, tfull = bfull + 16,
                 tempty = bfull + 32, drain = bfull + 48;
  __shared__ uint32_t s_tmem;
  __shared__ volatile uint32_t s_stop;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    s_stop = 0;
    for (int i = 0; i < NS; i++) { mbar_init(full + 8 * i, 1); mbar_init(empty + 8 * i, 1); }
    mbar_init(bfull, 1);
    mbar_init(bfree, 1);
    mbar_init(drain, 1);
    for (int i = 0; i < 2; i++) { mbar_init(tfull + 8 * i, 1); mbar_init(tempty + 8 * i, 4 * NOUT); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "n"(TCOLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  const uint32_t per = g.items / gridDim.x, rest = g.items % gridDim.x;
  const uint32_t first = blockIdx.x * per + min(blockIdx.x, rest);
  const uint32_t last = first + per + (blockIdx.x < rest ? 1u : 0u);
  const uint32_t mM = (1u << g.Mp) - 1;
  const uint32_t ncols = 1u << (g.m - K);   // fewer than 128 (one tile, partly empty) below 2^(7 + K) elements
  const uint32_t rows = min(128u, ncols) * 32u;
  // the matrix of an item: output group and kappa of its tile
  auto key_of = [&](uint32_t item) -> uint32_t {
    const uint32_t c0 = (item % g.ntiles) * 128u, og = item / g.ntiles;
    return ((c0 >> g.Mp) >> g.S) * Sh::GROUPS + og;
  };

  if (warp == 0 && lane == 0) {   // ---- producer
    uint32_t cur = 0xffffffffu, nkey = 0, it = 0;
    bool ok = true, waited = false;
    for (uint32_t item = first; item < last && ok; item++) {
      const uint32_t key = key_of(item);
      if (key != cur) {
        if (nkey) ok = mbar_wait(bfree, (nkey - 1) & 1, &s_stop, g.wait_limit);
        if (!ok) break;
        mbar_expect(bfull, Sh::BBYTES);
        const uint8_t* src = g.mat + (size_t)key * Sh::BBYTES;
        for (int t = 0; t < R; t++)
          asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sB + t * Sh::BSLICE),
                       "l"(src + (size_t)t * Sh::BSLICE), "r"(Sh::BSLICE), "r"(bfull)
                       : "memory");
        cur = key;
        nkey++;
      }
      if (!waited) {   // the matrices are constant; the elements come from the pass before
        asm volatile("griddepcontrol.wait;" ::: "memory");
        waited = true;
      }
      const uint32_t c0 = (item % g.ntiles) * 128u;
      for (int t = 0; t < R; t += NM_TS, it++) {
        const uint32_t slot = it % NS, round = it / NS;
        ok = mbar_wait(empty + 8 * slot, (round & 1) ^ 1, &s_stop, g.wait_limit);
        if (!ok) break;
        mbar_expect(full + 8 * slot, NM_TS * (g.first ? NM_ROWS : rows));
#pragma unroll
        for (int j = 0; j < NM_TS; j++) {
          const uint32_t dst = sA + slot * NM_SLOT + j * NM_ROWS;
          if (g.first)
            asm volatile(
                "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
                "l"(&amap), "r"(0), "r"(c0), "r"(t + j), "r"(full + 8 * slot)
                : "memory");
          else
            asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                         "l"(g.in + (((size_t)(t + j) << (g.m - K)) + c0) * 32), "r"(rows), "r"(full + 8 * slot)
                         : "memory");
        }
      }
    }
    // No copy may be in flight when the block ends. The consumers have waited for all of them unless some
    // warp gave up, perhaps after this one's last copy.
    if (nkey) mbar_drain(bfull, (nkey - 1) & 1);
    for (uint32_t j = it > (uint32_t)NS ? it - NS : 0; j < it; j++) mbar_drain(full + 8 * (j % NS), (j / NS) & 1);
  } else if (warp == 1 && lane == 0) {   // ---- MMA issue
    constexpr uint32_t idesc = (2u << 4) | ((32u * NOUT / 8) << 17) | ((128u / 16) << 24);   // u8 x u8 -> s32
    uint32_t cur = 0xffffffffu, nkey = 0, it = 0, n = 0;
    bool ok = true;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // the limited waits start when the pass before is done
    for (uint32_t item = first; item < last && ok; item++, n++) {
      const uint32_t key = key_of(item);
      if (key != cur) {
        ok = mbar_wait(bfull, nkey & 1, &s_stop, g.wait_limit);
        if (!ok) break;
        cur = key;
        nkey++;
      }
      const uint32_t buf = n & 1;
      ok = mbar_wait(tempty + 8 * buf, ((n >> 1) & 1) ^ 1, &s_stop, g.wait_limit);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d = tmem + buf * (32 * NOUT);
      for (int t = 0; t < R; t += NM_TS, it++) {
        const uint32_t slot = it % NS;
        ok = mbar_wait(full + 8 * slot, (it / NS) & 1, &s_stop, g.wait_limit);
        if (!ok) break;
#pragma unroll
        for (int j = 0; j < NM_TS; j++)
          asm volatile(
              "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
              "l"(nm_desc(sA + slot * NM_SLOT + j * NM_ROWS)), "l"(nm_desc(sB + (t + j) * Sh::BSLICE)), "r"(idesc), "r"(t + j)
              : "memory");
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(empty + 8 * slot) : "memory");
      }
      if (!ok) break;
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tfull + 8 * buf) : "memory");
      if (item + 1 < last && key_of(item + 1) != key)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bfree) : "memory");
    }
    // Nor an MMA, when tensor memory is freed: the epilogue has waited for the last one unless it gave up.
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(drain) : "memory");
    mbar_drain(drain, 0);
  } else if (warp >= 4) {   // ---- epilogue
    // jobs: output j of a tile's quarter (32 rows), taken in turn by the quarter's warps
    constexpr uint32_t STEP = nm_epi<TW>() / 4;
    const uint32_t quarter = warp & 3, jobs = (last - first) * NOUT;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // the output may be what an earlier pass still reads
#pragma unroll 1
    for (uint32_t job = (warp - 4) >> 2; job < jobs; job += STEP) {
      const uint32_t n = job / NOUT, j = job % NOUT, item = first + n, buf = n & 1;
      uint32_t c = (item % g.ntiles) * 128u + quarter * 32u + lane;
      const bool valid = c < ncols;
      c = valid ? c : 0;
      const uint32_t o = (item / g.ntiles) * NOUT + j;
      uint32_t kap = c >> g.Mp, rem = c & mM, dst;   // kappa', and what is left below it
      if (g.inverse) {
        rem |= o << g.Mp;
        dst = (kap << (g.Mp + K)) | rem;
      } else {
        kap |= o << g.s;
        dst = ((rem >> g.r_bits) << g.t_sh) | (kap << g.r_bits) | (rem & ((1u << g.r_bits) - 1));
      }
      Fe<PL> w;
      if (TW) w = fe_load_nc<PL>(g.tw + (size_t)(((kap >> g.tw_S) << (g.inverse ? g.Mp + K : g.Mp)) | rem) * 8);
      const bool ok = mbar_wait(tfull + 8 * buf, (n >> 1) & 1, &s_stop, g.wait_limit);
      if (!__all_sync(0xffffffffu, ok)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t sums[32];
      tmem_ld32(tmem + ((quarter * 32u) << 16) + buf * (32 * NOUT) + j * 32, sums);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty + 8 * buf);
      Fe<P> v = nm_fold<P>(sums, !TW && g.last);
      if (TW) {
        Fe<PL> a;
#pragma unroll
        for (int i = 0; i < 8; i++) a.v[i] = v.v[i];
        a = fe_mul(a, w);
#pragma unroll
        for (int i = 0; i < 8; i++) v.v[i] = a.v[i];
      }
      if (!valid) continue;
      uint32_t* p = g.out + (size_t)dst * 8;
      const uint32_t x = g.last ? 0u : dst & 4u;   // the swizzle of the next pass's rows: bit 2 of the index
      *reinterpret_cast<uint4*>(p + x) = make_uint4(v.v[0], v.v[1], v.v[2], v.v[3]);
      *reinterpret_cast<uint4*>(p + (x ^ 4u)) = make_uint4(v.v[4], v.v[5], v.v[6], v.v[7]);
    }
  }
  __syncwarp();
  __syncthreads();
  if (warp == 2)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TCOLS) : "memory");
  if (threadIdx.x == 0 && s_stop && g.fault) *(volatile uint32_t*)g.fault = 1u;
}

// The matrices of a pass, in the layout k_ntt_mat copies: image [kappa][output group][input element]
// [32 NOUT rows x 32 bytes, 32-byte swizzle]. One warp per (kappa, output, input) block of 32 x 32
// bytes: lane j forms w 2^(8j) mod r (standard form), the warp transposes the bytes.
// net: F[k1][t] (Montgomery, 2^2k elements), pw: powers of the fold's base, by exponent t kappa.
template <class P>
__global__ void k_ntt_mat_build(const uint32_t* __restrict__ net, const uint32_t* __restrict__ pw, int k, int u,
                                int inverse, int nout, uint8_t* __restrict__ dst) {
  __shared__ uint32_t sm[8][32][9];
  const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t R = 1u << k;
  const uint32_t blk = blockIdx.x * 8 + wid;
  if (blk >= (R * R) << u) return;
  const uint32_t in = blk & (R - 1), out = (blk >> k) & (R - 1), kappa = blk >> (2 * k);
  const uint32_t k1 = inverse ? in : out, t = inverse ? out : in;
  Fe<P> w = fe_mul(fe_load_nc<P>(net + (size_t)(k1 * R + t) * 8), fe_load_nc<P>(pw + (size_t)(t * kappa) * 8));
  Fe<P> sh = fe_zero<P>();
#pragma unroll
  for (int i = 0; i < 8; i++)
    if (i == (int)(lane >> 2)) sh.v[i] = 1u << (8 * (lane & 3));
  w = fe_mul(w, sh);   // (w R) 2^(8 lane) / R
#pragma unroll
  for (int i = 0; i < 8; i++) sm[wid][lane][i] = w.v[i];
  __syncwarp();
  uint32_t row[8];   // output byte `lane` of each of the 32 shifts
#pragma unroll
  for (int i = 0; i < 8; i++) {
    row[i] = 0;
#pragma unroll
    for (int b = 0; b < 4; b++) row[i] |= ((sm[wid][4 * i + b][lane >> 2] >> (8 * (lane & 3))) & 0xffu) << (8 * b);
  }
  const uint32_t groups = R / nout, n = (out % nout) * 32 + lane;
  uint8_t* slice = dst + ((size_t)(kappa * groups + out / nout) * R + in) * ((size_t)nout * 1024);
  const uint32_t x = (n >> 2) & 1;
  *reinterpret_cast<uint4*>(slice + n * 32 + (x ? 16 : 0)) = make_uint4(row[0], row[1], row[2], row[3]);
  *reinterpret_cast<uint4*>(slice + n * 32 + (x ? 0 : 16)) = make_uint4(row[4], row[5], row[6], row[7]);
}

// Group twiddles in position order: T[i] = h^(((i mod 2^lo) (i >> lo)) << S), h^e = A[e mod 2^a] B[e >> a]
template <class P>
__global__ void k_ntt_mat_twiddles(uint32_t* __restrict__ T, const uint32_t* __restrict__ A,
                                   const uint32_t* __restrict__ B, int a, int lo, int S, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t e = ((i & ((1u << lo) - 1)) * (i >> lo)) << S;
  fe_store<P>(T + (size_t)i * 8, fe_mul(fe_load_nc<P>(A + (size_t)(e & ((1u << a) - 1)) * 8),
                                        fe_load_nc<P>(B + (size_t)(e >> a) * 8)));
}

template <class P, int K, int NOUT, bool TW>
static zkg_status nm_launch(const CUtensorMap& map, const NttMatArgs& g, int sms, cudaStream_t st) {
  using Sh = NttMatShape<K, NOUT>;
  ZKB_CUDA(cudaFuncSetAttribute(k_ntt_mat<P, K, NOUT, TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::SMEM));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(std::min<uint32_t>((uint32_t)sms, g.items));
  cfg.blockDim = dim3(nm_threads<TW>());
  cfg.dynamicSmemBytes = Sh::SMEM;
  cfg.stream = st;
  // the next pass's blocks start (barriers, tensor memory, matrices) while this pass's last ones end
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_ntt_mat<P, K, NOUT, TW>, map, g);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (e != cudaSuccess) return set_status(ZKG_ERR_CUDA, "ntt_mat", cudaGetErrorString(e));
  return ZKG_OK;
}

template <class P, bool TW>
static zkg_status nm_dispatch(const CUtensorMap& map, const NttMatArgs& g, int nout, int sms, cudaStream_t st) {
  if (g.k == 4) return nout == 8 ? nm_launch<P, 4, 8, TW>(map, g, sms, st) : nm_launch<P, 4, 4, TW>(map, g, sms, st);
  return nout == 8 ? nm_launch<P, 3, 8, TW>(map, g, sms, st) : nm_launch<P, 3, 4, TW>(map, g, sms, st);
}

template <class P>
zkg_status ntt_mat_launch_pass(const NttPlan& pl, int exec, const uint32_t* in, uint32_t* out, int sms,
                               const NttRun& run, cudaStream_t st) {
  const NttMatPass& q = pl.mpasses[exec];
  static const PFN_cuTensorMapEncodeTiled encode = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &r) != cudaSuccess ||
        r != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled>(f);
  }();
  if (!encode) return set_status(ZKG_ERR_CUDA, "ntt_mat", "no cuTensorMapEncodeTiled");
  CUtensorMap map = {};
  const cuuint64_t dims[3] = {8, 1ull << (pl.m - q.k), 1ull << q.k}, strides[2] = {32, 32ull << (pl.m - q.k)};
  const cuuint32_t box[3] = {8, 128, 1}, es[3] = {1, 1, 1};
  if (exec == 0 && encode(&map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint32_t*>(in), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return set_status(ZKG_ERR_CUDA, "ntt_mat", "cuTensorMapEncodeTiled failed");
  NttMatArgs g;
  g.mat = q.d_mat;
  g.out = out;
  g.tw = q.tw >= 0 ? pl.d_gtw[q.tw] : nullptr;
  g.fault = run.fault;
  g.wait_limit = run.wait_limit;
  g.m = pl.m;
  g.k = q.k;
  g.Mp = q.Mp;
  g.S = q.S;
  g.u = q.u;
  g.inverse = pl.inverse;
  g.in = reinterpret_cast<const uint8_t*>(in);
  g.s = q.s;
  g.first = exec == 0;
  g.last = exec == (int)pl.mpasses.size() - 1;
  g.tw_S = q.tw_S;
  // forward layouts: the digit a pass transforms on top, below it (kappa << M') | r, so that every pass
  // reads 4 KB runs and a quarter of a tile writes runs of at least 2^M' elements
  g.t_sh = g.r_bits = 0;
  if (!pl.inverse && !g.last) {
    g.t_sh = pl.m - pl.mpasses[exec + 1].k;
    g.r_bits = pl.mpasses[exec + 1].Mp;
  }
  g.ntiles = 1u << std::max(0, pl.m - q.k - 7);
  g.items = g.ntiles * ((1u << q.k) / q.nout);
  if (g.tw) return nm_dispatch<P, true>(map, g, q.nout, sms, st);
  return nm_dispatch<P, false>(map, g, q.nout, sms, st);
}

template <class P>
zkg_status ntt_mat_build(const uint32_t* net, const uint32_t* pw, int k, int u, int inverse, int nout, uint8_t* dst,
                         cudaStream_t st) {
  const uint32_t blocks = (1u << (2 * k)) << u;
  return launch("ntt_mat_build", k_ntt_mat_build<P>, dim3((blocks + 7) / 8), dim3(256), 0, st, net, pw, k, u, inverse,
                nout, dst);
}
template <class P>
zkg_status ntt_mat_twiddles(uint32_t* T, const uint32_t* A, const uint32_t* B, int a, int lo, int S, uint32_t n,
                            cudaStream_t st) {
  using PD = typename DpfOf<P>::type;
  return launch("ntt_mat_twiddles", k_ntt_mat_twiddles<PD>, dim3((n + 255) / 256), dim3(256), 0, st, T, A, B, a, lo, S, n);
}

}  // namespace zkb
