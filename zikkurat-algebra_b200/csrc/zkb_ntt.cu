// NTT planning and entry points (kernels: zkb_ntt_mat.cuh, zkb_ntt_kernels.cuh).
//
// Reference: lib/cbits/curves/poly/mont/bn128_poly_mont.c:418-473 (forward: recursive radix-2
// decimation in time, twiddles g^j, natural order in and out) and :565-622 (inverse: recursive
// decimation in frequency, each stage halves, twiddles g^-j / 2).
//
// Factorisation used here. Write the reference's forward network with generator g on
// N = 2^m points as F_g. For N = N1*N2 (N1 = 2^k) it satisfies, for every g,
//     F_g(x)[k1 + N1*k2] = F_{g^N1}( r -> g^(r*k1) * F_{g^N2}( t -> x[r + N2*t] )[k1] )[k2]
// with r < N2, t, k1 < N1 and the literal power g^(r*k1) (exponent < N, never reduced), which
// follows from unrolling the recursion; for a generator of order N it is the four-step DFT.
// Applying it recursively gives passes of 2^k-point networks with a twiddle multiply between
// passes. The reference's inverse network is the transpose of F_{g^-1} times (1/2)^m, so the
// inverse runs the transposed passes in reverse order: twiddle first, then a 2^k-point
// decimation-in-frequency network. Every butterfly and twiddle is an exact field operation on
// the same powers of g as the reference, so results are bit-identical, for any `gen`.
//
// Pass p (forward order) has k bits, s bits already done and M' = m - s - k bits after it.
// Column c in [0, 2^(m-k)), row t / output k1 in [0, 2^k):
//     forward reads  x[in(c,t)],  in(c,t)  = (c mod 2^M') + ((c >> M') << (M'+k)) + (t << M')
//     forward writes y[out(c,k1)], out(c,k1) = c + (k1 << (m-k)), times g^(((c mod 2^M')*k1) << s)
// A CTA owns a tile of consecutive columns, so every global access is a run of consecutive
// 32-byte elements. From 2^9 elements on a pass is a matrix product on the tensor cores
// (zkb_ntt_mat.cuh); below, and in a batch's persistent kernel, its tile lives in shared memory and each
// thread runs 2 butterfly stages at a time on 4 elements held in registers.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <cstdlib>
#include <vector>

#include "zkb_dpf.cuh"
#include "zkb_field.cuh"
#include "zkb_host_ec.h"
#include "zkb_ntt.h"
#include "zkb_runtime.h"

namespace zkb {

// --------------------------------------------------------------------------- planning

static int g_ntt_kmax = 8;
// NTT passes with FP64-pipe products (tables in radix R' = 2^260, zkb_dpf.cuh); ZKB_NTT_DPF=0
// keeps every table in the reference's radix and the products on the integer pipes
static int g_ntt_dpf = [] {
  const char* v = std::getenv("ZKB_NTT_DPF");
  return v ? std::atoi(v) : 1;
}();
static bool g_ntt_kmax_set = false;       // an explicit zkg_set_ntt_kmax overrides tuning
static int g_ntt_tuned[2][NTT_MMAX + 1] = {{0}};    // tuned largest pass per curve and m (0 = untuned)

static std::once_flag g_ntt_tune_once[2];

static int effective_kmax(int curve, int m) {
  std::call_once(g_ntt_tune_once[curve], [curve] {   // persisted tuning (ZKG_TUNE_CACHE), once
    const int sms = device_sm_count();
    for (int mm = 0; mm <= NTT_MMAX; mm++) {
      int k = 0;
      if (tune_cache_get("ntt", curve, mm, sms, &k, 1) && k >= 1 && k <= NTT_KMAX) g_ntt_tuned[curve][mm] = k;
    }
  });
  if (!g_ntt_kmax_set && m >= 0 && m <= NTT_MMAX && g_ntt_tuned[curve][m] > 0) return g_ntt_tuned[curve][m];
  return g_ntt_kmax;
}

static std::vector<NttPass> ntt_schedule(int m, int kmax) {
  std::vector<NttPass> ps;
  if (m == 0) return ps;
  const int np = (m + kmax - 1) / kmax;
  int s = 0;
  for (int p = 0; p < np; p++) {
    const int rem = m - s, left = np - p;
    const int k = (rem + left - 1) / left;   // larger passes first
    NttPass q;
    q.k = k;
    q.s = s;
    q.Mp = m - s - k;
    ps.push_back(q);
    s += k;
  }
  return ps;
}

template <int NL>
static host::El<NL> el_from_u64(const uint64_t* p) {
  host::El<NL> r;
  std::memcpy(r.v, p, sizeof(r.v));
  return r;
}

static zkg_status upload(uint32_t** dst, const std::vector<host::El<4>>& v) {
  ZKB_CUDA(cudaMalloc(dst, v.size() * 32));
  ZKB_CUDA(cudaMemcpy(*dst, v.data(), v.size() * 32, cudaMemcpyHostToDevice));
  return ZKG_OK;
}

// Passes as matrix products (zkb_ntt_mat.cuh); ZKB_NTT_MAT=0 keeps the register form
static int g_ntt_mat = [] {
  const char* v = std::getenv("ZKB_NTT_MAT");
  return v ? std::atoi(v) : 1;
}();
// Sizes of the matrix form: from 2^9 on (2^9 20 -> 18 us, 2^8 equal, 2^7 13 -> 16). An explicit largest pass (zkg_set_ntt_kmax) and the
// integer products (ZKB_NTT_DPF=0) name the register form.
static constexpr int NTT_MAT_MMIN = 9;
static bool ntt_use_mat(int m) { return g_ntt_mat && g_ntt_dpf && !g_ntt_kmax_set && m >= NTT_MAT_MMIN; }

// Bits of the groups: from 2^14 elements on 7 to 12 each (128 columns share a matrix), two up to 2^24,
// three above: the fewest passes, then the smallest matrices. A group of G bits runs ceil(G / 4) passes
// of 4 and 3 bits, the 4s first. Below 2^14 every pass is a group, with a twiddle product between any
// two: a transform that small is all latency, and a pass takes ~6 us (2^12: 67 -> 22 us with three
// passes of 4 bits, the register form has two of 6).
static std::vector<int> ntt_mat_digits(int G) {
  const int np = (G + 3) / 4;
  std::vector<int> d(np, 3);
  for (int i = 0; i < G - 3 * np; i++) d[i] = 4;
  return d;
}
static std::vector<int> ntt_mat_groups(int m) {
  auto cost = [](int G) {
    double bytes = 0;
    int u = 0;
    for (int k : ntt_mat_digits(G)) { bytes += std::ldexp(1024.0, 2 * k + u); u += k; }
    return (double)((G + 3) / 4) * 1e12 + bytes;
  };
  std::vector<int> best;
  if (m < 14) return ntt_mat_digits(m);
  double bc = 1e300;
  for (int a = 7; a <= 12; a++)
    for (int b = 7; b <= 12; b++) {
      const int c = m - a - b;
      if (m <= 24 ? c != 0 : (c < 7 || c > 12)) continue;
      const double t = cost(a) + cost(b) + (c ? cost(c) : 0.0);
      if (t < bc) {
        bc = t;
        best = {a, b};
        if (c) best.push_back(c);
      }
    }
  return best;
}

// out[k1 2^k + t] = x0 F[k1][t], the matrix of the 2^k-point decimation-in-time network with twiddles w^j:
// column t of 2^l points is column t / 2 of half as many, its lower half times the literal powers of
// w^(2^(k - l)) for odd t, and the upper half that or its negative. (The network applied to every unit vector
// took a new plan 0.1 to 0.2 ms: with its first transform 2^12 365 -> 219 us, 2^18 515 -> 333.)
static void net_matrix(const host::Field<4>& F, const host::El<4>& w, int k, const host::El<4>& x0, host::El<4>* out) {
  const int R = 1 << k;
  std::vector<host::El<4>> wl(k + 1, w);   // wl[l] = w^(2^(k - l))
  for (int l = k - 1; l >= 1; l--) wl[l] = host::mul(F, wl[l + 1], wl[l + 1]);
  std::vector<host::El<4>> a((size_t)R * R), b((size_t)R * R);
  a[0] = x0;
  for (int l = 1; l <= k; l++) {
    const int n = 1 << l, h = n / 2;
    host::El<4> p = host::one(F);
    for (int r = 0; r < h; r++) {
      for (int t = 0; t < h; t++) {
        const host::El<4>& e = a[(size_t)r * h + t];
        const host::El<4> o = r ? host::mul(F, e, p) : e;
        b[(size_t)r * n + 2 * t] = b[(size_t)(r + h) * n + 2 * t] = e;
        b[(size_t)r * n + 2 * t + 1] = o;
        b[(size_t)(r + h) * n + 2 * t + 1] = host::sub(F, host::zero<4>(), o);
      }
      p = host::mul(F, p, wl[l]);
    }
    std::swap(a, b);
  }
  std::copy(a.begin(), a.end(), out);
}

static host::El<4> pow_2k(const host::Field<4>& F, host::El<4> x, int k) {
  for (int i = 0; i < k; i++) x = host::mul(F, x, x);
  return x;
}

// Matrices and group twiddles of a matrix-form plan; h is the network's generator, scale the
// inverse's (1/2)^m, folded into the first pass's matrix. One device block holds everything, filled
// from one upload of network matrices and powers (a batch builds a plan per transform: separate
// allocations made its first run a third longer).
template <class P>
static zkg_status build_mat(const host::Field<4>& F, NttPlan* pl, const host::El<4>& h, const host::El<4>& scale,
                            const host::El<4>& rp, cudaStream_t st) {
  const int m = pl->m;
  const std::vector<int> groups = ntt_mat_groups(m);
  const int sms = device_sm_count();
  pl->mat = true;
  std::vector<host::El<4>> hv;   // what the build kernels read
  auto powers = [&](size_t n, const host::El<4>& x0, const host::El<4>& g) {
    const size_t at = hv.size();
    host::El<4> x = x0;
    for (size_t i = 0; i < n; i++) { hv.push_back(x); x = host::mul(F, x, g); }
    return at;
  };
  size_t bytes = 0;
  auto take = [&](size_t n) { const size_t o = bytes; bytes += (n + 1023) & ~size_t(1023); return o; };
  struct Src { size_t net, pw, dst; };
  std::vector<Src> src;               // per pass, forward order
  std::vector<NttMatPass> fwd;
  size_t gtw[4] = {0, 0, 0, 0};
  int s = 0;
  for (size_t gi = 0; gi < groups.size(); gi++) {
    const int S = s;
    const std::vector<int> digits = ntt_mat_digits(groups[gi]);
    for (size_t di = 0; di < digits.size(); di++) {
      NttMatPass q = {};
      q.k = digits[di];
      q.s = s;
      q.Mp = m - s - q.k;
      q.S = S;
      q.u = s - S;
      const int R = 1 << q.k;
      // half the outputs per CTA when a whole set of them leaves SMs idle
      q.nout = (1 << std::max(0, m - q.k - 7)) * (R / 8) < sms ? 4 : 8;
      q.tw = -1;
      const size_t b = pl->inverse ? gi - 1 : gi;   // the boundary this pass's outputs cross, if any
      if (pl->inverse ? (di == 0 && gi > 0) : (di + 1 == digits.size() && gi + 1 < groups.size())) {
        q.tw = (int)b;
        q.tw_S = 0;
        for (size_t j = 0; j < b; j++) q.tw_S += groups[j];
      }
      Src f;
      f.net = hv.size();
      hv.resize(f.net + (size_t)R * R);
      net_matrix(F, pow_2k(F, h, m - q.k), q.k, s == 0 && pl->inverse ? scale : host::one(F), hv.data() + f.net);
      f.pw = powers((size_t)1 << (q.k + q.u), host::one(F), pow_2k(F, h, S + q.Mp));
      f.dst = take((size_t)1024 << (2 * q.k + q.u));
      src.push_back(f);
      fwd.push_back(q);
      pl->passes.push_back({q.k, q.s, q.Mp});
      s += q.k;
    }
    if (gi + 1 < groups.size()) gtw[gi] = take((size_t)32 << (m - S));
  }
  // powers for the twiddles: h^e = A[e mod 2^a] B[e >> a], both in FP64 radix (x R -> x R')
  const int a = (m + 1) / 2;
  const size_t A = powers((size_t)1 << a, rp, h), B = powers((size_t)1 << (m - a), rp, pow_2k(F, h, a));
  const size_t o_hv = take(hv.size() * 32);
  if (cudaMalloc(&pl->d_mblk, bytes) != cudaSuccess) {
    (void)cudaGetLastError();
    pl->d_mblk = nullptr;
    return set_status(ZKG_ERR_NOMEM, "ntt plan", "matrices");
  }
  pl->bytes = bytes;
  char* base = static_cast<char*>(pl->d_mblk);
  const uint32_t* dh = reinterpret_cast<const uint32_t*>(base + o_hv);
  ZKB_CUDA(cudaMemcpyAsync(base + o_hv, hv.data(), hv.size() * 32, cudaMemcpyHostToDevice, st));
  for (size_t i = 0; i < fwd.size(); i++) {
    NttMatPass& q = fwd[i];
    q.d_mat = reinterpret_cast<uint8_t*>(base + src[i].dst);
    ZKB_TRY(ntt_mat_build<P>(dh + src[i].net * 8, dh + src[i].pw * 8, q.k, q.u, pl->inverse, q.nout, q.d_mat, st));
  }
  s = 0;
  for (size_t gi = 0; gi + 1 < groups.size(); gi++) {   // after group gi: h^((r kappa) << S)
    pl->d_gtw[gi] = reinterpret_cast<uint32_t*>(base + gtw[gi]);
    ZKB_TRY(ntt_mat_twiddles<P>(pl->d_gtw[gi], dh + A * 8, dh + B * 8, a, m - s - groups[gi], s, 1u << (m - s), st));
    s += groups[gi];
  }
  if (pl->inverse) std::reverse(fwd.begin(), fwd.end());
  pl->mpasses = fwd;
  ZKB_CUDA(cudaStreamSynchronize(st));
  return ZKG_OK;
}

template <class P>
static zkg_status build_plan_uncached(const host::Field<4>& F, int curve, int m, const uint64_t* gen, int inverse,
                                      int kmax, bool mat, cudaStream_t stream, NttPlan** out) {
  NttPlan* pl = new NttPlan();
  pl->curve = curve;
  pl->m = m;
  pl->inverse = inverse;
  pl->kmax = kmax;
  std::memcpy(pl->gen, gen, 32);
  pl->dpf = g_ntt_dpf != 0;
  // tables in radix R' when the passes multiply on the FP64 pipe: x R -> x R R' / R
  using PD = typename DpfOf<P>::type;
  host::El<4> rp = host::zero<4>();   // R' mod r as a standard integer
  for (int w = 0; w < 8; w++) rp.v[w >> 1] |= (uint64_t)PD::one(w) << (32 * (w & 1));
  auto conv = [&](std::vector<host::El<4>>& v) {
    if (pl->dpf)
      for (auto& e : v) e = host::mul(F, e, rp);
  };
  host::El<4> g = el_from_u64<4>(gen);
  host::El<4> h = inverse ? host::inv(F, g) : g;   // network generator
  // (1/2)^m, the inverse's final scale (bn128_poly_mont.c:565-622 halves at every level)
  host::El<4> scale = host::one(F);
  if (inverse) {
    host::El<4> two = host::zero<4>();
    two.v[0] = 2;
    scale = host::pow_u64(F, host::inv(F, host::from_std(F, two)), (uint64_t)m);
  }
  if (mat) {
    const zkg_status st = build_mat<P>(F, pl, h, scale, rp, stream);
    if (st != ZKG_OK) { delete pl; return st; }
    *out = pl;
    return ZKG_OK;
  }
  pl->passes = ntt_schedule(m, kmax);
  // small-network tables: w_k = h^(2^(m-k)), powers 0 .. 2^(k-1)-1
  for (const NttPass& q : pl->passes) {
    if (pl->d_om[q.k]) continue;
    host::El<4> w = h;
    for (int i = 0; i < m - q.k; i++) w = host::mul(F, w, w);
    std::vector<host::El<4>> tab((size_t)1 << (q.k - 1));
    host::El<4> x = host::one(F);
    for (auto& e : tab) { e = x; x = host::mul(F, x, w); }
    conv(tab);
    zkg_status st = upload(&pl->d_om[q.k], tab);
    if (st != ZKG_OK) { delete pl; return st; }
  }
  if (pl->passes.size() >= 2) {
    const uint32_t N = 1u << m;
    const int a = (m + 1) / 2;
    std::vector<host::El<4>> A((size_t)1 << a), Bt((size_t)1 << (m - a));
    host::El<4> x = host::one(F);
    for (auto& e : A) { e = x; x = host::mul(F, x, h); }
    const host::El<4> step = x;   // h^(2^a)
    x = host::one(F);
    for (auto& e : Bt) { e = x; x = host::mul(F, x, step); }
    // the inverse's last pass multiplies its inputs by the twiddles anyway: a copy of the table
    // scaled by (1/2)^m (A[j] (1/2)^m times Bt[i]) folds the final scale into that product
    std::vector<host::El<4>> As;
    if (inverse)
      for (const auto& e : A) As.push_back(host::mul(F, e, scale));
    conv(A);
    conv(Bt);
    conv(As);
    uint32_t *dA = nullptr, *dB = nullptr, *dAs = nullptr;
    zkg_status st = upload(&dA, A);
    if (st == ZKG_OK) st = upload(&dB, Bt);
    if (st == ZKG_OK && inverse) st = upload(&dAs, As);
    if (st == ZKG_OK && (cudaMalloc(&pl->d_tw, (size_t)N * 32) != cudaSuccess ||
                         (inverse && cudaMalloc(&pl->d_tw_last, (size_t)N * 32) != cudaSuccess))) {
      (void)cudaGetLastError();
      st = set_status(ZKG_ERR_NOMEM, "ntt plan", "twiddle table");
    }
    if (st == ZKG_OK)
      st = pl->dpf ? ntt_launch_table<PD>(pl->d_tw, dA, dB, a, N, stream)
                   : ntt_launch_table<P>(pl->d_tw, dA, dB, a, N, stream);
    if (st == ZKG_OK && inverse)
      st = pl->dpf ? ntt_launch_table<PD>(pl->d_tw_last, dAs, dB, a, N, stream)
                   : ntt_launch_table<P>(pl->d_tw_last, dAs, dB, a, N, stream);
    if (st == ZKG_OK && cudaStreamSynchronize(stream) != cudaSuccess) st = set_status(ZKG_ERR_CUDA, "ntt plan", "sync");
    if (dA) cudaFree(dA);
    if (dB) cudaFree(dB);
    if (dAs) cudaFree(dAs);
    if (st != ZKG_OK) { delete pl; return st; }
    pl->bytes += (size_t)N * 32 * (inverse ? 2 : 1);
  }
  if (inverse) {
    std::vector<host::El<4>> sc(1, scale);
    conv(sc);
    zkg_status st = upload(&pl->d_scale, sc);
    if (st != ZKG_OK) { delete pl; return st; }
  }
  *out = pl;
  return ZKG_OK;
}

template <class P>
static zkg_status build_plan(Context& cx, const host::Field<4>& F, int curve, int m, const uint64_t* gen, int inverse,
                             NttPlan** out) {
  for (NttPlan* p : cx.ntt_plans)
    if (p->curve == curve && p->m == m && p->inverse == inverse && p->kmax == effective_kmax(curve, m) &&
        p->dpf == (g_ntt_dpf != 0) && p->mat == ntt_use_mat(m) && std::memcmp(p->gen, gen, 32) == 0) {
      *out = p;
      return ZKG_OK;
    }
  NttPlan* pl = nullptr;
  ZKB_TRY(build_plan_uncached<P>(F, curve, m, gen, inverse, effective_kmax(curve, m), ntt_use_mat(m), cx.stream, &pl));
  // bounded cache: drop the oldest plans beyond 64 plans or 4 GiB of tables (a 2^24 forward and
  // inverse pair holds 1.5 GiB)
  cx.ntt_plans.push_back(pl);
  auto table_bytes = [&] {
    size_t b = 0;
    for (NttPlan* p : cx.ntt_plans) b += p->bytes;
    return b;
  };
  while (cx.ntt_plans.size() > 1 && (cx.ntt_plans.size() > 64 || table_bytes() > ((size_t)4 << 30))) {
    delete cx.ntt_plans.front();
    cx.ntt_plans.erase(cx.ntt_plans.begin());
  }
  *out = pl;
  return ZKG_OK;
}

// The calls on the context's stream, one at a time: its own fault word, cleared.
static zkg_status ntt_context_run(Context& cx, NttRun& run) {
  if (!cx.ntt_fault) ZKB_CUDA(cudaMallocHost(&cx.ntt_fault, sizeof(uint32_t)));
  *cx.ntt_fault = 0;
  run.fault = cx.ntt_fault;
  return ZKG_OK;
}

// Runs the plan d_src -> d_tgt; scratch (N elements) needed when there are >= 2 passes.
template <class P>
static zkg_status ntt_run(Context& cx, const NttPlan& pl, const uint32_t* d_src, uint32_t* d_tgt, uint32_t* scratch,
                          cudaStream_t st, const NttRun& run) {
  const int np = (int)pl.passes.size();
  const size_t N = (size_t)1 << pl.m;
  if (np == 0) {   // m = 0: copy (bn128_poly_mont.c:420-423)
    ZKB_CUDA(cudaMemcpyAsync(d_tgt, d_src, N * 32, cudaMemcpyDeviceToDevice, st));
    return ZKG_OK;
  }
  const uint32_t* in = d_src;
  for (int i = 0; i < np; i++) {
    // the i-th executed pass writes tgt when (np-1-i) is even, scratch otherwise
    uint32_t* out = ((np - 1 - i) % 2 == 0) ? d_tgt : scratch;
    const NttPass& q = pl.inverse ? pl.passes[np - 1 - i] : pl.passes[i];
    if (pl.mat) ZKB_TRY(ntt_mat_launch_pass<P>(pl, i, in, out, cx.sm_count, run, st));
    else if (pl.dpf) ZKB_TRY(ntt_launch_pass<typename DpfOf<P>::type>(pl, q, in, out, pl.inverse && i == np - 1, st));
    else ZKB_TRY(ntt_launch_pass<P>(pl, q, in, out, pl.inverse && i == np - 1, st));
    in = out;
  }
  return ZKG_OK;
}

template <class P>
static zkg_status ntt_entry(const host::Field<4>& F, int curve, int m, const uint64_t* gen, const uint64_t* src,
                            uint64_t* tgt, int inverse, bool device_ptrs) {
  NvtxRange nvtx("zkb.ntt");
  if (m < 0 || m > NTT_MMAX) return set_status(ZKG_ERR_ARG, "ntt", "m out of range [0, 30]");
  if (!gen || !src || !tgt) return set_status(ZKG_ERR_ARG, "ntt", "null pointer");
  if (src == tgt) return set_status(ZKG_ERR_ARG, "ntt", "src and tgt must not alias");
  Context* cxp = nullptr;
  ZKB_TRY(get_context(&cxp));
  Context& cx = *cxp;
  std::lock_guard<std::mutex> lk(cx.mu);
  NttPlan* pl = nullptr;
  ZKB_TRY(build_plan<P>(cx, F, curve, m, gen, inverse, &pl));
  NttRun run;
  ZKB_TRY(ntt_context_run(cx, run));
  const size_t N = (size_t)1 << m, bytes = N * 32, rb = (bytes + 255) & ~size_t(255);
  const bool need_scratch = pl->passes.size() >= 2;
  if (device_ptrs) {
    ZKB_TRY(cx.arena.reserve(need_scratch ? rb : 256));
    cx.arena.reset();
    uint32_t* scratch = static_cast<uint32_t*>(cx.arena.take(need_scratch ? bytes : 32));
    const cudaStream_t st = cx.compute();
    if (!cx.user_stream) ZKB_CUDA(cudaDeviceSynchronize());   // inputs may come from any stream
    ZKB_CUDA(cudaEventRecord(cx.ev_a, st));
    ZKB_TRY(ntt_run<P>(cx, *pl, reinterpret_cast<const uint32_t*>(src), reinterpret_cast<uint32_t*>(tgt), scratch,
                       st, run));
    ZKB_CUDA(cudaEventRecord(cx.ev_b, st));
    ZKB_CUDA(cudaStreamSynchronize(st));
  } else {
    ZKB_TRY(cx.arena.reserve(3 * rb));
    cx.arena.reset();
    uint32_t* d_src = static_cast<uint32_t*>(cx.arena.take(bytes));
    uint32_t* d_tgt = static_cast<uint32_t*>(cx.arena.take(bytes));
    uint32_t* scratch = static_cast<uint32_t*>(cx.arena.take(bytes));
    const cudaStream_t st = cx.compute();
    ZKB_TRY(copy_h2d(cx, d_src, src, bytes, st));
    ZKB_CUDA(cudaEventRecord(cx.ev_a, st));
    ZKB_TRY(ntt_run<P>(cx, *pl, d_src, d_tgt, scratch, st, run));
    ZKB_CUDA(cudaEventRecord(cx.ev_b, st));
    ZKB_TRY(copy_d2h(cx, tgt, d_tgt, bytes, st));
  }
  ZKB_CUDA(cudaEventElapsedTime(&cx.last_kernel_ms, cx.ev_a, cx.ev_b));
  ZKB_TRY(ntt_fault_report(cx.ntt_fault));
  return set_status(ZKG_OK, nullptr, nullptr);
}

// ------------------------------------------------------------- shifted / asymmetric NTT
// out[i] = in[i] * eta^i with eta^i = A[i mod 2^a] * Bt[i >> a]
template <class P>
__global__ void k_ntt_scale_pow(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t N,
                                const uint32_t* __restrict__ A, const uint32_t* __restrict__ Bt, int a) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const Fe<P> pw = fe_mul(fe_load_nc<P>(A + (size_t)(i & ((1u << a) - 1)) * 8), fe_load_nc<P>(Bt + (size_t)(i >> a) * 8));
  fe_store<P>(out + (size_t)i * 8, fe_mul(fe_load_nc<P>(in + (size_t)i * 8), pw));
}

// out[i K + k] = in[i]
__global__ void k_ntt_interleave(const uint4* __restrict__ in, uint4* __restrict__ out, uint32_t Ns, uint32_t K,
                                 uint32_t k) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Ns) return;
  out[((size_t)i * K + k) * 2] = in[(size_t)i * 2];
  out[((size_t)i * K + k) * 2 + 1] = in[(size_t)i * 2 + 1];
}

// Powers eta^j (j < 2^a) and eta^(j 2^a) (j < 2^(m-a)) for the scaling kernel.
static void pow_tables(const host::Field<4>& F, const host::El<4>& eta, int m, int a, std::vector<host::El<4>>& A,
                       std::vector<host::El<4>>& Bt) {
  A.assign((size_t)1 << a, host::El<4>());
  Bt.assign((size_t)1 << (m - a), host::El<4>());
  host::El<4> x = host::one(F);
  for (auto& e : A) { e = x; x = host::mul(F, x, eta); }
  const host::El<4> step = x;
  x = host::one(F);
  for (auto& e : Bt) { e = x; x = host::mul(F, x, step); }
}

// Shifted (coset) NTT on host buffers: forward = NTT of src[i] eta^i
// (bn128_poly_mont.c:477-488); inverse = inverse NTT, then output i times eta^i (:626-641).
template <class P>
static zkg_status ntt_shifted_entry(const host::Field<4>& F, int curve, const uint64_t* eta, int m,
                                   const uint64_t* gen, const uint64_t* src, uint64_t* tgt, int inverse) {
  if (m < 0 || m > NTT_MMAX) return set_status(ZKG_ERR_ARG, "ntt_shifted", "m out of range [0, 30]");
  if (!eta || !gen || !src || !tgt) return set_status(ZKG_ERR_ARG, "ntt_shifted", "null pointer");
  Context* cxp = nullptr;
  ZKB_TRY(get_context(&cxp));
  Context& cx = *cxp;
  std::lock_guard<std::mutex> lk(cx.mu);
  NttPlan* pl = nullptr;
  ZKB_TRY(build_plan<P>(cx, F, curve, m, gen, inverse, &pl));
  NttRun run;
  ZKB_TRY(ntt_context_run(cx, run));
  const size_t N = (size_t)1 << m, bytes = N * 32, rb = (bytes + 255) & ~size_t(255);
  const int a = (m + 1) / 2;
  std::vector<host::El<4>> A, Bt;
  host::El<4> e;
  std::memcpy(e.v, eta, 32);
  pow_tables(F, e, m, a, A, Bt);
  const size_t tb = ((A.size() + Bt.size()) * 32 + 511) & ~size_t(255);
  ZKB_TRY(cx.arena.reserve(4 * rb + tb));
  cx.arena.reset();
  uint32_t* d_a = static_cast<uint32_t*>(cx.arena.take(bytes));
  uint32_t* d_b = static_cast<uint32_t*>(cx.arena.take(bytes));
  uint32_t* d_c = static_cast<uint32_t*>(cx.arena.take(bytes));
  uint32_t* scratch = static_cast<uint32_t*>(cx.arena.take(bytes));
  uint32_t* dA = static_cast<uint32_t*>(cx.arena.take(A.size() * 32));
  uint32_t* dB = static_cast<uint32_t*>(cx.arena.take(Bt.size() * 32));
  const cudaStream_t st = cx.compute();
  ZKB_CUDA(cudaMemcpyAsync(dA, A.data(), A.size() * 32, cudaMemcpyHostToDevice, st));
  ZKB_CUDA(cudaMemcpyAsync(dB, Bt.data(), Bt.size() * 32, cudaMemcpyHostToDevice, st));
  ZKB_TRY(copy_h2d(cx, d_a, src, bytes, st));
  ZKB_CUDA(cudaEventRecord(cx.ev_a, st));
  const dim3 g((uint32_t)((N + 255) / 256));
  if (!inverse) {
    ZKB_TRY(launch("ntt_scale_pow", k_ntt_scale_pow<P>, g, dim3(256), 0, st, (const uint32_t*)d_a, d_b, (uint32_t)N,
                   (const uint32_t*)dA, (const uint32_t*)dB, a));
    ZKB_TRY(ntt_run<P>(cx, *pl, d_b, d_c, scratch, st, run));
  } else {
    ZKB_TRY(ntt_run<P>(cx, *pl, d_a, d_b, scratch, st, run));
    ZKB_TRY(launch("ntt_scale_pow", k_ntt_scale_pow<P>, g, dim3(256), 0, st, (const uint32_t*)d_b, d_c, (uint32_t)N,
                   (const uint32_t*)dA, (const uint32_t*)dB, a));
  }
  ZKB_CUDA(cudaEventRecord(cx.ev_b, st));
  ZKB_TRY(copy_d2h(cx, tgt, d_c, bytes, st));
  ZKB_CUDA(cudaEventElapsedTime(&cx.last_kernel_ms, cx.ev_a, cx.ev_b));
  ZKB_TRY(ntt_fault_report(cx.ntt_fault));
  return set_status(ZKG_OK, nullptr, nullptr);
}

// Asymmetric NTT (bn128_poly_mont.c:492-555): for k < K = 2^(m_tgt - m_src), the forward NTT
// (generator gen_src) of src[i] gen_tgt^(k i), written to tgt[i K + k].
template <class P>
static zkg_status ntt_asym_entry(const host::Field<4>& F, int curve, int m_src, int m_tgt, const uint64_t* gen_src,
                                 const uint64_t* gen_tgt, const uint64_t* src, uint64_t* tgt) {
  if (m_src < 0 || m_tgt < m_src || m_tgt > NTT_MMAX)
    return set_status(ZKG_ERR_ARG, "ntt_asymmetric", "need 0 <= m_src <= m_tgt <= 30");
  if (!gen_src || !gen_tgt || !src || !tgt) return set_status(ZKG_ERR_ARG, "ntt_asymmetric", "null pointer");
  Context* cxp = nullptr;
  ZKB_TRY(get_context(&cxp));
  Context& cx = *cxp;
  std::lock_guard<std::mutex> lk(cx.mu);
  NttPlan* pl = nullptr;
  ZKB_TRY(build_plan<P>(cx, F, curve, m_src, gen_src, 0, &pl));
  NttRun run;
  ZKB_TRY(ntt_context_run(cx, run));
  const size_t Ns = (size_t)1 << m_src, K = (size_t)1 << (m_tgt - m_src), bs = Ns * 32;
  const size_t rbs = (bs + 255) & ~size_t(255), bt = Ns * K * 32, rbt = (bt + 255) & ~size_t(255);
  const int a = (m_src + 1) / 2;
  const size_t tb = ((((size_t)1 << a) + ((size_t)1 << (m_src - a))) * 32 + 511) & ~size_t(255);
  ZKB_TRY(cx.arena.reserve(4 * rbs + rbt + tb));
  cx.arena.reset();
  uint32_t* d_src = static_cast<uint32_t*>(cx.arena.take(bs));
  uint32_t* d_sh = static_cast<uint32_t*>(cx.arena.take(bs));
  uint32_t* d_out = static_cast<uint32_t*>(cx.arena.take(bs));
  uint32_t* scratch = static_cast<uint32_t*>(cx.arena.take(bs));
  uint32_t* d_tgt = static_cast<uint32_t*>(cx.arena.take(bt));
  uint32_t* dA = static_cast<uint32_t*>(cx.arena.take(((size_t)32) << a));
  uint32_t* dB = static_cast<uint32_t*>(cx.arena.take(((size_t)32) << (m_src - a)));
  const cudaStream_t st = cx.compute();
  ZKB_TRY(copy_h2d(cx, d_src, src, bs, st));
  ZKB_CUDA(cudaEventRecord(cx.ev_a, st));
  host::El<4> gt, eta = host::one(F);
  std::memcpy(gt.v, gen_tgt, 32);
  std::vector<host::El<4>> A, Bt;
  const dim3 g((uint32_t)((Ns + 255) / 256));
  for (size_t k = 0; k < K; k++) {
    if (k) eta = host::mul(F, eta, gt);
    pow_tables(F, eta, m_src, a, A, Bt);
    ZKB_CUDA(cudaMemcpyAsync(dA, A.data(), A.size() * 32, cudaMemcpyHostToDevice, st));
    ZKB_CUDA(cudaMemcpyAsync(dB, Bt.data(), Bt.size() * 32, cudaMemcpyHostToDevice, st));
    ZKB_TRY(launch("ntt_scale_pow", k_ntt_scale_pow<P>, g, dim3(256), 0, st, (const uint32_t*)d_src, d_sh,
                   (uint32_t)Ns, (const uint32_t*)dA, (const uint32_t*)dB, a));
    ZKB_TRY(ntt_run<P>(cx, *pl, d_sh, d_out, scratch, st, run));
    ZKB_TRY(launch("ntt_interleave", k_ntt_interleave, g, dim3(256), 0, st, (const uint4*)d_out, (uint4*)d_tgt,
                   (uint32_t)Ns, (uint32_t)K, (uint32_t)k));
    ZKB_CUDA(cudaStreamSynchronize(st));   // the host-side tables are rewritten for the next k
  }
  ZKB_CUDA(cudaEventRecord(cx.ev_b, st));
  ZKB_TRY(copy_d2h(cx, tgt, d_tgt, bt, st));
  ZKB_CUDA(cudaEventElapsedTime(&cx.last_kernel_ms, cx.ev_a, cx.ev_b));
  ZKB_TRY(ntt_fault_report(cx.ntt_fault));
  return set_status(ZKG_OK, nullptr, nullptr);
}

zkg_status ntt_plan_new(int curve, int m, const uint64_t* gen, int inverse, int kmax, cudaStream_t st,
                        NttPlan** out, bool tiles) {
  if (m < 0 || m > NTT_MMAX) return set_status(ZKG_ERR_ARG, "ntt", "m out of range [0, 30]");
  const bool mat = !tiles && kmax <= 0 && ntt_use_mat(m);
  if (kmax <= 0) kmax = effective_kmax(curve, m);
  if (curve == ZKG_BN254) return build_plan_uncached<BnFr>(host::BN_FR, curve, m, gen, inverse, kmax, mat, st, out);
  if (curve == ZKG_BLS12_381) return build_plan_uncached<BlsFr>(host::BLS_FR, curve, m, gen, inverse, kmax, mat, st, out);
  return set_status(ZKG_ERR_ARG, "ntt", "unknown curve");
}

zkg_status ntt_fault_report(uint32_t* word) {
  volatile uint32_t* w = word;
  if (!w || !*w) return ZKG_OK;
  *w = 0;
  return set_status(ZKG_ERR_TIMEOUT, "ntt", "a bounded wait inside a pass ran out");
}

zkg_status ntt_plan_execute(const NttPlan& pl, const uint32_t* d_src, uint32_t* d_tgt, uint32_t* scratch,
                            cudaStream_t st, const NttRun& run) {
  Context* cx = nullptr;
  ZKB_TRY(get_context(&cx));
  if (pl.curve == ZKG_BN254) return ntt_run<BnFr>(*cx, pl, d_src, d_tgt, scratch, st, run);
  return ntt_run<BlsFr>(*cx, pl, d_src, d_tgt, scratch, st, run);
}

}  // namespace zkb

extern "C" {

zkg_status zkg_ntt(zkg_curve curve, int m, const uint64_t* gen, const uint64_t* src, uint64_t* tgt, int inverse) {
  if (curve == ZKG_BN254) return zkb::ntt_entry<zkb::BnFr>(zkb::host::BN_FR, curve, m, gen, src, tgt, inverse, false);
  if (curve == ZKG_BLS12_381)
    return zkb::ntt_entry<zkb::BlsFr>(zkb::host::BLS_FR, curve, m, gen, src, tgt, inverse, false);
  return zkb::set_status(ZKG_ERR_ARG, "zkg_ntt", "unknown curve");
}

zkg_status zkg_ntt_device(zkg_curve curve, int m, const uint64_t* gen, const uint64_t* d_src, uint64_t* d_tgt,
                          int inverse) {
  if (curve == ZKG_BN254) return zkb::ntt_entry<zkb::BnFr>(zkb::host::BN_FR, curve, m, gen, d_src, d_tgt, inverse, true);
  if (curve == ZKG_BLS12_381)
    return zkb::ntt_entry<zkb::BlsFr>(zkb::host::BLS_FR, curve, m, gen, d_src, d_tgt, inverse, true);
  return zkb::set_status(ZKG_ERR_ARG, "zkg_ntt_device", "unknown curve");
}

zkg_status zkg_ntt_shifted(zkg_curve curve, const uint64_t* eta, int m, const uint64_t* gen, const uint64_t* src,
                           uint64_t* tgt, int inverse) {
  if (curve == ZKG_BN254) return zkb::ntt_shifted_entry<zkb::BnFr>(zkb::host::BN_FR, curve, eta, m, gen, src, tgt, inverse);
  if (curve == ZKG_BLS12_381)
    return zkb::ntt_shifted_entry<zkb::BlsFr>(zkb::host::BLS_FR, curve, eta, m, gen, src, tgt, inverse);
  return zkb::set_status(ZKG_ERR_ARG, "zkg_ntt_shifted", "unknown curve");
}

zkg_status zkg_ntt_asymmetric(zkg_curve curve, int m_src, int m_tgt, const uint64_t* gen_src, const uint64_t* gen_tgt,
                              const uint64_t* src, uint64_t* tgt) {
  if (curve == ZKG_BN254)
    return zkb::ntt_asym_entry<zkb::BnFr>(zkb::host::BN_FR, curve, m_src, m_tgt, gen_src, gen_tgt, src, tgt);
  if (curve == ZKG_BLS12_381)
    return zkb::ntt_asym_entry<zkb::BlsFr>(zkb::host::BLS_FR, curve, m_src, m_tgt, gen_src, gen_tgt, src, tgt);
  return zkb::set_status(ZKG_ERR_ARG, "zkg_ntt_asymmetric", "unknown curve");
}

zkg_status zkg_release_cache(void) {
  zkb::Context* cx = nullptr;
  zkg_status st = zkb::get_context(&cx);
  if (st != ZKG_OK) return st;
  std::lock_guard<std::mutex> lk(cx->mu);
  cudaDeviceSynchronize();
  for (zkb::NttPlan* p : cx->ntt_plans) delete p;
  cx->ntt_plans.clear();
  if (cx->arena.base) cudaFree(cx->arena.base);
  cx->arena.base = nullptr;
  cx->arena.cap = cx->arena.used = 0;
  return ZKG_OK;
}

int zkg_set_ntt_kmax(int k) {
  const int prev = zkb::g_ntt_kmax;
  if (k >= 1 && k <= zkb::NTT_KMAX) {
    zkb::g_ntt_kmax = k;
    zkb::g_ntt_kmax_set = true;
  } else if (k == 0) {
    zkb::g_ntt_kmax = 8;
    zkb::g_ntt_kmax_set = false;
  }
  return prev;
}

// Times the largest pass size 7..11 for each m in [m_min, m_max] (forward transform on random
// device data) and keeps the fastest per size.
zkg_status zkg_autotune_ntt(zkg_curve curve, int m_min, int m_max, int* chosen) {
  if ((curve != ZKG_BN254 && curve != ZKG_BLS12_381) || m_min < 1 || m_max < m_min || m_max > 26)
    return zkb::set_status(ZKG_ERR_ARG, "zkg_autotune_ntt", "need 1 <= m_min <= m_max <= 26");
  uint32_t *d_x = nullptr, *d_y = nullptr;
  const size_t bytes = (size_t)32 << m_max;
  if (cudaMalloc(&d_x, bytes) != cudaSuccess || cudaMalloc(&d_y, bytes) != cudaSuccess) {
    if (d_x) cudaFree(d_x);
    return zkb::set_status(ZKG_ERR_NOMEM, "zkg_autotune_ntt", "buffers");
  }
  cudaMemset(d_x, 0x11, bytes);   // below both moduli word-wise; timing does not depend on values
  const uint64_t gen[4] = {0x0123456789abcdefULL, 0x0fedcba987654321ULL, 0x1111111111111111ULL, 0x0222222222222222ULL};
  const bool was_set = zkb::g_ntt_kmax_set;
  const int was_k = zkb::g_ntt_kmax;
  zkg_status st = ZKG_OK;
  for (int m = m_min; m <= m_max && st == ZKG_OK; m++) {
    float best = 1e30f;
    int bestk = 8;
    for (int k = 6; k <= zkb::NTT_KMAX && st == ZKG_OK; k++) {
      zkb::g_ntt_kmax = k;
      zkb::g_ntt_kmax_set = true;
      float t = 1e30f;
      for (int rep = 0; rep < 3 && st == ZKG_OK; rep++) {
        st = zkg_ntt_device(curve, m, gen, reinterpret_cast<const uint64_t*>(d_x), reinterpret_cast<uint64_t*>(d_y), 0);
        if (rep > 0) t = std::min(t, zkg_last_kernel_ms());
      }
      if (st == ZKG_OK && t < best) { best = t; bestk = k; }
    }
    if (st == ZKG_OK) {
      zkb::effective_kmax(curve, m);   // loads the persisted entries first, so they are not lost
      zkb::g_ntt_tuned[curve][m] = bestk;
      zkb::tune_cache_put("ntt", curve, m, zkb::device_sm_count(), &bestk, 1);
      if (chosen) chosen[m - m_min] = bestk;
    }
  }
  zkb::g_ntt_kmax = was_k;
  zkb::g_ntt_kmax_set = was_set;
  cudaFree(d_x);
  cudaFree(d_y);
  return st;
}

}  // extern "C"
