// Runtime: per-device context, scratch arena, status reporting.
#include "zkb_runtime.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <thread>

namespace zkb {

static thread_local zkg_status t_last_status = ZKG_OK;
static thread_local char t_last_error[512] = {0};
std::atomic<uint64_t> g_launches{0};

zkg_status set_status(zkg_status s, const char* where, const char* detail) {
  t_last_status = s;
  if (s != ZKG_OK)
    std::snprintf(t_last_error, sizeof(t_last_error), "%s: %s", where ? where : "", detail ? detail : "");
  else
    t_last_error[0] = 0;
  return s;
}

zkg_status allow_smem(const void* kernel, size_t bytes) {
  ZKB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return ZKG_OK;
}

zkg_status Arena::reserve(size_t bytes) {
  if (bytes <= cap) return ZKG_OK;
  size_t free_bytes = 0, all = 0;   // what cannot fit is refused with the present buffer kept
  if (cudaMemGetInfo(&free_bytes, &all) == cudaSuccess && bytes > cap + free_bytes)
    return set_status(ZKG_ERR_NOMEM, "arena reserve", "more than the device has free");
  if (base) {
    cudaFree(base);
    base = nullptr;
    cap = 0;
  }
  size_t want = bytes + (bytes >> 3);   // 12.5% headroom against regrowth
  cudaError_t e = cudaMalloc(&base, want);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    base = nullptr;
    e = cudaMalloc(&base, bytes);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      base = nullptr;
      return set_status(ZKG_ERR_NOMEM, "arena reserve", cudaGetErrorString(e));
    }
    want = bytes;
  }
  cap = want;
  used = 0;
  return ZKG_OK;
}

static std::mutex g_ctx_mu;
static Context* g_ctx[64] = {nullptr};

zkg_status get_context(Context** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return set_status(ZKG_ERR_CUDA, "cudaGetDevice", cudaGetErrorString(e));
  if (dev < 0 || dev >= 64) return set_status(ZKG_ERR_ARG, "get_context", "device index out of range");
  std::lock_guard<std::mutex> lk(g_ctx_mu);
  if (!g_ctx[dev]) {
    Context* cx = new Context();
    cx->device = dev;
    ZKB_CUDA(cudaDeviceGetAttribute(&cx->sm_count, cudaDevAttrMultiProcessorCount, dev));
    ZKB_CUDA(cudaStreamCreateWithFlags(&cx->stream, cudaStreamNonBlocking));
    ZKB_CUDA(cudaStreamCreateWithFlags(&cx->copy_stream, cudaStreamNonBlocking));
    ZKB_CUDA(cudaEventCreateWithFlags(&cx->ev_copy, cudaEventDisableTiming));
    ZKB_CUDA(cudaEventCreate(&cx->ev_a));
    ZKB_CUDA(cudaEventCreate(&cx->ev_b));
    for (auto& e : cx->ev_phase) ZKB_CUDA(cudaEventCreate(&e));
    for (auto& e : cx->ev_part) ZKB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (auto& e : cx->ev_scal) ZKB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (auto& e : cx->ev_acc) ZKB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (auto& e : cx->ev_fold) ZKB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    ZKB_CUDA(cudaStreamCreateWithFlags(&cx->side_stream, cudaStreamNonBlocking));
    g_ctx[dev] = cx;
  }
  *out = g_ctx[dev];
  return ZKG_OK;
}

// ------------------------------------------------------------ staged host <-> device copies
namespace {
// A fixed pool of host threads for large memcpys (started on first use, lives to exit).
class CopyPool {
 public:
  static CopyPool& get() {   // never destroyed: its detached threads wait on it until exit
    static CopyPool* p = new CopyPool();
    return *p;
  }
  // dst[0, n) = src[0, n), split over the pool and the calling thread. Each call waits only for
  // its own pieces (a latch per call), so callers on other threads or devices never wait for
  // each other's copies.
  void memcpy_par(void* dst, const void* src, size_t n) {
    const size_t piece_min = size_t(2) << 20;
    const int parts = (int)std::min<size_t>(nthreads_ + 1, std::max<size_t>(1, n / piece_min));
    if (parts <= 1) {
      std::memcpy(dst, src, n);
      return;
    }
    const size_t piece = (n + parts - 1) / parts;
    Latch latch;
    {
      std::lock_guard<std::mutex> lk(mu_);
      for (int k = 1; k < parts; k++) {
        const size_t o = (size_t)k * piece;
        if (o >= n) break;
        jobs_.push_back({static_cast<char*>(dst) + o, static_cast<const char*>(src) + o, std::min(piece, n - o), &latch});
        latch.pending++;
      }
    }
    cv_.notify_all();
    std::memcpy(dst, src, std::min(piece, n));
    std::unique_lock<std::mutex> lk(mu_);
    latch.cv.wait(lk, [&] { return latch.pending == 0; });
  }

 private:
  struct Latch {   // pieces of one call still being copied (guarded by mu_)
    int pending = 0;
    std::condition_variable cv;
  };
  struct Job {
    char* dst;
    const char* src;
    size_t n;
    Latch* latch;
  };
  CopyPool() {
    const unsigned hw = std::thread::hardware_concurrency();
    nthreads_ = (int)std::max(1u, std::min(7u, hw > 1 ? hw / 2 : 1u));
    for (int i = 0; i < nthreads_; i++) std::thread([this] { run(); }).detach();
  }
  void run() {
    for (;;) {
      Job j;
      {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return !jobs_.empty(); });
        j = jobs_.back();
        jobs_.pop_back();
      }
      std::memcpy(j.dst, j.src, j.n);
      {
        // notify under the lock: the waiting caller owns the latch and may return (destroying
        // it) as soon as it sees pending == 0
        std::lock_guard<std::mutex> lk(mu_);
        if (--j.latch->pending == 0) j.latch->cv.notify_all();
      }
    }
  }
  int nthreads_ = 1;
  std::mutex mu_;
  std::condition_variable cv_;
  std::vector<Job> jobs_;
};

const bool g_stage = [] {
  const char* v = std::getenv("ZKB_STAGE");
  return !(v && v[0] == '0');
}();
constexpr size_t STAGE_CHUNK = size_t(32) << 20;
constexpr size_t STAGE_MIN = size_t(4) << 20;   // below this the driver's own staging is as good

bool page_locked(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

// Page-locked staging slots and their events, created once per context. A slot or event that was
// created before a failure is kept and reused by the next call (nothing is created twice).
zkg_status stage_reserve(Context& cx) {
  if (cx.stage_bytes >= STAGE_CHUNK) return ZKG_OK;
  for (int k = 0; k < Context::NSTAGE; k++) {
    if (!cx.stage[k]) {
      void* p = nullptr;
      const cudaError_t e = cudaMallocHost(&p, STAGE_CHUNK);
      if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return set_status(ZKG_ERR_NOMEM, "cudaMallocHost (staging)", cudaGetErrorString(e));
      }
      cx.stage[k] = p;
    }
    if (!cx.stage_ev[k]) {
      cudaEvent_t ev = nullptr;
      const cudaError_t e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
      if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return set_status(ZKG_ERR_CUDA, "cudaEventCreate (staging)", cudaGetErrorString(e));
      }
      cx.stage_ev[k] = ev;
    }
  }
  cx.stage_bytes = STAGE_CHUNK;
  return ZKG_OK;
}
}  // namespace

zkg_status copy_h2d(Context& cx, void* dst, const void* src, size_t bytes, cudaStream_t st) {
  if (!g_stage || bytes < STAGE_MIN || page_locked(src)) {
    ZKB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
    return ZKG_OK;
  }
  ZKB_TRY(stage_reserve(cx));
  for (size_t o = 0; o < bytes; o += STAGE_CHUNK) {
    const size_t n = std::min(STAGE_CHUNK, bytes - o);
    const int k = (int)(cx.stage_next++ % Context::NSTAGE);
    ZKB_CUDA(cudaEventSynchronize(cx.stage_ev[k]));   // the slot's previous DMA is done
    CopyPool::get().memcpy_par(cx.stage[k], static_cast<const char*>(src) + o, n);
    ZKB_CUDA(cudaMemcpyAsync(static_cast<char*>(dst) + o, cx.stage[k], n, cudaMemcpyHostToDevice, st));
    ZKB_CUDA(cudaEventRecord(cx.stage_ev[k], st));
  }
  return ZKG_OK;
}

zkg_status copy_d2h(Context& cx, void* dst, const void* src, size_t bytes, cudaStream_t st) {
  if (!g_stage || bytes < STAGE_MIN || page_locked(dst)) {
    ZKB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
    ZKB_CUDA(cudaStreamSynchronize(st));
    return ZKG_OK;
  }
  ZKB_TRY(stage_reserve(cx));
  // DMA chunk c into a slot, then copy chunk c - 1 out of its slot while chunk c is in flight
  const size_t nch = (bytes + STAGE_CHUNK - 1) / STAGE_CHUNK;
  int slot_of[2] = {0, 0};
  for (size_t c = 0; c <= nch; c++) {
    if (c < nch) {
      const size_t o = c * STAGE_CHUNK, n = std::min(STAGE_CHUNK, bytes - o);
      const int k = (int)(cx.stage_next++ % Context::NSTAGE);
      ZKB_CUDA(cudaEventSynchronize(cx.stage_ev[k]));
      ZKB_CUDA(cudaMemcpyAsync(cx.stage[k], static_cast<const char*>(src) + o, n, cudaMemcpyDeviceToHost, st));
      ZKB_CUDA(cudaEventRecord(cx.stage_ev[k], st));
      slot_of[c & 1] = k;
    }
    if (c > 0) {
      const size_t o = (c - 1) * STAGE_CHUNK, n = std::min(STAGE_CHUNK, bytes - o);
      const int k = slot_of[(c - 1) & 1];
      ZKB_CUDA(cudaEventSynchronize(cx.stage_ev[k]));
      CopyPool::get().memcpy_par(static_cast<char*>(dst) + o, cx.stage[k], n);
    }
  }
  return ZKG_OK;
}

// ----------------------------------------------------------------- persisted tuning
namespace {
std::mutex g_tune_mu;
bool g_tune_loaded = false;
std::map<std::string, std::vector<int>> g_tune_map;   // "<kind> <curve> <size> <sms>" -> values

std::string tune_key(const char* kind, int curve, int size, int sms) {
  char b[96];
  std::snprintf(b, sizeof(b), "%s %d %d %d", kind, curve, size, sms);
  return b;
}

void tune_load_locked() {
  if (g_tune_loaded) return;
  g_tune_loaded = true;
  const char* path = std::getenv("ZKG_TUNE_CACHE");
  if (!path || !path[0]) return;
  FILE* f = std::fopen(path, "r");
  if (!f) return;
  char line[512];
  while (std::fgets(line, sizeof(line), f)) {
    char kind[32];
    int curve, size, sms, used = 0;
    if (std::sscanf(line, "%31s %d %d %d%n", kind, &curve, &size, &sms, &used) != 4) continue;
    std::vector<int> v;
    const char* q = line + used;
    int x, n;
    while (std::sscanf(q, "%d%n", &x, &n) == 1) {
      v.push_back(x);
      q += n;
    }
    g_tune_map[tune_key(kind, curve, size, sms)] = v;
  }
  std::fclose(f);
}
}  // namespace

bool tune_cache_get(const char* kind, int curve, int size, int sms, int* vals, int nvals) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  tune_load_locked();
  auto it = g_tune_map.find(tune_key(kind, curve, size, sms));
  if (it == g_tune_map.end() || (int)it->second.size() < nvals) return false;
  for (int i = 0; i < nvals; i++) vals[i] = it->second[i];
  return true;
}

void tune_cache_put(const char* kind, int curve, int size, int sms, const int* vals, int nvals) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  tune_load_locked();
  g_tune_map[tune_key(kind, curve, size, sms)] = std::vector<int>(vals, vals + nvals);
  const char* path = std::getenv("ZKG_TUNE_CACHE");
  if (!path || !path[0]) return;
  const std::string tmp = std::string(path) + ".tmp";
  FILE* f = std::fopen(tmp.c_str(), "w");
  if (!f) return;
  for (const auto& kv : g_tune_map) {
    std::fprintf(f, "%s", kv.first.c_str());
    for (int x : kv.second) std::fprintf(f, " %d", x);
    std::fprintf(f, "\n");
  }
  std::fclose(f);
  std::rename(tmp.c_str(), path);
}

int device_sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return sms;
}

const bool g_dev_checks = [] {
  const char* v = std::getenv("ZKB_DEVICE_CHECKS");
  return v && v[0] == '1';
}();

uint32_t* dev_check_word(Context& cx) {
  if (!g_dev_checks) return nullptr;
  if (!cx.d_check) {
    if (cudaMalloc(&cx.d_check, 4) != cudaSuccess || cudaMemset(cx.d_check, 0, 4) != cudaSuccess) {
      (void)cudaGetLastError();
      cx.d_check = nullptr;
    }
  }
  return cx.d_check;
}

zkg_status dev_check_report(Context& cx, const char* where) {
  if (!g_dev_checks || !cx.d_check) return ZKG_OK;
  uint32_t w = 0;
  ZKB_CUDA(cudaMemcpy(&w, cx.d_check, 4, cudaMemcpyDeviceToHost));
  if (!w) return ZKG_OK;
  ZKB_CUDA(cudaMemset(cx.d_check, 0, 4));
  char msg[128];
  std::snprintf(msg, sizeof(msg), "device bounds check failed (word 0x%x: 1 bucket, 2 entry, 4 point, 8 segment)", w);
  return set_status(ZKG_ERR_CUDA, where, msg);
}

zkg_status pinned_reserve(Context& cx, size_t bytes) {
  if (bytes <= cx.pinned_cap) return ZKG_OK;
  if (cx.pinned) cudaFreeHost(cx.pinned);
  cx.pinned = nullptr;
  cx.pinned_cap = 0;
  ZKB_CUDA(cudaMallocHost(&cx.pinned, bytes));
  cx.pinned_cap = bytes;
  return ZKG_OK;
}

}  // namespace zkb

namespace zkb {
// Issue-rate probes: every thread runs 8 independent dependency chains of one instruction kind.
//   kind 0 mad.lo.u32 (IMAD), 1 mad.hi.u32, 2 mad.wide.u32, 3 fma.rn.f64
template <int KIND>
__global__ void k_pipe_probe(uint32_t* out, int iters, uint32_t a, uint32_t b) {
  uint32_t x[8];
  uint64_t w[8];
  double d[8];
#pragma unroll
  for (int j = 0; j < 8; j++) { x[j] = threadIdx.x + j; w[j] = x[j]; d[j] = (double)x[j]; }
  const double da = 1.0000001, db = 1e-9;
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int j = 0; j < 8; j++) {
      if (KIND == 0) asm volatile("mad.lo.u32 %0, %0, %1, %2;" : "+r"(x[j]) : "r"(a), "r"(b));
      if (KIND == 1) asm volatile("mad.hi.u32 %0, %0, %1, %2;" : "+r"(x[j]) : "r"(a), "r"(b));
      if (KIND == 2) { const uint32_t lo = (uint32_t)w[j]; asm volatile("mad.wide.u32 %0, %1, %2, %0;" : "+l"(w[j]) : "r"(lo), "r"(a)); }
      if (KIND == 3) asm volatile("fma.rn.f64 %0, %0, %1, %2;" : "+d"(d[j]) : "d"(da), "d"(db));
    }
  }
  uint64_t s = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) s ^= x[j] ^ w[j] ^ (uint64_t)d[j];
  if (s == 0x9e3779b9u) out[0] = (uint32_t)s;   // keeps the chains live
}

}  // namespace zkb

extern "C" {

zkg_status zkg_last_status(void) { return zkb::t_last_status; }
const char* zkg_last_error(void) { return zkb::t_last_error; }
uint64_t zkg_kernel_launches(void) { return zkb::g_launches.load(); }

float zkg_last_kernel_ms(void) {
  zkb::Context* cx = nullptr;
  if (zkb::get_context(&cx) != ZKG_OK) return -1.f;
  return cx->last_kernel_ms;
}

zkg_status zkg_set_stream(void* stream) {
  zkb::Context* cx = nullptr;
  zkg_status st = zkb::get_context(&cx);
  if (st != ZKG_OK) return st;
  std::lock_guard<std::mutex> lk(cx->mu);
  cx->user_stream = static_cast<cudaStream_t>(stream);
  return ZKG_OK;
}

int zkg_last_phase_ms(float* out, int max) {
  zkb::Context* cx = nullptr;
  if (zkb::get_context(&cx) != ZKG_OK) return 0;
  const int n = cx->nphase < max ? cx->nphase : max;
  for (int i = 0; i < n; i++) out[i] = cx->last_phase_ms[i];
  return n;
}

double zkg_pipe_probe(int kind) {
  zkb::Context* cx = nullptr;
  if (zkb::get_context(&cx) != ZKG_OK || kind < 0 || kind > 3) return -1.0;
  std::lock_guard<std::mutex> lk(cx->mu);
  uint32_t* d = nullptr;
  if (cudaMalloc(&d, 64) != cudaSuccess) return -1.0;
  const int iters = 4096, threads = 256, blocks = cx->sm_count * 8;
  double best = 0.0;
  for (int rep = 0; rep < 4; rep++) {
    cudaEventRecord(cx->ev_a, cx->stream);
    switch (kind) {
      case 0: zkb::k_pipe_probe<0><<<blocks, threads, 0, cx->stream>>>(d, iters, 0x01000193u, 0x811c9dc5u); break;
      case 1: zkb::k_pipe_probe<1><<<blocks, threads, 0, cx->stream>>>(d, iters, 0x01000193u, 0x811c9dc5u); break;
      case 2: zkb::k_pipe_probe<2><<<blocks, threads, 0, cx->stream>>>(d, iters, 0x01000193u, 0x811c9dc5u); break;
      default: zkb::k_pipe_probe<3><<<blocks, threads, 0, cx->stream>>>(d, iters, 0x01000193u, 0x811c9dc5u); break;
    }
    zkb::g_launches.fetch_add(1);
    cudaEventRecord(cx->ev_b, cx->stream);
    if (cudaStreamSynchronize(cx->stream) != cudaSuccess) { cudaFree(d); return -1.0; }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, cx->ev_a, cx->ev_b);
    const double n = (double)blocks * threads * iters * 8.0;
    if (rep > 0 && ms > 0) best = std::max(best, n / (ms * 1e-3));
  }
  cudaFree(d);
  return best;
}

double zkg_imad_probe(void) { return zkg_pipe_probe(0); }

}  // extern "C"
