// gsknn_api.cu -- the C ABI of libgsknn.so (declared in include/gsknn.h).
//
// Host-pointer entry points (the reference API) copy the referenced row range of each point
// table, the index lists and the heap rows to the GPU, run the device pipeline, copy D/I back
// and return when done. Device-pointer entry points (gsknn_*_device) enqueue the same pipeline
// on a caller stream. Scratch memory comes from a cache keyed by (device, stream, slot).
#include "gsknn.h"
#include "knn_internal.h"

#include <cmath>
#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <tuple>
#include <type_traits>
#include <thread>
#include <vector>

#if defined(__x86_64__)
#include <emmintrin.h>
#endif

namespace gsknn {

// ------------------------------------------------------------------------------------------
// status
// ------------------------------------------------------------------------------------------
static thread_local int t_status = 0;
static thread_local char t_msg[512] = "ok";

int set_status(int code, const char *fmt, ...) {
  t_status = code;
  if (fmt) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(t_msg, sizeof(t_msg), fmt, ap);
    va_end(ap);
  } else {
    snprintf(t_msg, sizeof(t_msg), "%s", code == 0 ? "ok" : "error");
  }
  return code;
}

#define CU(call)                                                                          \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess)                                                                \
      return set_status(e_ == cudaErrorMemoryAllocation ? GSKNN_ERR_NOMEM : GSKNN_ERR_CUDA, \
                        "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__,  \
                        __LINE__);                                                        \
  } while (0)

// ------------------------------------------------------------------------------------------
// scratch cache
// ------------------------------------------------------------------------------------------
enum Slot { SLOT_KERNEL = 0, SLOT_HQTAB, SLOT_HCTAB, SLOT_HQNRM, SLOT_HCNRM,
            SLOT_HQIDX, SLOT_HCIDX, SLOT_HD, SLOT_HI, SLOT_AUX, SLOT_HGATHER };

struct Buf {
  void *p = nullptr;
  size_t n = 0;
};
static std::mutex g_mu;
static std::map<std::tuple<int, uintptr_t, int>, Buf> g_bufs;

static cudaError_t scratch(int slot, size_t bytes, cudaStream_t st, void **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(g_mu);
  Buf &b = g_bufs[std::make_tuple(dev, (uintptr_t)st, slot)];
  if (b.n < bytes) {
    // what cannot be had is refused before the present buffer is given up: a call that then takes
    // fewer rows at a time runs in it, call after call
    size_t left = 0, all = 0;
    if (cudaMemGetInfo(&left, &all) == cudaSuccess && bytes > left + b.n)
      return cudaErrorMemoryAllocation;
    if (b.p) {
      e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) return e;
      cudaFree(b.p);
      b.p = nullptr;
      b.n = 0;
    }
    size_t nb = std::max(bytes, (size_t)4096);
    e = cudaMalloc(&b.p, nb);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      return e;
    }
    b.n = nb;
  }
  *out = b.p;
  return cudaSuccess;
}

// Status of the calls of one stream: the device word the kernels report to, and its host-visible
// mirror (pinned), which the last kernel of a call writes, so that reading the status is one
// synchronisation and no copy. Kept like the scratch buffers.
struct StatusWords {
  int *dev, *mirror_dev, *mirror_host;
};
static std::map<std::pair<int, uintptr_t>, StatusWords> g_status;

static cudaError_t status_words(cudaStream_t st, StatusWords *out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(g_mu);
  const auto key = std::make_pair(dev, (uintptr_t)st);
  auto it = g_status.find(key);
  if (it == g_status.end()) {
    StatusWords w{};
    e = cudaMalloc((void **)&w.dev, 256);
    if (e == cudaSuccess) e = cudaHostAlloc((void **)&w.mirror_host, 64, cudaHostAllocMapped);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer((void **)&w.mirror_dev, w.mirror_host, 0);
    if (e != cudaSuccess) {
      if (w.mirror_host) cudaFreeHost(w.mirror_host);
      if (w.dev) cudaFree(w.dev);
      (void)cudaGetLastError();
      return e;
    }
    *w.mirror_host = 0;
    it = g_status.emplace(key, w).first;
  }
  *out = it->second;
  return cudaSuccess;
}

static void release_all_for_device(int dev) {
  std::lock_guard<std::mutex> lk(g_mu);
  for (auto it = g_status.begin(); it != g_status.end();) {
    if (it->first.first == dev) {
      cudaStreamSynchronize((cudaStream_t)it->first.second);
      cudaFree(it->second.dev);
      cudaFreeHost(it->second.mirror_host);
      it = g_status.erase(it);
    } else {
      ++it;
    }
  }
  for (auto it = g_bufs.begin(); it != g_bufs.end();) {
    if (std::get<0>(it->first) == dev) {
      cudaStreamSynchronize((cudaStream_t)std::get<1>(it->first));
      cudaFree(it->second.p);
      it = g_bufs.erase(it);
    } else {
      ++it;
    }
  }
}

// ------------------------------------------------------------------------------------------
// launch tracing: CUDA events around every kernel launch of the library, on its stream
// ------------------------------------------------------------------------------------------
struct TraceRec {
  const char *name;
  cudaEvent_t a, b;
  int nk;  // kernels of the library launched between a and b
};
static std::mutex g_tmu;
static bool g_trace = false;
static std::vector<TraceRec> g_recs;
static std::vector<cudaEvent_t> g_evpool;

static cudaEvent_t ev_get() {
  if (!g_evpool.empty()) {
    cudaEvent_t e = g_evpool.back();
    g_evpool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  return e;
}

struct TraceScope {
  const char *name;
  cudaStream_t st;
  int nk;
  cudaEvent_t a = nullptr;
  TraceScope(const char *n, cudaStream_t s, int kernels = 1) : name(n), st(s), nk(kernels) {
    if (!g_trace) return;
    std::lock_guard<std::mutex> lk(g_tmu);
    a = ev_get();
    cudaEventRecord(a, st);
  }
  ~TraceScope() {
    if (!a) return;
    std::lock_guard<std::mutex> lk(g_tmu);
    cudaEvent_t b = ev_get();
    cudaEventRecord(b, st);
    g_recs.push_back({name, a, b, nk});
  }
};

// Pinned host staging of the calling thread (the gathered rows of a host call), kept between
// calls and freed when the thread exits.
struct PinnedStage {
  void *p = nullptr;
  size_t n = 0;
  ~PinnedStage() {
    if (p) cudaFreeHost(p);
  }
};
static thread_local PinnedStage t_stage;

static cudaError_t pinned_stage(size_t bytes, void **out) {
  if (t_stage.n < bytes) {
    if (t_stage.p) cudaFreeHost(t_stage.p);
    t_stage.p = nullptr;
    t_stage.n = 0;
    cudaError_t e = cudaHostAlloc(&t_stage.p, bytes, cudaHostAllocDefault);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      return e;
    }
    t_stage.n = bytes;
  }
  *out = t_stage.p;
  return cudaSuccess;
}

static size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

// Host threads of the host-pointer path: one per hardware thread, at most 32.
static unsigned host_threads() {
  unsigned nt = std::thread::hardware_concurrency();
  if (nt == 0) nt = 1;
  return nt > 32 ? 32 : nt;
}

// memcpy of `bytes` split over the host threads (one thread below 4 MiB).
static void par_copy(void *dst, const void *src, size_t bytes) {
  unsigned nt = host_threads();
  if (bytes < ((size_t)4 << 20)) nt = 1;
  auto work = [&](unsigned w) {
    const size_t a = bytes * w / nt, b = bytes * (w + 1) / nt;
    std::memcpy(static_cast<char *>(dst) + a, static_cast<const char *>(src) + a, b - a);
  };
  std::vector<std::thread> pool;
  for (unsigned w = 1; w < nt; w++) pool.emplace_back(work, w);
  work(0);
  for (auto &t : pool) t.join();
}

// Rows qidx[0..nq) of Xq, then cidx[0..nc) of Xc, and their norms, gathered by the host threads
// into pinned hrows / hn and copied to drows / dn on stream st. The rows go in chunks: every
// thread gathers its part of chunk j, and the calling thread enqueues chunk j's copy as soon as
// all parts are in, so the copies overlap the gathering of the next chunks. Returns the first
// copy error.
template <typename T>
static cudaError_t gather_rows_to_device(const T *Xq, const T *Xq2, const int *qidx, int nq,
                                         const T *Xc, const T *Xc2, const int *cidx, int nc,
                                         int d, T *hrows, T *hn, T *drows, T *dn,
                                         cudaStream_t st) {
  const size_t n = (size_t)nq + nc, row_bytes = (size_t)d * sizeof(T);
  const bool big = n * row_bytes >= ((size_t)8 << 20);
  const unsigned nt = big ? host_threads() : 1;
  const int nch = n * row_bytes >= ((size_t)32 << 20) ? 8 : 1;
  std::unique_ptr<std::atomic<unsigned>[]> done(new std::atomic<unsigned>[nch]);
  for (int j = 0; j < nch; j++) done[j].store(0);
#if defined(__x86_64__)
  // The staging rows are written once and then read only by the DMA engine: non-temporal
  // stores skip the read-for-ownership of every destination line (a third of the host memory
  // traffic of this copy). Used when rows and the staging base are 16-byte aligned.
  const bool stream = row_bytes % 16 == 0 && (reinterpret_cast<uintptr_t>(hrows) & 15) == 0;
#endif
  auto part = [&](unsigned w, int j) {
    const size_t c0 = n * j / nch, c1 = n * (j + 1) / nch;
    const size_t a = c0 + (c1 - c0) * w / nt, b = c0 + (c1 - c0) * (w + 1) / nt;
    for (size_t i = a; i < b; i++) {
      const bool q = i < (size_t)nq;
      const size_t r = q ? (size_t)qidx[i] : (size_t)cidx[i - nq];
      const T *src = (q ? Xq : Xc) + r * d;
#if defined(__x86_64__)
      if (stream) {
        const __m128i *s4 = reinterpret_cast<const __m128i *>(src);
        __m128i *d4 = reinterpret_cast<__m128i *>(hrows + i * d);
        for (size_t v = 0; v < row_bytes / 16; v++)
          _mm_stream_si128(d4 + v, _mm_loadu_si128(s4 + v));
      } else {
        std::memcpy(hrows + i * d, src, row_bytes);
      }
#else
      std::memcpy(hrows + i * d, src, row_bytes);
#endif
      hn[i] = (q ? Xq2 : Xc2)[r];
    }
#if defined(__x86_64__)
    _mm_sfence();  // the streamed rows are visible before the chunk is handed to the DMA
#endif
    done[j].fetch_add(1, std::memory_order_release);
  };
  std::vector<std::thread> pool;
  for (unsigned w = 1; w < nt; w++)
    pool.emplace_back([&, w] {
      for (int j = 0; j < nch; j++) part(w, j);
    });
  cudaError_t err = cudaSuccess;
  for (int j = 0; j < nch; j++) {
    part(0, j);
    while (done[j].load(std::memory_order_acquire) < nt) std::this_thread::yield();
    const size_t c0 = n * j / nch, c1 = n * (j + 1) / nch;
    if (err == cudaSuccess)
      err = cudaMemcpyAsync(drows + c0 * d, hrows + c0 * d, (c1 - c0) * row_bytes,
                            cudaMemcpyHostToDevice, st);
  }
  for (auto &t : pool) t.join();
  if (err == cudaSuccess) err = cudaMemcpyAsync(dn, hn, n * sizeof(T), cudaMemcpyHostToDevice, st);
  return err;
}

// table[(idx[i] - lo)] = rows[i] (and the norms), one warp per row
template <typename T>
__global__ void scatter_rows(const T *__restrict__ rows, const T *__restrict__ rows2,
                             const int *__restrict__ idx, int n, int d, int lo, T *__restrict__ tab,
                             T *__restrict__ tab2) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;
  const size_t r = (size_t)(idx[i] - lo);
  for (int p = lane; p < d; p += 32) tab[r * d + p] = rows[(size_t)i * d + p];
  if (lane == 0) tab2[r] = rows2[i];
}

static cudaStream_t host_stream() {
  static thread_local std::map<int, cudaStream_t> streams;
  int dev = 0;
  cudaGetDevice(&dev);
  auto it = streams.find(dev);
  if (it != streams.end()) return it->second;
  cudaStream_t s = nullptr;
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) s = nullptr;
  streams[dev] = s;
  return s;
}

static int sm_count() {
  static std::atomic<int> known[64];
  int dev = 0, n = 148;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && known[dev].load(std::memory_order_relaxed) > 0)
    return known[dev].load(std::memory_order_relaxed);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  if (n <= 0) n = 148;
  if (dev >= 0 && dev < 64) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Number of candidate splits per query tile of the CUDA-core kernels. A CTA's time is its tiles
// (about 10 + d/4 us each at 1 or 2 CTAs per SM) plus what its lists take to fill: a split of t
// candidates inserts about k (1 + ln(t/k)) of them into each query's list, however short it is,
// so every further split costs the filling again. Splitting to level the waves alone (9, 16, 9,
// 7 splits) was 1.1 to 2.2 times slower on calls of several waves: 20,000 x 20,000 at d = 32,
// k = 64 takes 11,630 us in 16 splits and 5,280 in the 2 chosen here; 20,000 x 20,000, k = 16
// 3,605 and 2,389; 2,000 x 20,000 at d = 100, k = 100 1,780 and 1,352; FP64 4,000 x 8,000 at
// d = 20, k = 100 2,035 and 1,193 (1-norm calls). Few query tiles take all slots where the lists
// are short (one query, 1,000,000 candidates, k = 16: 855 us in 64 splits, 576 in about 200);
// merging lists beyond 64 entries costs more than that gives (8 queries, 46,095 candidates,
// k = 94: 388 us in 64 splits, 407 in 91).
static int choose_splits(int qtiles, int rtiles, int slots, int d, int k, int br, int minb,
                         double merge) {
  int best_s = 1;
  double best = 1e300;
  const int smax = std::min(rtiles, k <= 64 ? std::max(64, slots / qtiles) : 64);
  const double tile = 10.0 + 0.25 * d, insert = 1.6 * minb * k;  // us, of `minb` CTAs per SM
  for (int s = 1; s <= smax; s++) {
    const int t = (rtiles + s - 1) / s;
    if (s > 1 && t == (rtiles + s - 2) / (s - 1)) continue;  // no fewer tiles per CTA
    const long long items = (long long)qtiles * s;
    const double waves = (double)((items + slots - 1) / slots);
    const double fill = insert * (1.0 + std::log(std::max(1.0, (double)t * br / k)));
    const double cost = waves * (t * tile + fill) * (1.0 + 0.002 * s) + merge * s;
    if (cost < best) {
      best = cost;
      best_s = s;
    }
  }
  return best_s;
}

// Tracer hook for pipelines that bracket groups of launches themselves (the tensor-core path).
static void trace_hook(void *, const char *name, bool begin, cudaStream_t st, int nkernels) {
  if (!g_trace) return;
  std::lock_guard<std::mutex> lk(g_tmu);
  static thread_local std::vector<std::pair<const char *, cudaEvent_t>> pending;
  if (begin) {
    cudaEvent_t a = ev_get();
    cudaEventRecord(a, st);
    pending.push_back({name, a});
    return;
  }
  for (size_t i = pending.size(); i-- > 0;) {
    if (std::strcmp(pending[i].first, name) == 0) {
      cudaEvent_t b = ev_get();
      cudaEventRecord(b, st);
      g_recs.push_back({name, pending[i].second, b, nkernels});
      pending.erase(pending.begin() + (long)i);
      return;
    }
  }
}

// ------------------------------------------------------------------------------------------
// device pipeline: pack -> fused select -> finalize (queries = heap rows)
// ------------------------------------------------------------------------------------------
// Sizes and workspace of the CUDA-core pipeline (offsets from the start of its workspace).
struct SimtPlan {
  SimtGeom g;
  int nkc, qtiles, rtiles, S, tps;
  size_t oA, oB, oQN, oCN, oCI, oPD, oPI, bytes;
};

template <typename T>
static SimtPlan simt_plan(int nq, int nc, int d, int k) {
  SimtPlan P{};
  P.g = simt_geometry<T>(k);
  if (P.g.kp == 0) return P;
  const SimtGeom &g = P.g;
  P.nkc = (d + g.dk - 1) / g.dk;
  P.qtiles = (nq + g.bq - 1) / g.bq;
  P.rtiles = (nc + g.br - 1) / g.br;
  const int minb = std::max(1, g.minb);
  P.S = choose_splits(std::max(1, P.qtiles), P.rtiles, sm_count() * minb, d, k, g.br, minb,
                      // us per list that a query merges: a sorting network of kp entries
                      0.08 * (g.kp / 32) * std::log2((double)g.kp) * (sizeof(T) / 4));
  P.tps = (P.rtiles + P.S - 1) / P.S;
  size_t off = 0;
  auto take = [&](size_t bytes) { size_t o = off; off = align256(off + bytes); return o; };
  P.oA = take((size_t)P.qtiles * P.nkc * g.dk * g.bq * sizeof(T));
  P.oB = take((size_t)P.rtiles * P.nkc * g.dk * g.br * sizeof(T));
  P.oQN = take((size_t)P.qtiles * g.bq * sizeof(T));
  P.oCN = take((size_t)P.rtiles * g.br * sizeof(T));
  P.oCI = take((size_t)P.rtiles * g.br * 4);
  P.oPD = take((size_t)P.S * nq * k * sizeof(T));
  P.oPI = take((size_t)P.S * nq * k * 4);
  P.bytes = off;
  return P;
}

// The CUDA-core kernels of one call; with `rows` / `nrows` (device) only for those heap rows.
template <typename T>
static int simt_run(const SimtPlan &P, int nq, int nc, int d, int k, const T *Xq, const T *Xq2,
                    long long nrows_q, const int *qidx, const T *Xc, const T *Xc2,
                    long long nrows_c, const int *cidx, T *D, int *I, int ldD, char *base,
                    const StatusWords &sw, cudaStream_t st, int metric,
                    const int *rows = nullptr, const int *nrows = nullptr) {
  int *status = sw.dev;
  const SimtGeom &g = P.g;
  T *Apack = reinterpret_cast<T *>(base + P.oA);
  T *Bpack = reinterpret_cast<T *>(base + P.oB);
  T *qn = reinterpret_cast<T *>(base + P.oQN);
  T *cn = reinterpret_cast<T *>(base + P.oCN);
  uint32_t *cid = reinterpret_cast<uint32_t *>(base + P.oCI);
  T *partD = reinterpret_cast<T *>(base + P.oPD);
  uint32_t *partI = reinterpret_cast<uint32_t *>(base + P.oPI);
  {
    TraceScope ts(rows ? "tc_fallback" : "pack_panels", st);
    CU(launch_pack<T>(Xq, Xq2, d, nrows_q, qidx, nq, g.bq, g.dk, P.nkc, Apack, qn, nullptr,
                      status, st, nrows, rows));
  }
  {
    TraceScope ts(rows ? "tc_fallback" : "pack_panels", st);
    CU(launch_pack<T>(Xc, Xc2, d, nrows_c, cidx, nc, g.br, g.dk, P.nkc, Bpack, cn, cid, status,
                      st, nrows));
  }
  SimtArgs<T> sa{};
  sa.Apack = Apack; sa.Bpack = Bpack; sa.qn = qn; sa.cn = cn; sa.cid = cid;
  sa.Din = D; sa.ldD = ldD; sa.Q = nq; sa.k = k; sa.nkc = P.nkc;
  sa.ntiles_r = P.rtiles; sa.tiles_per_split = P.tps; sa.partD = partD; sa.partI = partI;
  sa.metric = metric;
  sa.dQ = nrows;
  sa.rowmap = rows;
  {
    TraceScope ts(rows ? "tc_fallback" : "fused_knn_simt", st);
    CU(launch_simt<T>(sa, g.kp, P.qtiles, P.S, st));
  }
  FinalizeArgs<T> fa{};
  fa.Din = D; fa.Iin = I; fa.ldD = ldD; fa.Q = nq; fa.k = k; fa.S = P.S;
  fa.partD = partD; fa.partI = partI; fa.Dout = D; fa.Iout = I;
  fa.dQ = nrows;
  fa.rowmap = rows;
  fa.status = status;
  fa.mirror = sw.mirror_dev;
  {
    TraceScope ts(rows ? "tc_fallback" : "finalize_heap", st);
    CU(launch_finalize<T>(fa, g.kp, st));
  }
  return set_status(GSKNN_OK, nullptr);
}

template <typename T>
int knn_device_simt(int nq, int nc, int d, int k, const T *Xq, const T *Xq2, long long nrows_q,
                    const int *qidx, const T *Xc, const T *Xc2, long long nrows_c,
                    const int *cidx, T *D, int *I, int ldD, cudaStream_t st, int metric = 0) {
  if (nq == 0 || nc == 0 || d == 0 || k == 0)
    return set_status(GSKNN_EARLY_RETURN, "early return: m, n, d or k is 0");
  if (nq < 0 || nc < 0 || d < 0 || k < 0 || ldD < k)
    return set_status(GSKNN_ERR_ARG, "invalid sizes (n=%d m=%d d=%d k=%d ldD=%d)", nq, nc, d,
                      k, ldD);
  // the 1-norm reads no norms
  if (!Xq || !qidx || !Xc || !cidx || !D || !I || (metric == 0 && (!Xq2 || !Xc2)))
    return set_status(GSKNN_ERR_ARG, "null pointer argument");
  if (metric) Xq2 = Xc2 = nullptr;
  const SimtPlan P = simt_plan<T>(nq, nc, d, k);
  if (P.g.kp == 0)
    return set_status(GSKNN_ERR_UNSUPPORTED, "k=%d exceeds the fused kernel's list size", k);
  void *ws = nullptr;
  StatusWords sw;
  CU(scratch(SLOT_KERNEL, P.bytes, st, &ws));
  CU(status_words(st, &sw));
  int *status = sw.dev;
  CU(cudaMemsetAsync(status, 0, sizeof(int), st));
  return simt_run<T>(P, nq, nc, d, k, Xq, Xq2, nrows_q, qidx, Xc, Xc2, nrows_c, cidx, D, I, ldD,
                     static_cast<char *>(ws), sw, st, metric);
}

static int g_mode = GSKNN_MODE_AUTO;

// A tensor-core call runs in chunks of heap rows (they are independent) where the logs of all rows
// together would take more than LOG_BUDGET, or where its workspace cannot be had: all chunks but the
// last have `rows` rows, whole waves of query tiles where they are that many (1,000,000 x 131,072,
// d = 32, k = 64: 58.9 ms, in equal chunks 61.8), and every chunk packs the candidates again (80 us
// for 262,144 x 64).
constexpr size_t LOG_BUDGET = (size_t)16 << 30;
constexpr int MIN_CHUNK = 1024;
struct RowChunks {
  int rows, tail;  // tail: rows of the last chunk
  TcPlan P, T;     // plans of the whole chunks and of the last
};

// Plans the call and gets its workspace; `whole`, when set, is the plan of all rows, and
// `extra(rows, tail)` the bytes that a chunk takes behind its plan's. cudaErrorInvalidValue: no
// plan.
template <typename Extra>
static cudaError_t tc_workspace(int mode, const TcPlan *whole, int nq, int nc, int d, int k,
                                cudaStream_t st, Extra extra, RowChunks *c, void **ws) {
  const int wave = 128 * sm_count();
  c->rows = nq;
  for (;;) {
    const int rows = c->rows;
    c->tail = nq - (nq - 1) / rows * rows;
    c->P = whole && rows == nq ? *whole : tc_plan(rows, nc, d, k, mode, sm_count());
    if (!c->P.ok) return cudaErrorInvalidValue;
    c->T = c->tail == rows ? c->P : tc_plan(c->tail, nc, d, k, mode, sm_count());
    double part = 0.5;
    if (c->P.log_bytes > LOG_BUDGET && rows > MIN_CHUNK) {
      part = std::min(0.99, (double)LOG_BUDGET / (double)c->P.log_bytes);
    } else {
      const cudaError_t e =
          scratch(SLOT_KERNEL,
                  std::max(align256(c->P.bytes) + extra(rows, false),
                           c->tail == rows ? 0 : align256(c->T.bytes) + extra(c->tail, true)),
                  st, ws);
      if (e != cudaErrorMemoryAllocation || rows <= MIN_CHUNK) return e;
    }
    const int fewer = (int)(rows * part), unit = fewer >= wave ? wave : 128;
    c->rows = std::max(fewer / unit * unit, MIN_CHUNK);
  }
}

// Tensor-core approximate pass + FP64 re-rank (float inputs). `dbg`, when set, also receives
// the approximate distance of every (query, candidate) pair (row stride dbg_ld) and `margin`
// the per-query band width 2E.
static int knn_device_tc(int mode, const TcPlan *plan, int nq, int nc, int d, int k,
                         const float *Xq, const float *Xq2, long long nrows_q, const int *qidx, const float *Xc,
                         const float *Xc2, long long nrows_c, const int *cidx, float *D, int *I,
                         int ldD, cudaStream_t st, float *dbg = nullptr, long long dbg_ld = 0,
                         float *margin = nullptr) {
  if (nq == 0 || nc == 0 || d == 0 || k == 0)
    return set_status(GSKNN_EARLY_RETURN, "early return: m, n, d or k is 0");
  if (nq < 0 || nc < 0 || d < 0 || k < 0 || ldD < k)
    return set_status(GSKNN_ERR_ARG, "invalid sizes (n=%d m=%d d=%d k=%d ldD=%d)", nq, nc, d,
                      k, ldD);
  if (!Xq || !Xq2 || !qidx || !Xc || !Xc2 || !cidx || !D || !I)
    return set_status(GSKNN_ERR_ARG, "null pointer argument");
  RowChunks ch;
  void *ws = nullptr;
  StatusWords sw;
  const cudaError_t we =
      tc_workspace(mode, plan, nq, nc, d, k, st, [](int, bool) { return (size_t)0; }, &ch, &ws);
  if (!ch.P.ok)
    return set_status(GSKNN_ERR_UNSUPPORTED,
                      "tensor-core mode %d does not support d=%d k=%d (shared memory)", mode, d,
                      k);
  CU(we);
  CU(status_words(st, &sw));
  int *status = sw.dev;  // cleared by the first kernel
  // GSKNN_TC_COUNTERS=1: per-call diagnostics of the tensor-core epilogue on stderr
  static const bool want_counters = std::getenv("GSKNN_TC_COUNTERS") != nullptr;
  unsigned long long *counters = nullptr;
  if (want_counters) {
    void *cv = nullptr;
    CU(scratch(SLOT_AUX, 128, st, &cv));
    counters = static_cast<unsigned long long *>(cv);
  }
  for (int q0 = 0; q0 < nq; q0 += ch.rows) {
    const int n = std::min(ch.rows, nq - q0);
    const TcPlan &P = n == ch.rows ? ch.P : ch.T;
    if (counters) CU(cudaMemsetAsync(counters, 0, 128, st));
    CU(tc_run(P, n, nc, d, k, Xq, Xq2, nrows_q, qidx + q0, Xc, Xc2, nrows_c, cidx,
              D + (size_t)q0 * ldD, I + (size_t)q0 * ldD, ldD, ws, status,
              dbg ? dbg + (size_t)q0 * dbg_ld : nullptr, dbg_ld, counters, st, trace_hook, nullptr,
              sw.mirror_dev, q0 == 0));
    if (counters) {
      unsigned long long h[16] = {};
      int nfb = 0;
      CU(cudaMemcpyAsync(h, counters, sizeof(h), cudaMemcpyDeviceToHost, st));
      CU(cudaMemcpyAsync(&nfb, static_cast<char *>(ws) + P.o_fbc, sizeof(int),
                         cudaMemcpyDeviceToHost, st));
      CU(cudaStreamSynchronize(st));
      const double ctas = (double)P.qtiles * P.S, warps = ctas * TC_EPI_WARPS;
      std::fprintf(stderr,
                   "gsknn tc: mode=%d n=%d m=%d d=%d k=%d S=%d N=%d NST=%d: logged/query=%.1f "
                   "flushes/warp=%.1f slow-chunks/warp=%.1f "
                   "chunks/warp=%.1f rerank-scanned/query=%.1f exact/query=%.1f fallback=%d | "
                   "cycles/CTA: mma-loop=%.0f mma-wait-tma=%.0f mma-wait-epilogue=%.0f | "
                   "cycles/warp: epi-loop=%.0f epi-wait-mma=%.0f\n",
                   mode, n, nc, d, k, P.S, P.N, P.NST, (double)h[0] / n,
                   (double)h[2] / warps, (double)h[3] / warps, (double)h[4] / warps,
                   (double)h[5] / n, (double)h[6] / n, nfb, (double)h[10] / ctas,
                   (double)h[7] / ctas, (double)h[8] / ctas, (double)h[11] / warps,
                   (double)h[9] / warps);
    }
    if (margin)
      CU(cudaMemcpyAsync(margin + q0, static_cast<char *>(ws) + P.o_margin, (size_t)n * 4,
                         cudaMemcpyDeviceToDevice, st));
  }
  return set_status(GSKNN_OK, nullptr);
}

// The tensor-core mode AUTO takes for a shape (GSKNN_MODE_FP32: none fits), and its plan.
static int auto_mode(int nq, int nc, int d, int k, TcPlan *P) {
  // Split BF16 (three MMAs per product) keeps the re-rank band narrowest. One FP16 MMA per product
  // (and half the panel bytes) pays from d = 128 where the contraction bounds the call, about
  // 1.3e10 (pair, padded dimension) products, or the packing does, 2.5e7 (candidate, padded
  // dimension) entries; beyond d = 256, where split tiles are narrow, 9e6. B200, us, split -> FP16:
  // 16,384 x 60,000, d = 256 1,532 -> 795; 4,096 x 65,536, d = 128 318 -> 260; 16 x 250,000,
  // d = 200 613 -> 397; 16 x 30,000, d = 300 208 -> 169; but 2,000 x 30,000, d = 128 167 -> 175,
  // 16 x 30,000, d = 128 127 -> 164 and 16 x 4,096 96 -> 108 (the escalation's launches). Below
  // d = 128 its band overflows the logs on clusters, and all that it gains on other points is less
  // than what those lose: 16,384 x 60,000, d = 100, k = 32 uniform 785 -> 625, mixture of sigma 0.05
  // 795 -> 734, 0.02 868 -> 2,625, 0.014 1,145 -> 2,160, 0.01 4,173 -> 190,959; doubles 5,003 x
  // 50,021, d = 100, k = 50, sigma 0.05 531 -> 593, 0.02 608 -> 1,748.
  const double d_pad = (d + 63) / 64 * 64, entries = nc * d_pad, products = nq * entries;
  const bool big = d >= 128 && (products >= 1.3e10 || entries >= (d > 256 ? 9e6 : 2.5e7));
  const int order[4] = {big ? GSKNN_TC_FP16 : GSKNN_TC_BF16X3,
                        big ? GSKNN_TC_BF16X3 : GSKNN_TC_FP16, GSKNN_TC_TF32, GSKNN_MODE_FP32};
  for (int i = 0; i < 3; i++) {
    *P = tc_plan(nq, nc, d, k, order[i], sm_count());
    if (P->ok) return order[i];
  }
  return GSKNN_MODE_FP32;
}

// A double call through the tensor cores: approximate distances with a rigorous bound, exact FP64
// distances of the band in the CUDA-core kernel's own order of operations, so the results are the
// same bits. Queries that the passes could not bound (their band overflows in the narrowest
// format; values beyond the floats' range; NaN) run through the CUDA-core kernels, which are
// launched behind them over the list of such rows, mostly empty. Returns -1 when the form does not
// apply (shared memory, k) or its scratch cannot be had: the caller takes the CUDA cores.
static int knn_device_tc_double(int nq, int nc, int d, int k, const double *Xq, const double *Xq2,
                                long long nrows_q, const int *qidx, const double *Xc,
                                const double *Xc2, long long nrows_c, const int *cidx, double *D,
                                int *I, int ldD, cudaStream_t st) {
  if (nq <= 0 || nc <= 0 || d <= 0 || k <= 0 || ldD < k || !Xq || !Xq2 || !qidx || !Xc || !Xc2 ||
      !cidx || !D || !I)
    return -1;  // (the CUDA-core path reports)
  TcPlan P;
  const int mode = auto_mode(nq, nc, d, k, &P);
  if (mode == GSKNN_MODE_FP32) return -1;
  if (simt_geometry<double>(k).kp == 0) return -1;
  RowChunks ch;
  void *ws = nullptr;
  StatusWords sw;
  SimtPlan F[2];  // of the whole chunks and of the last
  const cudaError_t se = tc_workspace(
      mode, &P, nq, nc, d, k, st,
      [&](int rows, bool tail) { return (F[tail] = simt_plan<double>(rows, nc, d, k)).bytes; }, &ch,
      &ws);
  if (se == cudaErrorMemoryAllocation) return -1;
  CU(se);
  CU(status_words(st, &sw));
  int *status = sw.dev;  // cleared by the first kernel
  for (int q0 = 0; q0 < nq; q0 += ch.rows) {
    const int n = std::min(ch.rows, nq - q0);
    const TcPlan &R = n == ch.rows ? ch.P : ch.T;
    const int *left = nullptr, *nleft = nullptr;
    double *Dq = D + (size_t)q0 * ldD;
    int *Iq = I + (size_t)q0 * ldD;
    CU(tc_run_double(R, n, nc, d, k, Xq, Xq2, nrows_q, qidx + q0, Xc, Xc2, nrows_c, cidx, Dq, Iq,
                     ldD, ws, status, &left, &nleft, st, trace_hook, nullptr, q0 == 0));
    const int rc = simt_run<double>(F[n != ch.rows], n, nc, d, k, Xq, Xq2, nrows_q, qidx + q0, Xc,
                                    Xc2, nrows_c, cidx, Dq, Iq, ldD,
                                    static_cast<char *>(ws) + align256(R.bytes), sw, st, 0, left,
                                    nleft);
    if (rc != GSKNN_OK) return rc;
  }
  return set_status(GSKNN_OK, nullptr);
}

template <typename T>
int knn_device_large(int nq, int nc, int d, int k, const T *Xq, const T *Xq2, long long nrows_q,
                     const int *qidx, const T *Xc, const T *Xc2, long long nrows_c,
                     const int *cidx, T *D, int *I, int ldD, int four_ary, cudaStream_t st,
                     int metric = 0) {
  if (nq == 0 || nc == 0 || d == 0 || k == 0)
    return set_status(GSKNN_EARLY_RETURN, "early return: m, n, d or k is 0");
  const int need = four_ary ? k + KNN_HEAP_OFFSET : k;
  if (nq < 0 || nc < 0 || d < 0 || k < 0 || ldD < need)
    return set_status(GSKNN_ERR_ARG, "invalid sizes (n=%d m=%d d=%d k=%d ldD=%d)", nq, nc, d,
                      k, ldD);
  if (!Xq || !qidx || !Xc || !cidx || !D || !I || (metric == 0 && (!Xq2 || !Xc2)))
    return set_status(GSKNN_ERR_ARG, "null pointer argument");
  if (large_select_smem(k, sizeof(T)) > 227 * 1024)
    return set_status(GSKNN_ERR_UNSUPPORTED, "k=%d exceeds the selection kernel (k <= %d)", k,
                      sizeof(T) == 8 ? 16384 : 16384);
  const LargePlan P = large_plan<T>(nq, nc, d, k, (size_t)1 << 30);
  void *ws = nullptr;
  StatusWords sw;
  CU(scratch(SLOT_KERNEL, P.bytes, st, &ws));
  CU(status_words(st, &sw));
  int *status = sw.dev;
  CU(cudaMemsetAsync(status, 0, sizeof(int), st));
  {
    // two packing launches, then a distance block and a selection per chunk of query rows
    TraceScope ts("select_rows", st, 2 + 2 * ((nq + P.chunk_rows - 1) / P.chunk_rows));
    CU(large_run<T>(P, nq, nc, d, k, Xq, Xq2, nrows_q, qidx, Xc, Xc2, nrows_c, cidx, D, I, ldD,
                    four_ary, ws, status, st, metric));
  }
  CU(cudaMemcpyAsync(sw.mirror_host, status, sizeof(int), cudaMemcpyDeviceToHost, st));
  return set_status(GSKNN_OK, nullptr);
}

template <typename T>
int knn_device(int nq, int nc, int d, int k, const T *Xq, const T *Xq2, long long nrows_q,
               const int *qidx, const T *Xc, const T *Xc2, long long nrows_c, const int *cidx,
               T *D, int *I, int ldD, cudaStream_t st, int metric = 0) {
  if (metric != 0) {  // the 1-norm: CUDA cores only (it is no inner product)
    if (simt_geometry<T>(k).kp == 0)
      return knn_device_large<T>(nq, nc, d, k, Xq, Xq2, nrows_q, qidx, Xc, Xc2, nrows_c, cidx,
                                 D, I, ldD, 0, st, metric);
    return knn_device_simt<T>(nq, nc, d, k, Xq, Xq2, nrows_q, qidx, Xc, Xc2, nrows_c, cidx, D,
                              I, ldD, st, metric);
  }
  if constexpr (std::is_same<T, float>::value) {
    // explicit modes are honoured; AUTO takes the tensor-core form with the exact FP64 re-rank
    // where it fits, else the CUDA-core FP32 kernel
    TcPlan P;
    const int set = g_mode;
    const int mode = set != GSKNN_MODE_AUTO  ? set
                     : nq > 0 && nc > 0 && d > 0 && k > 0 ? auto_mode(nq, nc, d, k, &P)
                                                          : GSKNN_MODE_BF16X3;
    if (mode != GSKNN_MODE_FP32)
      return knn_device_tc(mode, set == GSKNN_MODE_AUTO ? &P : nullptr, nq, nc, d, k, Xq, Xq2,
                           nrows_q, qidx, Xc, Xc2, nrows_c, cidx, D, I, ldD, st);
  }
  // lists beyond the fused kernels' capacity: explicit distance block + row selection
  if (simt_geometry<T>(k).kp == 0)
    return knn_device_large<T>(nq, nc, d, k, Xq, Xq2, nrows_q, qidx, Xc, Xc2, nrows_c, cidx, D,
                               I, ldD, 0, st);
  if constexpr (std::is_same<T, double>::value) {
    // From 32,768 pairs on the tensor-core form is the faster one (B200, us, CUDA cores -> tensor
    // cores: 1 x 300, d = 3 91 -> 103; 16 x 4,096, d = 32 136 -> 113; 4,096 x 4,096, d = 32
    // 426 -> 130; 1,000 x 20,000, k = 200 1,928 -> 476; 5,003 x 50,021, d = 100, k = 50
    // 7,853 -> 565; 8,192 x 65,536, d = 3 2,584 -> 357).
    // GSKNN_MODE_FP32 asks for the CUDA cores, here too.
    if (g_mode != GSKNN_MODE_FP32 && (long long)nq * nc >= 32768) {
      const int rc = knn_device_tc_double(nq, nc, d, k, Xq, Xq2, nrows_q, qidx, Xc, Xc2, nrows_c,
                                          cidx, D, I, ldD, st);
      if (rc != -1) return rc;
    }
  }
  return knn_device_simt<T>(nq, nc, d, k, Xq, Xq2, nrows_q, qidx, Xc, Xc2, nrows_c, cidx, D, I,
                            ldD, st);
}

// Reads back the device status word of `st` (after synchronising it).
static int device_status(cudaStream_t st) {
  StatusWords sw;
  CU(status_words(st, &sw));
  CU(cudaStreamSynchronize(st));
  const int h = *static_cast<volatile int *>(sw.mirror_host);
  if (h == GSKNN_ERR_INDEX)
    return set_status(GSKNN_ERR_INDEX, "an alpha/beta index lies outside its point table");
  if (h == GSKNN_ERR_TIMEOUT)
    return set_status(GSKNN_ERR_TIMEOUT, "a bounded device-side wait gave up");
  if (h != 0) return set_status(h, "device-side error %d", h);
  return GSKNN_OK;
}

// ------------------------------------------------------------------------------------------
// host-pointer path
// ------------------------------------------------------------------------------------------
static bool index_range(const int *idx, int n, int *lo, int *hi) {
  int a = idx[0], b = idx[0];
  for (int i = 1; i < n; i++) {
    const int v = idx[i];
    a = v < a ? v : a;
    b = v > b ? v : b;
  }
  *lo = a;
  *hi = b;
  return a >= 0;
}

template <typename T>
// path: 0 = the default dispatch, 1 = explicit distance block + selection into binary heaps,
// 2 = the same into 4-ary heaps with the 3-slot header (rows of ldD >= k + 3).
// metric: 0 = squared 2-norm, 1 = 1-norm (heap_t.type KNN_1NORM).
int knn_host(int nq, int nc, int d, int k, const T *Xq, const T *Xq2, const int *qidx,
             const T *Xc, const T *Xc2, const int *cidx, T *D, int *I, int ldD, int path = 0,
             int metric = 0) {
  if (nq == 0 || nc == 0 || d == 0 || k == 0)
    return set_status(GSKNN_EARLY_RETURN, "early return: m, n, d or k is 0");
  if (nq < 0 || nc < 0 || d < 0 || k < 0 || ldD < (path == 2 ? k + KNN_HEAP_OFFSET : k))
    return set_status(GSKNN_ERR_ARG, "invalid sizes");
  if (!Xq || !Xq2 || !qidx || !Xc || !Xc2 || !cidx || !D || !I)
    return set_status(GSKNN_ERR_ARG, "null pointer argument");
  // GSKNN_HOST_TRACE=1: one stderr line per call with the host-side phases in milliseconds
  static const bool host_trace = std::getenv("GSKNN_HOST_TRACE") != nullptr;
  using hclock = std::chrono::steady_clock;
  const auto h0 = hclock::now();
  auto hms = [&](hclock::time_point t) {
    return std::chrono::duration<double, std::milli>(t - h0).count();
  };
  hclock::time_point h_gather = h0, h_copy = h0, h_enq = h0, h_done = h0;
  int qlo, qhi, clo, chi;
  if (!index_range(qidx, nq, &qlo, &qhi) || !index_range(cidx, nc, &clo, &chi))
    return set_status(GSKNN_ERR_INDEX, "negative point index");
  cudaStream_t st = host_stream();
  const bool same = (Xq == Xc) && (Xq2 == Xc2);
  if (same) {
    qlo = clo = std::min(qlo, clo);
    qhi = chi = std::max(qhi, chi);
  }
  void *pqi, *pci, *pD, *pI;
  CU(scratch(SLOT_HQIDX, (size_t)nq * 4, st, &pqi));
  CU(scratch(SLOT_HCIDX, (size_t)nc * 4, st, &pci));
  CU(scratch(SLOT_HD, (size_t)nq * ldD * sizeof(T), st, &pD));
  CU(scratch(SLOT_HI, (size_t)nq * ldD * 4, st, &pI));
  CU(cudaMemcpyAsync(pqi, qidx, (size_t)nq * 4, cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(pci, cidx, (size_t)nc * 4, cudaMemcpyHostToDevice, st));
  // Device copy of each table over the row range the index lists reach, so that global row ids
  // index it directly. When the lists reference well under that range (random subsets of a
  // large table), only the referenced rows travel: gathered on the host into pinned staging,
  // one copy, then scattered into place on the device. Otherwise the range is copied as is.
  const size_t qrows = (size_t)(qhi - qlo + 1), crows = (size_t)(chi - clo + 1);
  const size_t range_rows = same ? qrows : qrows + crows;
  const bool sparse = (size_t)(nq + nc) * 10 < range_rows * 6;
  void *pqt = nullptr, *pqn = nullptr, *pct = nullptr, *pcn = nullptr;
  CU(scratch(SLOT_HQTAB, qrows * d * sizeof(T), st, &pqt));
  CU(scratch(SLOT_HQNRM, qrows * sizeof(T), st, &pqn));
  if (!same) {
    CU(scratch(SLOT_HCTAB, crows * d * sizeof(T), st, &pct));
    CU(scratch(SLOT_HCNRM, crows * sizeof(T), st, &pcn));
  } else {
    pct = pqt;
    pcn = pqn;
  }
  // Pinned staging of this call: the heaps first (both directions go through it, so their
  // copies run at DMA speed), then, on the sparse path, the gathered rows and their norms. The
  // heaps' copy to the device overlaps the gathering of the rows.
  const size_t n = (size_t)nq + nc;
  const size_t hd_bytes = (size_t)nq * ldD * sizeof(T), hi_bytes = (size_t)nq * ldD * 4;
  const size_t rows_off = al256(al256(hd_bytes) + hi_bytes);
  const size_t bytes = rows_off + (sparse ? n * d * sizeof(T) + n * sizeof(T) : 0);
  void *stage = nullptr;
  CU(cudaStreamSynchronize(st));  // the staging buffer of the previous call is free
  CU(pinned_stage(bytes, &stage));
  T *hD = static_cast<T *>(stage);
  int *hI = reinterpret_cast<int *>(static_cast<char *>(stage) + al256(hd_bytes));
  par_copy(hD, D, hd_bytes);
  par_copy(hI, I, hi_bytes);
  CU(cudaMemcpyAsync(pD, hD, hd_bytes, cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(pI, hI, hi_bytes, cudaMemcpyHostToDevice, st));
  if (sparse) {
    void *dg = nullptr;
    CU(scratch(SLOT_HGATHER, n * d * sizeof(T) + n * sizeof(T), st, &dg));
    T *hrows = reinterpret_cast<T *>(static_cast<char *>(stage) + rows_off);
    T *hn = hrows + n * d;
    T *grows = static_cast<T *>(dg);
    T *gn = grows + n * d;
    CU(gather_rows_to_device<T>(Xq, Xq2, qidx, nq, Xc, Xc2, cidx, nc, d, hrows, hn, grows, gn,
                                st));
    h_gather = hclock::now();
    scatter_rows<T><<<(nq + 7) / 8, 256, 0, st>>>(grows, gn, static_cast<const int *>(pqi), nq,
                                                  d, qlo, static_cast<T *>(pqt),
                                                  static_cast<T *>(pqn));
    scatter_rows<T><<<(nc + 7) / 8, 256, 0, st>>>(grows + (size_t)nq * d, gn + nq,
                                                  static_cast<const int *>(pci), nc, d, clo,
                                                  static_cast<T *>(pct), static_cast<T *>(pcn));
    CU(cudaGetLastError());
  } else {
    CU(cudaMemcpyAsync(pqt, Xq + (size_t)qlo * d, qrows * d * sizeof(T), cudaMemcpyHostToDevice,
                       st));
    CU(cudaMemcpyAsync(pqn, Xq2 + qlo, qrows * sizeof(T), cudaMemcpyHostToDevice, st));
    if (!same) {
      CU(cudaMemcpyAsync(pct, Xc + (size_t)clo * d, crows * d * sizeof(T),
                         cudaMemcpyHostToDevice, st));
      CU(cudaMemcpyAsync(pcn, Xc2 + clo, crows * sizeof(T), cudaMemcpyHostToDevice, st));
    }
  }
  const T *dXq = static_cast<const T *>(pqt) - (size_t)qlo * d;
  const T *dXq2 = static_cast<const T *>(pqn) - qlo;
  const T *dXc = static_cast<const T *>(pct) - (size_t)clo * d;
  const T *dXc2 = static_cast<const T *>(pcn) - clo;
  int rc = GSKNN_OK;
  h_copy = hclock::now();
  if (path == 0)
    rc = knn_device<T>(nq, nc, d, k, dXq, dXq2, (long long)qhi + 1, static_cast<int *>(pqi),
                       dXc, dXc2, (long long)chi + 1, static_cast<int *>(pci),
                       static_cast<T *>(pD), static_cast<int *>(pI), ldD, st, metric);
  else
    rc = knn_device_large<T>(nq, nc, d, k, dXq, dXq2, (long long)qhi + 1,
                             static_cast<int *>(pqi), dXc, dXc2, (long long)chi + 1,
                             static_cast<int *>(pci), static_cast<T *>(pD),
                             static_cast<int *>(pI), ldD, path == 2 ? 1 : 0, st, metric);
  if (rc != GSKNN_OK) {
    cudaStreamSynchronize(st);
    return rc;
  }
  h_enq = hclock::now();
  rc = device_status(st);
  if (rc != GSKNN_OK) return rc;
  h_done = hclock::now();
  CU(cudaMemcpyAsync(hD, pD, hd_bytes, cudaMemcpyDeviceToHost, st));
  CU(cudaMemcpyAsync(hI, pI, hi_bytes, cudaMemcpyDeviceToHost, st));
  CU(cudaStreamSynchronize(st));
  par_copy(D, hD, hd_bytes);
  par_copy(I, hI, hi_bytes);
  if (host_trace)
    std::fprintf(stderr,
                 "gsknn host: n=%d m=%d sparse=%d gather %.3f copies-enqueued %.3f "
                 "kernels-enqueued %.3f device-done %.3f heaps-back %.3f ms\n",
                 nq, nc, sparse ? 1 : 0, hms(h_gather), hms(h_copy), hms(h_enq), hms(h_done),
                 hms(hclock::now()));
  return set_status(GSKNN_OK, nullptr);
}

// Distance block of host tables: C[j*ldc + i] for rows j < nq (qidx) and columns i < nc (cidx).
template <typename T>
int sq2nrm_host(int nq, int nc, int d, const T *Xq, const T *Xq2, const int *qidx, const T *Xc,
                const T *Xc2, const int *cidx, T *C, int ldc) {
  if (nq == 0 || nc == 0 || d == 0)
    return set_status(GSKNN_EARLY_RETURN, "early return: m, n or k is 0");
  if (nq < 0 || nc < 0 || d < 0 || ldc < nc)
    return set_status(GSKNN_ERR_ARG, "invalid sizes (ldc must be >= m)");
  if (!Xq || !Xq2 || !qidx || !Xc || !Xc2 || !cidx || !C)
    return set_status(GSKNN_ERR_ARG, "null pointer argument");
  int qlo, qhi, clo, chi;
  if (!index_range(qidx, nq, &qlo, &qhi) || !index_range(cidx, nc, &clo, &chi))
    return set_status(GSKNN_ERR_INDEX, "negative point index");
  cudaStream_t st = host_stream();
  const size_t qrows = (size_t)(qhi - qlo + 1), crows = (size_t)(chi - clo + 1);
  void *pq, *pq2, *pc, *pc2, *pqi, *pci, *pC, *ws;
  StatusWords sw;
  CU(scratch(SLOT_HQTAB, qrows * d * sizeof(T), st, &pq));
  CU(scratch(SLOT_HQNRM, qrows * sizeof(T), st, &pq2));
  CU(scratch(SLOT_HCTAB, crows * d * sizeof(T), st, &pc));
  CU(scratch(SLOT_HCNRM, crows * sizeof(T), st, &pc2));
  CU(scratch(SLOT_HQIDX, (size_t)nq * 4, st, &pqi));
  CU(scratch(SLOT_HCIDX, (size_t)nc * 4, st, &pci));
  CU(scratch(SLOT_HD, (size_t)nq * nc * sizeof(T), st, &pC));
  CU(status_words(st, &sw));
  CU(cudaMemcpyAsync(pq, Xq + (size_t)qlo * d, qrows * d * sizeof(T), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(pq2, Xq2 + qlo, qrows * sizeof(T), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(pc, Xc + (size_t)clo * d, crows * d * sizeof(T), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(pc2, Xc2 + clo, crows * sizeof(T), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(pqi, qidx, (size_t)nq * 4, cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(pci, cidx, (size_t)nc * 4, cudaMemcpyHostToDevice, st));
  int *status = sw.dev;
  CU(cudaMemsetAsync(status, 0, sizeof(int), st));
  const LargePlan P = large_plan<T>(nq, nc, d, 1, 0);
  CU(scratch(SLOT_KERNEL, P.bytes, st, &ws));
  {
    TraceScope ts("dist_block", st, 3);  // two packing launches and the distance block
    CU(block_run<T>(P, nq, nc, d, static_cast<const T *>(pq) - (size_t)qlo * d,
                    static_cast<const T *>(pq2) - qlo, (long long)qhi + 1,
                    static_cast<const int *>(pqi), static_cast<const T *>(pc) - (size_t)clo * d,
                    static_cast<const T *>(pc2) - clo, (long long)chi + 1,
                    static_cast<const int *>(pci), static_cast<T *>(pC), nc, ws, status, st));
  }
  CU(cudaMemcpyAsync(sw.mirror_host, status, sizeof(int), cudaMemcpyDeviceToHost, st));
  int rc = device_status(st);
  if (rc != GSKNN_OK) return rc;
  CU(cudaMemcpy2DAsync(C, (size_t)ldc * sizeof(T), pC, (size_t)nc * sizeof(T),
                       (size_t)nc * sizeof(T), (size_t)nq, cudaMemcpyDeviceToHost, st));
  CU(cudaStreamSynchronize(st));
  return set_status(GSKNN_OK, nullptr);
}

}  // namespace gsknn

using namespace gsknn;

// ==========================================================================================
// C ABI
// ==========================================================================================
extern "C" {

int gsknn_last_error(void) { return t_status; }
const char *gsknn_last_error_string(void) { return t_msg; }

int gsknn_set_mode(int mode) {
  if (mode < GSKNN_MODE_AUTO || mode > GSKNN_MODE_BF16X3)
    return set_status(GSKNN_ERR_ARG, "unknown mode %d", mode);
  g_mode = mode;
  return set_status(GSKNN_OK, nullptr);
}
int gsknn_get_mode(void) { return g_mode; }

int gsknn_s_device(int m, int n, int d, int k, const float *XA, const float *XA2, long long nA,
                   const int *alpha, const float *XB, const float *XB2, long long nB,
                   const int *beta, float *D, int *I, int ldD, void *stream) {
  return knn_device<float>(n, m, d, k, XB, XB2, nB, beta, XA, XA2, nA, alpha, D, I, ldD,
                           (cudaStream_t)stream);
}

int gsknn_d_device(int m, int n, int d, int k, const double *XA, const double *XA2,
                   long long nA, const int *alpha, const double *XB, const double *XB2,
                   long long nB, const int *beta, double *D, int *I, int ldD, void *stream) {
  return knn_device<double>(n, m, d, k, XB, XB2, nB, beta, XA, XA2, nA, alpha, D, I, ldD,
                            (cudaStream_t)stream);
}

int gsknn_s_device_metric(int type, int m, int n, int d, int k, const float *XA,
                          const float *XA2, long long nA, const int *alpha, const float *XB,
                          const float *XB2, long long nB, const int *beta, float *D, int *I,
                          int ldD, void *stream) {
  if (type != KNN_2NORM && type != KNN_1NORM)
    return set_status(GSKNN_ERR_ARG, "type must be KNN_2NORM or KNN_1NORM");
  return knn_device<float>(n, m, d, k, XB, XB2, nB, beta, XA, XA2, nA, alpha, D, I, ldD,
                           (cudaStream_t)stream, type == KNN_1NORM ? 1 : 0);
}

int gsknn_d_device_metric(int type, int m, int n, int d, int k, const double *XA,
                          const double *XA2, long long nA, const int *alpha, const double *XB,
                          const double *XB2, long long nB, const int *beta, double *D, int *I,
                          int ldD, void *stream) {
  if (type != KNN_2NORM && type != KNN_1NORM)
    return set_status(GSKNN_ERR_ARG, "type must be KNN_2NORM or KNN_1NORM");
  return knn_device<double>(n, m, d, k, XB, XB2, nB, beta, XA, XA2, nA, alpha, D, I, ldD,
                            (cudaStream_t)stream, type == KNN_1NORM ? 1 : 0);
}

int gsknn_stream_status(void *stream) { return device_status((cudaStream_t)stream); }

int gsknn_tc_distances(int mode, int m, int n, int d, int k, const float *XA, const float *XA2,
                       long long nA, const int *alpha, const float *XB, const float *XB2,
                       long long nB, const int *beta, float *D, int *I, int ldD, float *C,
                       long long ldc, float *margin, void *stream) {
  if (mode < GSKNN_MODE_TF32 || mode > GSKNN_MODE_FP16)
    return set_status(GSKNN_ERR_ARG, "gsknn_tc_distances: mode must be a tensor-core mode");
  if (C && ldc < m) return set_status(GSKNN_ERR_ARG, "gsknn_tc_distances: ldc < m");
  return knn_device_tc(mode, nullptr, n, m, d, k, XB, XB2, nB, beta, XA, XA2, nA, alpha, D, I, ldD,
                       (cudaStream_t)stream, C, ldc, margin);
}

void gsknn_trace_enable(int on) {
  std::lock_guard<std::mutex> lk(g_tmu);
  g_trace = on != 0;
}

int gsknn_trace_read(char *buf, int len) {
  std::lock_guard<std::mutex> lk(g_tmu);
  struct Acc { int n = 0; double ms = 0.0; };
  std::map<std::string, Acc> acc;
  int total = 0;
  for (auto &r : g_recs) {
    cudaEventSynchronize(r.b);
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, r.a, r.b) == cudaSuccess) {
      Acc &x = acc[r.name];
      x.n += r.nk;
      x.ms += ms;
    }
    g_evpool.push_back(r.a);
    g_evpool.push_back(r.b);
    total++;
  }
  g_recs.clear();
  std::string out = "{";
  bool first = true;
  for (auto &kv : acc) {
    char tmp[256];
    snprintf(tmp, sizeof(tmp), "%s\"%s\": {\"launches\": %d, \"ms\": %.6f}", first ? "" : ", ",
             kv.first.c_str(), kv.second.n, kv.second.ms);
    out += tmp;
    first = false;
  }
  out += "}";
  if (buf && len > 0) snprintf(buf, (size_t)len, "%s", out.c_str());
  return total;
}

void gsknn_release_workspace(void) {
  int dev = 0;
  cudaGetDevice(&dev);
  release_all_for_device(dev);
}

// ---- reference entry points (frame/gsknn.c) ----
void sgsknn_var1(int m, int n, int k, int r, float *XA, float *XA2, int *alpha, float *XB,
                 float *XB2, int *beta, float *D, int *I) {
  knn_host<float>(m, n, k, r, XA, XA2, alpha, XB, XB2, beta, D, I, r);
}

void dgsknn_var1(int m, int n, int k, int r, double *XA, double *XA2, int *alpha, double *XB,
                 double *XB2, int *beta, double *D, int *I) {
  knn_host<double>(m, n, k, r, XA, XA2, alpha, XB, XB2, beta, D, I, r);
}

void sgsknn(int m, int n, int k, int r, float *XA, float *XA2, int *alpha, float *XB,
            float *XB2, int *beta, heap_t *heap) {
  if (!heap) {
    set_status(GSKNN_ERR_ARG, "null heap");
    return;
  }
  knn_host<float>(n, m, k, r, XB, XB2, beta, XA, XA2, alpha, heap->D_s, heap->I, heap->ldk, 0,
                  heap->type == KNN_1NORM ? 1 : 0);
}

void dgsknn(int m, int n, int k, int r, double *XA, double *XA2, int *alpha, double *XB,
            double *XB2, int *beta, heap_t *heap) {
  if (!heap) {
    set_status(GSKNN_ERR_ARG, "null heap");
    return;
  }
  if (r > KNN_VAR_THRES) {
    dgsknn_var3(m, n, k, r, XA, XA2, alpha, XB, XB2, beta, heap);
    return;
  }
  knn_host<double>(n, m, k, r, XB, XB2, beta, XA, XA2, alpha, heap->D, heap->I, heap->ldk, 0,
                   heap->type == KNN_1NORM ? 1 : 0);
}

// frame/gsknn.c:597-659. The heap's own layout decides the selection: 4-ary with the header
// when heapCreate_d built it that way (heap->d == 4), binary otherwise (attached heaps).
void dgsknn_var3(int m, int n, int k, int r, double *XA, double *XA2, int *amap, double *XB,
                 double *XB2, int *bmap, heap_t *heap) {
  if (!heap) {
    set_status(GSKNN_ERR_ARG, "null heap");
    return;
  }
  knn_host<double>(n, m, k, r, XB, XB2, bmap, XA, XA2, amap, heap->D, heap->I, heap->ldk,
                   heap->d == 4 ? 2 : 1, heap->type == KNN_1NORM ? 1 : 0);
}

void dgssq2nrm(int m, int n, int k, double *XA, double *XA2, int *amap, double *XB,
               double *XB2, int *bmap, double *C, int ldc) {
  sq2nrm_host<double>(n, m, k, XB, XB2, bmap, XA, XA2, amap, C, ldc);
}

// frame/gsknn_ref.c:63-162: D/I are n rows of r (binary heaps), candidates on the alpha side.
void sgsknn_ref(int m, int n, int k, int r, float *XA, float *XA2, int *alpha, float *XB,
                float *XB2, int *beta, float *D, int *I) {
  if (r == 0) {
    set_status(GSKNN_EARLY_RETURN, "early return: r is 0");
    return;
  }
  knn_host<float>(n, m, k, r, XB, XB2, beta, XA, XA2, alpha, D, I, r, 1);
}

void dgsknn_ref(int m, int n, int k, int r, double *XA, double *XA2, int *alpha, double *XB,
                double *XB2, int *beta, double *D, int *I) {
  if (r == 0) {
    set_status(GSKNN_EARLY_RETURN, "early return: r is 0");
    return;
  }
  knn_host<double>(n, m, k, r, XB, XB2, beta, XA, XA2, alpha, D, I, r, 1);
}

// frame/gsknn_ref_stl.cpp:81-214: the same reference algorithm with an STL heap per row.
void sgsknn_ref_stl(int m, int n, int k, int r, float *XA, float *XA2, int *alpha, float *XB,
                    float *XB2, int *beta, float *D, int *I) {
  sgsknn_ref(m, n, k, r, XA, XA2, alpha, XB, XB2, beta, D, I);
}

void dgsknn_ref_stl(int m, int n, int k, int r, double *XA, double *XA2, int *alpha,
                    double *XB, double *XB2, int *beta, double *D, int *I) {
  dgsknn_ref(m, n, k, r, XA, XA2, alpha, XB, XB2, beta, D, I);
}

}  // extern "C"
