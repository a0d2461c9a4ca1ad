// bf_api.cu -- host side of the C ABI declared in include/beamform.h.
//
// Owns the per-device state (error word, staging and operand scratch), picks
// the kernel family, and implements the drop-in form_beams() of cpu.cxx:15-16
// on top of the explicit entry points.  No entry point exits the process or
// falls back to the CPU: a shape no GPU kernel takes returns
// BF_ERR_UNSUPPORTED.
#include "bf_internal.h"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace bf {
namespace {

int to_status(cudaError_t e) {
  if (e == cudaSuccess) return BF_OK;
  if (e == cudaErrorMemoryAllocation) return BF_ERR_OUT_OF_MEMORY;
  if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return BF_ERR_NO_DEVICE;
  return BF_ERR_CUDA;
}

#define BF_TRY(expr)                          \
  do {                                        \
    const cudaError_t e_ = (expr);            \
    if (e_ != cudaSuccess) return to_status(e_); \
  } while (0)

// Growable device buffer.
struct DevBuf {
  void *p = nullptr;
  size_t cap = 0;
  cudaError_t reserve(size_t n) {
    if (n <= cap) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    const cudaError_t e = cudaMalloc(&p, std::max<size_t>(n, 256));
    if (e == cudaSuccess) cap = std::max<size_t>(n, 256);
    return e;
  }
  template <class T>
  T *as() const {
    return static_cast<T *>(p);
  }
};

// One pipeline lane of the host-pointer path: a stream and the E chunk in flight on it.
struct Lane {
  cudaStream_t s = nullptr;
  cudaEvent_t done = nullptr;
  DevBuf E;
};

constexpr int kLanes = 3;

// Scratch of a captured call (Scratch), once its graph is gone: a CUDA call cannot
// be made where that is noticed, so the next call on the device frees it.
struct GraphScratch {
  struct DeviceCtx *c;
  void *p;
  GraphScratch *next;
};

// What the host reads back after a call, and the blocks of pinned memory it is read
// from: pinned, so that the copy back is one asynchronous transfer and the call waits
// once; the device's, so that a thread neither pins memory on its first call nor frees
// it, which waits for the device, at its end.
struct DevResult {
  int err;
  uint32_t adler;
  unsigned long long adl[2];
};
struct alignas(64) HostBlock {
  DevResult r;
};
constexpr int kHostBlocks = 32;  // calls of a device that read at the same time; more read into their stack

// Memory that stays with one stream (its id, which no later stream gets) from call to
// call: in stream order each call can use what the one before prepared into.
struct Home {
  unsigned long long id = 0;
  bool taken = false;
  void *p = nullptr;
  size_t cap = 0;
};
constexpr int kHomes = 4;

struct DeviceCtx {
  std::mutex mu;
  bool ready = false;
  bool lanes_ready = false;
  Lane lanes[kLanes];
  // The fields of the device's DevResult.
  int *err = nullptr;              // error word written by kernels
  uint32_t *adler = nullptr;       // adler32 result of the separate pass
  unsigned long long *adl = nullptr;  // fused adler32 sums {sum d_i, sum i d_i} of the last checked call
  HostBlock *host = nullptr;       // null: no pinned memory to be had
  std::atomic<uint32_t> host_used{0};
  cudaMemPool_t pool = nullptr;    // of the calls' operands (Scratch)
  cudaStream_t pool_s = nullptr;   // allocations that belong to no caller's stream
  std::atomic<GraphScratch *> dropped{nullptr};
  Home homes[kHomes];              // of the first streams that made calls; under mu
  DevBuf E, A, G, J;        // staging for host-pointer calls
  DevBuf W;                 // what synchronous calls prepare: they end before they let go of mu
  DevBuf partials;          // adler32 partial sums
};

constexpr int kMaxDevices = 64;
DeviceCtx g_ctx[kMaxDevices];

// Lets this thread allocate and free while another one captures a graph in global
// mode, which would refuse it and lose that capture.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Unused memory the pool of a device keeps from one call to the next; what is above
// goes back to the device when a stream is waited for.
constexpr uint64_t kPoolKeep = uint64_t(1) << 30;
// The most that is kept until exit: of synchronous calls, and of each stream with a home.
constexpr size_t kKeptBytes = size_t(256) << 20;
constexpr size_t kHomeBytes = size_t(64) << 20;

cudaError_t make_pool(int dev, DeviceCtx &c) {
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  if (!c.pool_s) {
    const cudaError_t e = cudaStreamCreateWithFlags(&c.pool_s, cudaStreamNonBlocking);
    if (e != cudaSuccess) return e;
  }
  if (c.pool) return cudaSuccess;
  cudaMemPool_t pool = nullptr;
  uint64_t keep = kPoolKeep;
  int off = 0;  // streams stay independent: one does not wait for another's memory
  cudaError_t e = cudaMemPoolCreate(&pool, &props);
  if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &off);
  if (e == cudaSuccess) c.pool = pool;
  else if (pool) (void)cudaMemPoolDestroy(pool);
  return e;
}

void CUDART_CB drop_graph_scratch(void *arg) {
  GraphScratch *g = static_cast<GraphScratch *>(arg);
  g->next = g->c->dropped.load();
  while (!g->c->dropped.compare_exchange_weak(g->next, g)) {
  }
}

// Device memory of one asynchronous call on stream s, in stream order: calls on one
// stream use the same memory one after the other, calls on several streams never
// share it (one operand per device let the second call's preparation overwrite what
// the first one's kernel still read).  Allocation and free cost 0.5 us of host time
// together and no launch, the first ones after a wait 3 us more.  A call under capture gets memory that belongs to its
// graph: a replay reads it at any later time, beside any other call.
class Scratch {
 public:
  Scratch() = default;
  Scratch(const Scratch &) = delete;
  Scratch &operator=(const Scratch &) = delete;
  ~Scratch() {
    if (!p_ || graph_) return;
    RelaxedCapture relaxed;
    (void)cudaFreeAsync(p_, s_);
  }
  cudaError_t reserve(DeviceCtx &c, size_t n, cudaStream_t s) {
    RelaxedCapture relaxed;
    s_ = s;
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamGetCaptureInfo(s, &st, nullptr, &graph, nullptr, nullptr, nullptr);
    if (e == cudaSuccess)
      e = st == cudaStreamCaptureStatusNone     ? cudaMallocFromPoolAsync(&p_, n, c.pool, s)
          : st == cudaStreamCaptureStatusActive ? of_graph(c, n, graph)
                                                : cudaErrorStreamCaptureInvalidated;
    if (e != cudaSuccess) (void)cudaGetLastError();
    return e;
  }
  uint8_t *get() const { return static_cast<uint8_t *>(p_); }

 private:
  cudaError_t of_graph(DeviceCtx &c, size_t n, cudaGraph_t graph) {
    graph_ = true;
    GraphScratch *const g = new (std::nothrow) GraphScratch{&c, nullptr, nullptr};
    if (!g) return cudaErrorMemoryAllocation;
    cudaError_t e = cudaMallocFromPoolAsync(&g->p, n, c.pool, c.pool_s);
    if (e != cudaSuccess) {
      delete g;
      return e;
    }
    p_ = g->p;
    cudaUserObject_t owner = nullptr;
    e = cudaStreamSynchronize(c.pool_s);  // any stream may use it from here on
    if (e == cudaSuccess) e = cudaUserObjectCreate(&owner, g, drop_graph_scratch, 1, cudaUserObjectNoDestructorSync);
    if (e != cudaSuccess) {
      drop_graph_scratch(g);
      return e;
    }
    e = cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove);
    if (e != cudaSuccess) (void)cudaUserObjectRelease(owner, 1);
    return e;
  }
  void *p_ = nullptr;
  cudaStream_t s_ = nullptr;
  bool graph_ = false;  // the graph's memory, not the call's
};

// A host block for one call: pinned where one is free.
class HostResult {
 public:
  explicit HostResult(DeviceCtx &c) : c_(c) {
    if (!c.host) return;
    for (uint32_t used = c.host_used.load(); used != ~uint32_t(0);) {
      const uint32_t bit = ~used & (used + 1);  // the lowest free one
      if (c.host_used.compare_exchange_weak(used, used | bit)) {
        bit_ = bit;
        int i = 0;
        while (!(bit >> i & 1)) ++i;
        p_ = &c.host[i].r;
        return;
      }
    }
  }
  HostResult(const HostResult &) = delete;
  HostResult &operator=(const HostResult &) = delete;
  ~HostResult() { c_.host_used.fetch_and(~bit_); }
  DevResult *get() { return p_; }
  bool pinned() const { return bit_ != 0; }

 private:
  DeviceCtx &c_;
  DevResult stack_{};
  DevResult *p_ = &stack_;
  uint32_t bit_ = 0;
};
static_assert(kHostBlocks == 32, "one bit each");

int current_ctx(DeviceCtx **out) {
  int dev = -1;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return to_status(e);
  if (dev < 0 || dev >= kMaxDevices) return BF_ERR_NO_DEVICE;
  DeviceCtx &c = g_ctx[dev];
  if (!c.ready) {
    std::lock_guard<std::mutex> lk(c.mu);
    if (!c.ready) {
      BF_TRY(make_pool(dev, c));
      DevResult *res = nullptr;
      BF_TRY(cudaMalloc(&res, sizeof(DevResult)));
      BF_TRY(cudaMemset(res, 0, sizeof(DevResult)));
      if (cudaMallocHost(&c.host, kHostBlocks * sizeof(HostBlock)) != cudaSuccess) {
        (void)cudaGetLastError();
        c.host = nullptr;
      }
      c.err = &res->err;
      c.adler = &res->adler;
      c.adl = res->adl;
      c.ready = true;
    }
  }
  *out = &c;
  return BF_OK;
}

std::mutex g_dims_mu;
bool g_dims_set = false;
bf_dims g_dims{};
std::atomic<int> g_kernel{BF_KERNEL_AUTO};
thread_local int t_last_status = BF_OK;
thread_local const char *t_last_kernel = "none";

const char *simt_name() { return g_kernel.load() == BF_KERNEL_SIMT4 ? "simt4" : "simt"; }

bool dims_valid(const bf_dims *d) {
  return d && d->ntimes >= 0 && d->nfrequencies >= 0 && d->ndishes >= 0 && d->npolarizations >= 0 &&
         d->nbeams >= 0;
}

size_t esize(const bf_dims &d) {
  return static_cast<size_t>(d.ntimes) * d.nfrequencies * d.ndishes * d.npolarizations;
}
size_t asize(const bf_dims &d) { return static_cast<size_t>(d.nfrequencies) * d.nbeams * d.ndishes; }
size_t gsize(const bf_dims &d) { return static_cast<size_t>(d.nfrequencies) * d.nbeams; }
size_t jsize(const bf_dims &d) {
  return static_cast<size_t>(d.nbeams) * d.nfrequencies * d.npolarizations * d.ntimes;
}

// Sizes the operand layout for F x B x D weights.
void plan_weights(TcWeights &w, int64_t F, int64_t B, int64_t D) {
  w.F = F;
  w.B = B;
  w.D = D;
  w.Dk = (D + 7) / 8 * 8;
  tc_plan_beams(B, &w.nb_pass, &w.npass);
  w.nw = static_cast<int>((B + 7) / 8 * 8 * 2);
  w.nw_pad = w.npass * 2 * w.nb_pass;
}

size_t weights_bytes(const TcWeights &w) { return static_cast<size_t>(w.F) * w.nw * 2 * w.Dk; }

// The operand in one block: W, then (on a 256-byte boundary) the digit rows and gains.
size_t extra_at(const TcWeights &w) { return (weights_bytes(w) + 255) / 256 * 256; }
size_t operand_bytes(const TcWeights &w) { return extra_at(w) + tc_extra_bytes(w); }
void set_operand(TcWeights &w, uint8_t *p) {
  w.W = p;
  tc_set_extra(w, p + extra_at(w));
}

int choose_tensor(const bf_dims &d, bool *use_tc) {
  const int k = g_kernel.load();
  const bool ok = tc_supported(d);
  if (k == BF_KERNEL_TENSOR && !ok) return BF_ERR_UNSUPPORTED;
  if ((k == BF_KERNEL_SIMT || k == BF_KERNEL_SIMT4) && (d.npolarizations < 1 || d.npolarizations > 2))
    return BF_ERR_UNSUPPORTED;
  if (k == BF_KERNEL_AUTO && !ok && (d.npolarizations < 1 || d.npolarizations > 2)) return BF_ERR_UNSUPPORTED;
  *use_tc = (k == BF_KERNEL_TENSOR) || (k == BF_KERNEL_AUTO && ok);
  return BF_OK;
}

// The home of stream s for n bytes: null where it has none, is being captured, or the
// memory cannot be had.  The caller holds c.mu until its launches are queued.
uint8_t *home_memory(DeviceCtx &c, size_t n, cudaStream_t s) {
  unsigned long long id = 0;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone ||
      cudaStreamGetId(s, &id) != cudaSuccess)
    return nullptr;
  for (Home &h : c.homes) {
    if (h.taken && h.id != id) continue;
    h.taken = true;
    h.id = id;
    if (h.cap < n) {
      RelaxedCapture relaxed;
      if (h.p) (void)cudaFreeAsync(h.p, s);
      h.p = nullptr;
      h.cap = 0;
      if (cudaMallocFromPoolAsync(&h.p, n, c.pool, s) != cudaSuccess) {
        h.p = nullptr;
        return nullptr;
      }
      h.cap = n;
    }
    return static_cast<uint8_t *>(h.p);
  }
  return nullptr;
}

// Memory for what one call prepares.  Synchronous calls (`ends_here`: the caller waits
// for the stream before it lets go of c.mu, also after an error) share a buffer of the
// device, the first streams keep theirs (`locked`: the caller holds c.mu until its
// launches are queued), any other call has its own: from the pool in every call,
// checked calls took 55 us for 52, and an explicit call on an idle stream 55 for 50.
cudaError_t call_memory(DeviceCtx &c, Scratch &own, bool locked, bool ends_here, size_t n, cudaStream_t s, uint8_t **p) {
  if (c.dropped.load(std::memory_order_relaxed)) {
    RelaxedCapture relaxed;
    for (GraphScratch *g = c.dropped.exchange(nullptr); g;) {
      GraphScratch *const next = g->next;
      (void)cudaFreeAsync(g->p, c.pool_s);
      delete g;
      g = next;
    }
  }
  cudaError_t e = cudaSuccess;
  *p = nullptr;
  if (ends_here && n <= kKeptBytes) {
    e = c.W.reserve(n);
    *p = c.W.as<uint8_t>();
  } else {
    if (locked && n <= kHomeBytes) *p = home_memory(c, n, s);
    if (!*p) {
      e = own.reserve(c, n, s);
      *p = own.get();
    }
  }
  if (e != cudaSuccess || !*p) (void)cudaGetLastError();
  return e;
}

// A shape the tensor-core kernel does not take in place, on it all the same
// (TcPadded); *ran = false where the dp4a kernel has to take it: the rule says so,
// the memory cannot be had, or the stream is being captured (a graph would hold the
// copy of E for as long as it lives).  `rw`: resident weights, whose operand is used
// instead of preparing A; no checksum then.  `locked`: the caller holds c.mu.
int run_padded(DeviceCtx &c, bool locked, bool ends_here, const bf_dims &d, uint8_t *J, const uint8_t *E, const uint8_t *A,
               const float *G, const TcWeights *rw, cudaStream_t s, int a_layout, int j_layout,
               unsigned long long *adl, bool *fused, bool *ran) {
  *ran = false;
  const TcPadded r = tc_padded(d, E, rw != nullptr);
  if (!r.ok) return BF_OK;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    (void)cudaGetLastError();
    return BF_OK;
  }
  TcWeights w;
  if (rw) {
    w = *rw;
  } else {
    plan_weights(w, d.nfrequencies, d.nbeams, d.ndishes);
  }
  const size_t copy = r.copy ? (r.bytes + 255) / 256 * 256 : 0;  // the copy of E first, then the operand
  const size_t need = copy + (rw ? 0 : operand_bytes(w));
  Scratch own;
  uint8_t *mem = nullptr;
  if (need && call_memory(c, own, locked, ends_here, need, s, &mem) != cudaSuccess) return BF_OK;
  *ran = true;
  t_last_kernel = "tensor";
  if (adl && fused) *fused = true;
  if (!rw) {
    set_operand(w, mem + copy);
    w.G = G;
    BF_TRY(launch_prep_weights(w, A, s, a_layout, adl));
  }
  const int64_t P = d.npolarizations, per_t = d.nfrequencies * d.ndishes * P;
  for (int64_t t0 = 0; t0 < d.ntimes; t0 += r.times) {
    const int64_t nt = std::min(r.times, d.ntimes - t0);
    const uint8_t *Ec = E + t0 * per_t;
    if (r.copy) {
      BF_TRY(launch_pad_e(d, Ec, esize(d) - static_cast<size_t>(t0 * per_t), nt, mem, s));
      Ec = mem;
    }
    if (P == 1) {
      const TcRows rows{d.ntimes, nt};
      const int64_t pairs = (nt + 1) / 2;
      BF_TRY(launch_tc(w, pairs, J + t0, Ec, c.err, s, (d.ntimes + 1) / 2, kJ2, adl, J, &rows));
    } else {
      BF_TRY(launch_tc(w, nt, J + (j_layout == kJ2 ? 2 * t0 : t0), Ec, c.err, s, d.ntimes, j_layout, adl, J));
    }
  }
  return BF_OK;
}

// All four arrays on the device; asynchronous on s.  With `adl` set, a tensor-core
// launch also sums J for its adler32 (into sums that it zeroes) and *fused reports
// that it did; the SIMT kernel does not.  The caller holds c.mu.
int run_device(DeviceCtx &c, bool ends_here, const bf_dims &d, uint8_t *J, const uint8_t *E, const uint8_t *A, const float *G,
               cudaStream_t s, int a_layout = kALinear, int j_layout = kJLinear, unsigned long long *adl = nullptr,
               bool *fused = nullptr) {
  if (fused) *fused = false;
  if (jsize(d) == 0) return BF_OK;
  bool use_tc = false;
  const int st = choose_tensor(d, &use_tc);
  if (st != BF_OK) return st;
  const bool aligned = ((reinterpret_cast<uintptr_t>(E) | reinterpret_cast<uintptr_t>(J)) & 15u) == 0;
  if (use_tc && !aligned && g_kernel.load() == BF_KERNEL_TENSOR) return BF_ERR_UNSUPPORTED;
  use_tc = use_tc && aligned;
  if (!use_tc) {
    if (g_kernel.load() == BF_KERNEL_AUTO) {
      bool ran = false;
      const int ps = run_padded(c, true, ends_here, d, J, E, A, G, nullptr, s, a_layout, j_layout, adl, fused, &ran);
      if (ran || ps != BF_OK) return ps;
    }
    t_last_kernel = simt_name();
    return to_status(launch_simt(d, J, E, A, G, s, 0, a_layout, j_layout));
  }
  TcWeights w;
  plan_weights(w, d.nfrequencies, d.nbeams, d.ndishes);
  Scratch own;
  uint8_t *mem = nullptr;
  BF_TRY(call_memory(c, own, true, ends_here, operand_bytes(w), s, &mem));
  set_operand(w, mem);
  w.G = G;
  if (adl && fused) *fused = true;
  BF_TRY(launch_prep_weights(w, A, s, a_layout, adl));
  t_last_kernel = "tensor";
  return to_status(launch_tc(w, d.ntimes, J, E, c.err, s, 0, j_layout, adl, J));
}

// Waits for the stream and reads the device results; a kernel's error clears the
// error word and is the status.  `behind_kernel`: the stream's last work is a
// kernel, and another one writes the results faster than a copy; behind a copy a
// copy is faster (host call 294 against 296 us).
int read_and_clear_err(DeviceCtx &c, cudaStream_t s, DevResult *out = nullptr, bool behind_kernel = false) {
  HostResult block(c);
  DevResult *const h = block.get();
  static_assert(sizeof(DevResult) % 4 == 0 && sizeof(DevResult) <= 128, "words of one warp");
  if (behind_kernel && block.pinned())
    BF_TRY(launch_write_words(c.err, h, sizeof(DevResult) / 4, s));
  else
    BF_TRY(cudaMemcpyAsync(h, c.err, sizeof(DevResult), cudaMemcpyDeviceToHost, s));
  BF_TRY(cudaStreamSynchronize(s));
  if (out) *out = *h;
  if (h->err != 0) {
    BF_TRY(cudaMemsetAsync(c.err, 0, sizeof(int), s));
    BF_TRY(cudaStreamSynchronize(s));
    return BF_ERR_DEVICE_TIMEOUT;
  }
  return BF_OK;
}

// Times per pipeline chunk of the host-pointer path: about 256 MB of E per
// chunk (a multiple of 64 times), or all of T when that is one chunk anyway.
// BF_HOST_CHUNK_BYTES overrides the chunk size (tuning and tests).
int64_t chunk_times(const bf_dims &d) {
  const int64_t per_t = std::max<int64_t>(1, d.nfrequencies * d.ndishes * d.npolarizations);
  int64_t bytes = int64_t(256) << 20;
  if (const char *env = std::getenv("BF_HOST_CHUNK_BYTES")) bytes = std::max<int64_t>(1, std::atoll(env));
  int64_t tc = std::max<int64_t>(64, (bytes / per_t) / 64 * 64);
  return tc * 3 / 2 >= d.ntimes ? d.ntimes : tc;
}

// Copies bytes [off, off + len) of each of `rows` rows (`pitch` bytes apart)
// from the device J to the caller's J in pinned host memory (its device
// mapping): one 16-byte load and streaming store per step, so a warp writes
// whole 64-byte lines across the host link.  off, len, pitch and both base
// addresses are multiples of 16.
__global__ void __launch_bounds__(256) drain_rows(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst,
                                                  int64_t rows, int64_t pitch, int64_t off, int64_t len) {
  const int64_t per_row = len / 16;
  const int64_t total = rows * per_row;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / per_row;
    const int64_t o = r * pitch + off + 16 * (i - r * per_row);
    __stcs(reinterpret_cast<uint4 *>(dst + o), __ldcs(reinterpret_cast<const uint4 *>(src + o)));
  }
}

// Device address of the caller's J when it is pinned host memory that the
// drain can write directly (16-byte aligned, rows a multiple of 16 bytes);
// null otherwise (pageable memory: one copy at the end instead).
uint8_t *mapped_host_j(uint8_t *J, const bf_dims &d, int j_layout) {
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, J) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  const int64_t pitch = j_layout == kJ2 ? d.ntimes * d.npolarizations : d.ntimes;
  if (at.type != cudaMemoryTypeHost || !at.devicePointer || (pitch & 15) ||
      (reinterpret_cast<uintptr_t>(at.devicePointer) & 15))
    return nullptr;
  return static_cast<uint8_t *>(at.devicePointer);
}

// Host-pointer pass pipelined over time chunks: E[t0..t1][f][d][p] is
// contiguous, so each chunk goes in with one copy on one of kLanes streams and
// is beamformed while the next chunk copies; every chunk writes its times of J
// (rows of ntimes bytes) in a device buffer.  When the caller's J is pinned,
// a drain kernel behind each chunk writes the chunk's row segments straight
// into it, so J leaves over the link while later chunks of E arrive;
// otherwise J is copied out once at the end.
// A, G and the tensor-core operand are uploaded / prepared once.  Synchronous;
// the caller holds c.mu.
int run_host_pipelined(DeviceCtx &c, const bf_dims &d, uint8_t *J, const uint8_t *E, const uint8_t *A,
                       const float *G, cudaStream_t caller, int a_layout, int j_layout,
                       unsigned long long *adl = nullptr, bool *fused = nullptr) {
  if (fused) *fused = false;
  if (!c.lanes_ready) {
    for (Lane &l : c.lanes) {
      BF_TRY(cudaStreamCreateWithFlags(&l.s, cudaStreamNonBlocking));
      BF_TRY(cudaEventCreateWithFlags(&l.done, cudaEventDisableTiming));
    }
    c.lanes_ready = true;
  }
  bool use_tc = false;
  int st = choose_tensor(d, &use_tc);
  if (st != BF_OK) return st;
  const int64_t T = d.ntimes, per_t = d.nfrequencies * d.ndishes * d.npolarizations;
  const int64_t tc = chunk_times(d);
  BF_TRY(c.A.reserve(asize(d)));
  BF_TRY(c.G.reserve(gsize(d) * sizeof(float)));
  BF_TRY(c.J.reserve(jsize(d)));
  Lane &l0 = c.lanes[0];
  // work already queued on the caller's stream comes first
  BF_TRY(cudaEventRecord(l0.done, caller));
  BF_TRY(cudaStreamWaitEvent(l0.s, l0.done, 0));
  BF_TRY(cudaMemcpyAsync(c.A.p, A, asize(d), cudaMemcpyHostToDevice, l0.s));
  BF_TRY(cudaMemcpyAsync(c.G.p, G, gsize(d) * sizeof(float), cudaMemcpyHostToDevice, l0.s));
  TcWeights w;
  if (use_tc) {
    plan_weights(w, d.nfrequencies, d.nbeams, d.ndishes);
    BF_TRY(c.W.reserve(operand_bytes(w)));
    set_operand(w, c.W.as<uint8_t>());
    w.G = c.G.as<float>();
    // every chunk's launch adds into the same sums, positions from the start of J
    BF_TRY(launch_prep_weights(w, c.A.as<uint8_t>(), l0.s, a_layout, adl));
    if (adl && fused) *fused = true;
  }
  BF_TRY(cudaEventRecord(l0.done, l0.s));
  for (int i = 1; i < kLanes; ++i) BF_TRY(cudaStreamWaitEvent(c.lanes[i].s, l0.done, 0));
  t_last_kernel = use_tc ? "tensor" : simt_name();
  uint8_t *jmap = mapped_host_j(J, d, j_layout);
  const int64_t P = d.npolarizations;
  const int64_t jrows = j_layout == kJ2 ? d.nbeams * d.nfrequencies : d.nbeams * d.nfrequencies * P;
  const int64_t jpitch = j_layout == kJ2 ? T * P : T;
  const int64_t jscale = j_layout == kJ2 ? P : 1;  // bytes per time in a row
  for (int64_t t0 = 0, k = 0; t0 < T; t0 += tc, ++k) {
    Lane &l = c.lanes[k % kLanes];
    const int64_t nt = std::min(tc, T - t0);
    BF_TRY(l.E.reserve(static_cast<size_t>(nt * per_t)));
    BF_TRY(cudaMemcpyAsync(l.E.p, E + t0 * per_t, static_cast<size_t>(nt * per_t), cudaMemcpyHostToDevice, l.s));
    // the chunk's first time: byte t0 of each J row, byte t0 * P of each J2 row
    uint8_t *Jc = c.J.as<uint8_t>() + (j_layout == kJ2 ? t0 * d.npolarizations : t0);
    if (use_tc) {
      BF_TRY(launch_tc(w, nt, Jc, l.E.as<uint8_t>(), c.err, l.s, T, j_layout, adl, c.J.as<uint8_t>()));
    } else {
      const bf_dims dc{nt, d.nfrequencies, d.ndishes, d.npolarizations, d.nbeams};
      BF_TRY(launch_simt(dc, Jc, l.E.as<uint8_t>(), c.A.as<uint8_t>(), c.G.as<float>(), l.s, T, a_layout, j_layout));
    }
    if (jmap) {
      const int grid = 2 * num_sms();
      drain_rows<<<grid, 256, 0, l.s>>>(c.J.as<uint8_t>(), jmap, jrows, jpitch, t0 * jscale, nt * jscale);
      BF_TRY(cudaGetLastError());
    }
  }
  for (int i = 1; i < kLanes; ++i) {
    BF_TRY(cudaEventRecord(c.lanes[i].done, c.lanes[i].s));
    BF_TRY(cudaStreamWaitEvent(l0.s, c.lanes[i].done, 0));
  }
  if (!jmap) BF_TRY(cudaMemcpyAsync(J, c.J.p, jsize(d), cudaMemcpyDeviceToHost, l0.s));
  BF_TRY(cudaStreamSynchronize(l0.s));
  return read_and_clear_err(c, caller);
}

}  // namespace

bool simt_four_multiply() { return g_kernel.load() == BF_KERNEL_SIMT4; }

int device_error_word(int **out) {
  DeviceCtx *c = nullptr;
  const int st = current_ctx(&c);
  if (st != BF_OK) return st;
  *out = c->err;
  return BF_OK;
}

}  // namespace bf

using namespace bf;

// form_beams over any pointer kind and layout; with adler_out set, also the
// adler32 of the J it wrote (synchronous then).
static int form_beams_impl(const bf_dims *dims, uint8_t *J, const uint8_t *E, const uint8_t *A, const float *G,
                           int a_layout, int j_layout, int ptr_kind, bf_stream_t stream, uint32_t *adler_out);

extern "C" {

int bf_set_dims(const bf_dims *dims) {
  if (!dims_valid(dims)) return BF_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(g_dims_mu);
  g_dims = *dims;
  g_dims_set = true;
  return BF_OK;
}

int bf_last_status(void) { return t_last_status; }

const char *bf_last_kernel(void) { return t_last_kernel; }

const char *bf_status_string(int status) {
  switch (status) {
    case BF_OK: return "ok";
    case BF_ERR_INVALID_ARGUMENT: return "invalid argument";
    case BF_ERR_UNSUPPORTED: return "shape or alignment not supported by any GPU kernel";
    case BF_ERR_NO_DEVICE: return "no usable CUDA device";
    case BF_ERR_CUDA: return "CUDA runtime error";
    case BF_ERR_OUT_OF_MEMORY: return "out of memory";
    case BF_ERR_DEVICE_TIMEOUT: return "a device-side wait expired; results are invalid";
    case BF_ERR_NOT_CONFIGURED: return "form_beams() called before bf_set_dims()";
    case BF_ERR_SIZE_MISMATCH: return "weights were built for a different shape";
    case BF_ERR_TOO_LARGE: return "problem exceeds the fixed scratch of bf_form_beams_noalloc";
    default: return "unknown status";
  }
}

int bf_set_kernel(int kernel) {
  if (kernel < BF_KERNEL_AUTO || kernel > BF_KERNEL_SIMT4) return BF_ERR_INVALID_ARGUMENT;
  g_kernel.store(kernel);
  return BF_OK;
}

int bf_set_test_stall(int on) {
  tc_set_test_stall(on);
  return BF_OK;
}

int bf_set_test_one_cta(int on) {
  tc_set_test_one_cta(on);
  return BF_OK;
}

int bf_form_beams_ex(const bf_dims *dims, uint8_t *J, const uint8_t *E, const uint8_t *A, const float *G,
                     int ptr_kind, bf_stream_t stream) {
  return bf_form_beams_layout(dims, J, E, A, G, BF_A_LINEAR, BF_J_LINEAR, ptr_kind, stream);
}

int bf_form_beams_layout(const bf_dims *dims, uint8_t *J, const uint8_t *E, const uint8_t *A, const float *G,
                         int a_layout, int j_layout, int ptr_kind, bf_stream_t stream) {
  return form_beams_impl(dims, J, E, A, G, a_layout, j_layout, ptr_kind, stream, nullptr);
}

int bf_form_beams_adler(const bf_dims *dims, uint8_t *J, const uint8_t *E, const uint8_t *A, const float *G,
                        int a_layout, int j_layout, int ptr_kind, uint32_t *adler, bf_stream_t stream) {
  if (!adler) return BF_ERR_INVALID_ARGUMENT;
  return form_beams_impl(dims, J, E, A, G, a_layout, j_layout, ptr_kind, stream, adler);
}

}  // extern "C"

namespace bf {
namespace {

// Ends a checked call: the adler32 of the n bytes of device J, from the fused
// sums when the tensor-core kernel ran, else by the separate two-kernel pass, and
// the call's status.  Synchronises the stream.
int finish_adler(DeviceCtx &c, bool fused, const uint8_t *Jdev, size_t n, cudaStream_t s, uint32_t *out,
                 bool behind_kernel = false) {
  if (!fused) {
    BF_TRY(c.partials.reserve(static_cast<size_t>(adler_nchunks(n)) * 2 * sizeof(uint32_t)));
    BF_TRY(launch_adler_partials(Jdev, n, c.partials.as<uint32_t>(), s));
    BF_TRY(launch_adler_combine(c.partials.as<uint32_t>(), n, c.adler, s));
  }
  DevResult r{};
  const int st = read_and_clear_err(c, s, &r, behind_kernel || !fused);
  if (st == BF_OK) *out = fused ? adler_finish(r.adl[0], r.adl[1], n) : r.adler;
  return st;
}

// After a failed synchronous call: wait for what it had already queued (copies
// from the caller's E, drains into the caller's J, the operand's preparation) so
// that nothing touches the caller's buffers, or the device's, once the call has
// returned.
void settle_after_error(DeviceCtx &c, cudaStream_t s) {
  (void)cudaStreamSynchronize(s);
  if (c.lanes_ready)
    for (Lane &l : c.lanes) (void)cudaStreamSynchronize(l.s);
  (void)cudaGetLastError();
}

}  // namespace
}  // namespace bf

static int form_beams_impl(const bf_dims *dims, uint8_t *J, const uint8_t *E, const uint8_t *A, const float *G,
                           int a_layout, int j_layout, int ptr_kind, bf_stream_t stream, uint32_t *adler_out) {
  if (!dims_valid(dims)) return BF_ERR_INVALID_ARGUMENT;
  if ((a_layout != BF_A_LINEAR && a_layout != BF_A_A2) || (j_layout != BF_J_LINEAR && j_layout != BF_J_J2))
    return BF_ERR_INVALID_ARGUMENT;
  if (a_layout == BF_A_A2 && !a2_supported(dims->ndishes)) return BF_ERR_UNSUPPORTED;
  if (ptr_kind != BF_PTR_HOST && ptr_kind != BF_PTR_DEVICE) return BF_ERR_INVALID_ARGUMENT;
  const bf_dims d = *dims;
  if (jsize(d) == 0) {
    if (adler_out) *adler_out = 1u;  // adler32 of no bytes
    return BF_OK;
  }
  if (!J || (esize(d) && !E) || (asize(d) && !A) || !G) return BF_ERR_INVALID_ARGUMENT;
  DeviceCtx *c = nullptr;
  int st = current_ctx(&c);
  if (st != BF_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  std::lock_guard<std::mutex> lk(c->mu);
  unsigned long long *adl = adler_out ? c->adl : nullptr;
  bool fused = false;
  if (ptr_kind == BF_PTR_DEVICE) {
    st = run_device(*c, adler_out != nullptr, d, J, E, A, G, s, a_layout, j_layout, adl, &fused);
    if (!adler_out) return st;
    if (st == BF_OK) st = finish_adler(*c, fused, J, jsize(d), s, adler_out, true);
    if (st != BF_OK && st != BF_ERR_UNSUPPORTED) settle_after_error(*c, s);  // a refused shape queued nothing
    return st;
  }

  // Host pointers: stage in, compute, stage out, synchronously (cuda.cu:274-314 does the same around its
  // kernel), pipelined over time chunks when there is more than one.
  const int hs = [&]() -> int {
    if (chunk_times(d) < d.ntimes) {
      const int ps = run_host_pipelined(*c, d, J, E, A, G, s, a_layout, j_layout, adl, &fused);
      if (ps != BF_OK || !adler_out) return ps;
      return finish_adler(*c, fused, c->J.as<uint8_t>(), jsize(d), s, adler_out);
    }
    BF_TRY(c->E.reserve(esize(d)));
    BF_TRY(c->A.reserve(asize(d)));
    BF_TRY(c->G.reserve(gsize(d) * sizeof(float)));
    BF_TRY(c->J.reserve(jsize(d)));
    BF_TRY(cudaMemcpyAsync(c->E.p, E, esize(d), cudaMemcpyHostToDevice, s));
    BF_TRY(cudaMemcpyAsync(c->A.p, A, asize(d), cudaMemcpyHostToDevice, s));
    BF_TRY(cudaMemcpyAsync(c->G.p, G, gsize(d) * sizeof(float), cudaMemcpyHostToDevice, s));
    const int rs = run_device(*c, true, d, c->J.as<uint8_t>(), c->E.as<uint8_t>(), c->A.as<uint8_t>(), c->G.as<float>(),
                              s, a_layout, j_layout, adl, &fused);
    if (rs != BF_OK) return rs;
    BF_TRY(cudaMemcpyAsync(J, c->J.p, jsize(d), cudaMemcpyDeviceToHost, s));
    return adler_out ? finish_adler(*c, fused, c->J.as<uint8_t>(), jsize(d), s, adler_out) : read_and_clear_err(*c, s);
  }();
  if (hs != BF_OK) settle_after_error(*c, s);
  return hs;
}

extern "C" {

void form_beams(uint8_t *J, const uint8_t *E, const uint8_t *A, const float *G) {
  bf_dims d;
  {
    std::lock_guard<std::mutex> lk(g_dims_mu);
    if (!g_dims_set) {
      t_last_status = BF_ERR_NOT_CONFIGURED;
      return;
    }
    d = g_dims;
  }
  t_last_status = bf_form_beams_ex(&d, J, E, A, G, BF_PTR_HOST, nullptr);
}

int bf_stream_status(bf_stream_t stream) {
  DeviceCtx *c = nullptr;
  const int st = current_ctx(&c);
  if (st != BF_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return to_status(e);
  return read_and_clear_err(*c, s);
}

int bf_weights_create(bf_weights **out, int64_t nfrequencies, int64_t nbeams, int64_t ndishes, const uint8_t *A,
                      const float *G, int ptr_kind, bf_stream_t stream) {
  if (!out || nfrequencies <= 0 || nbeams <= 0 || ndishes <= 0 || !A || !G) return BF_ERR_INVALID_ARGUMENT;
  if (ptr_kind != BF_PTR_HOST && ptr_kind != BF_PTR_DEVICE) return BF_ERR_INVALID_ARGUMENT;
  DeviceCtx *c = nullptr;
  int st = current_ctx(&c);
  if (st != BF_OK) return st;
  bf_weights *w = new bf_weights();
  cudaGetDevice(&w->device);
  plan_weights(w->tc, nfrequencies, nbeams, ndishes);
  const size_t na = static_cast<size_t>(nfrequencies) * nbeams * ndishes;
  const size_t ng = static_cast<size_t>(nfrequencies) * nbeams;
  cudaError_t e = cudaMalloc(&w->A, na);
  if (e == cudaSuccess) e = cudaMalloc(&w->G, ng * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&w->tc.W, weights_bytes(w->tc));
  uint8_t *extra = nullptr;
  if (e == cudaSuccess) e = cudaMalloc(&extra, tc_extra_bytes(w->tc));
  if (e == cudaSuccess) tc_set_extra(w->tc, extra);
  if (e != cudaSuccess) {
    bf_weights_destroy(w);
    return to_status(e);
  }
  w->tc.G = w->G;
  st = bf_weights_update(w, A, G, ptr_kind, stream);
  if (st != BF_OK) {
    bf_weights_destroy(w);
    return st;
  }
  *out = w;
  return BF_OK;
}

// Whether all n bytes at p lie in one allocation of this device: what a copy from
// there would check.
static bool on_device(const void *p, size_t n, int device) {
  using Fn = CUresult (*)(unsigned int, CUpointer_attribute *, void **, CUdeviceptr);
  static const Fn fn = []() -> Fn {
    void *q = nullptr;
    cudaDriverEntryPointQueryResult r{};
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &q, 12000, cudaEnableDefault, &r) != cudaSuccess ||
        r != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<Fn>(q);
  }();
  unsigned type = 0;
  int ordinal = -1;
  CUdeviceptr start = 0;
  size_t size = 0;
  CUpointer_attribute at[4] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL,
                               CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
  void *out[4] = {&type, &ordinal, &start, &size};
  const CUdeviceptr at0 = reinterpret_cast<CUdeviceptr>(p);
  if (!fn || fn(4, at, out, at0) != CUDA_SUCCESS) return false;
  return type == CU_MEMORYTYPE_DEVICE && ordinal == device && at0 >= start && n <= size && at0 - start <= size - n;
}

int bf_weights_update(bf_weights *w, const uint8_t *A, const float *G, int ptr_kind, bf_stream_t stream) {
  if (!w || !A || !G) return BF_ERR_INVALID_ARGUMENT;
  if (ptr_kind != BF_PTR_HOST && ptr_kind != BF_PTR_DEVICE) return BF_ERR_INVALID_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t na = static_cast<size_t>(w->tc.F) * w->tc.B * w->tc.D;
  const size_t ng = static_cast<size_t>(w->tc.F) * w->tc.B;
  // The preparation reads every byte of A and G once: it writes the copies on the
  // way where it can read them in place, instead of two device copies in front of
  // it (update and pass, t=80 f=1 d=416 b=19 15.0 -> 10.8 us, t=1024 f=16 d=1024 b=512
  // 75.1 -> 67.9).
  if (ptr_kind == BF_PTR_DEVICE && (reinterpret_cast<uintptr_t>(G) & 3u) == 0 && on_device(A, na, w->device) &&
      on_device(G, ng * sizeof(float), w->device)) {
    TcWeights t = w->tc;
    t.G = G;
    return to_status(launch_prep_weights(t, A, s, kALinear, nullptr, w->A, w->G));
  }
  const cudaMemcpyKind k = ptr_kind == BF_PTR_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  BF_TRY(cudaMemcpyAsync(w->A, A, na, k, s));
  BF_TRY(cudaMemcpyAsync(w->G, G, ng * sizeof(float), k, s));
  BF_TRY(launch_prep_weights(w->tc, w->A, s));
  if (ptr_kind == BF_PTR_HOST) BF_TRY(cudaStreamSynchronize(s));
  return BF_OK;
}

int bf_weights_destroy(bf_weights *w) {
  if (!w) return BF_OK;
  if (w->A) cudaFree(w->A);
  if (w->G) cudaFree(w->G);
  if (w->tc.W) cudaFree(w->tc.W);
  if (w->tc.dig) cudaFree(w->tc.dig);
  delete w;
  return BF_OK;
}

int bf_form_beams_resident(const bf_weights *w, int64_t ntimes, uint8_t *J, const uint8_t *E, bf_stream_t stream) {
  if (!w || ntimes < 0 || (ntimes > 0 && (!J || !E))) return BF_ERR_INVALID_ARGUMENT;
  if (ntimes == 0) return BF_OK;
  DeviceCtx *c = nullptr;
  const int st = current_ctx(&c);
  if (st != BF_OK) return st;
  const bf_dims d{ntimes, w->tc.F, w->tc.D, 2, w->tc.B};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  bool use_tc = false;
  const int cs = choose_tensor(d, &use_tc);
  if (cs != BF_OK) return cs;
  if (use_tc && ((reinterpret_cast<uintptr_t>(E) | reinterpret_cast<uintptr_t>(J)) & 15u)) {
    if (g_kernel.load() == BF_KERNEL_TENSOR) return BF_ERR_UNSUPPORTED;
    use_tc = false;
  }
  if (use_tc) {
    t_last_kernel = "tensor";
    return to_status(launch_tc(w->tc, ntimes, J, E, c->err, s));
  }
  if (g_kernel.load() == BF_KERNEL_AUTO) {
    bool ran = false;
    std::unique_lock<std::mutex> lk(c->mu, std::try_to_lock);  // for the stream's home, where no other call has it
    const int ps = run_padded(*c, lk.owns_lock(), false, d, J, E, nullptr, nullptr, &w->tc, s, kALinear, kJLinear, nullptr,
                              nullptr, &ran);
    if (ran || ps != BF_OK) return ps;
  }
  t_last_kernel = simt_name();
  return to_status(launch_simt(d, J, E, w->A, w->G, s));
}

int bf_adler32_device(const uint8_t *data, size_t len, uint32_t *out, bf_stream_t stream) {
  if (!out || (len && !data)) return BF_ERR_INVALID_ARGUMENT;
  if (len == 0) {
    *out = 1u;
    return BF_OK;
  }
  DeviceCtx *c = nullptr;
  const int st = current_ctx(&c);
  if (st != BF_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  std::lock_guard<std::mutex> lk(c->mu);
  BF_TRY(c->partials.reserve(static_cast<size_t>(adler_nchunks(len)) * 2 * sizeof(uint32_t)));
  BF_TRY(launch_adler_partials(data, len, c->partials.as<uint32_t>(), s));
  BF_TRY(launch_adler_combine(c->partials.as<uint32_t>(), len, c->adler, s));
  HostResult block(*c);
  DevResult *const h = block.get();
  BF_TRY(cudaMemcpyAsync(&h->adler, c->adler, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  BF_TRY(cudaStreamSynchronize(s));
  *out = h->adler;
  return BF_OK;
}

int bf_fill_random_device(uint8_t *dst, size_t n, uint64_t seed, uint64_t stream_id, bf_stream_t stream) {
  if (n && !dst) return BF_ERR_INVALID_ARGUMENT;
  return to_status(launch_fill_random(dst, n, seed, stream_id, static_cast<cudaStream_t>(stream)));
}

int bf_fill_random_host(uint8_t *dst, size_t n, uint64_t seed, uint64_t stream_id) {
  if (n && !dst) return BF_ERR_INVALID_ARGUMENT;
  auto mix64 = [](uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  };
  const uint64_t key = mix64(seed * 2u + stream_id + 1u);
  const size_t nwords = (n + 7) / 8;
  const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
  const size_t per = (nwords + hw - 1) / hw;
  std::vector<std::thread> th;
  for (unsigned i = 0; i < hw; ++i) {
    const size_t j0 = i * per, j1 = std::min(nwords, j0 + per);
    if (j0 >= j1) break;
    th.emplace_back([=]() {
      for (size_t j = j0; j < j1; ++j) {
        const uint64_t w = mix64(key + static_cast<uint64_t>(j + 1) * 0x9E3779B97F4A7C15ull);
        if (8 * j + 8 <= n) {
          uint8_t b[8];
          for (int k = 0; k < 8; ++k) b[k] = static_cast<uint8_t>(w >> (8 * k));
          std::memcpy(dst + 8 * j, b, 8);
        } else {
          for (size_t k = 0; 8 * j + k < n; ++k) dst[8 * j + k] = static_cast<uint8_t>(w >> (8 * k));
        }
      }
    });
  }
  for (auto &t : th) t.join();
  return BF_OK;
}

int bf_gains_host(const bf_dims *dims, float *G) {
  if (!dims_valid(dims) || !G) return BF_ERR_INVALID_ARGUMENT;
  // arraysizes.cxx:31-32: float(n) / Gsize / ndishes * (15 + n % 15) / 30, left to right in float
  const int64_t gs = dims->nfrequencies * dims->nbeams;
  const float fg = static_cast<float>(static_cast<uint64_t>(gs));
  const float fd = static_cast<float>(static_cast<uint64_t>(dims->ndishes));
  for (int64_t n = 0; n < gs; ++n) {
    float g = static_cast<float>(static_cast<uint64_t>(n));
    g = g / fg;
    g = g / fd;
    g = g * static_cast<float>(static_cast<uint64_t>(15 + n % 15));
    g = g / 30.0f;
    G[n] = g;
  }
  return BF_OK;
}

}  // extern "C"
