// Runtime half of the C ABI: device, memory kinds, copies, event timing and
// CUDA-graph record/replay.  Stands where the reference's Vulkan runtime stood
// (vk.Device / vk.Buffer / vk.Graph); nothing here computes.
#include "common.cuh"

#include <chrono>
#include <cstdlib>
#include <thread>

#if defined(__x86_64__)
#include <immintrin.h>
#endif

static thread_local char g_err[1024] = "";

void vkg_set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

extern "C" const char* vkg_last_error(void) { return g_err; }

extern "C" const char* vkg_version(void) { return "vkgrad_b200 0.1 (sm_100a)"; }

extern "C" int vkg_device_count(int* count) {
  if (!count) VKG_FAIL("null count");
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  *count = n;
  return 0;
}

// ---- stamps ------------------------------------------------------------------------------

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Both stamps leave the kernels between them free to overlap: the first lets its successor set up
// meanwhile, the second is launched ahead and waits (a 256^3 GEMM call 15.4 -> 13.7 us).
__global__ void k_stamp_begin(vkg_stamp_dev* d) {
  pdl_trigger();
  d->t0 = global_ns();
}

// Runs after everything before it on the stream has completed.  The fence orders what that work
// left in mapped host memory before the number the host polls; with the fence between two stores
// of its own instead, the second waited for the first to cross the host link (6 us).
__global__ void k_stamp_end(vkg_stamp_dev* d, vkg_stamp_host* h) {
  pdl_wait();
  const uint64_t t1 = global_ns();
  const uint32_t n = d->seq + 1;
  d->seq = n;
  const uint64_t ticks = (t1 - d->t0) >> 5;
  __threadfence_system();
  asm volatile("st.volatile.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(h), "r"(n),
               "r"(ticks > 0xffffffffull ? 0xffffffffu : (uint32_t)ticks), "r"((uint32_t)t1), "r"((uint32_t)(t1 >> 32))
               : "memory");
}

bool vkg_is_stamp_kernel(const void* func) {
  return func == (const void*)k_stamp_begin || func == (const void*)k_stamp_end;
}

// Slots come in pages of 64 and go back to the free list with their running number.
static int stamp_acquire(vkg_device* dev, vkg_stamp* out) {
  vkg_stamp_pool& pool = *dev->stamps;
  std::lock_guard<std::mutex> lock(pool.mu);
  if (pool.free_slots.empty()) {
    constexpr int N = 64;
    void *h = nullptr, *hd = nullptr, *d = nullptr;
    VKG_CUDA(cudaHostAlloc(&h, N * sizeof(vkg_stamp_host), cudaHostAllocMapped | cudaHostAllocPortable));
    pool.pages_host.push_back(h);
    memset(h, 0, N * sizeof(vkg_stamp_host));
    VKG_CUDA(cudaHostGetDevicePointer(&hd, h, 0));
    VKG_CUDA(cudaMalloc(&d, N * sizeof(vkg_stamp_dev)));
    pool.pages_dev.push_back(d);
    VKG_CUDA(cudaMemset(d, 0, N * sizeof(vkg_stamp_dev)));
    for (int i = 0; i < N; ++i) {
      vkg_stamp s;
      s.host = (volatile vkg_stamp_host*)h + i;
      s.host_dev = (vkg_stamp_host*)hd + i;
      s.dev = (vkg_stamp_dev*)d + i;
      pool.free_slots.push_back(s);
    }
  }
  *out = pool.free_slots.back();
  pool.free_slots.pop_back();
  return 0;
}

static void stamp_release(vkg_stamp_pool* pool, const vkg_stamp& st) {
  if (!st.dev) return;
  std::lock_guard<std::mutex> lock(pool->mu);
  pool->free_slots.push_back(st);
}

vkg_stamp_pool::~vkg_stamp_pool() {
  for (void* p : pages_host) cudaFreeHost(p);
  for (void* p : pages_dev) cudaFree(p);
}

int vkg_stamp_begin(vkg_device* dev, vkg_stamp* st) {
  k_stamp_begin<<<1, 1, 0, dev->stream>>>(st->dev);
  return vkg_check_launch("stamp_begin");
}

int vkg_stamp_end(vkg_device* dev, vkg_stamp* st) {
  VKG_CUDA(vkg_launch(dev, VKG_K_SMALL | VKG_SHORT, k_stamp_end, dim3(1), dim3(1), 0, 1, st->dev, st->host_dev));
  return vkg_check_launch("stamp_end");
}

extern "C" int vkg_device_create(int ordinal, vkg_device** out) {
  if (!out) VKG_FAIL("null out");
  *out = nullptr;
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
    cudaGetLastError();
    VKG_FAIL("no CUDA device is visible; this library has no CPU fallback");
  }
  VKG_REQUIRE(ordinal >= 0 && ordinal < n, "device ordinal %d out of range (%d devices)",
              ordinal, n);
  VKG_CUDA(cudaSetDevice(ordinal));
  cudaDeviceProp prop;
  VKG_CUDA(cudaGetDeviceProperties(&prop, ordinal));
  VKG_REQUIRE(prop.major == 10,
              "device %d is compute capability %d.%d; this library is built for sm_100a only",
              ordinal, prop.major, prop.minor);
  vkg_device* d = new vkg_device();
  d->ordinal = ordinal;
  d->sm_count = prop.multiProcessorCount;
  d->cc_major = prop.major;
  d->cc_minor = prop.minor;
  d->total_bytes = prop.totalGlobalMem;
  d->gemm_smem_optin = prop.sharedMemPerBlockOptin;
  snprintf(d->name, sizeof(d->name), "%.127s", prop.name);
  VKG_CUDA(cudaStreamCreateWithFlags(&d->stream, cudaStreamNonBlocking));
  void* host = nullptr;
  VKG_CUDA(cudaHostAlloc(&host, 64, cudaHostAllocMapped | cudaHostAllocPortable));
  memset(host, 0, 64);
  d->err_host = (volatile uint32_t*)host;
  VKG_CUDA(cudaHostGetDevicePointer((void**)&d->err_dev, host, 0));
  cudaDriverEntryPointQueryResult qres;
  void* fn = nullptr;
  cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
  if (e != cudaSuccess || qres != cudaDriverEntryPointSuccess || !fn) {
    cudaGetLastError();
    delete d;
    VKG_FAIL("cuTensorMapEncodeTiled is not available from this driver");
  }
  d->encode_tiled = fn;
  if (stamp_acquire(d, &d->timer)) return 1;
  d->gemm_plans = vkg_gemm_plans_create();
  const char* pdl = getenv("VKG_PDL");
  if (pdl && pdl[0]) d->pdl = pdl[0] == '1' ? 1 : 0;     // default: short launches only
  const char* ts = getenv("VKG_TMA_STORE");
  d->tma_store = !(ts && ts[0] == '0');
  const char* a1 = getenv("VKG_ATTN_ONE_PASS");
  if (a1 && a1[0]) d->attn_one_pass = a1[0] == '1';
  const char* lim = getenv("VKG_SM_LIMIT");      // persistent kernels' grid cap, for experiments
  if (lim && lim[0]) d->sm_limit = atoi(lim);
  const char* mask = getenv("VKG_PDL_MASK");     // kernel families, for experiments
  if (mask && mask[0]) d->pdl_mask = (unsigned)strtoul(mask, nullptr, 0);
  *out = d;
  return 0;
}

extern "C" int vkg_set_pdl(vkg_device* dev, int on) {
  if (!dev) VKG_FAIL("null device");
  VKG_REQUIRE(!dev->capturing, "set_pdl: not while a graph is being recorded");
  dev->pdl = on != 0;
  return 0;
}

extern "C" int vkg_set_tuning(vkg_device* dev, int key, int64_t value) {
  if (!dev) VKG_FAIL("null device");
  // the SM limit is host state read when a launch is enqueued: it may change between the
  // launches of one recording
  VKG_REQUIRE(!dev->capturing || key == VKG_TUNE_SM_LIMIT,
              "set_tuning: not while a graph is being recorded");
  switch (key) {
    case VKG_TUNE_PDL: dev->pdl = value != 0; break;
    case VKG_TUNE_PDL_FAMILIES: dev->pdl_mask = (unsigned)value; break;
    case VKG_TUNE_TMA_STORE: dev->tma_store = value != 0; break;
    case VKG_TUNE_SM_LIMIT:
      VKG_REQUIRE(value >= 0, "set_tuning: the SM limit cannot be negative");
      dev->sm_limit = (int)value;
      break;
    case VKG_TUNE_PAIR_MIN_WAVES:
      VKG_REQUIRE(value >= 0, "set_tuning: the threshold cannot be negative");
      dev->pair_min_waves_x10 = (int)value;
      break;
    case VKG_TUNE_ATTN_ONE_PASS: dev->attn_one_pass = value != 0; break;
    case VKG_TUNE_PAIR_192: dev->pair192 = value != 0; break;
    case VKG_TUNE_WAIT_TIMEOUT_MS:
      VKG_REQUIRE(value > 0, "set_tuning: the wait limit must be positive");
      dev->wait_timeout_s = (double)value * 1e-3;
      break;
    default: VKG_FAIL("set_tuning: unknown key %d", key);
  }
  return 0;
}

extern "C" int vkg_device_destroy(vkg_device* dev) {
  if (!dev) return 0;
  cudaSetDevice(dev->ordinal);
  cudaStreamSynchronize(dev->stream);
  if (dev->err_host) cudaFreeHost((void*)dev->err_host);
  if (dev->stream) cudaStreamDestroy(dev->stream);
  vkg_gemm_plans_destroy(dev->gemm_plans);
  delete dev;
  return 0;
}

extern "C" int vkg_device_info(vkg_device* dev, char* name, size_t name_cap, int* sm_count,
                               size_t* total_bytes, int* cc_major, int* cc_minor) {
  if (!dev) VKG_FAIL("null device");
  if (name && name_cap) snprintf(name, name_cap, "%s", dev->name);
  if (sm_count) *sm_count = dev->sm_count;
  if (total_bytes) *total_bytes = dev->total_bytes;
  if (cc_major) *cc_major = dev->cc_major;
  if (cc_minor) *cc_minor = dev->cc_minor;
  return 0;
}

extern "C" void* vkg_device_stream(vkg_device* dev) {
  if (!dev) return nullptr;
  dev->stream_shared.store(true);
  return (void*)dev->stream;
}

static int check_err_flag(vkg_device* dev) {
  uint32_t code = dev->err_host[0];
  if (code != 0) {
    uint32_t detail = dev->err_host[1];
    dev->err_host[0] = 0;
    dev->err_host[1] = 0;
    VKG_FAIL("kernel reported error %u (detail 0x%x): a bounded device-side wait gave up",
             code, detail);
  }
  return 0;
}

// ---- host waits ------------------------------------------------------------------------
//
// The reference turns a fence that does not signal within 10 s into VkError (vk.py:884-888,
// 1335-1339).  Here a step can hang only in a collective whose peer never arrives, so waits
// on a device with a communicator poll against a deadline; on expiry the communicator is
// aborted (which lets the stream drain) and the call fails.
int vkg_wait_with_deadline(const vkg_wait_hooks* h, const char* what) {
  const auto t0 = std::chrono::steady_clock::now();
  for (long long polls = 0;; ++polls) {
    const int q = h->query(h->query_ctx);
    if (q == 0) return 0;
    if (q != 1) return 1;
    if (h->async_error && (polls & 63) == 63 && h->async_error(h->comm_ctx)) {
      if (h->abort) h->abort(h->comm_ctx);
      return 1;
    }
    const double waited = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (h->abort && waited > h->timeout_s) {
      h->abort(h->comm_ctx);
      vkg_set_error("%s: the device did not finish within %.1f s (a collective whose peer never "
                    "arrived?); the communicator was aborted", what, h->timeout_s);
      return 1;
    }
    // spin for the first 200 us (a training step's tail), then yield the core
    if (waited > 200e-6) std::this_thread::sleep_for(std::chrono::microseconds(waited > 0.05 ? 500 : 20));
  }
}

namespace {
struct DeviceQuery {
  vkg_device* dev;
  const vkg_stamp* st;
  unsigned polls;
};
// A stamp is polled in host memory; every so often the stream is asked as well, so that a failed
// launch or a fault is noticed (and a drained stream ends the wait in any case).
int query_device(void* ctx) {
  DeviceQuery* q = static_cast<DeviceQuery*>(ctx);
  if (q->st) {
    if ((int32_t)(q->st->host->seq - q->st->launched) >= 0) return 0;
    if ((++q->polls & 1023u) != 0u) {
#if defined(__x86_64__)
      _mm_pause();
#endif
      return 1;
    }
  }
  cudaError_t e = cudaStreamQuery(q->dev->stream);
  if (e == cudaSuccess) return 0;
  if (e == cudaErrorNotReady) {
    cudaGetLastError();
    return 1;
  }
  vkg_set_error("device wait failed: %s", cudaGetErrorString(e));
  return 2;
}
}  // namespace

int vkg_wait_device(vkg_device* dev, const vkg_stamp* st, const char* what) {
  const uint64_t entered = dev->entered.load();
  DeviceQuery q{dev, st, 0};
  if (!dev->on_abort) {          // no communicator: nothing can hang
    if (st) {
      int r;
      while ((r = query_device(&q)) == 1) {
      }
      if (r != 0) return 1;
    } else {
      VKG_CUDA(cudaStreamSynchronize(dev->stream));
    }
    dev->drained.store(entered);
    return 0;
  }
  vkg_wait_hooks h{query_device, &q, dev->on_async_error, dev->on_abort, dev->wait_ctx,
                   dev->wait_timeout_s};
  return vkg_wait_with_deadline(&h, what);
}

// The deadline loop against a scripted device, for tests without a GPU: the "stream" reports
// done after ready_after_polls queries (never, if negative), the "communicator" reports an
// asynchronous error from its async_error_at-th check on (never, if negative).  *aborted
// receives how often the abort hook ran.
namespace {
struct FakeWait {
  long long polls, ready_after, checks, error_at;
  int aborted;
};
int fake_query(void* ctx) {
  FakeWait* f = static_cast<FakeWait*>(ctx);
  return (f->ready_after >= 0 && f->polls++ >= f->ready_after) ? 0 : 1;
}
int fake_async_error(void* ctx) {
  FakeWait* f = static_cast<FakeWait*>(ctx);
  if (f->error_at >= 0 && f->checks++ >= f->error_at) {
    vkg_set_error("communicator reported an asynchronous error (scripted)");
    return 1;
  }
  return 0;
}
void fake_abort(void* ctx) { static_cast<FakeWait*>(ctx)->aborted++; }
}  // namespace

extern "C" int vkg_selftest_wait_deadline(int64_t ready_after_polls, int64_t async_error_at,
                                          double timeout_s, int* aborted) {
  FakeWait f{0, ready_after_polls, 0, async_error_at, 0};
  vkg_wait_hooks h{fake_query, &f, fake_async_error, fake_abort, &f, timeout_s};
  const int rc = vkg_wait_with_deadline(&h, "selftest");
  if (aborted) *aborted = f.aborted;
  return rc;
}

// Two threads that enter a fresh device together, `rounds` times: how often neither of them marked it
// as shared.  For tests without a GPU.
extern "C" int vkg_selftest_first_threads(int rounds, int* unmarked) {
  VKG_REQUIRE(rounds > 0 && unmarked, "selftest: bad arguments");
  std::atomic<const void*> first{nullptr};
  std::atomic<bool> shared{false};
  std::atomic<int> go{0}, done{0};
  *unmarked = 0;
  const auto enter = [&](const void* self) {
    for (int i = 1; i <= rounds; ++i) {
      while (go.load() < i) std::this_thread::yield();
      vkg_note_thread(first, shared, self);
      done.fetch_add(1);
    }
  };
  int a, b;
  std::thread t1(enter, &a), t2(enter, &b);
  for (int i = 1; i <= rounds; ++i) {
    first.store(nullptr);
    shared.store(false);
    go.store(i);
    while (done.load() < 2 * i) std::this_thread::yield();
    if (!shared.load()) ++*unmarked;
  }
  t1.join();
  t2.join();
  return 0;
}

int vkg_stamp_finish(vkg_device* dev, const vkg_stamp* st, const char* what, double* seconds) {
  if (vkg_wait_device(dev, st, what)) return 1;
  if (seconds) *seconds = (double)st->host->ticks * 32e-9;
  return check_err_flag(dev);
}

extern "C" int vkg_sync(vkg_device* dev) {
  // the last wait found everything entered so far done: what a caller reads after a submit
  // (model.read_loss) needs no second trip to the driver
  if (dev && !dev->on_abort && !dev->capturing && !dev->stream_shared.load() &&
      dev->drained.load() == dev->entered.load())
    return check_err_flag(dev);
  if (vkg_bind(dev)) return 1;
  if (vkg_wait_device(dev, nullptr, "sync")) return 1;
  return check_err_flag(dev);
}

extern "C" int vkg_alloc(vkg_device* dev, size_t bytes, int kind, void** dptr, void** hptr) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(dptr && hptr, "null output pointer");
  *dptr = nullptr;
  *hptr = nullptr;
  if (bytes == 0) bytes = 16;
  if (kind == 0) {
    VKG_CUDA(cudaMalloc(dptr, bytes));
  } else if (kind == 1) {
    VKG_CUDA(cudaHostAlloc(hptr, bytes, cudaHostAllocMapped | cudaHostAllocPortable));
    memset(*hptr, 0, bytes);
    VKG_CUDA(cudaHostGetDevicePointer(dptr, *hptr, 0));
  } else if (kind == 2) {
    VKG_CUDA(cudaMalloc(dptr, bytes));
    cudaError_t e = cudaHostAlloc(hptr, bytes, cudaHostAllocPortable);
    if (e != cudaSuccess) {
      cudaFree(*dptr);
      *dptr = nullptr;
      VKG_FAIL("cudaHostAlloc(%zu) failed: %s", bytes, cudaGetErrorString(e));
    }
    memset(*hptr, 0, bytes);
  } else {
    VKG_FAIL("unknown memory kind %d", kind);
  }
  return 0;
}

extern "C" int vkg_free(vkg_device* dev, void* dptr, void* hptr, int kind) {
  if (vkg_bind(dev)) return 1;
  if (kind == 0) {
    if (dptr) VKG_CUDA(cudaFree(dptr));
  } else if (kind == 1) {
    if (hptr) VKG_CUDA(cudaFreeHost(hptr));
  } else if (kind == 2) {
    if (dptr) VKG_CUDA(cudaFree(dptr));
    if (hptr) VKG_CUDA(cudaFreeHost(hptr));
  } else {
    VKG_FAIL("unknown memory kind %d", kind);
  }
  return 0;
}

extern "C" int vkg_host_alloc(vkg_device* dev, size_t bytes, void** hptr) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(hptr, "null output pointer");
  *hptr = nullptr;
  cudaError_t e = cudaHostAlloc(hptr, bytes ? bytes : 16, cudaHostAllocPortable);
  if (e == cudaSuccess) return 0;
  cudaGetLastError();            // callers carry on without: the next launch must not find it
  *hptr = nullptr;
  VKG_FAIL("cudaHostAlloc(%zu) failed: %s", bytes, cudaGetErrorString(e));
}

extern "C" int vkg_host_free(void* hptr) {
  if (hptr) VKG_CUDA(cudaFreeHost(hptr));
  return 0;
}

extern "C" int vkg_upload(vkg_device* dev, void* dptr, const void* hptr, size_t bytes) {
  if (vkg_bind(dev)) return 1;
  VKG_CUDA(cudaMemcpyAsync(dptr, hptr, bytes, cudaMemcpyHostToDevice, dev->stream));
  VKG_CUDA(cudaStreamSynchronize(dev->stream));
  return 0;
}

extern "C" int vkg_download(vkg_device* dev, void* hptr, const void* dptr, size_t bytes) {
  if (vkg_bind(dev)) return 1;
  VKG_CUDA(cudaMemcpyAsync(hptr, dptr, bytes, cudaMemcpyDeviceToHost, dev->stream));
  if (vkg_wait_device(dev, nullptr, "download")) return 1;
  return check_err_flag(dev);
}

// Pinned host memory read by a kernel instead of the copy engine: for the inputs of a step, a few
// KB to a few hundred KB, that sit between two kernels of a graph.  64 KB take 3.6 us against 4.8,
// and no hand-over between engines (401 KB inside a graph: 10 us against 15.5); from 1 MB on the
// engine is as fast and leaves the SMs alone.
constexpr size_t COPY_KERNEL_MAX = 1 << 20;

__global__ void __launch_bounds__(256) k_copy_in(const uint4* __restrict__ src, uint4* __restrict__ dst, int n) {
  pdl_trigger();
  pdl_wait();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = __ldcs(src + i);
}

static int copy_in(vkg_device* dev, void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
  if (bytes <= COPY_KERNEL_MAX && bytes >= 16 && bytes % 16 == 0 && (((uintptr_t)dst | (uintptr_t)src) & 15) == 0) {
    cudaPointerAttributes s, d;
    VKG_CUDA(cudaPointerGetAttributes(&s, src));
    VKG_CUDA(cudaPointerGetAttributes(&d, dst));
    if (s.type == cudaMemoryTypeHost && s.devicePointer && d.type == cudaMemoryTypeDevice) {
      const int n = (int)(bytes / 16);
      k_copy_in<<<vkg_blocks(n, 256, dev->sm_count), 256, 0, dev->stream>>>((const uint4*)s.devicePointer,
                                                                           (uint4*)dst, n);
      return vkg_check_launch("copy_in");
    }
  }
  VKG_CUDA(cudaMemcpyAsync(dst, src, bytes, kind, dev->stream));
  return 0;
}

extern "C" int vkg_copy(vkg_device* dev, void* dst, const void* src, size_t bytes) {
  if (vkg_bind(dev)) return 1;
  return copy_in(dev, dst, src, bytes, cudaMemcpyDefault);
}

extern "C" int vkg_copy_h2d_async(vkg_device* dev, void* dptr, const void* hptr, size_t bytes) {
  if (vkg_bind(dev)) return 1;
  return copy_in(dev, dptr, hptr, bytes, cudaMemcpyHostToDevice);
}

extern "C" int vkg_copy_d2h_async(vkg_device* dev, void* hptr, const void* dptr, size_t bytes) {
  if (vkg_bind(dev)) return 1;
  VKG_CUDA(cudaMemcpyAsync(hptr, dptr, bytes, cudaMemcpyDeviceToHost, dev->stream));
  return 0;
}

// A few KB of zeros (a bias gradient about to be accumulated into) between two kernels of a graph:
// a kernel of our own hides its launch, a memset node takes 1.9 us.
constexpr size_t ZERO_KERNEL_MAX = 256 << 10;
__global__ void __launch_bounds__(256) k_zero(uint4* __restrict__ p, int n) {
  pdl_trigger();
  pdl_wait();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) p[i] = make_uint4(0u, 0u, 0u, 0u);
}

extern "C" int vkg_memset0(vkg_device* dev, void* dptr, size_t bytes) {
  if (vkg_bind(dev)) return 1;
  if (bytes > 0 && bytes <= ZERO_KERNEL_MAX && ((bytes | (uintptr_t)dptr) & 15) == 0) {
    const int n = (int)(bytes / 16);
    VKG_CUDA(vkg_launch(dev, VKG_K_SMALL | VKG_SHORT, k_zero, dim3((n + 255) / 256), dim3(256), 0, 1,
                        (uint4*)dptr, n));
    return vkg_check_launch("zero");
  }
  VKG_CUDA(cudaMemsetAsync(dptr, 0, bytes, dev->stream));
  return 0;
}

extern "C" int vkg_timer_begin(vkg_device* dev) {
  if (vkg_bind(dev)) return 1;
  return vkg_stamp_begin(dev, &dev->timer);
}

extern "C" int vkg_timer_end(vkg_device* dev, double* seconds) {
  if (vkg_bind(dev)) return 1;
  if (vkg_stamp_end(dev, &dev->timer)) return 1;
  dev->timer.launched++;
  return vkg_stamp_finish(dev, &dev->timer, "timer_end", seconds);
}

extern "C" int vkg_graph_begin(vkg_device* dev) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(!dev->capturing, "a graph is already being recorded on this device");
  if (stamp_acquire(dev, &dev->capture_stamp)) return 1;
  cudaError_t e = cudaStreamBeginCapture(dev->stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) {
    stamp_release(dev->stamps.get(), dev->capture_stamp);
    VKG_FAIL("cudaStreamBeginCapture failed: %s", cudaGetErrorString(e));
  }
  dev->capturing = true;
  dev->captured_hp.clear();
  return vkg_stamp_begin(dev, &dev->capture_stamp);
}

extern "C" int vkg_graph_end(vkg_device* dev, vkg_graph** out) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(out, "null out");
  VKG_REQUIRE(dev->capturing, "no graph is being recorded");
  dev->capturing = false;
  const vkg_stamp stamp = dev->capture_stamp;
  dev->capture_stamp = vkg_stamp();
  std::vector<const float*> hps;
  hps.swap(dev->captured_hp);
  vkg_launch(dev, VKG_K_SMALL | VKG_SHORT, k_stamp_end, dim3(1), dim3(1), 0, 1, stamp.dev, stamp.host_dev);
  cudaGetLastError();            // a capture that broke earlier is reported by EndCapture
  cudaGraph_t graph = nullptr;
  cudaError_t ce = cudaStreamEndCapture(dev->stream, &graph);
  if (ce != cudaSuccess || graph == nullptr) {
    stamp_release(dev->stamps.get(), stamp);
    VKG_FAIL("capture produced no graph (an enqueue failed during recording): %s", cudaGetErrorString(ce));
  }
  vkg_graph* g = new vkg_graph();
  g->graph = graph;
  g->dev = dev;
  g->stamps = dev->stamps;
  g->stamp = stamp;
  size_t n = 0;
  if (cudaGraphGetNodes(graph, nullptr, &n) == cudaSuccess && n > 0) {
    std::vector<cudaGraphNode_t> nodes(n);
    if (cudaGraphGetNodes(graph, nodes.data(), &n) == cudaSuccess) {
      if (!hps.empty()) vkg_graph_find_hp(g, hps, nodes);
      for (size_t i = 0; i < n; ++i) {
        cudaGraphNodeType t;
        if (cudaGraphNodeGetType(nodes[i], &t) == cudaSuccess && t == cudaGraphNodeTypeKernel)
          g->kernel_nodes++;
      }
    }
  }
  cudaError_t e = cudaGraphInstantiate(&g->exec, graph, 0);
  if (e != cudaSuccess) {
    cudaGraphDestroy(graph);
    stamp_release(dev->stamps.get(), stamp);
    delete g;
    VKG_FAIL("cudaGraphInstantiate failed: %s", cudaGetErrorString(e));
  }
  *out = g;
  return 0;
}

static int graph_enqueue(vkg_device* dev, vkg_graph* g) {
  VKG_REQUIRE(g && g->exec && g->dev == dev, "graph is not finished, or belongs to another device");
  if (!g->hp.empty() && vkg_graph_refresh_hp(g)) return 1;
  VKG_CUDA(cudaGraphLaunch(g->exec, dev->stream));
  g->stamp.launched++;
  return 0;
}

extern "C" int vkg_graph_launch(vkg_device* dev, vkg_graph* g, double* seconds) {
  if (vkg_bind(dev)) return 1;
  if (graph_enqueue(dev, g)) return 1;
  return vkg_stamp_finish(dev, &g->stamp, "graph_launch", seconds);
}

extern "C" int vkg_graph_launch_d2h(vkg_device* dev, vkg_graph* g, void* dst, size_t dst_pitch,
                                    const void* src, size_t src_pitch, size_t src_group, size_t width,
                                    size_t rows, size_t groups, double* launch_s, double* copy_s) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(dst && src && width <= dst_pitch && width <= src_pitch, "graph_launch_d2h: bad arguments");
  if (graph_enqueue(dev, g)) return 1;
  for (size_t k = 0; k < groups; ++k)
    VKG_CUDA(cudaMemcpy2DAsync((char*)dst + k * rows * dst_pitch, dst_pitch, (const char*)src + k * src_group,
                               src_pitch, width, rows, cudaMemcpyDeviceToHost, dev->stream));
  if (vkg_stamp_end(dev, &dev->timer)) return 1;      // its end mark; the graph has the other two
  dev->timer.launched++;
  if (vkg_stamp_finish(dev, &dev->timer, "graph_launch_d2h", nullptr)) return 1;
  if (launch_s) *launch_s = (double)g->stamp.host->ticks * 32e-9;
  if (copy_s) *copy_s = (double)(int64_t)(dev->timer.host->t1 - g->stamp.host->t1) * 1e-9;
  return 0;
}

extern "C" int vkg_graph_launch_async(vkg_device* dev, vkg_graph* g) {
  if (vkg_bind(dev)) return 1;
  return graph_enqueue(dev, g);
}

extern "C" int vkg_graph_destroy(vkg_graph* g) {
  if (!g) return 0;
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  if (g->stamps) stamp_release(g->stamps.get(), g->stamp);
  delete g;
  return 0;
}

extern "C" int vkg_graph_kernel_count(vkg_graph* g, int* count) {
  VKG_REQUIRE(g && count, "null argument");
  *count = g->kernel_nodes;
  return 0;
}
