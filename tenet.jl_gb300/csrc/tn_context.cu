// Context, device memory accounting, workspace arena, errors.
#include <cstdarg>
#include <cstdlib>
#include <cstring>

#include "tn_internal.cuh"

static thread_local std::string g_create_error;

tn_status_t tn_set_error(tn_ctx* ctx, tn_status_t st, const char* fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (ctx)
    ctx->last_error = buf;
  else
    g_create_error = buf;
  return st;
}

namespace {

// Freed blocks kept for the next allocation of their size: cudaMalloc and cudaFree of a 128 MB
// result take 0.15 ms, as long as the product that fills it.  A block may still be in use by a stream
// that the context does not know of, so it is handed out again only after the device has drained.
constexpr size_t kPoolBytes = size_t(4) << 30;  // most bytes kept
// Undrained blocks of one size at which an allocation drains the device rather than take new memory: a
// drain is 9 µs, and one call in four (of 128 MB results) to thirty-two (of small ones) pays for it
constexpr size_t kDrainCount = 32, kDrainBytes = size_t(512) << 20;

// the size in which a request is allocated, so that blocks fit each other: the driver's own granularity
// (pages of 2 MiB, and pieces of them), so no memory is held that the request would not take
size_t block_size(size_t bytes) {
  const size_t unit = bytes >= (size_t(2) << 20) ? size_t(2) << 20 : 512;
  return (bytes + unit - 1) / unit * unit;
}

cudaError_t driver_free(tn_ctx* ctx, void* p) {
  const cudaError_t e = cudaFree(p);
  if (e == cudaSuccess) ctx->drained = ctx->pool_age;  // (cudaFree waits for the device)
  return e;
}

// Waits for the device as cudaFree does, which unlike cudaDeviceSynchronize may be called while another
// thread captures a stream (that call ends its capture with an error).  The second small block
// keeps the driver's page: 6 µs instead of 60.
cudaError_t device_drain(tn_ctx* ctx) {
  int current = ctx->device;
  cudaGetDevice(&current);
  if (current != ctx->device) cudaSetDevice(ctx->device);
  void* p = nullptr;
  cudaError_t e = cudaSuccess;
  if (!ctx->drain_block) e = cudaMalloc(&ctx->drain_block, 256);
  if (e == cudaSuccess) e = cudaMalloc(&p, 256);
  if (e == cudaSuccess) e = driver_free(ctx, p);
  if (current != ctx->device) cudaSetDevice(current);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

// gives pooled blocks back to the driver, oldest first, until at most `keep` bytes are pooled
cudaError_t pool_shrink(tn_ctx* ctx, size_t keep) {
  while (ctx->pool_bytes > keep && !ctx->pool.empty()) {
    auto oldest = ctx->pool.begin();
    for (auto it = ctx->pool.begin(); it != ctx->pool.end(); ++it)
      if (it->second.age < oldest->second.age) oldest = it;
    const cudaError_t e = driver_free(ctx, oldest->second.p);
    if (e != cudaSuccess) return e;
    ctx->pool_bytes -= oldest->first;
    ctx->capacity.erase(oldest->second.p);
    ctx->pool.erase(oldest);
  }
  return cudaSuccess;
}

// a pooled block of this size that no stream uses any more, or null
void* pool_take(tn_ctx* ctx, size_t size) {
  if (ctx->budget && ctx->in_use + ctx->pool_bytes > ctx->budget) return nullptr;
  const auto range = ctx->pool.equal_range(size);  // (in the order of their release)
  if (range.first == range.second) return nullptr;
  if (range.first->second.age >= ctx->drained) {
    const size_t count = (size_t)std::distance(range.first, range.second);
    if (!ctx->budget && count < kDrainCount && count * size < kDrainBytes) return nullptr;
    if (device_drain(ctx) != cudaSuccess) return nullptr;
  }
  void* p = range.first->second.p;
  ctx->pool_bytes -= size;
  ctx->pool.erase(range.first);
  return p;
}

}  // namespace

tn_status_t tn_dev_alloc(tn_ctx* ctx, size_t bytes, void** p) {
  if (bytes == 0) bytes = 256;
  if (ctx->budget && ctx->in_use + bytes > ctx->budget)
    return tn_set_error(ctx, TN_ENOMEM, "HBM budget exceeded: %zu in use + %zu > %zu",
                        ctx->in_use, bytes, ctx->budget);
  const size_t size = block_size(bytes);
  *p = pool_take(ctx, size);
  if (!*p) {
    if (ctx->budget && ctx->in_use + ctx->pool_bytes + bytes > ctx->budget)
      TN_CHECK_CUDA(ctx, pool_shrink(ctx, ctx->budget - ctx->in_use - bytes));
    cudaError_t e = cudaMalloc(p, size);
    if (e != cudaSuccess && !ctx->pool.empty()) {
      cudaGetLastError();
      TN_CHECK_CUDA(ctx, pool_shrink(ctx, 0));
      e = cudaMalloc(p, size);
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      return tn_set_error(ctx, TN_ENOMEM, "cudaMalloc(%zu) failed: %s", bytes,
                          cudaGetErrorString(e));
    }
    ctx->capacity[*p] = size;
  }
  ctx->allocs[*p] = bytes;
  ctx->in_use += bytes;
  return TN_OK;
}

tn_status_t tn_dev_free(tn_ctx* ctx, void* p) {
  if (!p) return TN_OK;
  auto it = ctx->allocs.find(p);
  if (it == ctx->allocs.end())
    return tn_set_error(ctx, TN_EINVAL, "tn_free: pointer %p not allocated by this context", p);
  ctx->in_use -= it->second;
  ctx->allocs.erase(it);
  const size_t size = ctx->capacity[p];
  if (size > kPoolBytes) {
    TN_CHECK_CUDA(ctx, driver_free(ctx, p));
    ctx->capacity.erase(p);
    return TN_OK;
  }
  ctx->pool.emplace(size, tn_ctx::pool_block{p, ctx->pool_age++});
  ctx->pool_bytes += size;
  if (ctx->pool_bytes > kPoolBytes) TN_CHECK_CUDA(ctx, pool_shrink(ctx, kPoolBytes));
  return TN_OK;
}

void ws_overflow(tn_ctx* ctx, size_t need) {
  cudaStreamSynchronize(ctx->stream);
  fprintf(stderr, "tenetgb: workspace overflow: %zu bytes taken, %zu reserved (a missing ws_reserve)\n", need,
          ctx->ws_cap);
  fflush(stderr);
  std::abort();
}

constexpr size_t kPinnedBytes = 1 << 16;

tn_status_t wait_error_word(tn_ctx* ctx, int** out) {
  *out = reinterpret_cast<int*>(static_cast<char*>(ctx->pinned) + kPinnedBytes) - 1;  // (unified addressing)
  return TN_OK;
}

tn_status_t wait_error_check(tn_ctx* ctx) {
  volatile int* w = reinterpret_cast<int*>(static_cast<char*>(ctx->pinned) + kPinnedBytes) - 1;
  if (*w == 0) return TN_OK;
  *w = 0;
  return tn_set_error(ctx, TN_ETIMEOUT, "a bounded wait inside a kernel (QR, SVD or tensor-pipe product) exceeded its limit");
}

tn_status_t read_back_sync(tn_ctx* ctx) {
  TN_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return wait_error_check(ctx);
}

tn_status_t ws_reserve(tn_ctx* ctx, size_t bytes, size_t spare) {
  ctx->ws_top = 0;
  TN_RETURN_IF(wait_error_check(ctx));
  if (bytes <= ctx->ws_cap) return TN_OK;
  auto with_margin = [](size_t b) { return b + b / 4 + (1 << 20); };
  // (without the spare part it holds what the budget would refuse to grow)
  if (bytes - spare <= ctx->ws_cap && ctx->budget && ctx->in_use - ctx->ws_cap + with_margin(bytes) > ctx->budget) return TN_OK;
  // growth: the stream must be idle before the old arena is released
  TN_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  // (the cached graphs point into the arena; the profiler's events do not and stay)
  for (auto& kv : ctx->graphs) cudaGraphExecDestroy(kv.second);
  ctx->graphs.clear();
  if (ctx->ws) TN_RETURN_IF(tn_dev_free(ctx, ctx->ws));
  ctx->ws = nullptr;
  ctx->ws_cap = 0;
  size_t cap = with_margin(bytes);
  void* p = nullptr;
  tn_status_t st = tn_dev_alloc(ctx, cap, &p);
  if (st == TN_ENOMEM && spare > 0) {
    cap = with_margin(bytes - spare);
    st = tn_dev_alloc(ctx, cap, &p);
  }
  TN_RETURN_IF(st);
  ctx->ws = (char*)p;
  ctx->ws_cap = cap;
  return TN_OK;
}

tn_status_t ctx_flags(tn_ctx* ctx, size_t n, int** out) {
  if (n > ctx->flags_cap) {
    TN_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (ctx->d_flags) TN_RETURN_IF(tn_dev_free(ctx, ctx->d_flags));
    ctx->d_flags = nullptr;
    size_t cap = n < 1024 ? 1024 : n * 2;
    void* p = nullptr;
    TN_RETURN_IF(tn_dev_alloc(ctx, cap * sizeof(int), &p));
    ctx->d_flags = (int*)p;
    ctx->flags_cap = cap;
  }
  *out = ctx->d_flags;
  return TN_OK;
}

extern "C" {

const char* tn_version(void) { return "tenetgb 0.1.0 (sm_103a)"; }

tn_status_t tn_create(tn_ctx** out, int device) {
  if (!out) return tn_set_error(nullptr, TN_EINVAL, "tn_create: null output");
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n == 0) {
    cudaGetLastError();
    return tn_set_error(nullptr, TN_ECUDA, "no CUDA device: %s", cudaGetErrorString(e));
  }
  if (device < 0 || device >= n)
    return tn_set_error(nullptr, TN_EINVAL, "device %d out of range (%d devices)", device, n);
  tn_ctx* ctx = new tn_ctx();
  ctx->device = device;
  cudaSetDevice(device);
  cudaDeviceProp prop;
  cudaGetDeviceProperties(&prop, device);
  ctx->num_sms = prop.multiProcessorCount;
  if (prop.major < 10) {
    delete ctx;
    return tn_set_error(nullptr, TN_EUNSUPPORTED,
                        "device %d is sm_%d%d; libtenetgb is built for sm_103a", device,
                        prop.major, prop.minor);
  }
  e = cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete ctx;
    return tn_set_error(nullptr, TN_ECUDA, "stream create: %s", cudaGetErrorString(e));
  }
  ctx->stream = ctx->own_stream;
  e = cudaMallocHost(&ctx->pinned, kPinnedBytes);
  if (e != cudaSuccess) {
    cudaStreamDestroy(ctx->own_stream);
    delete ctx;
    return tn_set_error(nullptr, TN_ECUDA, "pinned alloc: %s", cudaGetErrorString(e));
  }
  memset(ctx->pinned, 0, kPinnedBytes);
  *out = ctx;
  return TN_OK;
}

}  // extern "C"

void ctx_release(tn_ctx* ctx) {
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  for (auto& kv : ctx->graphs) cudaGraphExecDestroy(kv.second);
  ctx->graphs.clear();
  for (auto& r : ctx->prof_recs) {
    cudaEventDestroy(r.a);
    cudaEventDestroy(r.b);
  }
  for (cudaEvent_t e : ctx->prof_pool) cudaEventDestroy(e);
  for (auto& kv : ctx->capacity) cudaFree(kv.first);  // live and pooled blocks
  ctx->capacity.clear();
  ctx->pool.clear();
  ctx->allocs.clear();
  if (ctx->drain_block) cudaFree(ctx->drain_block);
  if (ctx->pinned) cudaFreeHost(ctx->pinned);
  if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
  delete ctx;
}

extern "C" {

tn_status_t tn_destroy(tn_ctx* ctx) {
  if (!ctx) return TN_OK;
  if (ctx->refs > 0) {
    ctx->destroy_requested = true;  // released by the last tn_mps_destroy
    return TN_OK;
  }
  ctx_release(ctx);
  return TN_OK;
}

tn_status_t tn_set_stream(tn_ctx* ctx, void* stream) {
  if (!ctx) return TN_EINVAL;
  ctx->stream = stream ? (cudaStream_t)stream : ctx->own_stream;
  return TN_OK;
}

void* tn_get_stream(tn_ctx* ctx) { return ctx ? (void*)ctx->stream : nullptr; }

tn_status_t tn_sync(tn_ctx* ctx) {
  if (!ctx) return TN_EINVAL;
  return read_back_sync(ctx);
}

tn_status_t tn_alloc(tn_ctx* ctx, size_t bytes, void** dptr) {
  if (!ctx || !dptr) return TN_EINVAL;
  return tn_dev_alloc(ctx, bytes, dptr);
}

tn_status_t tn_free(tn_ctx* ctx, void* dptr) {
  if (!ctx) return TN_EINVAL;
  TN_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return tn_dev_free(ctx, dptr);
}

tn_status_t tn_release_cached(tn_ctx* ctx) {
  if (!ctx) return TN_EINVAL;
  TN_CHECK_CUDA(ctx, pool_shrink(ctx, 0));
  return TN_OK;
}

tn_status_t tn_memcpy_h2d(tn_ctx* ctx, void* dst, const void* src, size_t bytes) {
  if (!ctx) return TN_EINVAL;
  TN_ARG(ctx, dst && src, "tn_memcpy_h2d: null pointer");
  TN_CHECK_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
  TN_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TN_OK;
}

tn_status_t tn_memcpy_d2h(tn_ctx* ctx, void* dst, const void* src, size_t bytes) {
  if (!ctx) return TN_EINVAL;
  TN_ARG(ctx, dst && src, "tn_memcpy_d2h: null pointer");
  TN_CHECK_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
  return read_back_sync(ctx);
}

tn_status_t tn_memcpy_d2d(tn_ctx* ctx, void* dst, const void* src, size_t bytes) {
  if (!ctx) return TN_EINVAL;
  TN_ARG(ctx, dst && src, "tn_memcpy_d2d: null pointer");
  TN_CHECK_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
  return TN_OK;
}

tn_status_t tn_set_hbm_budget(tn_ctx* ctx, size_t bytes) {
  if (!ctx) return TN_EINVAL;
  ctx->budget = bytes;
  if (bytes) TN_CHECK_CUDA(ctx, pool_shrink(ctx, bytes > ctx->in_use ? bytes - ctx->in_use : 0));
  return TN_OK;
}

tn_status_t tn_hbm_in_use(tn_ctx* ctx, size_t* bytes) {
  if (!ctx || !bytes) return TN_EINVAL;
  *bytes = ctx->in_use;
  return TN_OK;
}

tn_status_t tn_kernel_launches(tn_ctx* ctx, int64_t* count) {
  if (!ctx || !count) return TN_EINVAL;
  *count = ctx->launches;
  return TN_OK;
}

tn_status_t tn_set_autotune(tn_ctx* ctx, int32_t enable) {
  if (!ctx) return TN_EINVAL;
  ctx->autotune = enable != 0;
  return TN_OK;
}

// text form: one "key value1 value2" line per tuned shape
tn_status_t tn_tuning_dump(tn_ctx* ctx, char* buf, size_t len, size_t* needed) {
  if (!ctx) return TN_EINVAL;
  std::string out;
  for (auto& kv : ctx->tuning)
    out += kv.first + " " + std::to_string(kv.second.first) + " " + std::to_string(kv.second.second) + "\n";
  if (needed) *needed = out.size() + 1;
  if (buf && len > 0) {
    size_t c = out.size() < len - 1 ? out.size() : len - 1;
    memcpy(buf, out.data(), c);
    buf[c] = 0;
  }
  return TN_OK;
}

tn_status_t tn_tuning_load(tn_ctx* ctx, const char* text) {
  if (!ctx || !text) return TN_EINVAL;
  const char* p = text;
  while (*p) {
    char key[128];
    int a = 0, b = 0, used = 0;
    if (sscanf(p, "%127s %d %d%n", key, &a, &b, &used) != 3) break;
    // the autotuner's candidate set: panel widths 1…32 and slab widths 1, 2, 4 (powers of two)
    const bool pow2 = (a & (a - 1)) == 0 && (b & (b - 1)) == 0;
    if (a < 1 || a > 32 || b < 1 || b > 4 || !pow2)
      return tn_set_error(ctx, TN_EINVAL, "tn_tuning_load: bad entry %s %d %d", key, a, b);
    ctx->tuning[key] = {a, b};
    p += used;
    while (*p == '\n' || *p == ' ') ++p;
  }
  return TN_OK;
}

const char* tn_last_error_string(tn_ctx* ctx) {
  return ctx ? ctx->last_error.c_str() : g_create_error.c_str();
}

}  // extern "C"
