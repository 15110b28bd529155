// Context: device selection, stream, device-memory accounting, errors.
#include <algorithm>
#include <chrono>
#include <thread>

#include "tc_internal.h"

namespace {
// The process's contexts: an allocation that fails in one takes the blocks that
// the others keep on its device.  (Never destroyed: a context may outlive static
// objects.)
struct Contexts {
  std::mutex mu;
  std::vector<tc_ctx*> all;
};
Contexts& contexts() {
  static Contexts* c = new Contexts();
  return *c;
}

void trim_all(int device) {
  std::lock_guard<std::mutex> g(contexts().mu);
  for (tc_ctx* c : contexts().all)
    if (c->device == device) c->trim_pool();
}
}  // namespace

tc_status tc_ctx::alloc(void** p, size_t bytes, const char* what, bool pooled) {
  bool trim = false;
  {
    std::lock_guard<std::mutex> g(mu);
    if (fail_next > 0) {
      --fail_next;
      err = std::string("injected allocation failure: ") + what;
      return TC_ERR_OOM;
    }
    if (budget && in_use + bytes > budget) {
      char buf[256];
      snprintf(buf, sizeof(buf), "memory budget exceeded allocating %zu bytes for %s (%zu of %zu in use)",
               bytes, what, in_use, budget);
      err = buf;
      return TC_ERR_OOM;
    }
    if (pooled) {
      // the smallest kept block that holds `bytes` with at most a quarter to
      // spare; under a budget only one of that very size, since what a block is
      // larger would count against the budget and so make what fits depend on
      // the blocks of earlier objects
      const size_t spare = budget ? 0 : bytes / 4 + 4096;
      const auto it = pool.lower_bound(bytes);
      if (it != pool.end() && it->first <= bytes + spare) {
        *p = it->second.p;
        const size_t size = it->first;
        pool_bytes -= size;
        pool.erase(it);
        allocs[*p] = tc::Block{bytes, size};
        in_use += bytes;
        if (in_use > peak) peak = in_use;
        return TC_OK;
      }
    }
    trim = budget && pool_bytes && in_use + pool_bytes + bytes > budget;
  }
  if (trim) trim_pool();
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    trim_all(device);
    e = cudaMalloc(p, bytes);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(TC_ERR_OOM, "cudaMalloc(%zu) for %s: %s", bytes, what, cudaGetErrorString(e));
  }
  std::lock_guard<std::mutex> g(mu);
  allocs[*p] = tc::Block{bytes, bytes};
  in_use += bytes;
  if (in_use > peak) peak = in_use;
  return TC_OK;
}

void tc_ctx::release(void* p, bool pooled) {
  if (!p) return;
  // wait for what the context's stream still does with the block: its next owner
  // may hand it to a synchronous call.  (Nothing else is waited for, so pooled
  // memory must not be written on any other stream, the default one included.)
  const bool idle = pooled && cudaStreamSynchronize(stream) == cudaSuccess;
  std::vector<void*> back;  // kept blocks that make room for this one
  bool keep = false;
  {
    std::lock_guard<std::mutex> g(mu);
    auto it = allocs.find(p);
    if (it != allocs.end()) {
      in_use -= it->second.asked;
      const size_t bytes = it->second.size;
      allocs.erase(it);
      const size_t room = !budget ? tc::kPoolMax : std::min(tc::kPoolMax, budget > in_use ? budget - in_use : 0);
      keep = idle && bytes <= tc::kPoolBlockMax && bytes <= room;
      if (keep) {
        while (pool_bytes + bytes > room) {  // the longest kept first
          auto old = pool.begin();
          for (auto b = pool.begin(); b != pool.end(); ++b)
            if (b->second.order < old->second.order) old = b;
          back.push_back(old->second.p);
          pool_bytes -= old->first;
          pool.erase(old);
        }
        pool.emplace(bytes, tc::KeptBlock{p, pool_order++});
        pool_bytes += bytes;
      }
    }
  }
  if (!keep) cudaFree(p);
  for (void* q : back) cudaFree(q);
}

void tc_ctx::trim_pool() {
  std::multimap<size_t, tc::KeptBlock> blocks;
  {
    std::lock_guard<std::mutex> g(mu);
    blocks.swap(pool);
    pool_bytes = 0;
  }
  for (auto& kv : blocks) cudaFree(kv.second.p);
}

extern "C" {

tc_status tc_ctx_create(int device, size_t mem_budget, tc_ctx** out) {
  if (!out) return TC_ERR_INVALID_ARG;
  *out = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
    cudaGetLastError();
    return TC_ERR_CUDA;
  }
  if (device < 0 || device >= count) return TC_ERR_INVALID_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return TC_ERR_CUDA;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return TC_ERR_CUDA;
  if (prop.major < 10) return TC_ERR_CUDA;  // built for sm_100a only
  tc_ctx* c = new tc_ctx();
  c->device = device;
  c->sm_count = prop.multiProcessorCount;
  c->budget = mem_budget;
  if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete c;
    return TC_ERR_CUDA;
  }
  if (cudaStreamCreateWithFlags(&c->pred_stream, cudaStreamNonBlocking) != cudaSuccess) {
    cudaStreamDestroy(c->stream);
    delete c;
    return TC_ERR_CUDA;
  }
  {
    std::lock_guard<std::mutex> g(contexts().mu);
    contexts().all.push_back(c);
  }
  *out = c;
  return TC_OK;
}

void tc_ctx_destroy(tc_ctx* ctx) {
  if (!ctx) return;
  {
    std::lock_guard<std::mutex> g(contexts().mu);
    auto& all = contexts().all;
    all.erase(std::remove(all.begin(), all.end(), ctx), all.end());
  }
  cudaSetDevice(ctx->device);
  {
    std::lock_guard<std::mutex> g(ctx->pred_mu);
    tc::stop_latency_worker(ctx, nullptr);
  }
  cudaStreamSynchronize(ctx->stream);
  cudaStreamSynchronize(ctx->pred_stream);
  ctx->trim_pool();
  for (auto& kv : ctx->allocs) cudaFree(kv.first);
  ctx->allocs.clear();
  if (ctx->pin_io) cudaFreeHost(ctx->pin_io);
  if (ctx->lw_box) cudaFreeHost(ctx->lw_box);
  for (int b = 0; b < 2; ++b) {
    if (ctx->up_stage[b]) cudaFreeHost(ctx->up_stage[b]);
    if (ctx->up_ev[b]) cudaEventDestroy(ctx->up_ev[b]);
  }
  if (ctx->lw_stream) cudaStreamDestroy(ctx->lw_stream);
  cudaStreamDestroy(ctx->stream);
  cudaStreamDestroy(ctx->pred_stream);
  delete ctx;
}

const char* tc_last_error(const tc_ctx* ctx) {
  if (!ctx) return "null context";
  return ctx->err.c_str();
}

tc_status tc_ctx_memory(const tc_ctx* ctx, size_t* in_use, size_t* peak) {
  if (!ctx) return TC_ERR_INVALID_ARG;
  if (in_use) *in_use = ctx->in_use;
  if (peak) *peak = ctx->peak;
  return TC_OK;
}

tc_status tc_ctx_trim(tc_ctx* ctx) {
  if (!ctx) return TC_ERR_INVALID_ARG;
  cudaSetDevice(ctx->device);
  ctx->trim_pool();
  return TC_OK;
}

tc_status tc_ctx_fail_next_allocs(tc_ctx* ctx, int count) {
  if (!ctx || count < 0) return TC_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> g(ctx->mu);
  ctx->fail_next = count;
  return TC_OK;
}

// Polls the context stream instead of blocking in the driver so that a
// stuck device turns into TC_ERR_TIMEOUT rather than a hung caller.
tc_status tc_ctx_set_latency_worker(tc_ctx* ctx, int enabled) {
  if (!ctx) return TC_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> g(ctx->pred_mu);
  cudaSetDevice(ctx->device);
  if (!enabled) tc::stop_latency_worker(ctx, nullptr);
  ctx->lw_enabled = enabled != 0;
  return TC_OK;
}

tc_status tc_ctx_synchronize(tc_ctx* ctx, int timeout_ms) {
  if (!ctx) return TC_ERR_INVALID_ARG;
  // not while another thread's training call may be capturing the stream
  std::lock_guard<std::recursive_mutex> train_lock(ctx->train_mu);
  cudaSetDevice(ctx->device);
  const auto t0 = std::chrono::steady_clock::now();
  for (;;) {
    cudaError_t e = cudaStreamQuery(ctx->stream);
    if (e == cudaSuccess) e = cudaStreamQuery(ctx->pred_stream);
    if (e == cudaSuccess) return TC_OK;
    if (e != cudaErrorNotReady) return ctx->cuda_fail(e, "stream");
    const auto dt = std::chrono::duration_cast<std::chrono::milliseconds>(
                        std::chrono::steady_clock::now() - t0).count();
    if (timeout_ms >= 0 && dt >= timeout_ms)
      return ctx->fail(TC_ERR_TIMEOUT, "device work did not finish within %d ms", timeout_ms);
    std::this_thread::sleep_for(std::chrono::microseconds(50));
  }
}

}  // extern "C"
