// Copies between pageable host memory and the device.
//
// A caller's arrays are ordinary memory: the driver copies them through a pinned buffer of its
// own with one thread, which for a freshly allocated destination also takes every page
// fault (a 2048^2 solve spent 25 of 31 ms there: 33 MB in, 101 MB out). Copies of STAGE_MIN
// bytes and more go through a ring of pinned chunks instead: the DMA of one chunk overlaps the
// memory copies of others, which a few worker threads make. Smaller copies, and host memory that
// is already pinned, go to the driver directly.

#include <condition_variable>
#include <cstring>
#include <deque>
#include <mutex>
#include <system_error>
#include <thread>

#include "context.h"

namespace otm {

// STAGE_MIN: below it, waking the workers costs more than they save, and the allocator hands out
// memory whose pages are there (density in and mesh out of a solve: 512^2, 2 and 4 MB, 0.86 ms
// staged against 0.71 direct; 1024^2, 8 and 17 MB, 1.59 against 2.06; 2048^2 9.5 against 24.9).
// Chunks of 2 or 4 MB were no faster than 1 MB. WORKERS: density in and mesh and density out of a 2048^2
// solve without iterations take 20.6, 14.9, 11.8, 10.5, 8.2, 8.4 and 10.6 ms with 1, 2, 3, 4, 6, 8 and
// 12 workers on 16 cores, 4096^2 81, 59, 46, 36, 28, 27 and 36.
constexpr size_t STAGE_MIN = size_t(8) << 20;
constexpr size_t CHUNK_MIN = size_t(512) << 10, CHUNK_MAX = size_t(1) << 20;
constexpr int SLOTS = 16, WORKERS = 6;

struct HostCopier {
  struct Job {
    void* dst;
    const void* src;
    size_t bytes;
    int slot;
  };
  unsigned char* ring = nullptr;  // SLOTS chunks of pinned memory
  cudaEvent_t dma[SLOTS] = {};    // the slot's last transfer
  bool busy[SLOTS] = {};          // a memory copy of the slot is queued or running
  std::vector<std::thread> threads;
  std::mutex mu;
  std::condition_variable work, done;
  std::deque<Job> jobs;
  bool stop = false;

  HostCopier() {
    try {
      OTM_CUDA(cudaMallocHost((void**)&ring, CHUNK_MAX * SLOTS));
      for (auto& e : dma) OTM_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
      for (int k = 0; k < WORKERS; ++k) threads.emplace_back([this] { run(); });
    } catch (...) {
      release();
      throw;
    }
  }
  HostCopier(const HostCopier&) = delete;
  HostCopier& operator=(const HostCopier&) = delete;
  ~HostCopier() { release(); }

  void release() {
    {
      std::lock_guard<std::mutex> l(mu);
      stop = true;
    }
    work.notify_all();
    for (auto& t : threads) t.join();
    threads.clear();
    for (auto& e : dma)
      if (e) cudaEventDestroy(e);
    if (ring) cudaFreeHost(ring);
    ring = nullptr;
  }

  void run() {
    std::unique_lock<std::mutex> l(mu);
    while (true) {
      work.wait(l, [this] { return stop || !jobs.empty(); });
      if (jobs.empty()) return;
      const Job j = jobs.front();
      jobs.pop_front();
      l.unlock();
      std::memcpy(j.dst, j.src, j.bytes);
      l.lock();
      busy[j.slot] = false;
      done.notify_all();
    }
  }

  void queue(const Job& j) {
    {
      std::lock_guard<std::mutex> l(mu);
      busy[j.slot] = true;
      jobs.push_back(j);
    }
    work.notify_one();
  }
  void wait(int slot) {
    std::unique_lock<std::mutex> l(mu);
    done.wait(l, [&] { return !busy[slot]; });
  }
  // Every queued memory copy has ended (also when a transfer failed: the caller's memory is
  // not touched once the call has returned).
  void drain() {
    for (int s = 0; s < SLOTS; ++s) wait(s);
  }
  unsigned char* slot(int s) { return ring + CHUNK_MAX * s; }

  static size_t chunk_of(size_t bytes) {
    size_t c = (bytes / SLOTS + 4095) / 4096 * 4096;
    return c < CHUNK_MIN ? CHUNK_MIN : c > CHUNK_MAX ? CHUNK_MAX : c;
  }

  void in(void* dst, const unsigned char* src, size_t bytes, cudaStream_t st) {
    const size_t c = chunk_of(bytes);
    const size_t chunks = (bytes + c - 1) / c;
    auto size = [&](size_t k) { return k + 1 < chunks ? c : bytes - k * c; };
    try {
      for (size_t k = 0; k < chunks + SLOTS; ++k) {
        const int s = (int)(k % SLOTS);
        if (k >= SLOTS) {  // chunk k - SLOTS is in the slot: on its way to the device
          const size_t p = k - SLOTS;
          if (p < chunks) {
            wait(s);
            OTM_CUDA(cudaMemcpyAsync((unsigned char*)dst + p * c, slot(s), size(p), cudaMemcpyHostToDevice, st));
            OTM_CUDA(cudaEventRecord(dma[s], st));
          }
        }
        if (k < chunks) {
          OTM_CUDA(cudaEventSynchronize(dma[s]));  // the slot's last transfer has left it
          queue({slot(s), src + k * c, size(k), s});
        }
      }
    } catch (...) {
      drain();
      throw;
    }
  }

  void out(unsigned char* dst, const void* src, size_t bytes, cudaStream_t st) {
    const size_t c = chunk_of(bytes);
    const size_t chunks = (bytes + c - 1) / c;
    auto size = [&](size_t k) { return k + 1 < chunks ? c : bytes - k * c; };
    constexpr int AHEAD = SLOTS / 2;  // transfers in flight; the other slots are being emptied
    try {
      for (size_t k = 0; k < chunks + AHEAD; ++k) {
        if (k < chunks) {
          const int s = (int)(k % SLOTS);
          wait(s);
          OTM_CUDA(cudaEventSynchronize(dma[s]));
          OTM_CUDA(cudaMemcpyAsync(slot(s), (const unsigned char*)src + k * c, size(k), cudaMemcpyDeviceToHost, st));
          OTM_CUDA(cudaEventRecord(dma[s], st));
        }
        if (k >= AHEAD) {
          const size_t p = k - AHEAD;
          const int s = (int)(p % SLOTS);
          OTM_CUDA(cudaEventSynchronize(dma[s]));
          queue({dst + p * c, slot(s), size(p), s});
        }
      }
    } catch (...) {
      drain();
      throw;
    }
    drain();
  }
};

void HostCopierDelete::operator()(HostCopier* c) const { delete c; }

// The context's copier, made on the first large copy; null when its memory or threads cannot
// be had (the driver's copies then serve).
static HostCopier* copier(otm_context* ctx) {
  if (!ctx->copier && !ctx->copier_failed) {
    try {
      ctx->copier.reset(new HostCopier);
    } catch (const CudaError&) {
      cudaGetLastError();
      ctx->copier_failed = true;
    } catch (const std::exception&) {
      ctx->copier_failed = true;
    }
  }
  return ctx->copier.get();
}

static bool pageable(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

void copy_in(otm_context* ctx, void* dst, const void* src, size_t bytes) {
  if (!bytes) return;
  if (bytes >= STAGE_MIN && pageable(src))
    if (HostCopier* c = copier(ctx)) return c->in(dst, static_cast<const unsigned char*>(src), bytes, ctx->stream);
  OTM_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, ctx->stream));
}

void copy_out(otm_context* ctx, void* dst, const void* src, size_t bytes, cudaStream_t st) {
  if (!bytes) return;
  if (bytes >= STAGE_MIN && pageable(dst))
    if (HostCopier* c = copier(ctx)) return c->out(static_cast<unsigned char*>(dst), src, bytes, st);
  OTM_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, st));
}
void copy_out(otm_context* ctx, void* dst, const void* src, size_t bytes) {
  copy_out(ctx, dst, src, bytes, ctx->stream);
}

}  // namespace otm
