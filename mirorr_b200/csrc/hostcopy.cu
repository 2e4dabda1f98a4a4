// hostcopy.cu -- see hostcopy.cuh.
#include "hostcopy.cuh"

#include <sys/types.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <new>
#include <thread>

namespace mb2 {

struct HostCopier::Pool {
  unsigned char *pin = nullptr;
  cudaEvent_t ev[kSlots] = {};
  bool pending[kSlots] = {};  // ev was recorded behind a copy of the slot
  int device = 0;
  pid_t pid = 0;  // of the process that has the threads

  std::mutex mu;
  std::condition_variable wake, idle;
  std::thread threads[kWorkers];
  int nthreads = 0, busy = 0;
  unsigned long long round = 0;
  bool stop = false;
  void (*fn)(void *, int) = nullptr;
  void *arg = nullptr;
  int n = 0;
  std::atomic<int> next{0};

  // On the current device; false: nothing is left behind but what end() frees.
  bool start() {
    pid = getpid();
    void *p = nullptr;
    if (cudaGetDevice(&device) != cudaSuccess || cudaMallocHost(&p, kChunk * kSlots) != cudaSuccess)
      return false;
    pin = static_cast<unsigned char *>(p);
    for (auto &e : ev)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        e = nullptr;
        return false;
      }
    const int want = std::min(kWorkers, (int)std::thread::hardware_concurrency() / 2 - 1);
    try {
      for (; nthreads < want; ++nthreads) threads[nthreads] = std::thread([this] { work(); });
    } catch (const std::exception &) {
      // fewer threads than wanted (none: the caller fills the chunks alone)
    }
    return true;
  }

  void end() {
    {
      std::lock_guard<std::mutex> lock(mu);
      stop = true;
    }
    wake.notify_all();
    for (int i = 0; i < nthreads; ++i) threads[i].join();
    for (int i = 0; i < kSlots; ++i)
      if (ev[i]) {
        if (pending[i]) cudaEventSynchronize(ev[i]);
        cudaEventDestroy(ev[i]);
      }
    if (pin) cudaFreeHost(pin);
  }

  void work() {
    cudaSetDevice(device);
    unsigned long long seen = 0;
    std::unique_lock<std::mutex> lock(mu);
    for (;;) {
      wake.wait(lock, [&] { return stop || round != seen; });
      if (stop) return;
      seen = round;
      lock.unlock();
      for (int i; (i = next.fetch_add(1)) < n;) fn(arg, i);
      lock.lock();
      if (--busy == 0) idle.notify_one();
    }
  }

  // f(0) .. f(count - 1) over the threads and the caller, who calls own() after
  // each of its part; returns when all are done and every thread waits again.
  template <class F, class G>
  void share(int count, F f, G own) {
    {
      std::lock_guard<std::mutex> lock(mu);
      fn = [](void *a, int i) { (*static_cast<F *>(a))(i); };
      arg = &f;
      n = count;
      next.store(0);
      busy = nthreads;
      ++round;
    }
    wake.notify_all();
    for (int i; (i = next.fetch_add(1)) < count;) {
      f(i);
      own();
    }
    std::unique_lock<std::mutex> lock(mu);
    idle.wait(lock, [&] { return busy == 0; });
  }
};

HostCopier::Pool *HostCopier::pool(const void *host, cudaStream_t s) {
  if (failed_) return nullptr;
  if (pool_ && pool_->pid != getpid()) return nullptr;  // forked: the threads stayed behind
  // memory the device reaches by itself (pinned, managed) needs no staging, and
  // a stream under capture takes the copy as the one node it always was
  cudaPointerAttributes at;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess ||
      cudaStreamIsCapturing(s, &cap) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (at.type != cudaMemoryTypeUnregistered || cap != cudaStreamCaptureStatusNone) return nullptr;
  if (!pool_) {
    pool_ = new (std::nothrow) Pool;
    if (!pool_ || !pool_->start()) {
      cudaGetLastError();
      release();
      failed_ = true;
    }
  }
  return pool_;
}

void HostCopier::release() {
  if (!pool_) return;
  if (pool_->pid == getpid()) {
    pool_->end();
    delete pool_;
  }  // else a forked child, where neither the threads nor the device memory exist
  pool_ = nullptr;
}

mirorr_status HostCopier::to_device(void *dst, const void *src, size_t bytes, cudaStream_t s) {
  std::unique_lock<std::mutex> use(use_, std::defer_lock);
  Pool *pl = bytes >= kMinIn && use.try_lock() ? pool(src, s) : nullptr;
  if (!pl) {
    MB2_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
    return MIRORR_OK;
  }
  const long long chunks = (long long)((bytes + kChunk - 1) / kChunk);
  // The halves of the buffer in turn: one is filled while the other is on the
  // link.  Only this thread calls the runtime (its lock, taken by all of them,
  // cost 0.4 ms a round): the chunks go out in order as they are filled.
  std::atomic<bool> full[kHalf];
  for (long long c0 = 0; c0 < chunks; c0 += kHalf) {
    const int h = (int)((c0 / kHalf) & 1) * kHalf, n = (int)std::min<long long>(kHalf, chunks - c0);
    for (int i = 0; i < kHalf; ++i) {
      if (pl->pending[h + i]) MB2_CUDA_TRY(cudaEventSynchronize(pl->ev[h + i]));
      pl->pending[h + i] = false;
      full[i].store(false, std::memory_order_relaxed);
    }
    int sent = 0;
    cudaError_t e = cudaSuccess;
    auto send = [&] {
      for (; sent < n && e == cudaSuccess && full[sent].load(std::memory_order_acquire); ++sent) {
        const size_t off = (size_t)(c0 + sent) * kChunk;
        e = cudaMemcpyAsync(static_cast<unsigned char *>(dst) + off,
                            pl->pin + (size_t)(h + sent) * kChunk, std::min(kChunk, bytes - off),
                            cudaMemcpyHostToDevice, s);
      }
    };
    pl->share(n, [&](int i) {
      const size_t off = (size_t)(c0 + i) * kChunk;
      memcpy(pl->pin + (size_t)(h + i) * kChunk, static_cast<const unsigned char *>(src) + off,
             std::min(kChunk, bytes - off));
      full[i].store(true, std::memory_order_release);
    }, send);
    send();
    MB2_CUDA_TRY(e);
    MB2_CUDA_TRY(cudaEventRecord(pl->ev[h], s));  // behind the whole half
    pl->pending[h] = true;
  }
  return MIRORR_OK;
}

mirorr_status HostCopier::to_host(void *dst, const void *src, size_t bytes, cudaStream_t s) {
  std::unique_lock<std::mutex> use(use_, std::defer_lock);
  Pool *pl = bytes >= kMinOut && use.try_lock() ? pool(dst, s) : nullptr;
  if (!pl) {
    MB2_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s));
    MB2_CUDA_TRY(cudaStreamSynchronize(s));
    return MIRORR_OK;
  }
  const long long chunks = (long long)((bytes + kChunk - 1) / kChunk);
  std::atomic<int> err{(int)cudaSuccess};
  // the halves of the buffer in turn: one is emptied while the next copies are
  // on the link
  auto issue = [&](long long c0) -> mirorr_status {
    const int h = (int)((c0 / kHalf) & 1) * kHalf;
    if (pl->pending[h]) MB2_CUDA_TRY(cudaStreamWaitEvent(s, pl->ev[h], 0));
    for (int i = 0; i < kHalf && c0 + i < chunks; ++i) {
      const size_t off = (size_t)(c0 + i) * kChunk, len = std::min(kChunk, bytes - off);
      MB2_CUDA_TRY(cudaMemcpyAsync(pl->pin + (size_t)(h + i) * kChunk,
                                   static_cast<const unsigned char *>(src) + off, len,
                                   cudaMemcpyDeviceToHost, s));
      MB2_CUDA_TRY(cudaEventRecord(pl->ev[h + i], s));
      pl->pending[h + i] = true;
    }
    return MIRORR_OK;
  };
  MB2_TRY(issue(0));
  // the stream's earlier work is waited for here, by one thread
  MB2_CUDA_TRY(cudaEventSynchronize(pl->ev[0]));
  for (long long c0 = 0; c0 < chunks; c0 += kHalf) {
    if (c0 + kHalf < chunks) MB2_TRY(issue(c0 + kHalf));
    const int h = (int)((c0 / kHalf) & 1) * kHalf;
    pl->share((int)std::min<long long>(kHalf, chunks - c0), [&](int i) {
      const size_t off = (size_t)(c0 + i) * kChunk, len = std::min(kChunk, bytes - off);
      const cudaError_t e = cudaEventSynchronize(pl->ev[h + i]);
      if (e == cudaSuccess)
        memcpy(static_cast<unsigned char *>(dst) + off, pl->pin + (size_t)(h + i) * kChunk, len);
      else
        err.store((int)e);
    }, [] {});
    MB2_CUDA_TRY((cudaError_t)err.load());
  }
  return MIRORR_OK;
}

}  // namespace mb2
