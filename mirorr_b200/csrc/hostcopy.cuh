// hostcopy.cuh -- copies between device memory and a caller's ordinary
// (pageable) host memory, of which every host-array entry point makes some:
// volumes in, resampled volumes and point lists out.
//
// The runtime stages such a copy through pinned memory on the calling thread,
// so it runs at one core's copy rate on a link of 55 GB/s.  Here a few threads
// share the host side of the same staging: chunks of a pinned buffer, each
// filled or emptied by whichever thread is free while others are on the link.
// Measured (us, the runtime's copy -> this one, 16 cores, arrays not in the
// caches):
//   to the host    4 MB 235 -> 253, 8 MB 432 -> 296, 32 MB 1596 -> 943,
//                  256 MB 16164 -> 8856
//   to the device  8 MB 780 -> 1205, 16 MB 1536 -> 1509, 32 MB 3037 -> 1698,
//                  64 MB 5933 -> 2439: the chunks are filled at 40 GB/s, but the
//                  first of them, fresh in several cores' caches, take the link
//                  0.8 ms whatever the size
// so each direction has its own least size.
#pragma once

#include <cstddef>
#include <mutex>

#include "common.cuh"

namespace mb2 {

class HostCopier {
 public:
  // Copies src (host) to dst (device) in stream order; the caller may reuse src
  // on return (the device copy may still be on its way).
  mirorr_status to_device(void *dst, const void *src, size_t bytes, cudaStream_t s);
  // Copies src (device) to dst (host) after the stream's earlier work; dst is
  // filled on return.
  mirorr_status to_host(void *dst, const void *src, size_t bytes, cudaStream_t s);
  // Ends the threads and frees the staging buffer (no copy in flight).
  void release();
  ~HostCopier() { release(); }

 private:
  static constexpr size_t kChunk = 1 << 19;
  static constexpr int kHalf = 16, kSlots = 2 * kHalf;  // 16 MB of staging per context
  static constexpr size_t kMinIn = 24 << 20, kMinOut = 5 << 20;  // smaller ones go plainly
  static constexpr int kWorkers = 5;

  struct Pool;  // threads, staging chunks and their events

  // The pool, made on the first large copy; null: copy plainly.
  Pool *pool(const void *host, cudaStream_t s);

  Pool *pool_ = nullptr;
  bool failed_ = false;
  std::mutex use_;  // one copy at a time; a second thread's copies plainly
};

}  // namespace mb2
