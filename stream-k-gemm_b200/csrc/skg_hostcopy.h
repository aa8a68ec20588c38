// Copies between pageable host memory and the device for the blocking host-
// pointer entry points: several host threads move pieces through pinned slots,
// so that the transfer runs at the link's rate instead of one staging thread's
// (11 GB/s measured for cudaMemcpyAsync on pageable memory; the 57 MB of a
// 13824 x 256 GEMM took 4.9 ms of its 5.0 ms). Pinned and managed memory, and
// copies too small to gain, go to cudaMemcpy2DAsync directly.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <condition_variable>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "skg_runtime.h"

namespace skg {

// One direction's pinned slots of a device, kept between calls (guarded by the
// device's host_mu like its staging buffers; at most 8 MB a direction) and
// freed by host_slots_release (skgemm_stream_release of the default stream).
struct HostSlots {
  // Threads 4 / 6 / 8 / 12 with 1 MB slots: 57 MB up in 2.1 / 2.3 / 2.5 / 3.2 ms
  // (512 KB slots 3.0 ms with 8, 2 MB 2.6 ms).
  static constexpr int kMaxThreads = 4;
  static constexpr size_t kSlotBytes = 1 << 20;
  char* base = nullptr;  // [threads][2][kSlotBytes]
  cudaEvent_t ev[2 * kMaxThreads] = {};
  int threads = 0;
  int ensure();
  void release();
};

class HostCopy {
 public:
  // Copies of one direction on stream `s` (kind: H2D or D2H).
  HostCopy(DeviceState* dev, cudaMemcpyKind kind, cudaStream_t s);
  ~HostCopy();
  HostCopy(const HostCopy&) = delete;
  HostCopy& operator=(const HostCopy&) = delete;

  // A 2-D copy of `height` rows of `width` bytes as part of group g (groups
  // 0, 1, .. in order), before start().
  void add(int g, void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
           size_t height);
  // Begins. Groups of a gated copy wait for open(g).
  int start(bool gated = false);
  // The group's pieces may be enqueued from here on.
  int open(int g);
  // H2D: returns when every piece of group g is enqueued on the stream. Where the
  // driver copies, only then: an event recorded next marks this group, not the later
  // ones too.
  int wait_group(int g);
  // Every piece is enqueued (H2D) or in host memory (D2H).
  int finish();

 private:
  struct Piece {
    int group;
    char* dst;
    size_t dpitch;
    const char* src;
    size_t spitch, width, height;
  };
  void work(int w);
  void fail_with(cudaError_t e);
  int direct(int g);  // enqueues the groups up to g that are not yet

  DeviceState* dev_;
  cudaMemcpyKind kind_;
  cudaStream_t s_;
  HostSlots* slots_;
  std::vector<Piece> pieces_, whole_;
  std::vector<int> left_;  // pieces of each group still to do
  std::vector<std::thread> threads_;
  std::mutex mu_;
  std::condition_variable cv_;
  std::atomic<size_t> next_{0};
  int opened_ = 0;       // groups below may run
  int next_direct_ = 0;  // first group the driver has not been given
  bool staged_ = false, stop_ = false, gated_ = false;
  cudaError_t err_ = cudaSuccess;
  size_t bytes_ = 0;
};

// Streams, events and the upload of one chunked host-pointer call (host_mu held).
struct HostPipe {
  DeviceState* dev = nullptr;
  cudaStream_t sc = nullptr, si = nullptr;  // compute, uploads
  std::vector<cudaEvent_t> ev;
  std::unique_ptr<HostCopy> up;
  int init(DeviceState* d, int n);
  // The call's host -> device copies, on si.
  HostCopy& upload();
  // Ends the upload (its threads enqueue nothing more), waits for both streams, frees
  // the events and reports device-side errors. Returns st if it is one: the pinned
  // slots and the staging buffers are then free for the next call in any case.
  int finish(int st);
};

// Frees the pinned slots of the device (host_mu held by the caller).
void host_slots_release(DeviceState* dev);

}  // namespace skg
