// Threaded copies between pageable host memory and the device (skg_hostcopy.h).
#include "skg_hostcopy.h"

#include <algorithm>
#include <cstring>
#include <system_error>

namespace skg {

namespace {

HostSlots g_slots[64][2];  // [device][0: H2D, 1: D2H]

// Copies below this stay with the driver. Starting the threads costs about what 2 MB
// take at 11 GB/s; short uploads run faster than that in the driver (us for a whole
// call, driver / threads: 3.4 MB up 362 / 432, 8.0 MB 601 / 691, 20 MB 1261 / 1181, 29 MB
// 1745 / 1120), short downloads do not (3.4 MB up and down 424 / 383).
constexpr size_t kStagedMinUp = 9 << 20, kStagedMinDown = 2 << 20;

bool pageable(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

}  // namespace

int HostSlots::ensure() {
  if (base) return SKGEMM_OK;
  const int hw = (int)std::thread::hardware_concurrency();
  threads = std::max(1, std::min(kMaxThreads, hw / 2));
  SKG_CUDA(cudaHostAlloc((void**)&base, (size_t)threads * 2 * kSlotBytes, cudaHostAllocPortable));
  for (int i = 0; i < 2 * threads; ++i) {
    const cudaError_t e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
    if (e != cudaSuccess) {
      release();
      return cuda_fail(e, "host copy events");
    }
  }
  return SKGEMM_OK;
}

void HostSlots::release() {
  for (cudaEvent_t& e : ev) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  if (base) cudaFreeHost(base);
  base = nullptr;
  threads = 0;
}

void host_slots_release(DeviceState* dev) {
  for (HostSlots& h : g_slots[dev->device]) h.release();
}

HostCopy::HostCopy(DeviceState* dev, cudaMemcpyKind kind, cudaStream_t s)
    : dev_(dev), kind_(kind), s_(s),
      slots_(&g_slots[dev->device][kind == cudaMemcpyHostToDevice ? 0 : 1]) {}

HostCopy::~HostCopy() {
  {
    std::lock_guard<std::mutex> lk(mu_);
    stop_ = true;
  }
  cv_.notify_all();
  for (std::thread& t : threads_) t.join();
}

void HostCopy::add(int g, void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
                   size_t height) {
  if ((int)left_.size() <= g) left_.resize(g + 1, 0);
  if (!width || !height) return;
  whole_.push_back({g, (char*)dst, dpitch, (const char*)src, spitch, width, height});
  bytes_ += width * height;
}

int HostCopy::start(bool gated) {
  if (!gated) opened_ = (int)left_.size();
  const void* host = nullptr;
  if (!whole_.empty()) host = kind_ == cudaMemcpyHostToDevice ? whole_[0].src : whole_[0].dst;
  staged_ = host && bytes_ >= (kind_ == cudaMemcpyHostToDevice ? kStagedMinUp : kStagedMinDown);
  for (const Piece& p : whole_)
    staged_ = staged_ && pageable(kind_ == cudaMemcpyHostToDevice ? p.src : p.dst);
  // Without pinned slots or threads the driver copies.
  if (staged_ && slots_->ensure() != SKGEMM_OK) {
    cudaGetLastError();  // or the next launch's check would report it
    staged_ = false;
  }
  gated_ = gated;
  if (!staged_) return SKGEMM_OK;
  try {
    // Pieces of a slot; smaller ones where a thread would get fewer than four, so that
    // no thread is left waiting for another's last piece.
    const size_t even = (bytes_ / (4 * slots_->threads) + 4095) / 4096 * 4096;
    const size_t slot = std::min(HostSlots::kSlotBytes, std::max<size_t>(even, 256 << 10));
    for (const Piece& p : whole_) {
      if (p.width >= slot) {  // a row in several pieces
        for (size_t r = 0; r < p.height; ++r)
          for (size_t o = 0; o < p.width; o += slot)
            pieces_.push_back({p.group, p.dst + r * p.dpitch + o, p.dpitch,
                               p.src + r * p.spitch + o, p.spitch, std::min(slot, p.width - o), 1});
      } else {  // several rows in a piece
        const size_t n = slot / p.width;
        for (size_t r = 0; r < p.height; r += n)
          pieces_.push_back({p.group, p.dst + r * p.dpitch, p.dpitch, p.src + r * p.spitch,
                             p.spitch, p.width, std::min(n, p.height - r)});
      }
    }
    for (const Piece& p : pieces_) ++left_[p.group];
    const int n = std::min<int>(slots_->threads, (int)pieces_.size());
    for (int w = 0; w < n; ++w) threads_.emplace_back(&HostCopy::work, this, w);
  } catch (const std::exception&) {
    if (!threads_.empty()) return SKGEMM_OK;  // fewer threads share the pieces
    pieces_.clear();
    std::fill(left_.begin(), left_.end(), 0);
    staged_ = false;
  }
  return SKGEMM_OK;
}

int HostCopy::direct(int g) {
  for (; next_direct_ <= g; ++next_direct_)
    for (const Piece& p : whole_)
      if (p.group == next_direct_) {
        if (p.height == 1)
          SKG_CUDA(cudaMemcpyAsync(p.dst, p.src, p.width, kind_, s_));
        else
          SKG_CUDA(
              cudaMemcpy2DAsync(p.dst, p.dpitch, p.src, p.spitch, p.width, p.height, kind_, s_));
      }
  return SKGEMM_OK;
}

int HostCopy::open(int g) {
  if (!staged_) return direct(g);
  {
    std::lock_guard<std::mutex> lk(mu_);
    opened_ = std::max(opened_, g + 1);
  }
  cv_.notify_all();
  return SKGEMM_OK;
}

void HostCopy::fail_with(cudaError_t e) {
  {
    std::lock_guard<std::mutex> lk(mu_);
    if (err_ == cudaSuccess) err_ = e;
    stop_ = true;
  }
  cv_.notify_all();
}

int HostCopy::wait_group(int g) {
  if (!staged_) return direct(g);
  std::unique_lock<std::mutex> lk(mu_);
  cv_.wait(lk, [&] { return left_[g] == 0 || stop_; });
  return err_ == cudaSuccess ? SKGEMM_OK : cuda_fail(err_, "host copy");
}

int HostCopy::finish() {
  if (!staged_) return gated_ ? SKGEMM_OK : direct((int)left_.size() - 1);
  for (std::thread& t : threads_) t.join();
  threads_.clear();
  return err_ == cudaSuccess ? SKGEMM_OK : cuda_fail(err_, "host copy");
}

void HostCopy::work(int w) {
  cudaError_t e = cudaSetDevice(dev_->device);
  if (e != cudaSuccess) return fail_with(e);
  const bool up = kind_ == cudaMemcpyHostToDevice;
  bool used[2] = {false, false};
  const Piece* pend = nullptr;  // D2H: enqueued, not yet in host memory
  int pend_k = 0, k = 0;
  auto slot = [&](int i) { return slots_->base + (size_t)(2 * w + i) * HostSlots::kSlotBytes; };
  auto done = [&](const Piece& p) {
    bool last;
    {
      std::lock_guard<std::mutex> lk(mu_);
      last = --left_[p.group] == 0;
    }
    if (last) cv_.notify_all();
  };
  auto drain = [&]() -> bool {
    if (!pend) return true;
    if ((e = cudaEventSynchronize(slots_->ev[2 * w + pend_k])) != cudaSuccess) {
      fail_with(e);
      return false;
    }
    for (size_t r = 0; r < pend->height; ++r)
      memcpy(pend->dst + r * pend->dpitch, slot(pend_k) + r * pend->width, pend->width);
    done(*pend);
    pend = nullptr;
    return true;
  };
  for (;;) {
    const size_t i = next_.fetch_add(1);
    if (i >= pieces_.size()) break;
    const Piece& p = pieces_[i];
    {
      std::unique_lock<std::mutex> lk(mu_);
      if (stop_) return;
      if (p.group >= opened_) {
        lk.unlock();
        if (!drain()) return;
        lk.lock();
        cv_.wait(lk, [&] { return p.group < opened_ || stop_; });
        if (stop_) return;
      }
    }
    cudaEvent_t ev = slots_->ev[2 * w + k];
    if (up) {
      if (used[k] && (e = cudaEventSynchronize(ev)) != cudaSuccess) return fail_with(e);
      for (size_t r = 0; r < p.height; ++r)
        memcpy(slot(k) + r * p.width, p.src + r * p.spitch, p.width);
      e = p.height == 1 ? cudaMemcpyAsync(p.dst, slot(k), p.width, kind_, s_)
                        : cudaMemcpy2DAsync(p.dst, p.dpitch, slot(k), p.width, p.width, p.height,
                                            kind_, s_);
    } else {
      e = p.height == 1 ? cudaMemcpyAsync(slot(k), p.src, p.width, kind_, s_)
                        : cudaMemcpy2DAsync(slot(k), p.width, p.src, p.spitch, p.width, p.height,
                                            kind_, s_);
    }
    if (e == cudaSuccess) e = cudaEventRecord(ev, s_);
    if (e != cudaSuccess) return fail_with(e);
    used[k] = true;
    if (up) {
      done(p);
    } else {
      if (!drain()) return;
      pend = &p;
      pend_k = k;
    }
    k ^= 1;
  }
  drain();
}

int HostPipe::init(DeviceState* d, int n) {
  dev = d;
  for (cudaStream_t* ps : {&dev->host_stream, &dev->host_h2d, &dev->host_d2h})
    if (!*ps) SKG_CUDA(cudaStreamCreateWithFlags(ps, cudaStreamNonBlocking));
  sc = dev->host_stream;
  si = dev->host_h2d;
  ev.assign(n, nullptr);
  for (auto& e : ev) SKG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  return SKGEMM_OK;
}

HostCopy& HostPipe::upload() {
  up.reset(new HostCopy(dev, cudaMemcpyHostToDevice, si));
  return *up;
}

int HostPipe::finish(int st) {
  up.reset();  // before the wait: a copy enqueued behind it would outlive the call
  cudaStreamSynchronize(si);
  cudaStreamSynchronize(sc);
  for (auto& e : ev)
    if (e) cudaEventDestroy(e);
  ev.clear();
  if (st) return st;
  StreamWorkspace* ws = nullptr;
  {
    std::lock_guard<std::mutex> lk(dev->mu);
    auto it = dev->ws.find(sc);
    if (it != dev->ws.end()) ws = it->second;
  }
  return consume_device_error(ws, sc);
}

}  // namespace skg
