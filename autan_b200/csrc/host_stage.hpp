// Copies between pageable host memory and the device through pinned slots.
//
// A pageable cudaMemcpyAsync is staged by the driver on the calling thread, one piece after the other;
// a result array that has just been allocated adds a page fault every 4 KB. Here a few threads each
// take a part of the copy and move it through two pinned slots of their own, so that host copies, page
// faults and the bus overlap. Pinned memory of the caller's goes straight to the bus. The slots of a
// device are shared by all handles of the process that use it and freed with the last of them; a copy
// that finds them taken by another thread's goes the driver's way.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <exception>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace autan_b200 {

class HostStage {
 public:
  // The slots of the current device in one direction (0 to the device, 1 to the host: each its own,
  // so that a copy in and a copy out can run beside each other).
  static std::shared_ptr<HostStage> of_device(int direction) {
    static std::mutex guard;
    static std::map<int, std::weak_ptr<HostStage>> all;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lock(guard);
    std::weak_ptr<HostStage>& slot = all[2 * device + direction];
    std::shared_ptr<HostStage> p = slot.lock();
    if (!p) {
      p.reset(new HostStage(device));
      slot = p;
    }
    return p;
  }

  ~HostStage() {
    int was = -1;
    const bool moved = cudaGetDevice(&was) == cudaSuccess && was != device_;
    if (moved) cudaSetDevice(device_);
    for (Slot& s : slots_) {
      if (s.done != nullptr) {
        cudaEventSynchronize(s.done);
        cudaEventDestroy(s.done);
      }
      if (s.p != nullptr) cudaFreeHost(s.p);
    }
    if (moved) cudaSetDevice(was);
  }
  HostStage(const HostStage&) = delete;
  HostStage& operator=(const HostStage&) = delete;

  // dst (device) = src (host), ordered on `stream`; src has been read when it returns, unless it is
  // pinned (then, as cudaMemcpyAsync, when the stream gets there).
  // may_pin: whether the slots may be allocated for this copy where they are not yet (a few
  // milliseconds: callers that copy once go the driver's way).
  cudaError_t to_device(void* dst, const void* src, size_t bytes, cudaStream_t stream, bool may_pin) {
    return copy(static_cast<char*>(dst), static_cast<const char*>(src), bytes, stream, true, may_pin);
  }
  // dst (host) = src (device), after what `stream` holds; dst holds the data when it returns, unless it
  // is pinned (then when the stream has been waited for).
  cudaError_t to_host(void* dst, const void* src, size_t bytes, cudaStream_t stream, bool may_pin) {
    return copy(static_cast<char*>(dst), static_cast<const char*>(src), bytes, stream, false, may_pin);
  }

  static bool pinned(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
    return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeManaged;
  }

 private:
  static constexpr int kLanes = 4;
  static constexpr size_t kSlot = size_t(1) << 19;
  // below this the driver's own staging is as fast
  static constexpr size_t kLeast = size_t(1) << 20;

  struct Slot {
    void* p = nullptr;
    cudaEvent_t done = nullptr;
  };

  explicit HostStage(int device) : device_(device) {}

  cudaError_t ready() {
    for (Slot& s : slots_) {
      if (s.p == nullptr) {
        const cudaError_t e = cudaHostAlloc(&s.p, kSlot, cudaHostAllocDefault);
        if (e != cudaSuccess) return e;
      }
      if (s.done == nullptr) {
        const cudaError_t e = cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming);
        if (e != cudaSuccess) return e;
      }
    }
    return cudaSuccess;
  }

  cudaError_t direct(char* dst, const char* src, size_t bytes, cudaStream_t stream, bool in) {
    return cudaMemcpyAsync(dst, src, bytes, in ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, stream);
  }

  cudaError_t copy(char* dst, const char* src, size_t bytes, cudaStream_t stream, bool in, bool may_pin) {
    std::unique_lock<std::mutex> lock(busy_, std::try_to_lock);
    if (bytes < kLeast || !lock.owns_lock() || pinned(in ? static_cast<const void*>(src) : dst))
      return direct(dst, src, bytes, stream, in);
    if (slots_[2 * kLanes - 1].done == nullptr && !may_pin) return direct(dst, src, bytes, stream, in);
    if (ready() != cudaSuccess) {  // no pinned memory to be had
      (void)cudaGetLastError();
      return direct(dst, src, bytes, stream, in);
    }
    const int lanes = static_cast<int>(std::min<size_t>(kLanes, bytes / kSlot));
    const size_t part = (bytes / lanes + 4095) / 4096 * 4096;
    cudaError_t result[kLanes] = {};
    auto lane = [&](int l) {
      const size_t a = std::min(bytes, part * static_cast<size_t>(l));
      const size_t b = l == lanes - 1 ? bytes : std::min(bytes, a + part);
      result[l] = in ? in_lane(l, dst + a, src + a, b - a, stream) : out_lane(l, dst + a, src + a, b - a, stream);
    };
    std::vector<std::thread> team;
    int begun = 1;
    try {
      for (; begun < lanes; ++begun)
        team.emplace_back([&, l = begun] {
          result[l] = cudaSetDevice(device_);
          if (result[l] == cudaSuccess) lane(l);
        });
    } catch (const std::exception&) {
      // no thread to be had: the remaining parts follow on this one
    }
    lane(0);
    for (int l = begun; l < lanes; ++l) lane(l);
    for (std::thread& t : team) t.join();
    for (int l = 0; l < lanes; ++l)
      if (result[l] != cudaSuccess) return result[l];
    return cudaSuccess;
  }

  cudaError_t in_lane(int l, char* dst, const char* src, size_t bytes, cudaStream_t stream) {
    for (size_t at = 0, k = 0; at < bytes; at += kSlot, ++k) {
      Slot& s = slots_[2 * l + (k & 1)];
      const size_t n = std::min(kSlot, bytes - at);
      cudaError_t e = cudaEventSynchronize(s.done);  // the slot's last copy has left it
      if (e != cudaSuccess) return e;
      std::memcpy(s.p, src + at, n);
      e = cudaMemcpyAsync(dst + at, s.p, n, cudaMemcpyHostToDevice, stream);
      if (e == cudaSuccess) e = cudaEventRecord(s.done, stream);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }

  cudaError_t out_lane(int l, char* dst, const char* src, size_t bytes, cudaStream_t stream) {
    auto fetch = [&](size_t at, size_t k) {
      Slot& s = slots_[2 * l + (k & 1)];
      cudaError_t e = cudaMemcpyAsync(s.p, src + at, std::min(kSlot, bytes - at), cudaMemcpyDeviceToHost, stream);
      return e == cudaSuccess ? cudaEventRecord(s.done, stream) : e;
    };
    cudaError_t e = bytes > 0 ? fetch(0, 0) : cudaSuccess;
    for (size_t at = 0, k = 0; at < bytes && e == cudaSuccess; at += kSlot, ++k) {
      if (at + kSlot < bytes) e = fetch(at + kSlot, k + 1);
      if (e != cudaSuccess) break;
      Slot& s = slots_[2 * l + (k & 1)];
      e = cudaEventSynchronize(s.done);
      if (e == cudaSuccess) std::memcpy(dst + at, s.p, std::min(kSlot, bytes - at));
    }
    return e;
  }

  const int device_;
  std::mutex busy_;
  Slot slots_[2 * kLanes];
};

// Pinned memory of one handle's, got on first use; where none is to be had it stays without.
class HostRows {
 public:
  HostRows() = default;
  HostRows(const HostRows&) = delete;
  HostRows& operator=(const HostRows&) = delete;
  ~HostRows() {
    if (p_ != nullptr) cudaFreeHost(p_);
  }
  bool held() const { return p_ != nullptr; }
  // `bytes` (the same at every call) of it, or null.
  void* get(size_t bytes) {
    if (p_ == nullptr && !refused_ && cudaMallocHost(&p_, bytes) != cudaSuccess) {
      (void)cudaGetLastError();
      p_ = nullptr;
      refused_ = true;
    }
    return p_;
  }

 private:
  void* p_ = nullptr;
  bool refused_ = false;
};

}  // namespace autan_b200
