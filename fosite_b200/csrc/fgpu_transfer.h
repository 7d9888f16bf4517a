// fgpu_transfer.h -- copies between the device and a caller's pageable host arrays.
//
// cudaMemcpyAsync on pageable memory goes through one staging buffer of the driver on one host
// core: 4.8 GB/s into fresh pages (703 MB of a 256^3 state: 150 ms, thirteen of its steps).  Here up
// to kLanes host threads, each with its own pinned slot and stream, move interleaved pieces: one
// piece is on the bus while others are copied between pinned and pageable memory (whose page faults
// are what a core spends its time on).  The lanes (4 MiB of pinned memory each) are shared by all
// handles of the process: made at the first large transfer, used by one transfer at a time, freed
// with the last handle.  Transfers below kSmallDown / kSmallUp, pinned host memory, and calls that
// find the lanes in use or cannot make them take the driver's path.  Thresholds (16 host cores, driver
// / lanes): downloads 1.1 MB 0.27 / 0.13 ms, 8.5 MB 1.2 / 0.43, 67 MB 14.3 / 3.6; uploads, whose pages
// exist already, 4.3 MB 0.31 / 0.37 ms, 8.5 MB 0.61 / 0.60, 34 MB 2.9 / 1.2.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace fgpu {

class Transfer {
 public:
  static constexpr size_t kPiece = size_t(4) << 20, kLeast = size_t(256) << 10;
  static constexpr size_t kSmallDown = size_t(1) << 20, kSmallUp = size_t(8) << 20;
  static constexpr int kLanes = 8;

  static Transfer& shared() {
    static Transfer* t = new Transfer;   // (never destroyed: no CUDA calls at process exit)
    return *t;
  }
  // handles alive; the lanes go with the last
  void attach() {
    std::lock_guard<std::mutex> lock(mutex_);
    ++handles_;
  }
  void detach() {
    std::lock_guard<std::mutex> lock(mutex_);
    if (--handles_ == 0) release();
  }
  // bytes between device memory (ready in stream order of s) and host memory; returns when the copy
  // is complete.  to_host: device to host, else host to device (later work of s sees it).
  cudaError_t copy(void* host, void* dev, size_t bytes, bool to_host, int device, cudaStream_t s) {
    const cudaMemcpyKind kind = to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
    std::unique_lock<std::mutex> lock(mutex_, std::defer_lock);
    if (bytes >= (to_host ? kSmallDown : kSmallUp) && !pinned(host)) (void)lock.try_lock();
    const OnDevice on(lock.owns_lock() ? device : -1);
    if (!lock.owns_lock() || !prepare(device)) {
      cudaError_t e = cudaMemcpyAsync(to_host ? host : dev, to_host ? dev : host, bytes, kind, s);
      return e != cudaSuccess ? e : cudaStreamSynchronize(s);
    }
    cudaError_t e = cudaEventRecord(ready_, s);   // the lanes start after the work enqueued on s
    if (e != cudaSuccess) return e;
    // two pieces a lane or more
    const size_t piece = std::min(kPiece, std::max(kLeast, (bytes / (2 * lanes_.size()) + 4095) / 4096 * 4096));
    const size_t pieces = (bytes + piece - 1) / piece;
    const int n = (int)std::min<size_t>(lanes_.size(), pieces);
    std::vector<cudaError_t> err(n, cudaSuccess);
    const cudaStreamCaptureMode capture = capture_mode();
    auto work = [&](int t) {
      Lane& L = lanes_[t];
      cudaStreamCaptureMode mode = capture;   // the lane's threads wait under the caller's rules
      cudaError_t r = cudaThreadExchangeStreamCaptureMode(&mode);
      if (r == cudaSuccess) r = cudaSetDevice(device);
      if (r == cudaSuccess) r = cudaStreamWaitEvent(L.stream, ready_, 0);
      for (size_t p = t; p < pieces && r == cudaSuccess; p += n) {
        const size_t o = p * piece, m = std::min(piece, bytes - o);
        char *h = static_cast<char*>(host) + o, *d = static_cast<char*>(dev) + o;
        if (!to_host) std::memcpy(L.slot, h, m);
        r = cudaMemcpyAsync(to_host ? L.slot : d, to_host ? d : L.slot, m, kind, L.stream);
        if (r == cudaSuccess) r = cudaStreamSynchronize(L.stream);
        if (r == cudaSuccess && to_host) std::memcpy(h, L.slot, m);
      }
      err[t] = r;
    };
    std::vector<std::thread> threads;
    threads.reserve(n);
    int started = 1;
    try {
      for (; started < n; ++started) threads.emplace_back(work, started);
    } catch (...) {   // no more threads: this one takes the remaining lanes' pieces
    }
    work(0);
    for (int t = started; t < n; ++t) work(t);
    for (auto& t : threads) t.join();
    for (cudaError_t r : err)
      if (r != cudaSuccess) return r;
    return cudaSuccess;
  }

 private:
  struct Lane { char* slot; cudaStream_t stream; };
  struct OnDevice {   // the calling thread's device for the length of a transfer
    int before = -1;
    explicit OnDevice(int device) {
      if (device >= 0 && cudaGetDevice(&before) == cudaSuccess && before != device) cudaSetDevice(device);
    }
    ~OnDevice() {
      if (before >= 0) cudaSetDevice(before);
    }
  };
  std::mutex mutex_;
  std::vector<Lane> lanes_;
  cudaEvent_t ready_ = nullptr;
  int device_ = -1;
  long long handles_ = 0;

  static bool pinned(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
  }
  // What the calling thread may do while another thread captures a stream: a program that captures
  // graphs of its own (in the global mode, whose captures a wait on any stream breaks) transfers from a
  // thread that has switched itself to the relaxed mode.
  static cudaStreamCaptureMode capture_mode() {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return cudaStreamCaptureModeGlobal;
    const cudaStreamCaptureMode callers = mode;
    cudaThreadExchangeStreamCaptureMode(&mode);
    return callers;
  }
  // lanes on this device (the last device's are given back first)
  bool prepare(int device) {
    if (device_ == device && !lanes_.empty()) return true;
    release();
    if (cudaEventCreateWithFlags(&ready_, cudaEventDisableTiming) != cudaSuccess) {
      ready_ = nullptr;
      cudaGetLastError();
      return false;
    }
    device_ = device;
    const int want = std::max(1, std::min<int>(kLanes, (int)std::thread::hardware_concurrency() / 2));
    for (int t = 0; t < want; ++t) {
      Lane L;
      if (cudaMallocHost(reinterpret_cast<void**>(&L.slot), kPiece) != cudaSuccess) break;
      if (cudaStreamCreateWithFlags(&L.stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaFreeHost(L.slot);
        break;
      }
      lanes_.push_back(L);
    }
    cudaGetLastError();
    if (lanes_.empty()) release();
    return !lanes_.empty();
  }
  void release() {
    for (Lane& L : lanes_) {
      cudaStreamDestroy(L.stream);
      cudaFreeHost(L.slot);
    }
    lanes_.clear();
    if (ready_) cudaEventDestroy(ready_);
    ready_ = nullptr;
    device_ = -1;
  }
};

}  // namespace fgpu
