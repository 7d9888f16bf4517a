// fgpu_transfer.h -- copies between the device and a caller's pageable host arrays.
//
// cudaMemcpyAsync on pageable memory goes through one staging buffer of the driver on one host
// core: 2 to 5 GB/s into fresh pages (703 MB of a 256^3 state: 150 to 340 ms).  Here up
// to kLanes host threads, each with its own pinned slot and stream, move interleaved pieces: one
// piece is on the bus while others are copied between pinned and pageable memory (whose page faults
// are what a core spends its time on).  The lanes are shared by all handles of the process, used by
// one transfer at a time, and made at the first large transfer: pinning their slots is what they
// cost (2 MiB in all 2 ms, 32 MiB 18 ms; freeing them 4 ms), so a slot holds the pieces asked
// of it so far (256 KiB for transfers up to 4 MiB, 4 MiB from 32 MiB on), and the lanes outlive the
// handles: a program that opens, reads and closes one grid after another keeps them (freed with every
// last handle they cost 35 ms a 256^2 grid).  Each device has lanes of its own, so that handles on two
// devices transfer in turn as those of one; they belong to its context, and go unused once a program has
// reset that between two grids.  The lanes are given back when the last handle goes and no transfer
// has used them since the previous time that it went; at most 32 MiB and eight streams a device stay.
// Pinned host memory, transfers below the thresholds, and calls that find the lanes in use or cannot
// make them (devices past the kDevices-th too) take the driver's path.  Thresholds, by what bounds
// the driver's one core (16 host cores, ms, driver / lanes):
//   * downloads into pages that do not exist yet, its page faults: 0.5 MB 0.25 / 0.22, 1.1 MB 0.54 / 0.21,
//     8.3 MB 4.0 / 1.0, 110 MB 52 / 9.5;
//   * downloads into resident pages (an allocator that reuses memory, or the caller's own array), its copy:
//     2.2 MB 0.15 / 0.31, 5.5 MB 0.35 / 0.56, 12.6 MB 0.67 / 0.59 (one download after another; after
//     another core's use 0.68 / 0.79, 34 MB 1.8 / 1.4); the lanes leave the array in their cores'
//     caches, and its next reader pays for that (2.2 MB 0.11 / 0.32, 34 MB 1.7 / 2.0);
//   * uploads: 4.2 MB 0.24 / 0.29, 8.3 MB 0.46 / 0.43, 34 MB 3.0 / 1.2.
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>

namespace fgpu {

class Transfer {
 public:
  static constexpr size_t kPiece = size_t(4) << 20, kLeast = size_t(256) << 10;
  static constexpr size_t kFreshDown = size_t(1) << 20, kDown = size_t(10) << 20, kUp = size_t(8) << 20;
  static constexpr int kLanes = 8, kDevices = 16;

  // Handles alive.  Neither waits for a transfer: one in flight belongs to a handle that is alive, so
  // that the lanes are not due.
  void attach() { ++handles_; }
  void detach() {
    if (--handles_ != 0) return;
    std::unique_lock<std::mutex> lock(mutex_, std::try_to_lock);
    if (!lock.owns_lock() || handles_ != 0) return;
    if (!used_) release();
    used_ = false;
  }
  // bytes between device memory (ready in stream order of s) and host memory.  to_host: device to
  // host, complete on return; else host to device: later work of s sees it, and the host array is
  // read until s has been waited for.  Its callers are C entries: nothing here throws.
  cudaError_t copy(void* host, void* dev, size_t bytes, bool to_host, int device, cudaStream_t s) {
    const cudaMemcpyKind kind = to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
    std::unique_lock<std::mutex> lock(mutex_, std::defer_lock);
    const bool lanes = !to_host ? bytes >= kUp : bytes >= kDown || (bytes >= kFreshDown && fresh(host, bytes));
    if (lanes && !pinned(host)) (void)lock.try_lock();
    const OnDevice on(lock.owns_lock() ? device : -1);
    Device* const D = lock.owns_lock() ? prepare(device, bytes) : nullptr;
    if (!D) {
      cudaError_t e = cudaMemcpyAsync(to_host ? host : dev, to_host ? dev : host, bytes, kind, s);
      return e != cudaSuccess || !to_host ? e : cudaStreamSynchronize(s);
    }
    used_ = true;
    cudaError_t e = cudaEventRecord(D->ready, s);   // the lanes start after the work enqueued on s
    if (e != cudaSuccess) return e;
    const size_t piece = std::min(D->slot_bytes, piece_bytes(bytes, D->lanes));
    const size_t pieces = (bytes + piece - 1) / piece;
    const int n = (int)std::min<size_t>(D->lanes, pieces);
    cudaError_t err[kLanes] = {};
    const cudaStreamCaptureMode capture = capture_mode();
    auto work = [&](int t) {
      const cudaStream_t stream = D->stream[t];
      char* const slot = D->slots + t * D->slot_bytes;
      cudaStreamCaptureMode mode = capture;   // the lane's threads wait under the caller's rules
      cudaError_t r = cudaThreadExchangeStreamCaptureMode(&mode);
      if (r == cudaSuccess) r = cudaSetDevice(device);
      if (r == cudaSuccess) r = cudaStreamWaitEvent(stream, D->ready, 0);
      for (size_t p = t; p < pieces && r == cudaSuccess; p += n) {
        const size_t o = p * piece, m = std::min(piece, bytes - o);
        char *h = static_cast<char*>(host) + o, *d = static_cast<char*>(dev) + o;
        if (!to_host) std::memcpy(slot, h, m);
        r = cudaMemcpyAsync(to_host ? slot : d, to_host ? d : slot, m, kind, stream);
        if (r == cudaSuccess) r = cudaStreamSynchronize(stream);
        if (r == cudaSuccess && to_host) std::memcpy(h, slot, m);
      }
      err[t] = r;
    };
    std::thread threads[kLanes];
    int started = 1;
    try {
      for (; started < n; ++started) threads[started] = std::thread(work, started);
    } catch (...) {   // no more threads (or no memory for them): this one takes the remaining lanes' pieces
    }
    work(0);
    for (int t = started; t < n; ++t) work(t);
    for (int t = 1; t < started; ++t) threads[t].join();
    for (cudaError_t r : err)
      if (r != cudaSuccess) return r;
    return cudaSuccess;
  }

 private:
  struct Device {
    int id = -1, lanes = 0;
    unsigned long long context = 0;   // what the rest belongs to
    char* slots = nullptr;            // one pinned block, a slot of slot_bytes per lane
    size_t slot_bytes = 0;
    cudaStream_t stream[kLanes] = {};
    cudaEvent_t ready = nullptr;
  };
  // two pieces a lane or more
  static size_t piece_bytes(size_t bytes, size_t lanes) {
    return std::min(kPiece, std::max(kLeast, (bytes / (2 * lanes) + 4095) / 4096 * 4096));
  }
  struct OnDevice {   // the calling thread's device for the length of a transfer
    int before = -1;
    explicit OnDevice(int device) {
      if (device >= 0 && cudaGetDevice(&before) == cudaSuccess) cudaSetDevice(device);   // (makes its context current)
    }
    ~OnDevice() {
      if (before >= 0) cudaSetDevice(before);
    }
  };
  std::mutex mutex_;
  Device devices_[kDevices];   // those with lanes first
  std::atomic<long long> handles_{0};
  bool used_ = false;          // since the last handle last went

  // whether most of a host array's pages do not exist yet (sixteen of them are looked at)
  static bool fresh(const void* host, size_t bytes) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), first = reinterpret_cast<size_t>(host);
    int absent = 0;
    for (size_t q = 0; q < 16; ++q) {
      unsigned char resident = 1;
      const size_t at = (first + bytes / 32 * (2 * q + 1)) / page * page;
      if (mincore(reinterpret_cast<void*>(at), page, &resident) == 0 && !(resident & 1)) ++absent;
    }
    return absent > 8;
  }
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
  // Driver calls: the identity of the current context (never used twice in a process), and whether a
  // device's context exists (cudaSetDevice would make one).
  int (*get_id_)(void*, unsigned long long*) = nullptr;
  int (*get_state_)(int, unsigned*, int*) = nullptr;
  unsigned long long current_context() {
    if (!get_id_) get_id_ = reinterpret_cast<int (*)(void*, unsigned long long*)>(driver_call("cuCtxGetId"));
    unsigned long long id = 0;
    return get_id_ && get_id_(nullptr, &id) == 0 ? id : 0;
  }
  bool has_context(int device) {
    if (!get_state_) get_state_ = reinterpret_cast<int (*)(int, unsigned*, int*)>(driver_call("cuDevicePrimaryCtxGetState"));
    unsigned flags = 0;
    int active = 1;
    return !get_state_ || get_state_(device, &flags, &active) != 0 || active != 0;
  }
  static void* driver_call(const char* name) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &found) != cudaSuccess) cudaGetLastError();
    return p;
  }
  // the lanes of the current device and context with slots for pieces of a transfer of `bytes`, or
  // smaller slots where no larger ones are to be had
  Device* prepare(int device, size_t bytes) {
    const unsigned long long context = current_context();
    Device* D = devices_;
    while (D < devices_ + kDevices && D->id >= 0 && (D->id != device || D->context != context)) ++D;
    if (D == devices_ + kDevices) return nullptr;
    if (D->id < 0) {
      const int want = std::max(1, std::min<int>(kLanes, (int)std::thread::hardware_concurrency() / 2));
      if (cudaEventCreateWithFlags(&D->ready, cudaEventDisableTiming) != cudaSuccess) D->ready = nullptr;
      while (D->ready && D->lanes < want &&
             cudaStreamCreateWithFlags(&D->stream[D->lanes], cudaStreamNonBlocking) == cudaSuccess)
        ++D->lanes;
      if (D->lanes) {
        D->id = device;
        D->context = context;
      } else {
        free_lanes(*D);
        *D = Device();
      }
    }
    if (D->lanes) reserve(*D, piece_bytes(bytes, D->lanes));
    cudaGetLastError();
    return D->slots ? D : nullptr;
  }
  static void reserve(Device& D, size_t piece) {
    size_t want = kLeast;
    while (want < piece) want *= 2;
    char* block = nullptr;
    if (want <= D.slot_bytes || cudaMallocHost(reinterpret_cast<void**>(&block), want * D.lanes) != cudaSuccess) return;
    if (D.slots) cudaFreeHost(D.slots);
    D.slots = block;
    D.slot_bytes = want;
  }
  static void free_lanes(Device& D) {
    for (int t = 0; t < D.lanes; ++t) cudaStreamDestroy(D.stream[t]);
    if (D.ready) cudaEventDestroy(D.ready);
    if (D.slots) cudaFreeHost(D.slots);
  }
  // gives the lanes back; those of a context that is gone went with it
  void release() {
    for (Device& D : devices_) {
      if (D.id >= 0 && has_context(D.id)) {
        const OnDevice on(D.id);
        if (current_context() == D.context) free_lanes(D);
        cudaGetLastError();
      }
      D = Device();
    }
  }
};

}  // namespace fgpu
