"""The pinned lanes of large transfers (fosite_b200/csrc/fgpu_transfer.h) on the host: the header compiled
against a stand-in for the CUDA runtime that copies with memcpy and counts what it is asked for."""
import ctypes as C
import mmap
import os
import shutil
import subprocess
import tempfile
import threading
import time

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fosite_b200", "csrc")

RUNTIME = r'''
#pragma once
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <thread>
typedef int cudaError_t;
typedef struct Stream { int device; unsigned long long context; } *cudaStream_t;
typedef struct Event { int device; unsigned long long context; } *cudaEvent_t;
enum { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorInvalidResourceHandle = 400 };
enum { cudaStreamNonBlocking = 1, cudaEventDisableTiming = 2, cudaMemoryTypeUnregistered = 0 };
enum { cudaEnableDefault = 0 };
enum cudaDriverEntryPointQueryResult { cudaDriverEntryPointSuccess };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum cudaStreamCaptureMode { cudaStreamCaptureModeGlobal, cudaStreamCaptureModeThreadLocal, cudaStreamCaptureModeRelaxed };
struct cudaPointerAttributes { int type; };
namespace fake {
inline std::atomic<long long> pins{0}, frees{0}, bytes{0}, streams{0}, destroyed{0}, copies{0}, waits{0};
inline std::atomic<long long> piece{0};   // of the largest copy
inline std::atomic<int> held{0};          // copies wait while it is set
inline thread_local int device = 0;
inline thread_local cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
inline std::atomic<unsigned long long> context[32];   // of each device; a reset makes another
inline std::atomic<long long> stale{0};                 // uses of what went with a context
inline unsigned long long now() { return 100 * device + context[device]; }
struct Head { size_t n; unsigned long long context; int device; char pad[44]; };
}  // namespace fake
inline cudaError_t cudaGetLastError() { return 0; }
inline cudaError_t cudaSetDevice(int d) { fake::device = d; return 0; }
inline cudaError_t cudaGetDevice(int* d) { *d = fake::device; return 0; }
inline cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
  const cudaStreamCaptureMode old = fake::mode;
  fake::mode = *m;
  *m = old;
  return 0;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = 0; return 0; }
inline cudaError_t cudaMallocHost(void** p, size_t n) {
  fake::Head* h = static_cast<fake::Head*>(std::malloc(sizeof(fake::Head) + n));
  h->n = n;
  h->context = fake::now();
  h->device = fake::device;
  *p = h + 1;
  ++fake::pins;
  fake::bytes += n;
  return 0;
}
inline cudaError_t cudaFreeHost(void* p) {
  fake::Head* h = static_cast<fake::Head*>(p) - 1;
  fake::stale += h->context != 100 * h->device + fake::context[h->device];
  fake::bytes -= h->n;
  ++fake::frees;
  std::free(h);
  return 0;
}
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, int) { ++fake::streams; *s = new Stream{fake::device, fake::now()}; return 0; }
template <class T>
void used(T* h) { fake::stale += h && h->context != 100 * h->device + fake::context[h->device]; }
inline cudaError_t cudaStreamDestroy(cudaStream_t s) { used(s); ++fake::destroyed; delete s; return 0; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) { *e = new Event{fake::device, fake::now()}; return 0; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { used(e); delete e; return 0; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { used(e); return 0; }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, int) { used(s); used(e); return 0; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) { used(s); ++fake::waits; return 0; }
inline int context_id(void*, unsigned long long* id) { *id = fake::now(); return 0; }
inline int context_state(int d, unsigned*, int* active) { *active = fake::context[d] % 2 == 0; return 0; }
inline cudaError_t cudaGetDriverEntryPoint(const char* name, void** p, unsigned long long, cudaDriverEntryPointQueryResult*) {
  *p = std::strcmp(name, "cuCtxGetId") == 0 ? reinterpret_cast<void*>(context_id) : reinterpret_cast<void*>(context_state);
  return 0;
}
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t stream) {
  used(stream);
  if (stream && stream->device != fake::device) return cudaErrorInvalidResourceHandle;
  std::memcpy(d, s, n);
  ++fake::copies;
  while (fake::held) std::this_thread::yield();
  long long m = fake::piece;
  while (m < (long long)n && !fake::piece.compare_exchange_weak(m, (long long)n)) {}
  return 0;
}
'''

SRC = r'''
#include <new>
#include "fgpu_transfer.h"
using fgpu::Transfer;
static std::atomic<int> starved{0};
void* operator new(size_t n) {
  void* p = starved ? nullptr : std::malloc(n);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
extern "C" {
void* make() { return new Transfer; }
void attach(void* t) { static_cast<Transfer*>(t)->attach(); }
void detach(void* t) { static_cast<Transfer*>(t)->detach(); }
int copy(void* t, void* host, void* dev, size_t n, int to_host, int device) {
  try {
    return static_cast<Transfer*>(t)->copy(host, dev, n, to_host != 0, device, nullptr);
  } catch (...) {
    return -1;
  }
}
void starve(int on) { starved = on; }
// a device's context goes (odd: none yet), or another one comes
void reset(int device) { ++fake::context[device]; }
void hold(int on) { fake::held = on; }
long long count(int what) {
  std::atomic<long long>* c[] = {&fake::pins, &fake::frees, &fake::bytes, &fake::streams, &fake::destroyed,
                                 &fake::copies, &fake::waits, &fake::piece, &fake::stale};
  return *c[what];
}
}
'''
PINS, FREES, PINNED, STREAMS, DESTROYED, COPIES, WAITS, PIECE, STALE = range(9)
MB = 1 << 20


@pytest.fixture(scope="module")
def lib():
    d = tempfile.mkdtemp()
    for name, text in (("cuda_runtime.h", RUNTIME), ("t.cpp", SRC)):
        with open(os.path.join(d, name), "w") as f:
            f.write(text)
    out = os.path.join(d, "libt.so")
    subprocess.check_call([shutil.which("g++") or "g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-pthread", "-Wl,-Bsymbolic", "-I", d, "-I", CSRC,
                           "-o", out, os.path.join(d, "t.cpp")])
    L = C.CDLL(out)
    L.make.restype = C.c_void_p
    L.count.restype = C.c_longlong
    return L


class _Lanes:
    """A Transfer of its own, with the counts since it was made"""

    def __init__(self, lib):
        self.L, self.t = lib, C.c_void_p(lib.make())
        self.start = [lib.count(q) for q in range(9)]

    def count(self, what):
        return self.L.count(what) - self.start[what]

    def attach(self):
        self.L.attach(self.t)

    def detach(self):
        self.L.detach(self.t)

    def copy(self, n, to_host=True, device=0, resident=False):
        """Moves n bytes, each checked, into pages that do not exist yet or (resident) into existing ones"""
        src = np.frombuffer(np.random.default_rng(n).bytes(n), np.uint8)
        dst = np.frombuffer(mmap.mmap(-1, n, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS), np.uint8)
        if resident:
            dst[:] = 0
        host, dev = (dst, src) if to_host else (src, dst)
        rc = self.L.copy(self.t, host.ctypes.data_as(C.c_void_p), dev.ctypes.data_as(C.c_void_p), C.c_size_t(n),
                         C.c_int(to_host), C.c_int(device))
        assert np.array_equal(src, dst)
        return rc


@pytest.mark.parametrize("n", [1 * MB, 1 * MB + 1, 3 * MB - 7, 9 * MB + 13, 70 * MB + 5])
@pytest.mark.parametrize("to_host", [True, False])
def test_every_byte_moves(lib, n, to_host):
    t = _Lanes(lib)
    t.attach()
    assert t.copy(n, to_host) == 0
    t.detach()


def test_lanes_outlive_the_handles_that_use_them(lib):
    """One grid after another, each closed before the next is opened: the slots are pinned once."""
    t = _Lanes(lib)
    for _ in range(5):
        t.attach()
        assert t.copy(2 * MB) == 0 and t.copy(MB + 64) == 0
        t.detach()
    assert t.count(PINS) == 1 and t.count(FREES) == 0 and t.count(STREAMS) <= 8


def test_lanes_are_given_back(lib):
    """A last handle that goes after no transfer used the lanes takes them along."""
    t = _Lanes(lib)
    t.attach()
    t.copy(40 * MB)
    t.detach()
    assert t.count(PINNED) > 0
    t.attach()
    t.copy(MB // 2)
    t.detach()
    assert t.count(PINNED) == 0 and t.count(STREAMS) == t.count(DESTROYED)
    t.attach()
    assert t.copy(2 * MB) == 0
    t.detach()


def test_slots_grow_with_the_transfers(lib):
    """Small grids pin little: a slot holds what has been asked of it, 4 MiB at most."""
    t = _Lanes(lib)
    t.attach()
    t.copy(2 * MB)
    lanes = t.count(STREAMS)
    assert t.count(PINNED) == lanes * MB // 4
    t.copy(200 * MB)
    assert t.count(PINNED) == lanes * 4 * MB and t.count(PINS) == 2
    t.copy(2 * MB)
    assert t.count(PINNED) == lanes * 4 * MB and t.count(PINS) == 2
    t.detach()


def test_devices_in_turn(lib):
    """Handles on several devices that transfer in turn: the lanes of each device are made once, and
    every piece goes through a stream of its device."""
    t = _Lanes(lib)
    t.attach()
    t.copy(2 * MB, device=0)
    lanes = t.count(STREAMS)
    for device in (0, 1, 2, 1, 0, 2):
        assert t.copy(2 * MB, device=device) == 0
    assert t.count(PINS) == 3 and t.count(STREAMS) == 3 * lanes and t.count(FREES) == t.count(DESTROYED) == 0
    for device in range(3, 20):   # more devices than have room: the driver's path
        assert t.copy(2 * MB, device=device) == 0
    assert t.count(STREAMS) <= 16 * lanes
    t.detach()


def test_handles_come_and_go_during_a_transfer(lib):
    """Creating and closing a handle does not wait for another thread's transfer."""
    t = _Lanes(lib)
    t.attach()
    lib.hold(1)
    rc, done = [], threading.Event()
    mover = threading.Thread(target=lambda: rc.append(t.copy(3 * MB)))
    other = threading.Thread(target=lambda: (t.attach(), t.detach(), done.set()))
    try:
        mover.start()
        while t.count(COPIES) == 0:
            time.sleep(0.001)
        other.start()
        assert done.wait(20)
    finally:
        lib.hold(0)
        mover.join()
        other.join()
    assert rc == [0]
    t.detach()


@pytest.mark.parametrize("to_host", [True, False])
def test_no_memory_for_threads(lib, to_host):
    """A transfer that can start no threads moves every piece itself; no exception reaches the C entry."""
    t = _Lanes(lib)
    t.attach()
    assert t.copy(9 * MB, to_host) == 0
    lib.starve(1)
    try:
        rc = t.copy(9 * MB, to_host)
    finally:
        lib.starve(0)
    assert rc == 0
    t.detach()


def test_small_uploads_are_enqueued(lib):
    """A small upload does not wait for its stream (its caller does, after the kernel that unpacks it); a
    download does."""
    t = _Lanes(lib)
    t.attach()
    assert t.copy(4096, to_host=False) == 0 and t.count(WAITS) == 0
    assert t.copy(4096, to_host=True) == 0 and t.count(WAITS) == 1
    t.detach()


@pytest.mark.parametrize("n,resident,lanes", [(MB - 8, False, False), (MB, False, True), (MB, True, False), (9 * MB, True, False),
                                              (10 * MB, True, True), (10 * MB, False, True)])
def test_downloads_by_their_pages(lib, n, resident, lanes):
    """Lanes for pages that have to be made; one core's copy into pages that exist is as fast up to 10 MB."""
    t = _Lanes(lib)
    t.attach()
    assert t.copy(n, resident=resident) == 0
    assert (t.count(STREAMS) > 0) == lanes
    t.detach()


@pytest.mark.parametrize("n,lanes", [(8 * MB - 8, False), (8 * MB, True)])
def test_uploads_by_their_size(lib, n, lanes):
    t = _Lanes(lib)
    t.attach()
    assert t.copy(n, to_host=False) == 0
    assert (t.count(STREAMS) > 0) == lanes
    t.detach()


@pytest.mark.parametrize("name", ["libfosite_gpu.so", "libfosite_gpu_exact.so"])
def test_the_lanes_are_internal_to_a_library(name):
    """Both builds in one process keep their own lanes: the object is not a unique symbol, which the dynamic
    linker shares between all libraries that define it, of whatever version."""
    path = os.path.join(os.path.dirname(CSRC), "lib", name)
    if not os.path.exists(path) or not shutil.which("nm"):
        pytest.skip("no library or no nm here")
    names = subprocess.run(["nm", "-D", "--defined-only", path], check=True, capture_output=True, text=True).stdout
    assert "fgpu_create" in names
    assert not [n for n in names.splitlines() if " u " in n and "Transfer" in n]


def test_a_context_that_was_reset(lib):
    """A program that resets the device between two grids: nothing that went with the old context is used or
    freed, neither by the next transfer nor when the lanes are given back."""
    t = _Lanes(lib)
    t.attach()
    assert t.copy(2 * MB) == 0 and t.copy(2 * MB, device=1) == 0
    t.detach()
    lib.reset(0)
    lib.reset(0)
    t.attach()
    assert t.copy(3 * MB) == 0 and t.count(PINS) == 3
    t.detach()
    lib.reset(1)      # gone, and no other one yet
    t.attach()
    t.detach()        # the idle handle takes the living context's lanes along
    assert t.count(FREES) == 1 and t.count(STALE) == 0
    lib.reset(1)
    t.attach()
    assert t.copy(2 * MB, device=1) == 0 and t.count(STALE) == 0
    t.detach()
