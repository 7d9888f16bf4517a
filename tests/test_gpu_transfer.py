"""State transfers: the pinned lanes of large pageable arrays, the driver's path of small and pinned
ones, and transfers of several threads at once give back what was uploaded, byte for byte."""
import threading

import numpy as np
import pytest

from fosite_b200 import abi
from cases import _gauss3d, _khi


def _sim(case):
    from fosite_b200.sim import Simulation
    cfg, p, _ = case
    s = Simulation(cfg)
    c = np.random.default_rng(cfg.inum).uniform(1.0, 2.0, (s.vnum,) + s.shape)
    c[-1] += 10.0
    return s, c


def _interior(a, cfg):
    return a[:, 2:-2, 2:-2, 2:-2] if cfg.knum > 1 else a[:, :, 2:-2, 2:-2]


# ghost-padded bytes: around 1 MiB (downloads into fresh pages take the lanes from there), 4.2 MB in odd rows, 48 and
# 110 MB (uploads too, from 8 MiB)
@pytest.mark.gpu
@pytest.mark.parametrize("case", [_khi(n=(36, 36)), _khi(n=(1021, 27)), _khi(n=(252, 125)), _khi(n=(509, 251)),
                                  _gauss3d(n=(100, 100, 106)), _gauss3d(n=(131, 133, 137))],
                         ids=["50K", "1M-", "1M+", "4M", "48M", "110M"])
def test_round_trip(case):
    s, c = _sim(case)
    for _ in range(2):
        s.set_state(abi.CVAR, c)
        assert np.array_equal(_interior(s.get(abi.CVAR), s.cfg), _interior(c, s.cfg))
        c = c * 1.5
    s.close()


@pytest.mark.gpu
def test_pinned_host_arrays():
    import ctypes as C

    import torch
    s, c = _sim(_khi(n=(509, 251)))
    src = torch.from_numpy(c).pin_memory()
    dst = torch.empty_like(src).pin_memory()
    s._check(s.L.fgpu_upload_state(s.h, abi.CVAR, C.c_void_p(src.data_ptr()), src.numel()))
    s._check(s.L.fgpu_download(s.h, abi.CVAR, C.c_void_p(dst.data_ptr()), dst.numel()))
    assert np.array_equal(_interior(dst.numpy(), s.cfg), _interior(c, s.cfg))
    s.close()


@pytest.mark.gpu
def test_threads_transfer_at_once():
    sims = [_sim(_khi(n=(509 + 2 * k, 251))) for k in range(4)]
    bad = []

    def work(s, c):
        for _ in range(8):
            s.set_state(abi.CVAR, c)
            if not np.array_equal(_interior(s.get(abi.CVAR), s.cfg), _interior(c, s.cfg)):
                bad.append(s.shape)

    threads = [threading.Thread(target=work, args=sc) for sc in sims]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    for s, _ in sims:
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(36, 36), (509, 251), (1021, 517)], ids=["50K", "4M", "17M"])
def test_transfer_while_another_thread_captures(n):
    """A thread in the relaxed capture mode transfers while another one captures a graph in the global
    mode: the transfer works and the capture survives (the lanes' threads wait under the same mode)."""
    import ctypes as C

    import torch
    torch.cuda.init()
    L = C.CDLL([x.split()[-1] for x in open("/proc/self/maps") if "libcudart.so" in x][0])
    relaxed, glob = C.c_int(2), 0   # cudaStreamCaptureModeRelaxed, cudaStreamCaptureModeGlobal
    s, c = _sim(_khi(n=n))
    stream = torch.cuda.Stream()
    begun, finish, got = threading.Event(), threading.Event(), []

    def capture():
        graph = C.c_void_p()
        got.append(L.cudaStreamBeginCapture(C.c_void_p(stream.cuda_stream), glob))
        begun.set()
        finish.wait(60)
        got.append(L.cudaStreamEndCapture(C.c_void_p(stream.cuda_stream), C.byref(graph)))
        if graph:
            L.cudaGraphDestroy(graph)

    other = threading.Thread(target=capture)
    assert L.cudaThreadExchangeStreamCaptureMode(C.byref(relaxed)) == 0
    try:
        other.start()
        begun.wait(60)
        s.set_state(abi.CVAR, c)
        back = s.get(abi.CVAR)
    finally:
        finish.set()
        other.join()
        L.cudaThreadExchangeStreamCaptureMode(C.byref(relaxed))
    assert got == [0, 0]
    assert np.array_equal(_interior(back, s.cfg), _interior(c, s.cfg))
    s.close()


_RESET = """
import sys
import ctypes as C
import numpy as np
from fosite_b200 import abi, problems
from fosite_b200.sim import Simulation

runtime = C.CDLL(sys.argv[1])
got = []
for _ in range(3):
    cfg = problems.khi2d(n=8)[0]
    cfg.inum = cfg.jnum = 1024
    p = np.ones((4, 1028, 1028))
    p[1:3], p[3] = 0.1, 2.5
    s = Simulation(cfg)
    s.set_state(abi.PVAR, p)
    s.first_step()
    s.run(2)
    got.append(s.get(abi.PVAR))
    s.close()
    assert runtime.cudaSetDevice(0) == 0 and runtime.cudaDeviceReset() == 0
assert np.isfinite(got[0]).all() and np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
print("done")
"""


@pytest.mark.gpu
def test_device_reset_between_grids():
    """A program (of its own process) that resets the device once its grids are closed opens new ones: the
    lanes, which went with the old context, are made anew."""
    import glob
    import os
    import subprocess
    import sys

    import torch
    found = glob.glob(os.path.join(os.path.dirname(os.path.dirname(torch.__file__)), "nvidia", "cuda_runtime", "lib",
                                   "libcudart.so*")) + glob.glob("/usr/local/cuda/lib64/libcudart.so*")
    if not found:
        pytest.skip("no shared CUDA runtime here")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _RESET, found[0]], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]
