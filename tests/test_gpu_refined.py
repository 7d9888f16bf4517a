"""The refined reciprocal and reciprocal square root of the product build (fgpu_device.cuh) against
their error bounds, over the ends of the range that the stage kernels use them in: the source is compiled
into a small probe and its results compared in 64-bit mantissas (x87)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from fosite_b200 import abi, build
from cases import _gauss3d, _khi, _visc

SRC = r'''
#include "fgpu_device.cuh"
__global__ void probe(const double* x, double* y, int n, int root) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = root ? fgpu::rsqrt_refined(x[i]) : fgpu::rcp_refined(x[i]);
}
extern "C" int run(const double* x, double* y, int n, int root) {
  double* d;
  if (cudaMalloc(&d, 2 * sizeof(double) * n) != cudaSuccess) return 1;
  cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice);
  probe<<<(n + 255) / 256, 256>>>(d, d + n, n, root);
  const cudaError_t e = cudaMemcpy(y, d + n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e != cudaSuccess;
}
'''


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("refined")
    src, out = str(d / "probe.cu"), str(d / "probe.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.check_call([build.nvcc(), "-O3", "-std=c++17", "--expt-relaxed-constexpr", *build.ARCH, "-shared", "-Xcompiler",
                           "-fPIC", "-I", build.CSRC, "-I", os.path.join(build.HERE, "..", "include"), "-o", out, src])
    run = C.CDLL(out).run

    def call(x, root):
        y = np.empty_like(x)
        assert run(x.ctypes.data_as(C.c_void_p), y.ctypes.data_as(C.c_void_p), C.c_int(x.size), C.c_int(root)) == 0
        return y
    return call


def _values(lo, hi, n=4_000_000):
    """Mantissas over [1, 2) at exponents lo .. hi - 1, with the ends and neighbours of the powers of two"""
    rng = np.random.default_rng(17)
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))
    p = np.ldexp(1.0, np.arange(lo, hi))
    return np.concatenate([x, p, np.nextafter(p, np.inf), np.ldexp(np.nextafter(2.0, 0.0), np.arange(lo, hi))])


@pytest.mark.gpu
def test_reciprocal(probe):
    """1/d for every normal d whose reciprocal is normal, of either sign, DBL_MIN among them (the van Leer
    slope's smallest denominator).  The cubed error of the approximation stays below 2^-60 and 1 - d y is
    rounded in a term 2^-20 of the result, so that the closing addition's half ulp, at most 2^-53, is the error."""
    d = _values(-1022, 1022)
    d = np.concatenate([d, -d])
    y = probe(d, 0)
    err = np.abs(y.astype(np.longdouble) * d.astype(np.longdouble) - 1)
    assert np.isfinite(y).all() and float(err.max()) <= 2.0 ** -53 * (1 + 2.0 ** -10)
    assert probe(np.array([2.0 ** -1022]), 0)[0] == 2.0 ** 1022
    assert np.isnan(probe(np.array([0.0, np.inf, -np.inf, np.nan, 5e-324, -2.0 ** -1023]), 0)).all()


@pytest.mark.gpu
def test_reciprocal_square_root(probe):
    """1/sqrt(q) for every normal q: q y is rounded, at most 2^-53 of it, which the correction halves; the
    closing addition's half ulp comes on top: at most 1.5 x 2^-53."""
    q = _values(-1022, 1024)
    y = probe(q, 1)
    y80 = y.astype(np.longdouble)
    err = np.abs(y80 * y80 * q.astype(np.longdouble) - 1) / 2
    assert np.isfinite(y).all() and float(err.max()) <= 1.5 * 2.0 ** -53 * (1 + 2.0 ** -10)
    assert np.isnan(probe(np.array([0.0, np.inf, -1.0, np.nan]), 1)).all()
    assert not np.isfinite(probe(np.array([5e-324, 2.0 ** -1023]), 1)).any()   # an infinite sound speed is not good


def _ring():
    """A cylindrical mesh that starts half a cell from the axis: the centre of the first inner ghost
    column lies on it, with no width along the angle."""
    c = abi.default_config()
    c.inum, c.jnum, c.knum = 16, 24, 1
    c.geometry = abi.CYLINDRICAL
    c.xmin, c.xmax, c.ymin, c.ymax = 0.03125, 1.03125, 0.0, 2 * np.pi
    c.physics, c.gamma = abi.EULER, 1.4
    c.limiter, c.variables = abi.VANLEER, abi.CONSERVATIVE
    c.method, c.tdorder, c.tol_rel = abi.MODIFIED_EULER, 3, 10.0
    c.cfl, c.stoptime = 0.4, 1.0e3
    for f, t in enumerate((abi.NO_GRADIENTS, abi.NO_GRADIENTS, abi.PERIODIC, abi.PERIODIC)):
        c.bc[f] = t
    abi.finalize_config(c)
    p = np.ones((4, 1, 28, 20))
    p[1:3] = np.random.default_rng(0).uniform(-0.1, 0.1, (2, 1, 28, 20))
    return c, p, {}


@pytest.mark.gpu
@pytest.mark.parametrize("exact", [True, False])
def test_time_step_of_a_ghost_cell_without_width(exact):
    """CalcTimestep's maximum runs over the ghost cells too: the oracle's step is 0 there."""
    from fosite_b200.sim import Simulation
    pyoracle = pytest.importorskip("pyoracle")
    cfg, p, _ = _ring()
    o, g = pyoracle.Oracle(cfg), Simulation(cfg, exact=exact)
    for s in (o, g):
        s.set_state(abi.PVAR, p)
        s.first_step()
    assert o.status().dt == 0.0 and g.status().dt == 0.0
    assert g.calc_timestep() == 0.0
    g.close()


@pytest.mark.gpu
def test_stresses_of_a_ghost_cell_without_width():
    """Infinities and NaN of the viscous source are where the quotients of the exact build have them."""
    from fosite_b200.sim import Simulation
    cfg, p, _ = _visc(_ring(), 0.01)
    rhs = []
    for exact in (True, False):
        g = Simulation(cfg, exact=exact)
        g.set_state(abi.PVAR, p)
        rhs.append(g.compute_rhs()[:, :, 2:-2, 2:-2])
        g.close()
    a, b = rhs
    assert not np.isfinite(a).all()
    for kind in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(kind(a), kind(b))
    m = np.isfinite(a)
    assert np.abs(a[m] - b[m]).sum() <= 1e-12 * np.abs(a[m]).sum()


@pytest.mark.gpu
@pytest.mark.parametrize("case", [_khi(n=(33, 20)), _khi(n=(40, 22), variables=abi.PRIMITIVE, limiter=abi.MINMOD),
                                  _gauss3d(n=(34, 12, 9), method=abi.MODIFIED_EULER, tdorder=3)], ids=["cons", "prim", "3d"])
def test_sound_speeds_that_overflow(case):
    """A subnormal density: p/rho is infinite, and so is the sound speed; the time step is 0 and the start
    refused as by the oracle (s rsqrt(s rho) is 2e154 there)."""
    from fosite_b200.sim import Simulation
    pyoracle = pytest.importorskip("pyoracle")
    cfg, p, _ = case
    p = p.copy()
    p[0, p.shape[1] // 2, 9:11, 12:15] = 1e-308
    p[-1, p.shape[1] // 2, 9:11, 12:15] = 2.5
    o, g = pyoracle.Oracle(cfg), Simulation(cfg)
    for s in (o, g):
        s.set_state(abi.PVAR, p)
    assert g.calc_timestep() == 0.0
    assert g.first_step() == o.first_step() and g.status().dt == o.status().dt == 0.0
    g.close()
