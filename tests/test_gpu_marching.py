"""The marching stage kernels (layout 6: 2D strips of 30 columns, 3D tiles of 32 x 8) at the sizes
where their tiling can go wrong: one column more or less than a strip or tile, odd extents (rows
copied element by element), a single column left over, the smallest chunks; every boundary type.
The --fmad=false build equals the oracle bit for bit (absorbing faces: 1e-13, CUDA's exp/log)."""
import numpy as np
import pytest

from fosite_b200 import abi
from cases import _disk, _disk_fargo, _gauss3d, _khi
from test_gpu_parity import _compare

pyoracle = pytest.importorskip("pyoracle")

P, R, N, A = abi.PERIODIC, abi.REFLECTING, abi.NO_GRADIENTS, abi.ABSORBING


def _check(case, steps, tol, exact=True):
    from fosite_b200.sim import Simulation
    cfg, p, extra = case
    o, g = pyoracle.Oracle(cfg), Simulation(cfg, exact=exact)
    for s in (o, g):
        if "bccsound" in extra:
            s.set_sound_speeds(np.broadcast_to(extra["bccsound"], o.shape),
                               np.broadcast_to(extra["fcsound"], (4,) + tuple(o.shape)))
        s.set_state(abi.PVAR, p)
        assert s.first_step() == 0
    for k in range(steps):
        assert o.step() == g.step()
        if tol == 0.0:
            assert g.status().dt == o.status().dt and g.status().time == o.status().time
        _compare(cfg, o, g, tol, "step %d" % k)
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("bcs", [[P] * 4, [R] * 4, [N] * 4, [A] * 4, [R, N, P, P], [P, P, N, R]])
@pytest.mark.parametrize("n", [(4, 5), (29, 6), (30, 4), (31, 9), (32, 2), (33, 7), (59, 13), (60, 3), (61, 8), (62, 11)])
def test_strips(n, bcs, monkeypatch):
    monkeypatch.setenv("FGPU_STAGE_VARIANT", "6")
    tol = 1e-13 if A in bcs else 0.0
    for kw in (dict(), dict(variables=abi.PRIMITIVE, limiter=abi.MONOCENT)):
        _check(_khi(n=n, bcs=bcs, **kw), 2, tol)


@pytest.mark.gpu
@pytest.mark.parametrize("build", [_disk, _disk_fargo])
@pytest.mark.parametrize("n", [(30, 21), (31, 40), (61, 18)])
def test_strips_disk(n, build, monkeypatch):
    monkeypatch.setenv("FGPU_STAGE_VARIANT", "6")
    _check(build(n=n), 3, 1e-13)


@pytest.mark.gpu
@pytest.mark.parametrize("kchunk", [1, 3, 16])
@pytest.mark.parametrize("bcs", [[P] * 6, [R] * 6, [N] * 6, [A] * 6, [R, R, P, P, N, N]])
@pytest.mark.parametrize("n", [(4, 3, 2), (31, 9, 4), (33, 8, 5), (34, 7, 3), (65, 17, 4)])
def test_tiles(n, bcs, kchunk, monkeypatch):
    monkeypatch.setenv("FGPU_STAGE_VARIANT", "6")
    monkeypatch.setenv("FGPU_KCHUNK", str(kchunk))
    tol = 1e-13 if A in bcs else 0.0
    _check(_gauss3d(n=n, bcs=bcs, method=abi.MODIFIED_EULER, tdorder=3), 1, tol)
    _check(_gauss3d(n=n, bcs=bcs, variables=abi.CONSERVATIVE, limiter=abi.VANLEER), 1, tol)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(48, 40), (49, 33)])
def test_states_outside_the_straight_line_flux(n, monkeypatch):
    """Near-vacuum cells whose sound speeds the straight-line flux does not cover (pressure and
    density at 1e-200): the product build takes its checked form there, as the other layouts do."""
    from fosite_b200.sim import Simulation
    cfg, p, _ = _khi(n=n, variables=abi.PRIMITIVE, limiter=abi.MINMOD)
    p[0, 10:14, 10:20] = 1e-200
    p[1:3, 10:14, 10:20] = 0.0
    p[3, 10:14, 10:20] = 1e-160
    got = []
    for variant in ("0", "6"):
        monkeypatch.setenv("FGPU_STAGE_VARIANT", variant)
        g = Simulation(cfg)
        g.set_state(abi.PVAR, p)
        got.append(g.compute_rhs() if variant == "0" else None)
        g.first_step()
        g.step()
        got[-1] = g.get(abi.CVAR)
        g.close()
    a, b = got
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    m = np.isfinite(a)
    assert np.abs(a[m] - b[m]).sum() <= 1e-12 * np.abs(a[m]).sum()
