"""The marching stage kernels (layout 6: 2D strips of 30 columns, 3D tiles of 32 x 8) at the sizes
where their tiling can go wrong: one column more or less than a strip or tile, odd extents (rows
copied element by element), a single column left over, the smallest chunks; every boundary type.
The --fmad=false build equals the oracle bit for bit (absorbing faces: 1e-13, CUDA's exp/log)."""
import numpy as np
import pytest

from fosite_b200 import abi
from cases import _disk, _disk_fargo, _gauss3d, _khi
from test_gpu_parity import _compare, _interior, rel_l1

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


_FLAT = dict(method=abi.MODIFIED_EULER, tdorder=3)
_VACUA = {"2d_prim": _khi(n=(48, 40), variables=abi.PRIMITIVE, limiter=abi.MINMOD), "2d_odd": _khi(n=(49, 33)),
          "3d_prim": _gauss3d(n=(36, 20, 12), **_FLAT),
          "3d_cons": _gauss3d(n=(35, 20, 12), variables=abi.CONSERVATIVE, limiter=abi.VANLEER, **_FLAT)}


@pytest.mark.gpu
@pytest.mark.parametrize("variant", ["6", "2"])
@pytest.mark.parametrize("case", list(_VACUA))
def test_states_outside_the_straight_line_flux(case, variant, monkeypatch):
    """A hole whose density and pressure are 1e-200: their product underflows, which the straight-line
    sound speed does not cover, so that the marching kernels (6) take their checked flux at its faces (a
    face left to the straight-line form is NaN there).  The flow runs into the hole at the usual time step;
    the product build's state after it equals the oracle's to rounding, over the whole grid and in the hole
    alone, as that of the tiles (2), which have no straight-line form, does: 5e-16 and 9e-15 at most on
    both layouts (the hole's pressure is a small difference), bound ten times the larger."""
    from fosite_b200.sim import Simulation
    monkeypatch.setenv("FGPU_STAGE_VARIANT", variant)
    cfg, p, _ = _VACUA[case]
    hole = (slice(0, 1) if cfg.knum == 1 else slice(5, 9), slice(8, 14), slice(10, 20))
    inner = tuple(h if h.stop == 1 else slice(h.start - 2, h.stop - 2) for h in hole)
    p = p.copy()
    assert p[(0,) + hole].size >= 60
    p[(slice(None),) + hole] = 0.0
    p[(0,) + hole] = p[(-1,) + hole] = 1e-200
    o, g = pyoracle.Oracle(cfg), Simulation(cfg)
    assert g.stage_layout()[0] == int(variant)
    for s in (o, g):
        s.set_state(abi.PVAR, p)
        assert s.first_step() == 0
        assert s.step() == 0
    ref, got = (_interior(s.get(abi.CVAR), cfg) for s in (o, g))
    assert np.isfinite(got).all() and ref[(0,) + inner].min() < 1e-3
    inside = (slice(None),) + inner
    assert rel_l1(got, ref) <= 1e-13 and rel_l1(got[inside], ref[inside]) <= 1e-13
    g.close()
