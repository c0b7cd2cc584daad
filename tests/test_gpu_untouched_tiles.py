"""Tiles that the wave has not reached are skipped; where the reference makes 0 * inf there, so does the engine.

Forward: a velocity that overflows a product of the absorbing strips' factors.  Adjoint: a stored forward field
that overflowed (an unstable model) below a layer that the adjoint field has not crossed."""
import numpy as np
import pytest
import torch

from geopvi_gb300.params import Params

pytestmark = pytest.mark.gpu

BASE = dict(nx=150, nz=120, pml0=9, Lc=4, ns=2, nt=41, ds=60, ns0=40, depths=100, depthr=0, nr=150, dr=1, nr0=0,
            nt_interval=1, dx=10.0, dz=10.0, dt=1e-3, f0=60.0)


def solve(oracle, p, vel, obs, run_fwi=1):
    op = oracle.Params(**{k: getattr(p, k) for k in oracle.INT_FIELDS + oracle.FLOAT_FIELDS})
    with np.errstate(all="ignore"):
        return oracle.fwi_f32(op, vel.ravel(), obs, run_fwi)


@pytest.mark.parametrize("kw", [dict(), dict(checkpoint=True), dict(variant=0), dict(variant=3)])
@pytest.mark.parametrize("change", [dict(), dict(nt_interval=2), dict(nx=70, ds=20, ns0=20, nr=70)])
def test_overflowed_forward_field_under_a_zero_adjoint(engine_lib, cuda, oracle, change, kw):
    from geopvi_gb300.engine import Fwi2dEngine
    p = Params(**{**BASE, **change})
    vel = np.full((p.nz, p.nx), 2000.0, np.float32)
    vel[90:] = 15000.0  # unstable; the sources lie in it
    obs = np.zeros((p.ns, p.nt, p.nr), np.float32)
    obs[:, -4:, : p.nr // 2] = 1e-3  # the last samples only: the adjoint starts there
    syn, ref = solve(oracle, p, vel, obs.ravel(), 0)
    # the infinities have not reached the receivers, and not all cells' terms are NaN
    assert np.isnan(ref).any() and np.isfinite(ref).any() and np.isfinite(syn).all()
    eng = Fwi2dEngine(p, device=cuda, **kw)
    r = eng.run(torch.from_numpy(vel.ravel()).to(cuda)[None], torch.from_numpy(obs.ravel()).to(cuda), imaging=True)
    assert np.array_equal(np.isfinite(r.grad[0].cpu().numpy()), np.isfinite(ref))


def test_velocity_that_overflows_the_strip(engine_lib, cuda, oracle):
    from geopvi_gb300.engine import Fwi2dEngine
    p = Params(**{**BASE, "depths": 2, "nt": 60, "f0": 30.0})
    vel = np.full((p.nz, p.nx), 2000.0, np.float32)
    vel[40, 0] = 1e14  # (v dt)^2 is finite, the square of the strip's first factor is not
    obs = np.zeros(p.data_len, np.float32)
    syn, _ = solve(oracle, p, vel, obs)
    assert np.isnan(syn).any() and np.isfinite(syn).any()
    r = Fwi2dEngine(p, device=cuda).run(torch.from_numpy(vel.ravel()).to(cuda)[None], torch.from_numpy(obs).to(cuda),
                                        forward_only=True)
    got = r.syn[0].cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(syn))
    assert np.array_equal(got[np.isfinite(syn)], syn[np.isfinite(syn)])


def test_overflow_in_one_inversion_of_a_fused_call(engine_lib, cuda, oracle):
    """Inversions of one launch share the flag: the unstable one has its NaN, the other its own values."""
    import ctypes
    from geopvi_gb300 import _native
    p = Params(**BASE)
    q = Params(**{**BASE, "ns": 3, "ds": 30, "nt": 60})
    bad = np.full((p.nz, p.nx), 2000.0, np.float32)
    bad[90:] = 15000.0
    good = np.full((q.nz, q.nx), 2000.0, np.float32)
    parts = []
    for prm, vel in ((p, bad), (q, good)):
        obs = np.zeros((prm.ns, prm.nt, prm.nr), np.float32)
        obs[:, -4:, : prm.nr // 2] = 1e-3
        v, o = torch.from_numpy(vel.ravel()).to(cuda)[None], torch.from_numpy(obs.ravel()).to(cuda)
        parts.append((prm, v, o, torch.empty_like(v), solve(oracle, prm, vel, obs.ravel(), 0)[1]))
    arr = (_native.CInstance * 2)(*[_native.CInstance(prm.c(), 1, v.data_ptr(), o.data_ptr(), None, g.data_ptr(), None)
                                    for prm, v, o, g, _ in parts])
    flags = _native.FLAG_IMAGING
    work = torch.empty(int(engine_lib.gb_fwi2d_instances_workspace_bytes(arr, 2, 0, flags)) + (1 << 28),
                       dtype=torch.uint8, device=cuda)
    st = engine_lib.gb_fwi2d_run_instances(arr, 2, flags, 0, ctypes.c_void_p(work.data_ptr()), work.numel(),
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    _native.check(st, "gb_fwi2d_run_instances")
    for _, _, _, g, ref in parts:
        assert np.array_equal(np.isfinite(g[0].cpu().numpy()), np.isfinite(ref))


@pytest.mark.parametrize("change,flag", [(dict(), 0), (dict(depthr=-12), 2), (dict(nr=176, nr0=-13), 2)])
def test_tiles_on_the_rim_are_not_looked_at(engine_lib, cuda, oracle, change, flag):
    """A tile at the end of a field's rows has no memory of the field beside it to look at: none is skipped then."""
    from geopvi_gb300.engine import Fwi2dEngine
    p = Params(**{**BASE, "depths": 2, **change})
    vel = np.full((p.nz, p.nx), 2000.0, np.float32)
    obs = np.zeros(p.data_len, np.float32)
    eng = Fwi2dEngine(p, device=cuda)
    r = eng.run(torch.from_numpy(vel.ravel()).to(cuda)[None], torch.from_numpy(obs).to(cuda), forward_only=True)
    assert int(eng._work[4:8].view(torch.int32)) == flag
    assert np.array_equal(r.syn[0].cpu().numpy(), solve(oracle, p, vel, obs)[0])
