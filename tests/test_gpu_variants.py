"""FD step kernel variants and the tuner that picks among them.

Every variant (rows per interior block x blocks per SM) computes the same
values bit for bit, so results never depend on the tuner's choice.
"""
import os

import numpy as np
import pytest
import torch

import cases
from geopvi_gb300 import _native

pytestmark = pytest.mark.gpu

GOLDEN = os.path.dirname(cases.__file__)


def run(p, vel, obs, **kw):
    from geopvi_gb300.engine import Fwi2dEngine
    eng = Fwi2dEngine(p, device="cuda:0", graph=False, **kw)
    v = torch.from_numpy(np.ascontiguousarray(np.atleast_2d(vel), dtype=np.float32)).cuda()
    o = torch.from_numpy(np.ascontiguousarray(obs, dtype=np.float32)).cuda()
    r = eng.run(v, o, want_syn=True)
    torch.cuda.synchronize()
    return eng, r.misfit.cpu().numpy().copy(), r.grad.cpu().numpy().copy(), r.syn.cpu().numpy().copy()


@pytest.mark.parametrize("name", ["fwi_o8", "fwi_o12", "fwi_ragged", "img_o6"])
def test_every_variant_is_bit_identical(engine_lib, cuda, name):
    z = np.load(os.path.join(GOLDEN, f"{name}.npz"))
    p = cases.params_from_npz(z)
    vel = np.stack([z["start"], z["truth"]]).astype(np.float32)
    ref = None
    for v in range(_native.NUM_STEP_VARIANTS):
        _, m, g, syn = run(p, vel, z["obs"], variant=v)
        if ref is None:
            ref = (m, g, syn)
            assert np.array_equal(syn[0], z["syn"])  # variant 0 against the reference's own data
        else:
            assert np.array_equal(m, ref[0]) and np.array_equal(g, ref[1]) and np.array_equal(syn, ref[2]), v


def test_tuner_settles_and_results_do_not_move(engine_lib, cuda):
    from geopvi_gb300.engine import Fwi2dEngine
    z = np.load(os.path.join(GOLDEN, "fwi_o8.npz"))
    p = cases.params_from_npz(z)
    eng = Fwi2dEngine(p, device="cuda:0", graph=False)
    v = torch.from_numpy(np.stack([z["start"], z["truth"]]).astype(np.float32)).cuda()
    o = torch.from_numpy(z["obs"].astype(np.float32)).cuda()
    outs = []
    for _ in range(_native.NUM_STEP_VARIANTS + 2):
        r = eng.run(v, o)
        torch.cuda.synchronize()
        outs.append(r.grad.cpu().numpy().copy())
    assert all(np.array_equal(outs[0], x) for x in outs[1:])
    chosen = eng.tuned_variant(2)
    assert 0 <= chosen < _native.NUM_STEP_VARIANTS
    with pytest.raises(_native.EngineError):
        run(p, z["start"], z["obs"], variant=_native.NUM_STEP_VARIANTS)


def test_tuner_tries_a_variant_per_wave(engine_lib, cuda):
    """Six waves of one solve: every variant is tried within the first call."""
    from geopvi_gb300.engine import Fwi2dEngine
    z = np.load(os.path.join(GOLDEN, "fwi_o8.npz"))
    p = cases.params_from_npz(z)
    eng = Fwi2dEngine(p, device="cuda:0", graph=True, max_resident=1)
    v = torch.from_numpy(np.stack([z["start"], z["truth"]]).astype(np.float32)).cuda()
    o = torch.from_numpy(z["obs"].astype(np.float32)).cuda()
    g0 = eng.run(v, o).grad.cpu().numpy().copy()
    torch.cuda.synchronize()
    assert 0 <= eng.tuned_variant(2) < _native.NUM_STEP_VARIANTS
    g1 = eng.run(v, o).grad.cpu().numpy().copy()  # the tuned variant, now through a CUDA graph
    assert np.array_equal(g0, g1)
    ref = Fwi2dEngine(p, device="cuda:0", graph=False, variant=0).run(v, o).grad.cpu().numpy()
    assert np.array_equal(g0, ref)


def test_forced_variant_on_a_grid_of_many_tiles(engine_lib, cuda):
    """More two-row tiles in a solve than a grid's y extent holds: the values come from taller ones."""
    from geopvi_gb300.engine import Fwi2dEngine
    from geopvi_gb300.params import Params
    p = Params(nx=30000, nz=300, pml0=5, Lc=4, ns=1, nt=12, ds=1, ns0=15000, depths=2, depthr=0, nr=3000, dr=1, nr0=13500,
               nt_interval=1, dx=10.0, dz=10.0, dt=1e-3, f0=60.0)
    v = torch.full((1, p.nz * p.nx), 2500.0, device=cuda)
    o = torch.zeros(p.data_len, device=cuda)
    want = Fwi2dEngine(p, device=cuda).run(v, o, forward_only=True).syn
    got = Fwi2dEngine(p, device=cuda, variant=3).run(v, o, forward_only=True).syn
    assert want.abs().max() > 0 and torch.equal(got, want)


# Sizes around each line of the rule: samples and shots of a grid, the variant (rows 16, 8, 4, 2).
@pytest.mark.parametrize("nz,nx,ns,n,variant", [
    (32, 48, 2, 1, 3), (120, 250, 16, 1, 3), (120, 250, 16, 2, 2), (120, 250, 16, 3, 1), (120, 250, 16, 9, 1),
    (120, 250, 16, 10, 0), (200, 400, 20, 4, 1), (200, 400, 20, 5, 0),
])
def test_rule_of_the_tile_height(engine_lib, cuda, nz, nx, ns, n, variant):
    from geopvi_gb300 import workloads
    from geopvi_gb300.engine import Fwi2dEngine
    p = workloads.make_params(nz, nx, 20, 1e-3, ns, 30.0, pml0=20)
    g = torch.Generator(device=cuda).manual_seed(3)
    v = (2500 + 200 * torch.randn(n, nz * nx, generator=g, device=cuda)).clamp(1500, 4500)
    o = 0.01 * torch.randn(p.data_len, generator=g, device=cuda)
    eng = Fwi2dEngine(p, device=cuda)
    r = eng.run(v, o, want_syn=True)
    assert eng.tuned_variant(n) == variant
    other = Fwi2dEngine(p, device=cuda, variant=(variant + 1) % 4).run(v, o, want_syn=True)
    for name in ("syn", "grad", "misfit"):
        assert torch.equal(getattr(r, name), getattr(other, name)), name
