"""Waves that run as two halves on two streams give the bits of solves run one at a time.

Halves start at 32 solves, or where a launch of two solves or more has many tiles; the cases lie on both
sides of it, with an odd number of solves, several waves, and with a checkpointed field.
"""
import pytest

pytestmark = pytest.mark.gpu

# nz, nx, shots, samples, nt, engine options
CASES = [
    (40, 60, 11, 3, 90, dict()),                      # 33 small solves
    (40, 60, 11, 3, 90, dict(checkpoint=True)),
    (40, 60, 11, 6, 90, dict(max_resident=35)),       # a wave of 35 and one of 31
    (40, 60, 11, 6, 90, dict(max_resident=35, checkpoint=True)),
    (300, 420, 7, 1, 45, dict()),                     # 7 solves with many tiles
    (300, 420, 7, 1, 45, dict(checkpoint=True)),
]


@pytest.mark.parametrize("graph", (False, True))
@pytest.mark.parametrize("nz,nx,ns,n,nt,kw", CASES)
def test_halves_match_single_solves(engine_lib, cuda, nz, nx, ns, n, nt, kw, graph):
    import torch
    from geopvi_gb300 import workloads
    from geopvi_gb300.engine import Fwi2dEngine
    p = workloads.make_params(nz, nx, nt, 1e-3, ns, 12.0, pml0=10)
    g = torch.Generator(device=cuda).manual_seed(3)
    vel = (2500 + 200 * torch.randn(n, nz * nx, generator=g, device=cuda)).clamp(1500, 4500)
    obs = 0.01 * torch.randn(p.data_len, generator=g, device=cuda)
    one = Fwi2dEngine(p, device=cuda, graph=False, max_resident=1)
    ref = one.run(vel, obs, want_syn=True)
    r = Fwi2dEngine(p, device=cuda, graph=graph, **kw).run(vel, obs, want_syn=True)
    for name in ("syn", "grad", "misfit"):
        assert torch.equal(getattr(r, name), getattr(ref, name)), name


@pytest.mark.parametrize("kw", (dict(), dict(checkpoint=True), dict(max_resident=4)))
@pytest.mark.parametrize("ns,nsamples", ((5, 1), (3, 2)))
def test_halves_3d_match_single_solves(engine_lib, cuda, ns, nsamples, kw):
    import numpy as np
    import torch
    from geopvi_gb300 import fwi3d
    rng = np.random.default_rng(5)
    nx, ny, nz, nt = 70, 61, 64, 26
    p = fwi3d.Fwi3dParams(nx=nx, ny=ny, nz=nz, nt=nt, dt=1e-3, dx=10.0, dy=10.0, dz=10.0, pml0=8, Lc=4)
    src = np.stack([rng.integers(20, 45, ns) for _ in range(3)], 1).astype(np.int32)
    rec = np.stack([rng.integers(0, m, 40) for m in (nx, ny, nz)], 1).astype(np.int32)
    wavelet = rng.standard_normal(nt).astype(np.float32)
    vel = torch.from_numpy((2500 + 200 * rng.standard_normal((nsamples, nx * ny * nz))).astype(np.float32)).to(cuda)
    obs = torch.from_numpy(rng.standard_normal(ns * nt * len(rec)).astype(np.float32)).to(cuda)
    ref = fwi3d.Fwi3dEngine(p, src, rec, wavelet, device=cuda, max_resident=1).run(vel, obs, want_syn=True)
    r = fwi3d.Fwi3dEngine(p, src, rec, wavelet, device=cuda, **kw).run(vel, obs, want_syn=True)
    for name in ("syn", "grad", "misfit"):
        assert torch.equal(getattr(r, name), getattr(ref, name)), name


@pytest.mark.parametrize("nz,nx,ns,n,kw", [
    (40, 60, 11, 3, dict()),                       # 33 small solves, no plain tile in a row of tiles' width
    (40, 60, 11, 3, dict(checkpoint=True)),
    (12, 14, 3, 1, dict()),                        # band tiles only
    (131, 197, 33, 1, dict(max_resident=33)),      # plain tiles within odd edges
])
def test_exact_gradient_halves_match_single_solves(engine_lib, cuda, nz, nx, ns, n, kw):
    import torch
    from geopvi_gb300 import workloads
    from geopvi_gb300.engine import Fwi2dEngine
    p = workloads.make_params(nz, nx, 60, 1e-3, ns, 12.0, pml0=10)
    g = torch.Generator(device=cuda).manual_seed(4)
    vel = (2500 + 200 * torch.randn(n, nz * nx, generator=g, device=cuda)).clamp(1500, 4500)
    obs = 0.01 * torch.randn(p.data_len, generator=g, device=cuda)
    ref = Fwi2dEngine(p, device=cuda, graph=False, max_resident=1).run(vel, obs, exact=True)
    r = Fwi2dEngine(p, device=cuda, **kw).run(vel, obs, exact=True)
    assert torch.equal(r.grad, ref.grad) and torch.equal(r.misfit, ref.misfit)


@pytest.mark.parametrize("kw", (dict(), dict(checkpoint=True)))
@pytest.mark.parametrize("ns,nsamples", ((7, 2), (5, 3)))  # waves of 5, 5 and 4 solves (4 are below the line), of 5, 5, 5
def test_halves_3d_over_several_waves(engine_lib, cuda, ns, nsamples, kw):
    """Five of these solves (2 x 5 tiles, 80 planes each: 4000) run as halves of two and three, wave after wave."""
    import numpy as np
    import torch
    from geopvi_gb300 import fwi3d
    rng = np.random.default_rng(6)
    nx, ny, nz, nt = 70, 61, 64, 26
    p = fwi3d.Fwi3dParams(nx=nx, ny=ny, nz=nz, nt=nt, dt=1e-3, dx=10.0, dy=10.0, dz=10.0, pml0=8, Lc=4)
    src = np.stack([rng.integers(20, 45, ns) for _ in range(3)], 1).astype(np.int32)
    rec = np.stack([rng.integers(0, m, 40) for m in (nx, ny, nz)], 1).astype(np.int32)
    wavelet = rng.standard_normal(nt).astype(np.float32)
    vel = torch.from_numpy((2500 + 200 * rng.standard_normal((nsamples, nx * ny * nz))).astype(np.float32)).to(cuda)
    obs = torch.from_numpy(rng.standard_normal(ns * nt * len(rec)).astype(np.float32)).to(cuda)
    ref = fwi3d.Fwi3dEngine(p, src, rec, wavelet, device=cuda, max_resident=1, **kw).run(vel, obs, want_syn=True)
    eng = fwi3d.Fwi3dEngine(p, src, rec, wavelet, device=cuda, max_resident=5, **kw)
    assert eng.resident_for(nsamples) == 5
    r = eng.run(vel, obs, want_syn=True)
    for name in ("syn", "grad", "misfit"):
        assert torch.equal(getattr(r, name), getattr(ref, name)), name
