"""The 3-D step's tiles against the 3-D oracle, bit for bit: sides at the edges of
the 64 x 16 (or 12) tiles and of the z chunks, a right strip cut by a tile
boundary, strips wider than a warp's packed pass, sources in a tile's corner
cells, and every FD order."""
import numpy as np
import pytest
import torch

from geopvi_gb300 import fwi3d
from oracle import oracle3d as O

pytestmark = pytest.mark.gpu

#            nx  ny  nz  pml0 Lc nti
CASES = {
    "one_tile": (44, 6, 7, 5, 4, 1),
    "tile_edges": (108, 22, 9, 10, 4, 1),         # 128 x 42 updated columns and rows
    "cut_right_strip": (55, 11, 12, 7, 4, 2),     # 69 columns: the strip lies in two tiles
    "interior_tile": (180, 5, 6, 4, 4, 1),        # a tile of interior columns only
    "wide_strips": (30, 9, 8, 18, 3, 1),          # 2 x 18 strip cells a row pair: two packed passes
    "order10": (70, 13, 11, 6, 5, 3),
    "order12": (61, 19, 10, 3, 6, 1),
    "tall": (12, 8, 90, 4, 4, 1),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("checkpoint", [False, True])
def test_tiles_match_the_oracle(engine_lib, cuda, name, checkpoint):
    nx, ny, nz, pml0, Lc, nti = CASES[name]
    rng = np.random.default_rng(7)
    p = fwi3d.Fwi3dParams(nx=nx, ny=ny, nz=nz, nt=50, dt=1e-3, dx=10.0, dy=12.0, dz=9.0, pml0=pml0, Lc=Lc,
                          nt_interval=nti, ns=2, nr=12)
    src = np.array([[0, ny - 1, 0], [nx - 1, 0, nz - 1]])
    rec = np.stack([rng.integers(0, nx, 12), rng.integers(0, ny, 12), rng.integers(0, nz, 12)], 1)
    rec[5] = rec[2]  # a shared cell
    t = np.arange(p.nt) * p.dt - 1.0 / 25.0
    a = (np.pi * 25.0 * t) ** 2
    wav = ((1 - 2 * a) * np.exp(-a)).astype(np.float32)
    truth, vel = (1700 + 700 * rng.random((2, p.ncell))).astype(np.float32)
    obs = O.run(p, src, rec, wav, truth)[0]
    syn, grad, misfit = O.run(p, src, rec, wav, vel, obs, grad=True)
    eng = fwi3d.Fwi3dEngine(p, src, rec, wav, device=cuda, checkpoint=checkpoint)
    r = eng.run(torch.from_numpy(vel).to(cuda)[None], torch.from_numpy(obs).to(cuda), want_syn=True)
    assert np.array_equal(r.syn[0].cpu().numpy(), syn)
    assert np.array_equal(r.grad[0].cpu().numpy(), grad)
    assert abs(float(r.misfit[0]) - misfit) <= 1e-12 * abs(misfit)
