"""The FD step's tiles against the oracle: every FD order with interior tiles
of one and two units, odd sizes at the tiles' edges, every tile height, sources
and receivers in the rim, a divisor without the two-operation quotient, and a
field that has not reached most tiles."""
import numpy as np
import pytest
import torch

from geopvi_gb300.params import Params

pytestmark = pytest.mark.gpu

# The data are the oracle's bit for bit.  The gradient's adjoint rounds each
# update once where the oracle rounds every operation: both are off the exact
# value by some 2^-24 sqrt(steps) of the field, far below this.
GRAD_TOL = 2e-5

BASE = dict(nx=140, nz=61, pml0=9, Lc=4, ns=2, nt=260, ds=90, ns0=20, depths=2, depthr=1, nr=139, dr=1, nr0=0,
            nt_interval=1, dx=10.0, dz=10.0, dt=1e-3, f0=15.0)
CASES = {
    "order6": dict(Lc=3, nz=33, nx=97, ds=50, nr=97),
    "order8_nti2": dict(nt_interval=2, nt=257, nz=48),
    "order10_rect": dict(Lc=5, dx=12.5, dz=10.0, nz=35),
    "order12_nti3": dict(Lc=6, nt_interval=3, nx=201, ds=120, nr=100, dr=2),
    "one_unit": dict(nx=64, ds=30, nr=64, pml0=20, nz=17),
    "low_rows": dict(nz=3, pml0=4, depths=1, depthr=0),
    "source_in_rim": dict(depths=-11, depthr=-12, nz=30),
    "receivers_in_rim_columns": dict(nr=160, nr0=-12, nz=30),
    "receiver_row_inside": dict(depths=40, depthr=37),
    "no_two_op_quotient": dict(dx=11.7, dz=11.7, nz=30, nt=150),
    "untouched_tiles": dict(nx=420, nz=90, nt=90, ds=60, nr=420),
}


def models(p, seed):
    rng = np.random.default_rng(seed)
    base = 1800.0 + 1200.0 * np.linspace(0, 1, p.nz)[:, None] + 40.0 * rng.standard_normal((p.nz, p.nx))
    return base.astype(np.float32).ravel()


@pytest.mark.parametrize("variant", [None, 0, 1, 2, 3])
@pytest.mark.parametrize("name", sorted(CASES))
def test_tiles_match_the_oracle(engine_lib, cuda, oracle, name, variant):
    from geopvi_gb300.engine import Fwi2dEngine
    p = Params(**{**BASE, **CASES[name]})
    op = oracle.Params(**{k: getattr(p, k) for k in oracle.INT_FIELDS + oracle.FLOAT_FIELDS})
    v, t = models(p, 3), models(p, 4)
    obs = oracle.forward_f32(op, t)
    syn, grad = oracle.fwi_f32(op, v, obs, 1)
    eng = Fwi2dEngine(p, device=cuda, variant=variant)
    r = eng.run(torch.from_numpy(v).to(cuda)[None], torch.from_numpy(obs).to(cuda), want_syn=True)
    assert eng.status() == 0
    assert np.array_equal(r.syn[0].cpu().numpy(), syn)
    g = r.grad[0].cpu().numpy().astype(np.float64)
    assert np.linalg.norm(g - grad) <= GRAD_TOL * np.linalg.norm(grad)


def test_infinite_velocity_reaches_the_untouched_tiles(engine_lib, cuda):
    """0 * inf in a cell the wave has not reached is NaN, as in the reference."""
    from geopvi_gb300.engine import Fwi2dEngine
    p = Params(**{**BASE, **CASES["untouched_tiles"], "nt": 40})
    v = models(p, 3)
    v[20 * p.nx + 250] = np.inf  # 160 cells from the nearest source
    eng = Fwi2dEngine(p, device=cuda)
    zero = torch.zeros(p.data_len, device=cuda)
    syn = eng.run(torch.from_numpy(v).to(cuda)[None], zero, forward_only=True).syn
    assert torch.isnan(syn).any()
