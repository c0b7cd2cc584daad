"""The adjoint pass where the field overflows: infinities stay infinities, as in the reference's arithmetic.

One receiver is given data so large that the adjoint field overflows in its cell alone, in the pass's third step.
The fourth and last step spreads the infinity along the stencil, to the source's cell a few rows below.  Only time
index 0 is imaged, where the stored field is the source's injection, so the gradient at the source's cell is that
injection times the adjoint value there: an infinity of a sign, not NaN.
"""
import numpy as np
import pytest

from geopvi_gb300.params import Params

BASE = dict(nx=60, nz=40, pml0=9, Lc=4, ns=1, nt=4, ds=1, ns0=30, depths=1, depthr=-2, nr=1, dr=1, nr0=30,
            nt_interval=4, dx=10.0, dz=10.0, dt=1e-3, f0=15.0)
CASES = {
    "top_strip": dict(),
    "top_strip_order12": dict(Lc=6, depthr=-3),
    "left_strip": dict(nr0=-2, ns0=1, depthr=15, depths=15),
    "interior": dict(depthr=3),
    "interior_large_reciprocal": dict(depthr=3, dx=12.5, dz=12.5),  # RN(1/dx^2) is above 1/dx^2
    "no_two_op_quotient": dict(dx=11.7, dz=11.7),
}


def reference(oracle, name):
    p = Params(**{**BASE, **CASES[name]})
    vel = np.full(p.nz * p.nx, 2500.0, np.float32)
    # injected value: 0.26 of the largest float; two steps later its second difference exceeds that
    obs = np.zeros(p.data_len, np.float32)
    obs.reshape(p.ns, p.nt, p.nr)[0, -1, 0] = -0.26 * 3.4028235e38 / (p.dt * 2500.0) ** 2
    op = oracle.Params(**{k: getattr(p, k) for k in oracle.INT_FIELDS + oracle.FLOAT_FIELDS})
    with np.errstate(all="ignore"):
        return p, vel, obs, oracle.fwi_f32(op, vel, obs, 1)[1]


@pytest.mark.parametrize("name", sorted(CASES))
def test_the_case_holds_an_infinity(oracle, name):
    p, _, _, grad = reference(oracle, name)
    at = p.depths * p.nx + p.ns0
    assert np.isinf(grad[at])


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
def test_infinities_of_the_adjoint_field(engine_lib, cuda, oracle, name):
    import torch
    from geopvi_gb300.engine import Fwi2dEngine
    p, vel, obs, ref = reference(oracle, name)
    r = Fwi2dEngine(p, device=cuda).run(torch.from_numpy(vel).to(cuda)[None], torch.from_numpy(obs).to(cuda))
    grad = r.grad[0].cpu().numpy()
    at = p.depths * p.nx + p.ns0
    assert grad[at] == ref[at]
