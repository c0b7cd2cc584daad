"""Graphs of calls whose buffers move: the library keeps the ones used last, within a bound."""
import pytest

pytestmark = pytest.mark.gpu


def test_graphs_of_moving_models_stay_bounded(engine_lib, cuda):
    import torch
    from geopvi_gb300 import workloads
    from geopvi_gb300.engine import Fwi2dEngine
    p = workloads.make_params(24, 40, 3000, 1e-3, 33, 15.0, pml0=8)  # 33 solves: two halves, 12,000 launches
    obs = 0.01 * torch.randn(p.data_len, device=cuda)
    model = torch.full((1, p.nz * p.nx), 2500.0, device=cuda)
    moved = [model.clone() for _ in range(30)]
    eng = Fwi2dEngine(p, device=cuda, graph=True)
    want = eng.run(model, obs).grad.clone()
    for v in moved:
        assert torch.equal(eng.run(v, obs).grad, want)
        assert engine_lib.gb_fwi2d_graph_launches() <= 1 << 18
    assert engine_lib.gb_fwi2d_graph_launches() > 1 << 17  # full, so the first ones went
    for v in (moved[0], moved[-1]):  # one that went, one that stayed
        assert torch.equal(eng.run(v, obs).grad, want)
