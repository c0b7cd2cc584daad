"""Calls of one thread on different streams: each runs its halves beside the other's, not behind them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def setup(cuda, nz, nx, ns, n, nt):
    from geopvi_gb300 import workloads
    from geopvi_gb300.engine import Fwi2dEngine
    p = workloads.make_params(nz, nx, nt, 1e-3, ns, 12.0, pml0=10)
    g = torch.Generator(device=cuda).manual_seed(3)
    vel = (2500 + 200 * torch.randn(n, nz * nx, generator=g, device=cuda)).clamp(1500, 4500)
    obs = 0.01 * torch.randn(p.data_len, generator=g, device=cuda)
    return Fwi2dEngine(p, device=cuda, graph=False), vel, obs  # eager: a replayed graph has its own branches


def test_a_short_call_does_not_wait_for_a_long_one(engine_lib, cuda):
    long, vel, obs = setup(cuda, 400, 800, 40, 1, 700)
    short, v1, o1 = setup(cuda, 40, 60, 33, 1, 20)
    want = {e: e.run(v, o) for e, v, o in ((long, vel, obs), (short, v1, o1))}
    want = {e: (r.grad.clone(), r.misfit.clone()) for e, r in want.items()}
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    ends = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
    torch.cuda.synchronize()
    for _ in range(2):  # the first round creates the streams' own second streams
        with torch.cuda.stream(streams[0]):
            ends[2].record()
            r0 = long.run(vel, obs)
            ends[0].record()
        with torch.cuda.stream(streams[1]):
            r1 = short.run(v1, o1)
            ends[1].record()
        torch.cuda.synchronize()
    whole, left = ends[2].elapsed_time(ends[0]), ends[1].elapsed_time(ends[0])
    assert left > 0.1 * whole, (left, whole)  # the long call's queue was full of work when the short one ended
    for e, r in ((long, r0), (short, r1)):
        assert torch.equal(r.grad, want[e][0]) and torch.equal(r.misfit, want[e][1])


def test_more_streams_than_a_thread_keeps_second_streams(engine_lib, cuda):
    eng, vel, obs = setup(cuda, 40, 60, 33, 1, 20)
    want = eng.run(vel, obs).grad.clone()
    before = engine_lib.gb_fwi2d_side_stream_count()
    for _ in range(12):
        with torch.cuda.stream(torch.cuda.Stream()):
            got = eng.run(vel, obs).grad.clone()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    assert engine_lib.gb_fwi2d_side_stream_count() - before <= 8
