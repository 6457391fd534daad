"""The gather's scratch under stream capture: a two-pass gather (variant 0) is captured wherever the
context's buffers hold a one-pass gather of its size, captured gathers stay good when later
gathers need more ballots, and ballots allocated beside another thread's capture do not break it."""
import dataclasses
import threading

import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu


@pytest.fixture()
def case(gpu_lib):
    from renzoku_b200 import instances, rzk
    ctx = rzk.Context(0)   # a context of its own: its buffers are those of the calls below
    sc = sg.room_objects(60, 64, 64, seed_geo=41, seed_mat=42)
    agg = rzk.AggregateCuda(ctx, sc)
    recv = agg.primary(rzk.Camera(dataclasses.replace(sc.camera, width=64, height=64)))
    vpls, _ = instances.spawn_vpls(agg, 3, 4000)
    yield ctx, rzk.VirtualPointLightCuda(agg, rzk.CLAMP_RADIANCE, 0.05), recv, vpls
    agg.close()
    ctx.close()


def _capture(ev, recv, vpls, n_vpl, **kw):
    import torch
    st, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    out = torch.zeros((4096, 3), dtype=torch.float32, device="cuda")
    with torch.cuda.graph(graph, stream=st):
        ev.gather(recv, 4096, vpls, n_vpl, image_width=64, out=out, stream=st, **kw)
    return graph, out


@pytest.mark.parametrize("n_chunks", [0, 1])
def test_captured_where_one_pass_fits(case, n_chunks):
    import torch
    ctx, ev, recv, vpls = case
    want = ev.gather(recv, 4096, vpls, 1000, image_width=64, variant=3, n_chunks=n_chunks)
    torch.cuda.synchronize()
    graph, out = _capture(ev, recv, vpls, 1000, n_chunks=n_chunks)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert torch.equal(ev.gather(recv, 4096, vpls, 1000, image_width=64, n_chunks=n_chunks), want)
    ctx.check()


@pytest.mark.parametrize("variant", [0, 3])
def test_captured_gathers_outlive_larger_ballots(case, variant):
    import torch
    ctx, ev, recv, vpls = case
    want = ev.gather(recv, 4096, vpls, 500, image_width=64, variant=variant, n_chunks=1)
    torch.cuda.synchronize()
    graph, out = _capture(ev, recv, vpls, 500, variant=variant, n_chunks=1)
    for n in (1000, 2000, 4000):   # one chunk: the same partial sums, more ballots
        ev.gather(recv, 4096, vpls, n, image_width=64, n_chunks=1)
        fill = torch.full((64 << 20,), 7, dtype=torch.uint8, device="cuda")   # whatever was freed is taken
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want) and bool((fill == 7).all())
        del fill
    ctx.check()


def test_ballots_beside_another_capture(case):
    import torch
    ctx, ev, recv, vpls = case
    want = ev.gather(recv, 4096, vpls, 1000, image_width=64, variant=3)   # its buffers, without ballots
    other, out = torch.cuda.Stream(), torch.zeros((4096, 3), dtype=torch.float32, device="cuda")
    x = torch.zeros(1000, device="cuda")
    errors = []

    def gather():
        try:
            ev.gather(recv, 4096, vpls, 1000, image_width=64, out=out, stream=other)
        except Exception as e:
            errors.append(repr(e))

    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        x += 1
        t = threading.Thread(target=gather)
        t.start()
        t.join()
        x += 1
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert not errors and torch.equal(out, want) and bool((x == 2).all())
    ctx.check()
