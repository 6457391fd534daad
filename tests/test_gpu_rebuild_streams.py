"""A rebuild on one stream beside queries in flight on another: it writes what the queries read once
and with the bytes that are there, so they answer as without it."""
import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [60, 600])
def test_queries_in_flight_keep_their_answers(ctx, count):
    import torch
    from renzoku_b200 import instances, rzk
    sc = sg.room_objects(count, 64, 64, seed_geo=31, seed_mat=32)
    agg = rzk.AggregateCuda(ctx, sc)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(4)
    p, q = (torch.rand((200000, 3), generator=gen, device="cuda") for _ in range(2))
    vpls, _ = instances.spawn_vpls(agg, 3, 1000)
    recv = agg.primary(rzk.Camera(sc.camera))
    ev = rzk.VirtualPointLightCuda(agg, rzk.CLAMP_RADIANCE, 0.05)

    def queries(stream=None):
        return [*agg.hit_rays(p, q - p, stream=stream), agg.hit_segments(p, q, stream=stream),
                ev.gather(recv, 4096, vpls, 1000, image_width=64, stream=stream)]
    want = queries()
    blob = agg.serialize()
    d = q - p   # made before the streams part
    torch.cuda.synchronize()
    st, other = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(3):
        with torch.cuda.stream(st):
            got = [[*agg.hit_rays(p, d), agg.hit_segments(p, q), ev.gather(recv, 4096, vpls, 1000, image_width=64)]
                   for _ in range(60)]
        for _ in range(4):
            agg.rebuild(stream=other)
        torch.cuda.synchronize()
        for g in got:
            for a, b in zip(g, want):
                assert torch.equal(a.view(torch.int32) if a.dtype == torch.float32 else a,
                                   b.view(torch.int32) if b.dtype == torch.float32 else b)
    assert agg.serialize() == blob
    ctx.check()
