"""The server's count of launched kernels is what the device ran, in one pass and in two, with and
without the ordering of the VPLs, one at a time and batched."""
import dataclasses

import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,n_vpl,chunked", [(16, 100, False), (32, 1000, True), (512, 100, False), (512, 1000, True),
                                                (640, 5000, True)])
@pytest.mark.parametrize("batching", [False, True])
def test_counted_kernels_ran(ctx, side, n_vpl, chunked, batching):
    import torch
    from renzoku_b200 import instances, rzk
    sc = sg.room_boxes(side, side)
    agg = rzk.AggregateCuda(ctx, sc)
    vpls, _ = instances.spawn_vpls(agg, 3, n_vpl)
    out = torch.zeros((side * side, 3), dtype=torch.float32, device="cuda")
    r = rzk.RequestC()
    r.kind, r.scene, r.d_vpls, r.n_vpl = rzk.REQ_GATHER, agg.h.value, vpls.data_ptr(), n_vpl
    r.camera = rzk.camera_c(rzk.Camera(dataclasses.replace(sc.camera, width=side, height=side)))
    r.clamp_mode, r.tau, r.scale, r.d_rgb = rzk.CLAMP_RADIANCE, 0.05, 1.0, out.data_ptr()
    srv = rzk.Server(0, batching=batching)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        assert srv.wait(srv.submit(r), timeout_ms=60000)[0] == rzk.OK
        torch.cuda.synchronize()
    counted = srv.stats()["launches"]
    srv.close()
    ran = [e.name for e in prof.events() if "rzk::" in e.name]
    if not ran:
        pytest.skip("no CUDA activity records here")
    assert any("order_keys" in x for x in ran) == chunked
    assert counted == len(ran), sorted(ran)
    ctx.check()
