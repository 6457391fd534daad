"""The two-pass gather (variant 0 below some billions of pairs) gives the one-pass kernel's image
bit for bit and traces the same rays, at the edges of its tiles, items and chunks and on both
sides of its two summing kernels; the one-launch VPL order is the stable order by Hilbert key."""
import dataclasses

import numpy as np
import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu
ONE_PASS = 3


@pytest.fixture(scope="module")
def scene(ctx):
    from renzoku_b200 import instances, rzk
    sc = sg.room_objects(60, 24, 24, seed_geo=41, seed_mat=42)
    agg = rzk.AggregateCuda(ctx, sc)
    vpls, _ = instances.spawn_vpls(agg, 3, 5000)
    return sc, agg, vpls


@pytest.mark.parametrize("w,h,n_vpl,tiled,mode", [(1, 1, 1, True, 0), (7, 3, 31, True, 1), (8, 4, 32, True, 2),
                                                  (9, 5, 33, True, 3), (31, 1, 127, False, 3), (33, 7, 128, False, 1),
                                                  (40, 30, 129, True, 3), (37, 29, 1000, True, 2), (64, 48, 4097, True, 3),
                                                  (320, 200, 257, False, 1), (301, 203, 4096, True, 3)])
def test_two_pass_equals_one_pass(ctx, scene, w, h, n_vpl, tiled, mode):
    from renzoku_b200 import rzk
    sc, agg, vpls = scene
    recv = agg.primary(rzk.Camera(dataclasses.replace(sc.camera, width=w, height=h)))
    ev = rzk.VirtualPointLightCuda(agg, mode, 0.05)
    out, rays = [], []
    for variant in (0, ONE_PASS):
        ctx.rays(reset=True)
        out.append(ev.gather(recv, w * h, vpls, n_vpl, scale=0.25, image_width=w if tiled else 0, variant=variant).cpu().numpy())
        rays.append(ctx.rays())
    ctx.check()
    assert np.array_equal(out[0], out[1]) and rays[0] == rays[1]


@pytest.mark.parametrize("n_vpl", [129, 1000, 1024, 1025, 4095, 4096, 4097])
def test_rank_order_is_the_spatial_order(ctx, scene, n_vpl):
    import torch
    from test_gpu_core import spatial_order
    from renzoku_b200 import rzk
    sc, agg, vpls = scene
    v = rzk.records_from_device(vpls, sg.VPL_DTYPE)[:n_vpl].copy()
    v["p"][n_vpl // 3:n_vpl // 2] = v["p"][0]   # equal keys keep their order
    recv = agg.primary(rzk.Camera(sc.camera))
    ev = rzk.VirtualPointLightCuda(agg, rzk.CLAMP_RADIANCE, 0.05)
    order = spatial_order(v, agg.bounding_box())
    a = ev.gather(recv, 576, rzk.records_to_device(v), n_vpl, image_width=24)
    b = ev.gather(recv, 576, rzk.records_to_device(v[order]), n_vpl, image_width=24)
    assert torch.equal(a, b)
