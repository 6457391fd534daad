"""The facing test of the gathers (FaceTest in rzk_gather_dev.cuh) drops a pair only where the
exact test drops it: the image equals the per-thread kernel's, which has no such test, NaN for NaN,
in each kernel that has it - the two-pass tracing kernel (items of more than four VPLs), the
one-pass kernel with 16-VPL tiles (rzk_gather_noalloc) and those with 32."""
import ctypes
import dataclasses

import numpy as np
import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu
SIDE, N_VPL = 128, 1000   # six VPLs an item in two passes


def _images(ctx, agg, recv, vpls):
    """The per-thread kernel's image, then those of the kernels with the facing test, each with its rays."""
    import torch
    from renzoku_b200 import rzk
    ev = rzk.VirtualPointLightCuda(agg, rzk.CLAMP_FORM_FACTOR, 1.0)
    out = []
    for variant in (7, 0, 1, 3, "noalloc"):
        ctx.rays(reset=True)
        if variant == "noalloc":
            img = torch.empty((SIDE * SIDE, 3), dtype=torch.float32, device="cuda")
            assert rzk.load().rzk_gather_noalloc(agg.h, ctypes.c_void_p(recv.data_ptr()), SIDE * SIDE, SIDE,
                                                 ctypes.c_void_p(vpls.data_ptr()), N_VPL, rzk.CLAMP_FORM_FACTOR, 1.0,
                                                 1.0, ctypes.c_void_p(img.data_ptr()), rzk._stream_ptr()) == rzk.OK
        else:
            img = ev.gather(recv, SIDE * SIDE, vpls, N_VPL, image_width=SIDE, variant=variant)
        out.append((variant, img.cpu().numpy(), ctx.rays()))
    ctx.check()
    return out


def _surface_vpls(hit, rng):
    take = hit[rng.integers(0, len(hit), N_VPL)]
    vpls = np.zeros(N_VPL, sg.VPL_DTYPE)
    for a, b in (("p", "p"), ("n", "ns"), ("u", "u"), ("v", "v"), ("nn", "n"), ("wi", "wo"), ("mat", "mat")):
        vpls[a] = take[b]
    vpls["contrib"] = rng.uniform(0, 2, (N_VPL, 3))
    return vpls


@pytest.mark.parametrize("far", [1e7, 1e9, 1e14, 1e17, 1e20, 1e31, 1e37, np.inf, np.nan])
def test_far_positions_drop_nothing(ctx, far):
    from renzoku_b200 import rzk
    sc = dataclasses.replace(sg.room_objects(60, SIDE, SIDE, seed_geo=61, seed_mat=62))
    agg = rzk.AggregateCuda(ctx, sc)
    recv = agg.primary(rzk.Camera(sc.camera))
    rec = rzk.records_from_device(recv, sg.RECEIVER_DTYPE).copy()
    rng = np.random.default_rng(12)
    vpls = _surface_vpls(rec[rec["mat"] >= 0], rng)
    sign = rng.choice([-1.0, 1.0], (N_VPL, 3))
    vpls["p"][::9] = (vpls["p"] + far * sign * rng.uniform(0.5, 1, (N_VPL, 3)))[::9]
    for place in ("vpls", "receivers"):
        if place == "receivers":
            n = len(rec)
            vpls = _surface_vpls(rec[rec["mat"] >= 0], rng)
            rec["p"][5::97] = (rec["p"] + far * rng.choice([-1.0, 1.0], (n, 3)))[5::97]
            recv = rzk.records_to_device(rec)
        (_, want, _), *rest = _images(ctx, agg, recv, rzk.records_to_device(vpls))
        for variant, got, _ in rest:
            assert np.array_equal(got, want, equal_nan=True), (place, variant)


@pytest.mark.parametrize("kind,scale,shift", [("room", 1, 0), ("objects", 1, 0), ("objects", 0.02, 0), ("objects", 300, 0),
                                              ("objects", 1, 70), ("spheres", 5, -900)])
def test_units_and_places(ctx, kind, scale, shift):
    from renzoku_b200 import rzk
    sc = {"room": lambda: sg.room_boxes(SIDE, SIDE), "spheres": lambda: sg.room_spheres(300, SIDE, SIDE, seed=6),
          "objects": lambda: sg.room_objects(150, SIDE, SIDE, seed_geo=51, seed_mat=52)}[kind]()
    v = sc.prim_v.reshape(-1, 4, 3) * np.float32(scale) + np.float32(shift)
    cam = dataclasses.replace(sc.camera, eye=tuple(scale * x + shift for x in sc.camera.eye),
                              lookat=tuple(scale * x + shift for x in sc.camera.lookat))
    agg = rzk.AggregateCuda(ctx, dataclasses.replace(sc, prim_v=np.ascontiguousarray(v.reshape(-1, 12)), camera=cam))
    recv = agg.primary(rzk.Camera(cam))
    rec = rzk.records_from_device(recv, sg.RECEIVER_DTYPE)
    rng = np.random.default_rng(8)
    vpls = _surface_vpls(rec[rec["mat"] >= 0], rng)
    vpls["p"][::7] += rng.normal(0, 0.3 * scale, (N_VPL, 3))[::7]   # off the surfaces
    vpls["p"][::50] += 4 * scale                                    # and outside the scene
    vpls["mat"][::5] = -1
    images = _images(ctx, agg, recv, rzk.records_to_device(vpls))
    rays = images[1][2]
    assert 0 < rays < SIDE * SIDE * N_VPL
    for variant, got, n in images[1:]:
        # a receiver at a VPL has a NaN term; everything else is the same number
        assert np.array_equal(got, images[0][1], equal_nan=True) and n == rays, variant
