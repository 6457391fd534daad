"""The packet gather's visibility (packet_visible in rzk_gather_dev.cuh) against the per-thread
kernel, whose traversal is the reference's any-hit on the reference tree: the same image bit for
bit and the same rays, for scenes in small, large and shifted units (the shaft's margins), narrow
and wide packets, single and no triangles, receivers at the VPLs and VPLs outside the scene."""
import dataclasses

import numpy as np
import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu


def _scene(kind, scale, shift):
    sc = {"room": lambda: sg.room_boxes(40, 28), "objects": lambda: sg.room_objects(150, 40, 28, seed_geo=51, seed_mat=52),
          "spheres": lambda: sg.room_spheres(300, 40, 28, seed=6),
          "one": lambda: sg.room_boxes(40, 28)}[kind]()
    if kind == "one":
        keep = [0]
        sc = dataclasses.replace(sc, prim_kind=np.full(1, sg.PRIM_TRIANGLE, np.int32), prim_v=sc.prim_v[keep],
                                 prim_mat=sc.prim_mat[keep], prim_emit=sc.prim_emit[keep], prim_flags=sc.prim_flags[keep])
    v = sc.prim_v.reshape(-1, 4, 3) * np.float32(scale) + np.float32(shift)
    cam = dataclasses.replace(sc.camera, eye=tuple(scale * x + shift for x in sc.camera.eye),
                              lookat=tuple(scale * x + shift for x in sc.camera.lookat))
    return dataclasses.replace(sc, prim_v=np.ascontiguousarray(v.reshape(-1, 12)), camera=cam)


@pytest.mark.parametrize("kind,scale,shift", [("room", 1, 0), ("objects", 1, 0), ("spheres", 1, 0), ("one", 1, 0),
                                              ("objects", 0.02, 0), ("objects", 300, 0), ("objects", 1, 70), ("spheres", 5, -900)])
def test_packet_equals_per_thread(ctx, kind, scale, shift):
    from renzoku_b200 import rzk
    sc = _scene(kind, scale, shift)
    agg = rzk.AggregateCuda(ctx, sc)
    last = agg.lib.rzk_gather_variants()
    recv = agg.primary(rzk.Camera(sc.camera))
    rec = rzk.records_from_device(recv, sg.RECEIVER_DTYPE)
    rng = np.random.default_rng(8)
    hit = rec[rec["mat"] >= 0]
    take = hit[rng.integers(0, len(hit), 700)]
    vpls = np.zeros(700, sg.VPL_DTYPE)
    for a, b in (("p", "p"), ("n", "ns"), ("u", "u"), ("v", "v"), ("nn", "n"), ("wi", "wo"), ("mat", "mat")):
        vpls[a] = take[b]
    vpls["contrib"] = rng.uniform(0, 2, (700, 3))
    vpls["p"][::7] += rng.normal(0, 0.3 * scale, (100, 3))    # off the surfaces
    vpls["p"][::50] += 4 * scale                              # and outside the scene
    vpls["mat"][::5] = -1
    scattered = take.copy()                                    # receivers of a packet far apart
    for r, n, w in ((recv, len(rec), 40), (rzk.records_to_device(scattered), 700, 0)):
        for n_vpl in (1, 40, 700):
            v = rzk.records_to_device(vpls[:n_vpl])
            ev = rzk.VirtualPointLightCuda(agg, rzk.CLAMP_FORM_FACTOR, 1.0)
            want = ev.gather(r, n, v, n_vpl, image_width=0, variant=7)
            for variant in (0, 3):
                got = ev.gather(r, n, v, n_vpl, image_width=w, variant=variant)
                # a receiver at a VPL has a NaN term; everything else is the same number
                assert np.array_equal(got.cpu().numpy(), want.cpu().numpy(), equal_nan=True), (n_vpl, variant)
    assert last > 7
    ctx.check()
