"""Closest hits through the closest-hit tree (rzk_sah.cu, closest_hit in rzk_traverse.cuh) equal
the reference's visit order byte for byte where its answer is delicate: rays at edges and
vertices (equal distances), along surfaces, along the axes, from origins the tree covers and
does not, on scenes with and without such a tree, and at every remainder of the rays a warp owns."""
import numpy as np
import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu


def _scaled(sc, k):
    sc.prim_v *= np.float32(k)
    return sc


SCENES = {
    "room": lambda: sg.room_boxes(8, 8),                                   # too few triangles
    "objects": lambda: sg.room_objects(150, 8, 8, seed_geo=21, seed_mat=22),
    "spheres": lambda: sg.room_spheres(500, 8, 8, seed=9),
    "large_units": lambda: _scaled(sg.room_objects(60, 8, 8, seed_geo=23, seed_mat=24), 100.0),   # inflated too far
}


def _rays(sc, kind, n, rng):
    v = sc.prim_v[rng.integers(0, sc.n_prims, n), :9].reshape(n, 3, 3).astype(np.float64)
    size = np.abs(sc.prim_v).max()
    o = rng.uniform(0, size, (n, 3))
    w = rng.dirichlet([1, 1, 1], n)
    p = (v * w[:, :, None]).sum(1)
    if kind == "surface":
        o, d = p, rng.normal(size=(n, 3))
    elif kind == "edges":
        d = 0.5 * (v[:, 0] + v[:, 1]) - o
    elif kind == "vertices":
        d = v[:, 0] - o
    elif kind == "along":
        e, f = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        nn = np.cross(e, f)
        nn /= np.maximum(np.linalg.norm(nn, axis=1, keepdims=True), 1e-20)
        d = e * rng.uniform(-1, 1, (n, 1)) + f * rng.uniform(-1, 1, (n, 1))
        d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-20)
        off = 10.0 ** rng.uniform(-8, -1, (n, 1))
        o = p - 0.3 * size * d * rng.uniform(size=(n, 1)) + nn * off * size * 0.01
        d = d - nn * off * rng.uniform(-0.1, 0.1, (n, 1))
    elif kind == "axes":
        d = np.zeros((n, 3))
        d[np.arange(n), rng.integers(0, 3, n)] = rng.choice([-1, 1], n)
        d += rng.choice([0, 1e-7, -1e-7, 1e-5], (n, 3))
    else:                                                                  # "far"
        o = (rng.normal(size=(n, 3)) * 5 + 0.5) * size
        d = p - o
    return o.astype(np.float32), d.astype(np.float32)


@pytest.mark.parametrize("scene", sorted(SCENES))
def test_closest_equals_reference_order(ctx, oracle_built, scene):
    import torch
    from oracle import Oracle
    from renzoku_b200 import rzk
    sc = SCENES[scene]()
    agg, o = rzk.AggregateCuda(ctx, sc), Oracle(sc)
    rng = np.random.default_rng(3)
    for kind, n in (("surface", 20001), ("edges", 6007), ("vertices", 6000), ("along", 20000), ("axes", 5003), ("far", 5000),
                    ("surface", 1), ("surface", 31), ("surface", 33), ("far", 129)):
        p, d = _rays(sc, kind, n, rng)
        want_t, want = o.closest(p, d)
        t, recv = agg.hit_rays(torch.from_numpy(p).cuda(), torch.from_numpy(d).cuda())
        assert np.array_equal(t.cpu().numpy(), want_t), kind
        assert recv.cpu().numpy().tobytes() == want.tobytes(), kind
    ctx.check()
