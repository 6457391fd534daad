"""The any-hit tree's device build (rzk_sah.cu): visibility must equal the oracle's bit for
bit whatever the triangle count and layout - below, at and above the size one warp builds,
partial last rounds of the block build, and inputs that binning cannot separate."""
import numpy as np
import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu


def _scene(n, layout, seed):
    rng = np.random.default_rng(seed)
    v = rng.uniform(-0.08, 0.08, (n, 3, 3))
    if layout == "spread":
        v += rng.uniform(0.1, 0.9, (n, 1, 3))
    elif layout == "planar":       # no extent along y
        v[:, :, 1] = 0.0
        v += rng.uniform(0.1, 0.9, (n, 1, 3)) * [1, 0, 1] + [0, 0.5, 0]
    elif layout == "copies":       # one triangle n times: no split separates the centroids
        v[:] = v[0] + 0.5
    else:                          # "chain": bins peel off one triangle at a time
        v += 0.5 * 0.7 ** np.arange(n)[:, None, None] + [0.0, 0.3, 0.3]
    prim_v = np.zeros((n, 12), np.float32)
    prim_v[:, :9] = v.reshape(n, 9)
    mats = np.zeros(1, sg.MATERIAL_DTYPE)
    mats["kd"] = 0.5
    return sg.Scene("triangles", np.full(n, sg.PRIM_TRIANGLE, np.int32), prim_v, np.zeros(n, np.int32),
                    np.zeros((n, 3), np.float32), np.full(n, sg.SURF_TWO_SIDED, np.int32), mats,
                    sg.CameraSpec(width=8, height=8))


@pytest.mark.parametrize("n,layout", [(1, "spread"), (2, "spread"), (3, "spread"), (33, "spread"), (255, "spread"),
                                      (256, "spread"), (257, "spread"), (1025, "spread"), (40003, "spread"),
                                      (700, "planar"), (256, "copies"), (3000, "copies"), (120, "chain"), (600, "chain")])
def test_visibility_equals_oracle(ctx, oracle_built, n, layout):
    import torch
    from oracle import Oracle
    from renzoku_b200 import rzk
    sc = _scene(n, layout, n)
    agg = rzk.AggregateCuda(ctx, sc)
    rng = np.random.default_rng(n + 1)
    p = rng.uniform(0, 1, (4000, 3)).astype(np.float32)
    q = rng.uniform(0, 1, (4000, 3)).astype(np.float32)
    tp, tq = torch.from_numpy(p).cuda(), torch.from_numpy(q).cuda()
    want = Oracle(sc).occluded(p, q)[0].astype(np.uint8)
    assert np.array_equal(agg.hit_segments(tp, tq).cpu().numpy(), want)
    ctx.check()
    blob = agg.serialize()
    agg.rebuild()
    assert np.array_equal(agg.hit_segments(tp, tq).cpu().numpy(), want)
    assert agg.serialize() == blob   # the build does not depend on scheduling
