"""Batches large enough for the refilling query kernels (rzk_trace.cu: 393,216 rays in scenes of
65,536 triangles and more) give, byte for byte, what the one-ray-per-thread kernels give for the
same rays in pieces, at every remainder of the runs a warp owns."""
import numpy as np
import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [393216, 393217, 400001, 700033])
def test_refilled_batches_equal_their_pieces(ctx, n):
    import torch
    from renzoku_b200 import rzk

    sc = sg.room_objects(600, 8, 8, seed_geo=31, seed_mat=32)
    agg = rzk.AggregateCuda(ctx, sc)
    assert agg.n_tris >= 65536
    rng = np.random.default_rng(n)
    size = np.abs(sc.prim_v).max()
    p = torch.from_numpy((rng.uniform(0, size, (n, 3))).astype(np.float32)).cuda()
    q = torch.from_numpy((rng.uniform(0, size, (n, 3))).astype(np.float32)).cuda()
    d = (q - p) / (q - p).norm(dim=1, keepdim=True)
    occ = agg.hit_segments(p, q)
    t, recv = agg.hit_rays(p, d)
    for i in range(0, n, 150000):
        e = min(n, i + 150000)
        assert torch.equal(occ[i:e], agg.hit_segments(p[i:e].contiguous(), q[i:e].contiguous()))
        t1, r1 = agg.hit_rays(p[i:e].contiguous(), d[i:e].contiguous())
        assert torch.equal(t[i:e], t1)
        assert torch.equal(recv.view(torch.uint8).reshape(n, -1)[i:e], r1.view(torch.uint8).reshape(e - i, -1))
    assert 0 < int(occ.sum()) < n
