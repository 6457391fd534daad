"""Transport matrices large enough for packets of segments (rzk_gather.cu: 8,192 VPLs, 2,097,152
pairs, 65,536 triangles and more) equal, byte for byte, the same columns filled in pieces, which
are traced one pair per thread; so does the same fill under stream capture."""
import dataclasses

import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n_vpl,mode", [(257, 8192, 0), (256, 8193, 1), (211, 10016, 2), (300, 9999, 3)])
def test_packet_fill_equals_pieces(ctx, rows, n_vpl, mode):
    import torch
    from renzoku_b200 import instances, rzk

    sc = sg.room_objects(600, 20, 15, seed_geo=33, seed_mat=34)
    agg = rzk.AggregateCuda(ctx, sc)
    assert agg.n_tris >= 65536 and rows * n_vpl >= 2 << 20
    recv = agg.primary(rzk.Camera(dataclasses.replace(sc.camera, width=20, height=15)))
    vpls, _ = instances.spawn_vpls(agg, 5, 12000)
    ev = rzk.VirtualPointLightCuda(agg, mode, 0.05)
    mat, vis = ev.fill(recv, rows, vpls, n_vpl)
    pieces = [ev.fill(recv, rows, vpls[96 * j:], min(2000, n_vpl - j)) for j in range(0, n_vpl, 2000)]
    want, want_vis = (torch.cat(p) for p in zip(*pieces))
    assert torch.equal(mat.view(torch.int32), want.view(torch.int32)) and torch.equal(vis, want_vis)
    assert 0 < int(vis.sum()) < vis.numel()
    st = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        mat2, vis2 = ev.fill(recv, rows, vpls, n_vpl, stream=st)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(mat2.view(torch.int32), want.view(torch.int32)) and torch.equal(vis2, want_vis)
    ctx.check()
