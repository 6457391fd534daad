"""A call on one thread leaves another thread's stream capture whole: the matrix fill that takes
scratch for its packets (rzk_gather.cu: 8,192 VPLs, 2,097,152 pairs, 65,536 triangles)."""
import threading

import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu


def test_packet_fill_beside_a_capture(ctx):
    import torch
    from renzoku_b200 import instances, rzk
    rows, n_vpl = 256, 9000
    sc = sg.room_objects(600, 16, 16, seed_geo=33, seed_mat=34)
    agg = rzk.AggregateCuda(ctx, sc)
    assert agg.n_tris >= 65536 and rows * n_vpl >= 2 << 20
    recv = agg.primary(rzk.Camera(sc.camera))
    vpls, _ = instances.spawn_vpls(agg, 5, n_vpl)
    ev = rzk.VirtualPointLightCuda(agg, rzk.CLAMP_RADIANCE, 0.05)
    want, want_vis = ev.fill(recv, rows, vpls, n_vpl)
    mat, vis = torch.zeros_like(want), torch.zeros_like(want_vis)
    other = torch.cuda.Stream()
    status = []
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()

    def fill():
        p = [rzk._dptr(t) for t in (recv, vpls, mat, vis)]
        status.append(agg.lib.rzk_gather_matrix(agg.h, p[0], rows, p[1], n_vpl, rzk.CLAMP_RADIANCE, 0.05, p[2], p[3],
                                                other.cuda_stream))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        x += 1
        t = threading.Thread(target=fill)
        t.start()
        t.join()
        x += 1
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert status == [rzk.OK] and bool((x == 2).all())
    assert torch.equal(mat.view(torch.int32), want.view(torch.int32)) and torch.equal(vis, want_vis)
    ctx.check()
