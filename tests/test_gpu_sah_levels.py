"""The any-hit tree's device build (rzk_sah.cu) stops launching levels soon after the last one that
has nodes: a chain of shrinking triangles, of which each split peels off a few, keeps large nodes
past level 23."""
import numpy as np
import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ratio,most", [(600, 0.7, 32), (3000, 0.999, 16)])
def test_levels_launched(ctx, n, ratio, most):
    import torch
    from renzoku_b200 import rzk
    rng = np.random.default_rng(0)
    k = ratio ** np.arange(n)[:, None, None]
    v = 0.5 * k * [1, 0, 0] + [0, 0.3, 0.3] + rng.uniform(-0.08, 0.08, (n, 3, 3)) * k
    prim_v = np.zeros((n, 12), np.float32)
    prim_v[:, :9] = v.reshape(n, 9)
    mats = np.zeros(1, sg.MATERIAL_DTYPE)
    sc = sg.Scene("chain", np.full(n, sg.PRIM_TRIANGLE, np.int32), prim_v, np.zeros(n, np.int32),
                  np.zeros((n, 3), np.float32), np.full(n, sg.SURF_TWO_SIDED, np.int32), mats, sg.CameraSpec(width=8, height=8))
    agg = rzk.AggregateCuda(ctx, sc)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        agg.rebuild()
        torch.cuda.synchronize()
    names = [e.name for e in prof.events()]
    if not any("sah_small_kernel" in x for x in names):
        pytest.skip("no CUDA activity records here")
    assert 0 < sum("sah_large_kernel" in x for x in names) <= most
