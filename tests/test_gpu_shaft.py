"""The shaft of a packet's shadow segments (Shaft in rzk_gather_dev.cuh) where its margin meets
the segments exactly: the smallest offset of the receivers from the VPL along one axis equals the
margin 8e-6 times the packet's size, so that the widened interval starts at zero.  The packet
kernels give the per-thread kernel's image bit for bit there, and one float to either side."""
import numpy as np
import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu


def _grid(axis, size, k):
    """A two-sided wall of k x k quads half way up, over three quarters of the first side axis."""
    a, b = (axis + 1) % 3, (axis + 2) % 3
    v = np.zeros((k, k, 4, 3), np.float32)
    edge_a = np.linspace(-0.5, 0.25, k + 1) * size
    edge_b = np.linspace(-1.0, 1.0, k + 1) * size
    for c, (i, j) in enumerate(((0, 0), (1, 0), (1, 1), (0, 1))):
        v[:, :, c, a] = edge_a[i:k + i, None]
        v[:, :, c, b] = edge_b[None, j:k + j]
        v[:, :, c, axis] = 0.5 * size
    n = k * k
    mats = np.zeros(1, sg.MATERIAL_DTYPE)
    mats["kd"] = 0.5
    return sg.Scene("wall", np.full(n, sg.PRIM_QUAD, np.int32), v.reshape(n, 12), np.zeros(n, np.int32),
                    np.zeros((n, 3), np.float32), np.full(n, sg.SURF_TWO_SIDED, np.int32), mats,
                    sg.CameraSpec(width=8, height=8))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("size,k", [(1.0, 1), (1.0, 12), (0.37, 5), (55.5, 3)])
@pytest.mark.parametrize("step", [-1, 0, 1])
def test_margin_equal_to_the_smallest_offset(ctx, axis, size, k, step):
    from renzoku_b200 import rzk
    size = np.float32(size)
    agg = rzk.AggregateCuda(ctx, _grid(axis, size, k))
    a, b = (axis + 1) % 3, (axis + 2) % 3
    margin = np.float32(8e-6) * size
    if step:
        margin = np.nextafter(margin, np.float32(np.inf if step > 0 else -np.inf), dtype=np.float32)
    rng = np.random.default_rng(5)
    n = 96                                     # every packet of 32 holds the smallest offset
    recv = np.zeros(n, sg.RECEIVER_DTYPE)
    recv["p"][:, axis] = size
    recv["p"][:, a] = np.where(np.arange(n) % 8 == 0, margin, rng.uniform(0.01, 0.99, n).astype(np.float32) * size)
    recv["p"][:, b] = rng.uniform(-0.9, 0.9, n).astype(np.float32) * size
    for f in ("ng", "ns", "n", "wo"):
        recv[f][:, axis] = -1.0
    recv["u"][:, a] = recv["v"][:, b] = 1.0
    vpls = np.zeros(3, sg.VPL_DTYPE)           # all at the origin
    for f in ("n", "nn", "wi"):
        vpls[f][:, axis] = 1.0
    vpls["u"][:, a] = vpls["v"][:, b] = 1.0
    vpls["contrib"] = rng.uniform(0.5, 2.0, (3, 3))
    ev = rzk.VirtualPointLightCuda(agg, rzk.CLAMP_NONE, 0.0)
    r, v = rzk.records_to_device(recv), rzk.records_to_device(vpls)
    want = ev.gather(r, n, v, 3, variant=7).cpu().numpy()
    dark = (want == 0).all(1)
    assert dark[::8].all() and 0 < (~dark).sum() < n
    for variant in (0, 1, 3):
        got = ev.gather(r, n, v, 3, variant=variant).cpu().numpy()
        assert np.array_equal(got, want), variant
    ctx.check()
