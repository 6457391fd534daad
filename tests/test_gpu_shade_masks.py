"""The summing halves of the two-pass gather (shade_marked, shade_chunk in rzk_gather_dev.cuh) on
ballots that mark lanes without a receiver or without a material, as the words of an item whose
bounded wait gave up can: those lanes read no material and add nothing, the others' sums are those
of clean ballots."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def shade(ctx, tmp_path_factory):
    from renzoku_b200 import build
    so = tmp_path_factory.mktemp("shade") / "shade_masks.so"
    subprocess.run([build.NVCC, *build.FLAGS, "-shared", "-o", str(so), os.path.join(HERE, "shade_masks.cu")], check=True)
    return ctypes.CDLL(str(so)).shade


@pytest.mark.parametrize("n_recv,n_vpl", [(1, 1), (20, 31), (31, 32), (32, 33), (20, 100)])
def test_unwritten_ballots_mark_no_idle_lane(shade, n_recv, n_vpl):
    import torch
    from renzoku_b200 import rzk
    rng = np.random.default_rng(n_recv + n_vpl)
    recv = np.zeros(n_recv, sg.RECEIVER_DTYPE)
    recv["p"] = rng.uniform(0, 1, (n_recv, 3)) + [0, 1, 0]
    for f in ("ng", "ns", "n", "wo"):
        recv[f] = [0, -1, 0]
    recv["u"], recv["v"] = [1, 0, 0], [0, 0, 1]
    recv["mat"] = np.where(np.arange(n_recv) % 5 == 4, -1, 0)      # every fifth missed the scene
    vpls = np.zeros(n_vpl, sg.VPL_DTYPE)
    vpls["p"] = rng.uniform(0, 1, (n_vpl, 3)) * [1, 0.5, 1]
    for f in ("n", "nn", "wi"):
        vpls[f] = [0, 1, 0]
    vpls["u"], vpls["v"] = [1, 0, 0], [0, 0, 1]
    vpls["contrib"] = rng.uniform(0.1, 1, (n_vpl, 3))
    mats = np.zeros(1, sg.MATERIAL_DTYPE)
    mats["kd"] = 0.5
    active = np.zeros(32, bool)
    active[:n_recv] = recv["mat"] >= 0
    bits = np.uint32((active * (1 << np.arange(32, dtype=np.int64))).sum())
    noise = rng.integers(0, 1 << 32, n_vpl, dtype=np.uint64).astype(np.uint32)
    dev = [rzk.records_to_device(x) for x in (recv, vpls, mats)]
    out = []
    for words in (noise, noise & bits):
        m = torch.from_numpy(words.view(np.int32).copy()).cuda()
        o = torch.full((2, 32, 3), float("nan"), device="cuda")
        p = [ctypes.c_void_p(t.data_ptr()) for t in (*dev, m, o)]
        assert shade(p[0], n_recv, p[1], n_vpl, p[3], p[2], p[4]) == 0
        out.append(o.cpu().numpy())
    assert np.array_equal(out[0], out[1])
    assert (out[0][:, ~active] == 0).all() and np.array_equal(out[0][0], out[0][1])
    assert n_vpl < 31 or (out[0][0][active] > 0).all()
