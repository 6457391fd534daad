"""The pool of per-call scratch (CallScratch in rzk_internal.cuh): it keeps at most 256 MB that no
call uses, and serves threads and streams while the last context ends."""
import ctypes
import os
import subprocess
import sys

import pytest

from renzoku_b200 import scenegen as sg

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KEEP = 256 << 20


def test_large_scratch_is_given_back(ctx):
    import torch
    from renzoku_b200 import rzk
    agg = rzk.AggregateCuda(ctx, sg.room_objects(20, 8, 8, seed_geo=3, seed_mat=4))
    out = torch.zeros(96 * 1000, dtype=torch.uint8, device="cuda")
    count = torch.zeros(1, dtype=torch.int32, device="cuda")

    def spawn(n):   # one record of scratch per particle and bounce
        assert agg.lib.rzk_vpl_generate(agg.h, 7, n, 4, ctypes.c_void_p(out.data_ptr()), 1000,
                                        ctypes.c_void_p(count.data_ptr()), rzk._stream_ptr()) == rzk.OK
    spawn(1000)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    spawn(4 << 20)   # 1.2 GB
    assert before - torch.cuda.mem_get_info()[0] <= KEEP + (64 << 20)
    ctx.check()


def test_scratch_while_contexts_end(gpu_lib):
    env = dict(os.environ, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, os.path.join(ROOT, "tests", "pool_worker.py")], env=env, timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0 and "worker ok" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
