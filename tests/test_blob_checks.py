"""rzk_scene_deserialize on damaged blobs, checked on the host before anything reaches a device:
an any-hit tree of another size than its triangles give, links and triangles out of range."""
import ctypes
import struct

import numpy as np
import pytest

N, NODES = 2, 3   # two triangles under one inner node


def _tree(codes, slots):
    t = np.zeros((slots, 8), np.float32)
    t.view(np.int32)[1:1 + len(codes), 3] = codes[:slots - 1]
    return t.tobytes()


def _blob(nodes=(1, -1, -2), trav=(1, -1, -2), trav_slots=2 * N, n_nodes=NODES, perm=(1, 0), depth=1, light_tris=2):
    f = lambda k: bytes(4 * k)
    cap = 2 * N
    light = bytearray(16 * 11 + 16)
    struct.pack_into("<i", light, 16 * 11 + 12, light_tris)
    tb = 32 * trav_slots
    arrays = [f(9 * N), f(3 * N), f(N), bytes(16), bytes(48), f(3 * N), f(3 * N), f(N), f(3 * N), f(3 * N), f(N), f(N),
              np.array(perm, np.int32).tobytes(), f(cap), f(cap), f(cap), f(cap), f(cap), f(3 * cap), f(3 * cap),
              _tree(nodes, cap + 1), bytes(48 * N), bytes(32 * N), b"", _tree(trav, trav_slots), bytes(light), f(1), f(1)]
    head = struct.pack("<8s2I10i8f4Q", b"RZKSCN01", 1, len(arrays), N, n_nodes, 2, 1, 1, 1, 0, depth, 1, 0,
                       1e-3, 0, 0, 0, 1, 1, 1, 0, tb, 0, 0, 0)
    return head + b"".join(struct.pack("<Q", len(a)) + a for a in arrays)


def _restore(blob):
    from renzoku_b200 import rzk
    ctx, out = ctypes.create_string_buffer(1024), ctypes.c_void_p()   # a context no check looks into
    return rzk.load().rzk_scene_deserialize(ctx, blob, len(blob), None, ctypes.byref(out)), rzk.ERR_INVALID


@pytest.fixture(autouse=True)
def no_device():
    import torch
    if torch.cuda.is_available():
        pytest.skip("a blob that passes the checks would go on to the device")


@pytest.mark.parametrize("depth", [1, 0, 7, -3])
def test_whole_blob_passes_the_checks(depth):
    status, invalid = _restore(_blob(depth=depth))
    assert status not in (0, invalid)   # no device to restore to


@pytest.mark.parametrize("damage", [
    dict(trav_slots=N), dict(trav_slots=2 * N - 1), dict(trav_slots=2 * N + 1),       # sizes that agree with the header
    dict(trav=(1, -1, -3)), dict(trav=(1, -2 ** 31, -2)), dict(trav=(2, -1, -2)),     # triangles, children past the end
    dict(trav=(0, -1, -2)), dict(trav=(1, 1, -2)), dict(trav=(2 ** 31 - 1, -1, -2)), dict(trav=(-1, -1, -2)),
    dict(nodes=(1, -1, -4)), dict(nodes=(5, -1, -2)), dict(n_nodes=2), dict(n_nodes=4), dict(n_nodes=100000),
    dict(perm=(0, 2)), dict(perm=(-1, 0)), dict(light_tris=3), dict(light_tris=0)])
def test_damaged_blobs_are_refused(damage):
    status, invalid = _restore(_blob(**damage))
    assert status == invalid, damage
