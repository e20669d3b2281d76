"""GPU: point queries at the edges of the kernel's batches (4 queries to a corner step, 32 to a warp's
batch, 128 and 1024 to a CTA of its chunks), against the oracle; unordered and FP32 keys included."""
import os
import struct

import numpy as np
import pytest

from conftest import golden_asset

pytestmark = pytest.mark.gpu

COUNTS = (1, 3, 4, 5, 31, 32, 33, 127, 129, 1023, 1025, 60001)


def queries(dims, frames, n, seed, sci):
    rng = np.random.default_rng(seed)
    q = np.empty((n, 4), np.uint32)
    for k in range(3):
        q[:, k] = rng.integers(0, dims[k], n)
    q[:, 3] = rng.integers(0, frames + (0 if sci else 2), n)
    return q


@pytest.mark.parametrize("name", ["tiny_density", "tiny_levelset", "sci_small", "sci_coarse", "sci_dense",
                                  "sci_dense_tb"])
def test_batch_edges(name, vbt, cuda, oracle):
    torch = cuda
    path = golden_asset(name)
    a, f = vbt.Asset(path), oracle.load(path)
    sci = a.profile == 2
    scale = float(np.ptp(f.frame(0))) if sci else 0.0
    for n in COUNTS:
        q = queries(a.dims, a.frames, n, n, sci)
        out = torch.full((n + 1,), -7.0, device="cuda")
        a.query_points(torch.from_numpy(q.view(np.int32)).cuda(), out)
        a.sync_status()
        got, want = out.cpu().numpy(), f.query(q)
        assert got[n] == -7.0, (name, n)
        if sci:   # one rounding of the field's range (bit for bit in test_sci_kinds.py)
            assert np.abs(got[:n].astype(np.float64) - want).max() <= 1e-6 * scale, (name, n)
        else:
            assert np.array_equal(got[:n].view(np.uint32), want.view(np.uint32)), (name, n)
    if not sci:   # outside the volume: no such voxel in any frame
        q = queries(a.dims, a.frames, 99, 5, False)
        q[::3, 0] = a.dims[0]
        q[1::3, 1] = a.dims[1] + 100
        q[2::3, 2] = 2 ** 31
        out = torch.full((99,), -7.0, device="cuda")
        a.query_points(torch.from_numpy(q.view(np.int32)).cuda(), out)
        a.sync_status()
        assert not out.any()
    a.close()


def _swap_keys(raw):
    """The file with the first two keys of the first control of every GRID4 / FINE6 leaf swapped."""
    b = bytearray(raw)
    leaves = struct.unpack_from("<I", b, 8 + 4 * 8)[0]
    off = np.frombuffer(raw, "<u4", leaves + 1, 52)
    for i in range(leaves):
        p = 52 + 4 * (leaves + 1) + 4 * int(off[i])
        head = struct.unpack_from("<I", b, p)[0]
        if head & 3 in (0, 2) or (head >> 2) & 3 == 1:
            continue
        desc = struct.unpack_from("<I", b, p + 8)[0]
        if (desc >> 16) & 255 < 2:
            continue
        k = p + 8 + 12 * ((head >> 6) & 7) ** 3 + 3 * (desc & 0xFFFF)
        b[k:k + 3], b[k + 3:k + 6] = b[k + 3:k + 6], b[k:k + 3]
    return bytes(b)


def test_unordered_keys(vbt, cuda, oracle, tmp_path):
    torch = cuda
    path = os.path.join(tmp_path, "swapped.vbtp")
    with open(golden_asset("tiny_density"), "rb") as g, open(path, "wb") as h:
        h.write(_swap_keys(g.read()))
    a, f = vbt.Asset(path), oracle.load(path)
    q = queries(a.dims, a.frames, 5000, 3, False)
    out = torch.empty(5000, device="cuda")
    a.query_points(torch.from_numpy(q.view(np.int32)).cuda(), out)
    a.sync_status()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), f.query(q).view(np.uint32))
    a.close()
