"""GPU: caches and dense frames of few frames, and slices (the kernels that read single frames from the
payload), bit for bit against the oracle: frame counts on both sides of the change to streamed leaves,
frames out of range, descending and repeated lists, cropped leaves, rows that are not 16-byte aligned,
every layer of the volume, leaves with unordered keys."""
import os

import numpy as np
import pytest

from conftest import golden_asset
from test_point_batches import _swap_keys

pytestmark = pytest.mark.gpu

LISTS = {"one": [5], "two": [-2, 3], "three": [7, 4, 4], "four": [0, 1, 2, 3], "five": [9, 3, 2, 2, 40],
         "nine": list(range(9))}


@pytest.fixture(params=["tiny_density", "tiny_levelset", "swapped"])
def pair(request, vbt, oracle, tmp_path):
    path = golden_asset("tiny_density" if request.param == "swapped" else request.param)
    if request.param == "swapped":
        with open(path, "rb") as g:
            raw = _swap_keys(g.read())
        path = os.path.join(tmp_path, "swapped.vbtp")
        with open(path, "wb") as h:
            h.write(raw)
    a = vbt.Asset(path)
    yield a, oracle.load(path)
    a.close()


def same(got, want):
    return np.array_equal(np.ascontiguousarray(got).view(np.uint32), np.ascontiguousarray(want).view(np.uint32))


@pytest.mark.parametrize("frames", list(LISTS.values()), ids=list(LISTS))
def test_frames(pair, frames, cuda):
    a, f = pair
    X, Y, Z = a.dims
    a.build_page_table()
    cache = cuda.full((len(frames), a.active_count, 512), -7.0, device="cuda")
    a.decode_cache(frames, cache)
    a.sync_status()
    got = cache.cpu().numpy()
    for j, t in enumerate(frames):
        assert same(got[j], f.cache(t).reshape(got[j].shape)), t
    n = X * Y * Z
    for shift in (0, 1):
        buf = cuda.full((len(frames) * n + shift + 4,), -7.0, device="cuda")
        a.decode_frames(frames, buf[shift:])
        a.sync_status()
        got = buf.cpu().numpy()
        assert (got[:shift] == -7.0).all() and (got[shift + len(frames) * n:] == -7.0).all()
        for j, t in enumerate(frames):
            assert same(got[shift + j * n:shift + (j + 1) * n], f.frame(t).reshape(-1)), (shift, t)


def test_layers(pair, cuda):
    a, f = pair
    X, Y, Z = a.dims
    t0, t1 = 2, 5
    want = np.stack([f.frame(t).reshape(Z, Y, X) for t in range(t0, t1)])
    for z in range(Z):
        for shift in (0, 1):
            buf = cuda.full(((t1 - t0) * X * Y + shift + 4,), -7.0, device="cuda")
            a.query_slice(z, t0, t1, buf[shift:])
            a.sync_status()
            got = buf.cpu().numpy()
            end = shift + (t1 - t0) * X * Y
            assert (got[:shift] == -7.0).all() and (got[end:] == -7.0).all()
            assert same(got[shift:end].reshape(t1 - t0, Y, X), want[:, z]), (z, shift)
