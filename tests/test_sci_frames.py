"""GPU: exact scientific frames at the edges of the kernel's items (4, 8 or 16 frames of a leaf each):
frame counts around them, repeated and descending lists, cropped leaves, outputs whose rows are not
16-byte aligned -- dense frames and the cache against the oracle."""
import numpy as np
import pytest

from conftest import golden_asset

pytestmark = pytest.mark.gpu

LISTS = {"one": [3], "three": [0, 1, 2], "five": [15, 14, 2, 2, 0], "nine": list(range(4, 13)),
         "all": list(range(16)), "twice": list(range(16)) + list(range(15, -1, -1)) + [7]}


@pytest.mark.parametrize("name", ["sci_small", "sci_coarse", "sci_dense", "sci_dense_tb"])
@pytest.mark.parametrize("frames", list(LISTS.values()), ids=list(LISTS))
def test_frames(name, frames, vbt, cuda, oracle):
    torch = cuda
    path = golden_asset(name)
    a, f = vbt.Asset(path), oracle.load(path)
    X, Y, Z = a.dims
    n = X * Y * Z
    want = np.stack([f.frame(t) for t in frames]).reshape(len(frames), -1)
    tol = 1e-6 * float(np.ptp(want))     # a few roundings of the field's range
    for shift in (0, 1):                 # 16-byte aligned rows, and not
        buf = torch.full((len(frames) * n + shift + 4,), -7.0, device="cuda")
        a.decode_frames(frames, buf[shift:])
        a.sync_status()
        got = buf.cpu().numpy()
        assert (got[:shift] == -7.0).all() and (got[shift + want.size:] == -7.0).all()
        got = got[shift:shift + want.size].reshape(want.shape).astype(np.float64)
        assert np.abs(got - want).max() <= tol, (name, shift)
    cache = torch.full((len(frames), a.leaf_count, 512), -7.0, device="cuda")
    a.decode_cache(frames, cache)
    a.sync_status()
    got = cache.cpu().numpy()
    for j, t in enumerate(frames):
        assert np.abs(got[j].astype(np.float64) - f.cache(t)).max() <= tol, (name, t)
    a.close()
