"""Event bins of a bad file that reach past their leaf and past the payload: the search's reads there are the
checked ones, so the call ends with an out-of-bounds status, and every value is the oracle's (which reads zeros
past the payload, where the reference throws)."""
import struct

import numpy as np
import pytest

from sciimages import sci_image

pytestmark = pytest.mark.gpu


def bad_image(dims=(16, 8, 16), T=20, end=60000):
    """Events in every leaf; bin 5 of leaf 1 (whose own section lies inside the payload) ends at event `end`."""
    kinds = [dict(keep=4, events=200), dict(keep=6, events=200, swap=True)]
    image = sci_image(dims, T, kinds, 9)
    L, scales = struct.unpack_from("<I", image, 8 + 32)[0], struct.unpack_from("<I", image, 8 + 40)[0]
    off = image[52 + 4 * scales:52 + 4 * scales + 4 * (L + 1)].view(np.uint32)
    leaf = 52 + 4 * scales + 4 * (L + 1) + 4 * int(off[1])
    keep = ((struct.unpack_from("<I", image, leaf)[0] >> 2) & 63) + 1
    struct.pack_into("<H", image, leaf + 4 + 64 * (keep + 1) + 68 + 2 * 6, end)
    return image


def test_bad_bins(vbt, cuda, oracle):
    dims, T = (16, 8, 16), 20
    image = bad_image(dims, T)
    a, f = vbt.Asset(data=image), oracle.load(image=image)
    a.build_page_table()
    X, Y, Z = dims
    want = np.stack([f.frame(t) for t in range(T)])

    def same(got, ref):
        with pytest.raises(vbt.VbtError) as e:
            a.sync_status()
        assert e.value.status == 11
        assert np.array_equal(got.cpu().numpy().view(np.uint32), ref.reshape(got.shape).view(np.uint32))

    dense = cuda.empty(T, Z, Y, X, device="cuda")
    a.decode_frames(list(range(T)), dense)
    same(dense, want)
    rows = cuda.empty(T, Y, X, device="cuda")
    a.query_slice(3, 0, T, rows)
    same(rows, want[:, 3])
    q = np.stack(np.meshgrid(range(X), range(Y), range(Z), range(T), indexing="ij"), -1).reshape(-1, 4).astype(np.uint32)
    out = cuda.empty(len(q), device="cuda")
    a.query_points(cuda.from_numpy(q.view(np.int32)).cuda(), out)
    same(out, want[q[:, 3], q[:, 2], q[:, 1], q[:, 0]])
    a.close()
