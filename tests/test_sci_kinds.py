"""Every kind of scientific leaf -- 1 to 40 coefficients per control, the four event capacities, few and many
events to a bin and to the frames of an item, keys out of order, residual grids of 3^3 and 4^3 with 0 to 15 bits
and of the temporal basis -- as frames, cache, window, slice and point queries, against the oracle bit for bit
(the decode's sums and lerps are the oracle's operations in its order).  The lists differ in what a file
holds: `narrow` has at most four coefficients, codes of at most eight bits and a grid per frame."""
import numpy as np
import pytest

from sciimages import sci_image

pytestmark = pytest.mark.gpu

KINDS = {
    "narrow": [dict(keep=4), dict(keep=3, events=200), dict(keep=2, res=3, bits=6), dict(keep=1, res=4, bits=8),
               dict(keep=4, res=3, bits=3), dict(keep=4, events=700, tier=2, spread=(3, 9)), dict(keep=1),
               dict(keep=4, res=4, bits=5), dict(keep=4, events=100, swap=True), dict(keep=4, res=3, bits=2)],
    "wide": [dict(keep=12), dict(keep=6, events=200), dict(keep=5, events=64, tier=0), dict(keep=1, res=3, bits=6),
             dict(keep=3, res=4, bits=5, tkeep=4), dict(keep=7, res=3, bits=4, tkeep=16),
             dict(keep=8, res=4, bits=9, tkeep=5), dict(keep=2, events=900, tier=3, spread=(0, 5)),
             dict(keep=6, events=90, swap=True), dict(keep=9, res=4, bits=0, tkeep=3), dict(keep=33, res=3, bits=10),
             dict(keep=40, events=256), dict(keep=4, res=4, bits=15)],
    "basis": [dict(keep=4, res=4, bits=4, tkeep=8), dict(keep=2, res=3, bits=8, tkeep=1), dict(keep=1)],
    "events": [dict(keep=7, events=1024, tier=3), dict(keep=4, events=768, tier=2, fpb=16), dict(keep=8, events=64, tier=0)],
}


@pytest.mark.parametrize("name", list(KINDS))
@pytest.mark.parametrize("dims", [(24, 16, 32), (20, 9, 21)], ids=["whole", "cropped"])
def test_kinds(name, dims, vbt, cuda, oracle):
    T = 41
    image = sci_image(dims, T, KINDS[name], 3)
    a, f = vbt.Asset(data=image), oracle.load(image=image)
    a.build_page_table()
    X, Y, Z = dims
    L = a.leaf_count
    want = np.stack([f.frame(t) for t in range(T)])
    cache = np.stack([f.cache(t) for t in range(T)])

    def same(got, ref, *what):
        a.sync_status()
        got = got.cpu().numpy()
        bad = got.view(np.uint32) != ref.reshape(got.shape).view(np.uint32)
        assert not bad.any(), (name, *what, int(bad.sum()), np.argwhere(bad)[:3])

    for frames in ([0], [40, 2, 2], [5, 6, 7, 8, 9], list(range(T)), list(range(T)) + [12, 3, 40, 39]):
        dense = cuda.full((len(frames), Z, Y, X), -7.0, device="cuda")
        a.decode_frames(frames, dense)
        same(dense, want[frames], "frames", frames)
        out = cuda.full((len(frames), L, 512), -7.0, device="cuda")
        a.decode_cache(frames, out)
        same(out, cache[frames], "cache", frames)
    out = cuda.full((19, L, 512), -7.0, device="cuda")
    a.decode_window(11, 19, out)
    same(out, cache[11:30], "window")
    for z in (0, 5, Z - 1):
        rows = cuda.full((T, Y, X), -7.0, device="cuda")
        a.query_slice(z, 0, T, rows)
        same(rows, want[:, z], "slice", z)
    rng = np.random.default_rng(1)
    for n in (1, 5, 33, 40000):
        q = np.stack([rng.integers(0, k, n) for k in (X, Y, Z, T)], 1).astype(np.uint32)
        out = cuda.full((n,), -7.0, device="cuda")
        a.query_points(cuda.from_numpy(q.view(np.int32)).cuda(), out)
        same(out, want[q[:, 3], q[:, 2], q[:, 1], q[:, 0]], "points", n)
    a.close()
