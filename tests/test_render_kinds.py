"""Render-temporal leaves of every grid resolution, of FP32 keys, with fine grids and Mode2 shells -- files whose
leaves are mostly of the common shape (FP16 keys, 4^3 grids, 6^3 fine grids) and files whose leaves are not --
as caches, windows and dense frames of frame counts on both sides of the rules for few frames, slices and point queries,
against the oracle bit for bit."""
import numpy as np
import pytest

from renderimages import render_image

pytestmark = pytest.mark.gpu

KINDS = {
    "fp32": [dict(res=4, fp32=True), dict(res=4, fine=6, fp32=True, fp32_second=True), None,
             dict(res=4, shell=0.4, fp32=True, fp32_second=True), dict(res=4, fine=6, fp32_second=True)],
    "grids": [dict(res=5, fine=7), dict(res=3, fine=5), dict(res=7), dict(res=2, shell=1.0), None, dict(res=4, fine=5),
              dict(res=6, fine=6), dict(res=1, fine=2), dict(res=5, shell=0.2)],
    "mostly common": [dict(res=4), dict(res=4, fine=6), dict(res=4, shell=0.3), dict(res=4), dict(res=5, fine=6),
                      dict(res=4, shell=0.9), dict(res=4, fine=6), dict(res=4, fp32=True)],
}
COUNTS = (1, 2, 3, 4, 6, 7, 9, 33)


@pytest.mark.parametrize("name", list(KINDS))
@pytest.mark.parametrize("dims", [(24, 16, 24), (20, 9, 21)], ids=["whole", "cropped"])
def test_kinds(name, dims, vbt, cuda, oracle):
    T = 33
    image = render_image(dims, T, KINDS[name], 7)
    a, f = vbt.Asset(data=image), oracle.load(image=image)
    a.build_page_table()
    X, Y, Z = dims
    want = np.stack([f.frame(t) for t in range(T)])
    cache = np.stack([f.cache(t) for t in range(T)])

    def same(got, ref, *what):
        a.sync_status()
        got = got.cpu().numpy()
        bad = got.view(np.uint32) != ref.reshape(got.shape).view(np.uint32)
        assert not bad.any(), (name, *what, int(bad.sum()), np.argwhere(bad)[:3])

    for n in COUNTS:
        for frames in (list(range(T - n, T)), [(5 * j) % T for j in range(n)]):
            out = cuda.full((n, a.active_count, 512), -7.0, device="cuda")
            a.decode_cache(frames, out)
            same(out, cache[frames], "cache", frames)
            dense = cuda.full((n, Z, Y, X), -7.0, device="cuda")
            a.decode_frames(frames, dense)
            same(dense, want[frames], "dense", frames)
    for t0, n in ((0, 2), (3, 20), (1, 32)):
        out = cuda.full((n, a.active_count, 512), -7.0, device="cuda")
        a.decode_window(t0, n, out, frame_stride=out.stride(0))
        same(out, cache[t0:t0 + n], "window", t0, n)
    for z in range(Z):
        rows = cuda.full((5, Y, X), -7.0, device="cuda")
        a.query_slice(z, 14, 19, rows)
        same(rows, want[14:19, z], "slice", z)
    rng = np.random.default_rng(2)
    q = np.stack([rng.integers(0, k, 20000) for k in (X, Y, Z, T)], 1).astype(np.uint32)
    out = cuda.full((len(q),), -7.0, device="cuda")
    a.query_points(cuda.from_numpy(q.view(np.int32)).cuda(), out)
    same(out, want[q[:, 3], q[:, 2], q[:, 1], q[:, 0]], "points")
    a.close()
