"""The 6^3 fit of leaves whose controls take very different times: in part of a leaf every series is constant (a
few instructions), in the rest every frame is a key.  The kernel's bin spans lie where it staged the coarse
frames before, so a warp of quick series must not write its spans while a slow one still reads them.  Streams
and fitted grids against the CPU oracle's fits, bit for bit, and equal from run to run."""
import numpy as np
import pytest

from test_coarse_fit import check_leaf, control_profile, gpu_fit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 2, 5, 24, 25, 49])
def test_uneven_series(vbt, cuda, oracle, T):
    from oracle.oracle import VoKeyframeProfile
    dims = X, Y, Z = 64, 64, 32
    n = X * Y * Z // 512
    rng = np.random.default_rng(T)
    frames = rng.normal(0, 1, (T, Z, Y, X)).astype(np.float32)
    for bz in range(Z // 8):      # the quiet half of a leaf: its lower layers, its upper ones, every other layer
        quiet = [slice(0, 4), slice(4, 8), slice(0, 8, 2), slice(1, 8, 2)][bz]
        frames[:, 8 * bz:8 * bz + 8][:, quiet] = 0.25
    got = gpu_fit(vbt, cuda, frames.reshape(T, -1), dims, list(range(n)))
    recon = cuda.from_numpy(got["recon"]).cuda()
    grid = cuda.from_numpy(got["grid"]).cuda()
    leaves = cuda.arange(n, dtype=cuda.int32, device="cuda")
    runs = []
    for _ in range(3):
        o = dict(desc=cuda.full((n, 216), -1, dtype=cuda.int32, device="cuda"),
                 bins=cuda.full((n, 216, 8), 255, dtype=cuda.uint8, device="cuda"),
                 key_frames=cuda.zeros((n, 216 * T), dtype=cuda.int16, device="cuda"),
                 key_values=cuda.zeros((n, 216 * T), dtype=cuda.float32, device="cuda"),
                 key_count=cuda.full((n,), -1, dtype=cuda.int32, device="cuda"),
                 required=cuda.zeros(n, dtype=cuda.uint8, device="cuda"),
                 grid=cuda.full((n, 216, T), float("nan"), dtype=cuda.float32, device="cuda"))
        vbt.fine6_fit(recon, dims, leaves, control_profile(vbt.KeyframeProfile), grid, o["desc"], o["bins"],
                      o["key_frames"], o["key_values"], o["key_count"], o["required"], o["grid"])
        runs.append(o)
    cuda.cuda.synchronize()
    for o in runs[1:]:
        assert all(cuda.equal(o[k], runs[0][k]) for k in o)
    fine = {k: v.cpu().numpy() for k, v in runs[0].items()}
    vol = got["recon"].reshape(T, Z // 8, 8, Y // 8, 8, X // 8, 8).transpose(0, 1, 3, 5, 2, 4, 6).reshape(T, n, 512)
    for li in range(n):
        want = oracle.fine6_fit(np.ascontiguousarray(vol[:, li].T), (8, 8, 8), control_profile(VoKeyframeProfile),
                                got["grid"][li])
        check_leaf(fine, li, want, T)
