"""The GPU control fits at the edges of their shapes: frame counts around the frames of the coarse grid that
the 6^3 fit stages at a time (24), around a key mask word (32), one and two frames, and series with a key at
every frame, whose key runs cross mask words and whose bin spans pass a byte.  Streams and fitted grids
against the CPU oracle's fits, bit for bit."""
import numpy as np
import pytest

from test_coarse_fit import check_leaf, control_profile, gpu_fit, oracle_fit

pytestmark = pytest.mark.gpu


def series(T, V, noise, seed):
    rng = np.random.default_rng(seed)
    t = np.arange(T)[:, None]
    c, width = rng.uniform(0, T, V), rng.uniform(1, 6, V)
    return (rng.uniform(0.2, 1.0, V) * np.exp(-((t - c) / width) ** 2) + rng.normal(0, noise, (T, V))).astype(np.float32)


@pytest.mark.parametrize("T,noise", [(1, 0.01), (2, 0.01), (23, 0.01), (24, 0.0), (25, 0.3), (32, 0.3), (33, 0.3),
                                     (49, 0.05), (96, 0.5), (160, 0.5)])
def test_fine_fit(vbt, cuda, oracle, T, noise):
    from oracle.oracle import VoKeyframeProfile
    dims = X, Y, Z = 11, 8, 13
    leaves = list(range(4))
    frames = series(T, X * Y * Z, noise, T)
    got = gpu_fit(vbt, cuda, frames, dims, leaves)
    recon = cuda.from_numpy(got["recon"]).cuda()
    n = len(leaves)
    o = dict(desc=cuda.full((n, 216), -1, dtype=cuda.int32, device="cuda"),
             bins=cuda.full((n, 216, 8), 255, dtype=cuda.uint8, device="cuda"),
             key_frames=cuda.zeros((n, 216 * T), dtype=cuda.int16, device="cuda"),
             key_values=cuda.zeros((n, 216 * T), dtype=cuda.float32, device="cuda"),
             key_count=cuda.full((n,), -1, dtype=cuda.int32, device="cuda"),
             required=cuda.zeros(n, dtype=cuda.uint8, device="cuda"),
             grid=cuda.full((n, 216, T), float("nan"), dtype=cuda.float32, device="cuda"))
    vbt.fine6_fit(recon, dims, cuda.tensor(leaves, dtype=cuda.int32, device="cuda"),
                  control_profile(vbt.KeyframeProfile), cuda.from_numpy(got["grid"]).cuda(), o["desc"], o["bins"],
                  o["key_frames"], o["key_values"], o["key_count"], o["required"], o["grid"])
    cuda.cuda.synchronize()
    fine = {k: v.cpu().numpy() for k, v in o.items()}
    vol = got["recon"].reshape(T, Z, Y, X)
    for li in leaves:
        check_leaf(got, li, oracle_fit(oracle, got["recon"], dims, li), T)
        bx, bz = li % 2, li // 2
        sub = vol[:, 8 * bz:8 * bz + 8, :, 8 * bx:8 * bx + 8]
        lt = np.zeros((T, 8, 8, 8), np.float32)
        lt[:, :sub.shape[1], :, :sub.shape[3]] = sub
        want = oracle.fine6_fit(np.ascontiguousarray(lt.reshape(T, 512).T), (sub.shape[3], 8, sub.shape[1]),
                                control_profile(VoKeyframeProfile), got["grid"][li])
        check_leaf(fine, li, want, T)


@pytest.mark.parametrize("T", [255, 257, 700])
def test_key_at_every_frame(vbt, cuda, oracle, T):
    dims = (8, 8, 8)
    frames = series(T, 512, 0.5, T)
    got = gpu_fit(vbt, cuda, frames, dims, [0])
    assert int(got["key_count"][0]) > 32 * T
    check_leaf(got, 0, oracle_fit(oracle, got["recon"], dims, 0), T)
