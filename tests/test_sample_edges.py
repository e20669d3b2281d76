"""GPU: the density sampler at the edges of its fast path, bit for bit against the oracle: samples on and
one ulp beside control coordinates, leaf borders and the volume's faces, at +0, -0 and tiny positions,
and rays of length 0 (whose samples all coincide)."""
import numpy as np
import pytest

from conftest import golden_asset
from test_sample import check, params, run_both

pytestmark = pytest.mark.gpu


def places(extent):
    f = np.float32
    v = [f(0), f(-0.0), f(1e-38), f(1e-30), f(2.0 ** -64), f(2.0 ** -63), f(1e-6), f(0.5), f(extent - 1)]
    for leaf in range(0, extent, 8):
        v.append(f(leaf))
        for res in (4, 6):
            v += [f(leaf) + f(k) * (f(7) / f(res - 1)) for k in range(res)]
    v = np.array(v, np.float32)
    return np.concatenate([v, np.nextafter(v, f(-1)), np.nextafter(v, f(1e9))])


@pytest.mark.parametrize("name", ["tiny_density", "tiny_levelset"])
@pytest.mark.parametrize("steps,bins", [(1, 0), (3, 0), (17, 1)])
def test_places(name, steps, bins, vbt, cuda, oracle):
    a = vbt.Asset(golden_asset(name))
    dims, frames = a.dims, a.frames
    a.close()
    rng = np.random.default_rng(steps)
    rays = np.zeros((20000, 8), np.float32)
    for k in range(3):
        rays[:, k] = rng.choice(places(dims[k]), rays.shape[0])
    rays[:, 4] = 1.0
    rays[10000:, 7] = rng.choice(np.array([0.0, 1e-30, 8.0, 16.0], np.float32), 10000)   # along x, from these places
    p = params(vbt, render_mode=0, step_count=steps, frame_index=frames // 2, surface_model=bins)
    got, want = run_both(vbt, cuda, oracle, golden_asset(name), p, rays)
    check(got, want, (name, steps))
    assert np.abs(want).max() > 0
