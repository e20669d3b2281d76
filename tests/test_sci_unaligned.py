"""Scientific windows and caches at outputs that do not start on 16 bytes or whose frames are not a multiple of
four floats apart: the same bits as at an aligned output, and nothing written between the frames."""
import pytest

from conftest import golden_asset
from sciimages import sci_image

pytestmark = pytest.mark.gpu

CROPPED = [dict(keep=4), dict(keep=4, events=150), dict(keep=3, res=3, bits=4), dict(keep=4, res=4, bits=6)]


@pytest.mark.parametrize("name", ["sci_small", "sci_dense", "cropped"])
def test_same_bits(name, vbt, cuda):
    a = vbt.Asset(data=sci_image((20, 9, 17), 20, CROPPED)) if name == "cropped" else vbt.Asset(golden_asset(name))
    a.build_page_table()
    n, size = 9, a.leaf_count * 512
    want = cuda.empty(n, size, device="cuda")
    a.decode_window(2, n, want)
    assert want.data_ptr() % 16 == 0 and size % 4 == 0
    for shift in range(4):
        for stride in (size, size + 1, size + 2, size + 512):
            for call in ("window", "cache"):
                buf = cuda.full((shift + n * stride + 4,), -7.0, device="cuda")
                if call == "window":
                    a.decode_window(2, n, buf[shift:], frame_stride=stride)
                else:
                    a.decode_cache(list(range(2, 2 + n)), buf[shift:], frame_stride=stride)
                a.sync_status()
                rows = buf[shift:shift + n * stride].view(n, stride)
                assert cuda.equal(rows[:, :size].view(cuda.int32), want.view(cuda.int32)), (shift, stride, call)
                assert bool((rows[:, size:] == -7.0).all()) and bool((buf[:shift] == -7.0).all())
                assert bool((buf[shift + n * stride:] == -7.0).all())
    a.close()
