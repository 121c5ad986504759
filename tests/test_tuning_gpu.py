"""The matching shapes that entries get with the timing off (scan_shape)."""
import pytest

from zb3d import _native as N
from zb3d.device import DeviceFilter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,bs,R,metric,rows", [
    (3840, 2160, 4, 12, "ssd", 8),   # at once: 76,800 bytes, two CTAs per SM
    (3840, 2160, 4, 12, "sad", 8),
    (1920, 1080, 8, 13, "ssd", 8),   # 115,200 bytes
    (1920, 1080, 8, 14, "ssd", 4),   # queues: 109,568 bytes with 4 rows (at once with 8: 117,760)
    (3840, 2160, 8, 16, "ssd", 2),   # 95,744 bytes with 2 rows, 116,736 with 4
    (3840, 2160, 4, 24, "sad", 8),   # two CTAs only with 1 row: the most rows
    (3840, 2160, 4, 30, "sad", 8),   # one CTA per SM whatever the rows
    (640, 480, 8, 9, "ssd", 4),      # few CTAs
    (640, 480, 8, 16, "ssd", 2),
    (640, 480, 4, 24, "ssd", 1),
    (640, 480, 4, 30, "sad", 4),
])
def test_untimed_shapes(w, h, bs, R, metric, rows, monkeypatch, tmp_path):
    monkeypatch.setenv("ZB3D_AUTOTUNE", "0")
    monkeypatch.setenv("ZB3D_TUNE_CACHE", str(tmp_path / "tune.txt"))
    f = DeviceFilter(w, h, family=N.GRAY, sigma=[10.0], block_step=bs, bm_range=R, num_streams=1, match_form=0,
                     bm_error_s=metric)
    got = f.tuning(0)
    f.close()
    assert got == (0, rows)
    assert not (tmp_path / "tune.txt").exists()
