"""The matching shapes that entries get without a timing: the only candidate where the rules of
tune_entry leave one (many block rows per CTA give enough CTAs, or taller tiles leave one CTA per
SM), timing or not, and with the timing off 4 block rows only where that is a candidate."""
import pytest

from zb3d import _native as N
from zb3d.device import DeviceFilter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("autotune", ["0", "1"])
@pytest.mark.parametrize("w,h,bs,R,metric,rows,only", [
    (3840, 2160, 4, 12, "ssd", 8, True),   # 31 x 68 CTAs with 8 rows: over 8 per SM
    (3840, 2160, 4, 12, "sad", 8, True),
    (3840, 2160, 4, 24, "sad", 1, True),   # 113,408 bytes with 1 row, two CTAs per SM; 119,168 with 2
    (3840, 2160, 8, 16, "ssd", 2, True),   # 95,744 bytes with 2 rows; 116,736 with 4
    (3840, 2160, 4, 30, "sad", 8, True),   # 137,216 bytes with 1 row: one CTA per SM whatever the rows
    (640, 480, 4, 30, "sad", 4, False),
    (640, 480, 8, 16, "ssd", 2, False),    # the same tiles, few CTAs: 2 and 1 rows are candidates
    (640, 480, 8, 9, "ssd", 4, False),     # 96,768 bytes with 4 rows
])
def test_untimed_shapes(w, h, bs, R, metric, rows, only, autotune, monkeypatch, tmp_path):
    monkeypatch.setenv("ZB3D_AUTOTUNE", autotune)
    monkeypatch.setenv("ZB3D_TUNE_CACHE", str(tmp_path / "tune.txt"))
    f = DeviceFilter(w, h, family=N.GRAY, sigma=[10.0], block_step=bs, bm_range=R, num_streams=1, match_form=0,
                     bm_error_s=metric)
    got = f.tuning(0)
    f.close()
    if only or autotune == "0":
        assert got == (0, rows)
    else:
        assert got[0] == 0 and got[1] in (1, 2, 4, 8)
    assert (tmp_path / "tune.txt").exists() == (autotune == "1" and not only)
