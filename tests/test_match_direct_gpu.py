"""The scan kernel of spatial ssd / sad matching with a warp per block row and candidates inserted
at once: its lists equal the CPU oracle's exact lists, on the sizes, ranges and contents on which
test_match_scan_gpu.py checks the form with queues."""
import numpy as np
import pytest

import oracle as orc
from test_match_scan_gpu import content
from zb3d import _native as N
from zb3d.device import DeviceFilter, unpack_list

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [2, 4, 8])
@pytest.mark.parametrize("w,h,bs,R,metric,kind", [
    (77, 53, 8, 9, "ssd", "noise"),
    (140, 44, 4, 12, "ssd", "noise"),
    (141, 61, 8, 9, "sad", "levels"),
    (65, 40, 4, 1, "ssd", "noise"),
    (70, 41, 4, 2, "sad", "noise"),
    (150, 50, 4, 15, "ssd", "noise"),
    (150, 50, 4, 16, "ssd", "levels"),
    (131, 49, 4, 12, "ssd", "special"),
    (131, 49, 8, 9, "sad", "special"),
    (8, 8, 8, 9, "ssd", "noise"),
])
def test_direct_lists_equal_oracle(w, h, bs, R, metric, kind, rows, monkeypatch, tmp_path):
    import torch
    pitch = (w + 31) // 32 * 32
    c = torch.cuda.get_device_properties(0)
    path = tmp_path / "tune.txt"
    path.write_text(f"sm{c.major}{c.minor}-{c.multi_processor_count}sm_w{w}_h{h}_p{pitch}_bs{bs}_R{R}"
                    f"_m{('ssd', 'sad').index(metric)}_r0_c1_f0 0 {rows} 1\n")
    monkeypatch.setenv("ZB3D_TUNE_CACHE", str(path))
    f = DeviceFilter(w, h, family=N.GRAY, sigma=[10.0], block_step=bs, bm_range=R, num_streams=1, match_form=0,
                     bm_error_s=metric)
    assert f.tuning(0) == (0, rows)
    plane = content(kind, w, h, f.entries[0].pitch)
    d_src = torch.from_numpy(plane.reshape(-1)).cuda()
    nbx, nby = (w - 8 + bs - 1) // bs + 1, (h - 8 + bs - 1) // bs + 1
    d_list = torch.zeros((nby, nbx, 8, 2), dtype=torch.int32, device="cuda")
    f.match(0, d_src.data_ptr(), d_list.data_ptr())
    torch.cuda.synchronize()
    got = unpack_list(d_list.cpu().numpy())
    f.close()
    want = orc.match(orc.make_cfg(w, h, plane.shape[1], [10.0 / 255.0], bs, R, bm_error=metric), [plane])
    bad = np.any(got != want, axis=(2, 3))
    assert not bad.any(), f"{bad.sum()} of {bad.size} blocks differ; first {np.argwhere(bad)[:4].tolist()}"
