"""Block steps other than 4 and 8 on small planes (a warp per block, zb_match_blocks) and just past
the size where a lane pair takes over: lists equal the CPU oracle's exact lists."""
import numpy as np
import pytest

import oracle as orc
from zb3d import _native as N
from zb3d import synth
from zb3d.device import DeviceFilter, unpack_list

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["ssd", "sad", "zssd", "zsad"])
@pytest.mark.parametrize("w,h,bs,R", [(161, 53, 5, 9), (61, 47, 3, 7), (9, 8, 1, 4), (55, 55, 1, 2), (56, 57, 1, 2)])
def test_lists_equal_oracle(w, h, bs, R, metric):
    import torch
    f = DeviceFilter(w, h, family=N.GRAY, sigma=[10.0], block_step=bs, bm_range=R, num_streams=1, match_form=0,
                     bm_error_s=metric)
    plane = synth.noisy_plane(w, h, 10.0, clip=11, stride=f.entries[0].pitch)
    plane[:, :w] = np.round(plane[:, :w] * 40.0) / 40.0  # ties
    d_src = torch.from_numpy(plane.reshape(-1)).cuda()
    nbx, nby = (w - 8 + bs - 1) // bs + 1, (h - 8 + bs - 1) // bs + 1
    d_list = torch.zeros((nby, nbx, 8, 2), dtype=torch.int32, device="cuda")
    f.match(0, d_src.data_ptr(), d_list.data_ptr())
    torch.cuda.synchronize()
    got = unpack_list(d_list.cpu().numpy())
    f.close()
    want = orc.match(orc.make_cfg(w, h, plane.shape[1], [10.0 / 255.0], bs, R, bm_error=metric), [plane])
    assert np.array_equal(got, want)
