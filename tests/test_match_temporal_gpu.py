"""The row kernel of the temporal search (ssd, ps_num 1 and 2, ps_range 2 to 6): its lists equal the
CPU oracle's for every window size, at planes smaller than a window and with windows cut by the
plane's edges, with content full of ties, with infinities and NaN, and with a number of blocks
that leaves the last warp's groups idle.  A source that does not start on 16 bytes gives the same lists.
"""
import numpy as np
import pytest

import oracle as orc
from zb3d import _native as N
from zb3d import synth
from zb3d.device import DeviceFilter, unpack_list

pytestmark = pytest.mark.gpu


def window(kind, w, h, stride, tw):
    out = []
    for t in range(tw):
        p = synth.noisy_plane(w, h, 12.0, clip=9, frame=t, motion=True, stride=stride)
        if kind == "levels":
            p[:, :w] = np.round(p[:, :w] * 5.0) / 5.0
        if kind == "special":
            p[h // 2, w // 2] = np.inf
            p[h // 3, w // 3] = np.nan
        out.append(p)
    return out


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("w,h,bs,R,radius,ps_num,P,kind", [
    (77, 53, 8, 9, 2, 2, 4, "noise"),
    (77, 53, 8, 9, 1, 1, 4, "noise"),
    (64, 40, 4, 7, 1, 2, 2, "noise"),
    (61, 47, 8, 9, 3, 2, 3, "noise"),
    (90, 33, 4, 5, 1, 2, 5, "noise"),
    (71, 60, 8, 9, 2, 2, 6, "noise"),
    (66, 50, 8, 9, 1, 2, 7, "noise"),
    (80, 48, 8, 9, 2, 2, 4, "levels"),
    (80, 48, 8, 9, 2, 2, 4, "special"),
    (8, 8, 8, 9, 2, 2, 4, "noise"),
    (9, 19, 8, 9, 1, 2, 4, "noise"),
    (32, 32, 8, 4, 16, 2, 4, "noise"),
])
def test_temporal_lists_equal_oracle(w, h, bs, R, radius, ps_num, P, kind, offset):
    import torch
    tw = 2 * radius + 1
    f = DeviceFilter(w, h, family=N.GRAY, num_frames=tw, sigma=[12.0], block_step=bs, bm_range=R, radius=radius,
                     ps_num=ps_num, ps_range=P, num_streams=1, match_form=0)
    lay = f.entries[0]
    planes = window(kind, w, h, lay.pitch, tw)
    d_src = torch.zeros(f.src_elems + 4, dtype=torch.float32, device="cuda")
    d_src[offset:offset + f.src_elems].copy_(torch.from_numpy(np.stack(planes).reshape(-1)))
    nbx, nby = (w - 8 + bs - 1) // bs + 1, (h - 8 + bs - 1) // bs + 1
    d_list = torch.zeros((nby, nbx, 8, 2), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    f.match(0, d_src.data_ptr() + 4 * offset, d_list.data_ptr())
    torch.cuda.synchronize()
    got = unpack_list(d_list.cpu().numpy())
    f.close()
    want = orc.match(orc.make_cfg(w, h, lay.pitch, [12.0 / 255.0], bs, R, radius, ps_num, P), planes)
    bad = np.any(got != want, axis=(2, 3))
    assert not bad.any(), f"{bad.sum()} of {bad.size} blocks differ; first {np.argwhere(bad)[:4].tolist()}"
