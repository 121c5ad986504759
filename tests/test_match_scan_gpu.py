"""The scan kernel of spatial ssd / sad matching (block_step 4 and 8): its lists equal the CPU
oracle's exact lists with every number of block rows per CTA (and so every split of a block's
candidate rows into ranges), at displacement ranges around the row scan's step of four (odd
and even, the smallest, both tile layouts), with ragged widths (the clamped last block column),
with content full of equal distances, and with infinities and NaN among the pixels.  Threads
that launch differently shaped CTAs of one kernel at the same time do not disturb each other.
"""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import oracle as orc
import zb3d
from zb3d import _native as N
from zb3d import synth
from zb3d.device import DeviceFilter, unpack_list

pytestmark = pytest.mark.gpu


def content(kind, w, h, stride):
    p = synth.noisy_plane(w, h, 10.0, clip=5, stride=stride)
    if kind == "levels":  # a handful of levels: most distances have ties, many are zero
        p[:, :w] = np.round(p[:, :w] * 6.0) / 6.0
    if kind == "special":
        p[h // 2, w // 3] = np.inf
        p[3, 5] = -np.inf
        p[h - 9, w - 12] = np.nan
    return p


def force_rows(monkeypatch, path, rows):
    """A tuning cache that gives every geometry of this test `rows` block rows per CTA."""
    import torch
    c = torch.cuda.get_device_properties(0)
    monkeypatch.setenv("ZB3D_TUNE_CACHE", str(path))

    def add(w, h, pitch, bs, R, metric, clips=1, form=0):
        with open(path, "a") as f:
            f.write(f"sm{c.major}{c.minor}-{c.multi_processor_count}sm_w{w}_h{h}_p{pitch}_bs{bs}_R{R}_m{metric}"
                    f"_r0_c{clips}_f{form} 0 {rows}\n")
    return add


@pytest.mark.parametrize("rows", [1, 2, 4, 8])
@pytest.mark.parametrize("w,h,bs,R,metric,kind", [
    (77, 53, 8, 9, "ssd", "noise"),
    (140, 44, 4, 12, "ssd", "noise"),
    (133, 70, 4, 12, "sad", "noise"),
    (141, 61, 8, 9, "sad", "levels"),
    (65, 40, 4, 1, "ssd", "noise"),
    (70, 41, 4, 2, "sad", "noise"),
    (90, 57, 8, 3, "ssd", "levels"),
    (150, 50, 4, 15, "ssd", "noise"),
    (150, 50, 4, 16, "ssd", "levels"),
    (131, 49, 4, 12, "ssd", "special"),
    (131, 49, 8, 9, "sad", "special"),
    (8, 8, 8, 9, "ssd", "noise"),
])
def test_scan_lists_equal_oracle(w, h, bs, R, metric, kind, rows, monkeypatch, tmp_path):
    import torch
    pitch = (w + 31) // 32 * 32
    force_rows(monkeypatch, tmp_path / "tune.txt", rows)(w, h, pitch, bs, R, {"ssd": 0, "sad": 1}[metric])
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


def test_threads_with_differently_shaped_launches(monkeypatch, tmp_path):
    """Planes of one clip with 8 and 2 block rows per CTA (other shared-memory sizes of the same
    kernel), requested by 8 threads over 4 streams: every frame comes, and is the frame of one thread."""
    w, h, nf = 256, 144, 24
    add = force_rows(monkeypatch, tmp_path / "tune.txt", 8)
    add(w, h, 256, 4, 12, 0, form=-1)
    force_rows(monkeypatch, tmp_path / "tune.txt", 2)(w // 2, h // 2, 128, 4, 12, 0, form=-1)
    frames = [[synth.noisy_plane(pw, ph, 10.0, clip=6, frame=n, plane=p)
               for p, (pw, ph) in enumerate([(w, h), (w // 2, h // 2), (w // 2, h // 2)])] for n in range(nf)]
    clip = zb3d.Clip.from_frames(frames, family=zb3d.YUV, subsampling=(1, 1))
    kw = dict(sigma=[10.0] * 3, block_step=4, bm_range=12, extractor_exp=3)
    one = zb3d.BM3D(clip, num_streams=1, **kw)
    want = [[p.copy() for p in one.get_frame(n)] for n in range(nf)]
    many = zb3d.BM3D(clip, num_streams=4, **kw)
    with ThreadPoolExecutor(8) as pool:
        got = list(pool.map(many.get_frame, range(nf)))
    assert all(np.array_equal(a, b) for g, x in zip(got, want) for a, b in zip(g, x))
