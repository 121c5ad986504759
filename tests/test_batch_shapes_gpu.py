"""A batch whose entries take different match tiles: at once and with queues, 8, 4 and 2 block rows,
one and two CTAs per SM, and the largest searches the work list takes (block_step 8, bm_range 32;
4, 41), hard threshold and Wiener: every window equals the window run alone."""
import pytest

from zb3d import _native as N
from zb3d import synth
from zb3d.device import DeviceFilter, process_batch

pytestmark = pytest.mark.gpu

SHAPES = [  # width, height, block_step, bm_range
    (133, 77, 4, 12),   # at once, 8 rows
    (141, 90, 8, 9),    # at once
    (96, 61, 8, 1),     # at once
    (150, 83, 8, 14),   # queues, 4 rows
    (101, 58, 8, 16),   # queues, 2 rows
    (140, 75, 4, 24),   # queues, 8 rows, one CTA per SM
    (77, 69, 8, 32),    # queues, 4 rows, one CTA per SM
    (79, 101, 4, 41),
    (8, 8, 8, 9),
]


@pytest.mark.parametrize("picks", [list(range(len(SHAPES))), [0], [1], [3], [4], [5], [6], [7]])
def test_mixed_shapes(picks, monkeypatch, tmp_path):
    import torch
    monkeypatch.setenv("ZB3D_AUTOTUNE", "0")
    jobs = []
    for i in picks:
        w, h, bs, R = SHAPES[i]
        for final in (False, True):
            f = DeviceFilter(w, h, family=N.GRAY, sigma=[10.0], block_step=bs, bm_range=R, extractor_exp=3, ref=final,
                             num_streams=1, match_form=0)
            lay = f.entries[0]
            src = torch.zeros(f.src_elems, dtype=torch.float32)
            v = src[lay.src_offset:lay.src_offset + lay.src_elems].view(lay.nclips, h, lay.pitch)
            for c in range(lay.nclips):
                v[c] = torch.from_numpy(synth.noisy_plane(w, h, 10.0 - 6 * c, clip=i, frame=c, stride=lay.pitch))
            jobs.append((f, src.cuda(), torch.zeros(f.dst_elems, dtype=torch.float32, device="cuda")))
    want = []
    for f, src, dst in jobs:
        f.run(src.data_ptr(), dst.data_ptr())
        torch.cuda.synchronize()
        want.append(dst.clone())
        dst.zero_()
    torch.cuda.synchronize()
    process_batch([(f, s.data_ptr(), d.data_ptr()) for f, s, d in jobs])
    torch.cuda.synchronize()
    for (f, _, d), x in zip(jobs, want):
        assert torch.equal(d, x)
        f.close()
