"""A batch of more plane entries than one work list holds (48), hard threshold and Wiener filters
mixed, odd sizes among them: every window equals the window run alone, in the synchronous call and
in a captured batch.  Chunks that give up in the first list end the batch with its status."""
import numpy as np
import pytest

import zb3d
from zb3d import _native as N
from zb3d import synth
from zb3d.device import Batch, DeviceFilter, process_batch

pytestmark = pytest.mark.gpu


def _jobs(torch, count=22):
    jobs = []
    for i in range(count):
        final = i % 3 == 2
        w, h = 48 + 2 * (i % 5) * 7, 40 + 2 * (i % 4) * 5
        f = DeviceFilter(w, h, family=N.YUV, subsampling=(1, 1), sigma=[8.0 + i] * 3, block_step=4 if i % 2 else 8,
                         bm_range=5 + i % 3, extractor_exp=3, ref=final, num_streams=1, match_form=0)
        src = torch.zeros(f.src_elems, dtype=torch.float32)
        for lay in f.entries:
            v = src[lay.src_offset:lay.src_offset + lay.src_elems].view(lay.nclips, lay.height, lay.pitch)
            for c in range(lay.nclips):
                v[c] = torch.from_numpy(synth.noisy_plane(lay.width, lay.height, 10.0 - 4 * c, clip=i, frame=c,
                                                          plane=lay.plane[0], stride=lay.pitch))
        jobs.append((f, src.cuda(), torch.zeros(f.dst_elems, dtype=torch.float32, device="cuda")))
    return jobs


def test_several_work_lists():
    import torch
    jobs = _jobs(torch)
    assert sum(len(f.entries) for f, _, _ in jobs) > 48
    want = []
    for f, src, dst in jobs:
        f.run(src.data_ptr(), dst.data_ptr())
        torch.cuda.synchronize()
        want.append(dst.clone())
    calls = [(f, s.data_ptr(), d.data_ptr()) for f, s, d in jobs]

    def check():
        torch.cuda.synchronize()
        for (_, _, d), x in zip(jobs, want):
            assert torch.equal(d, x)
            d.zero_()
    for _, _, d in jobs:
        d.zero_()
    torch.cuda.synchronize()
    process_batch(calls)
    check()
    torch.cuda.synchronize()
    with pytest.raises(zb3d.Error, match="gave up waiting"):
        process_batch(calls, wait_polls=1 << 10, unsatisfiable=True)
    for _, _, d in jobs:
        d.zero_()
    torch.cuda.synchronize()
    b = Batch(calls)
    st = torch.cuda.Stream()
    try:
        for _ in range(2):
            b.launch(st.cuda_stream)
            st.synchronize()
            b.status()
            check()
            torch.cuda.synchronize()
    finally:
        b.close()
