"""The pilot's training convolutions on buffers that do not start on 16 bytes (they are copied
element by element) give what aligned buffers give, on sizes with partial tiles, for every layer
shape: outputs bit for bit; weight and bias gradients, whose partial sums meet in any order,
within FP32 rounding of sums of about 1000 terms."""
import numpy as np
import pytest

from zb3d import _native as N

pytestmark = pytest.mark.gpu
SHAPES = [(16, 48), (48, 48), (48, 16), (16, 32), (32, 32), (32, 16), (16, 16)]


@pytest.mark.parametrize("cin,cout", SHAPES)
@pytest.mark.parametrize("n,h,w", [(1, 5, 7), (2, 17, 33), (1, 16, 16)])
def test_unaligned_buffers(cin, cout, n, h, w):
    import torch
    rng = np.random.default_rng(cin + cout + h)
    lib = N.lib()

    def buf(a, shift):  # bf16, `shift` elements past a 16-byte boundary
        t = torch.zeros(a.size + 16, dtype=torch.bfloat16, device="cuda")
        v = t[shift:shift + a.size]
        v.copy_(torch.from_numpy(a.reshape(-1)).to("cuda"))
        return v
    x = rng.uniform(-1, 1, (n, h, w, cin)).astype(np.float32)
    wgt = rng.normal(0, 0.1, (cout, 9, cin)).astype(np.float32)
    dy = rng.normal(0, 1, (n, h, w, cout)).astype(np.float32)
    bias = torch.from_numpy(rng.normal(0, 0.1, cout).astype(np.float32)).cuda()
    got = []
    for shift in (0, 2):
        xb, wb, db_ = buf(x, shift), buf(wgt, shift), buf(dy, shift)
        y = torch.zeros((n, h, w, cout), dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        assert lib.zb3d_pilot_conv3x3(xb.data_ptr(), n, h, w, cin, wb.data_ptr(), bias.data_ptr(), cout, 1, None,
                                      y.data_ptr(), None, None, None) == 0
        dw = torch.zeros((cout, 9, cin), device="cuda")
        db = torch.zeros(cout, device="cuda")
        assert lib.zb3d_pilot_conv3x3_wgrad(xb.data_ptr(), db_.data_ptr(), n, h, w, cin, cout, dw.data_ptr(),
                                            db.data_ptr(), None) == 0
        torch.cuda.synchronize()
        got.append((y, dw, db))
    assert torch.equal(got[0][0], got[1][0])
    xr = torch.nn.functional.pad(torch.from_numpy(x).to(torch.bfloat16).double(), (0, 0, 1, 1, 1, 1))
    dr = torch.from_numpy(dy).to(torch.bfloat16).double()
    want = torch.stack([torch.einsum("nhwo,nhwi->oi", dr, xr[:, t // 3:t // 3 + h, t % 3:t % 3 + w]) for t in range(9)], 1)
    for _, dw, db in got:  # sums of n * h * w products of order one: rounding 2^-24 of the partial sums
        tol = 2.0 ** -22 * (n * h * w) ** 0.5 * 8
        assert float((dw.cpu().double() - want).abs().max()) < tol
        assert float((db.cpu().double() - dr.sum((0, 1, 2))).abs().max()) < tol
