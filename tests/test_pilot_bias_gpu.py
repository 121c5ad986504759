"""The bias gradients of the training convolutions are FP32 sums: against the 64-bit sums of the same
BF16 values, some of them far larger than the rest, the error is that of FP32 additions.

Bound: a term passes at most L = 14 tiles x 16 pixels of a thread + 36 threads + 296 blocks = 556
additions at the magnitude of the sum it ends in, each off by at most half a unit in the last
place with either sign: sqrt(L / 3) 2^-24 = 8.1e-7 of the largest partial sums, taken here of the
result's 2-norm."""
import pytest

from zb3d import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side,cin,cout", [(32, 128, 32, 32), (32, 128, 48, 48), (32, 64, 16, 32), (3, 37, 32, 16),
                                             (1, 8, 16, 16), (2, 17, 48, 16)])
def test_bias_sums(n, side, cin, cout):
    import torch
    err = ref = 0.0
    for seed in range(4):
        g = torch.Generator(device="cuda").manual_seed(seed)
        shape = (n, side, side, cout)
        dy = torch.randn(shape, device="cuda", generator=g)
        dy = (dy * torch.exp(4.0 * torch.randn(shape, device="cuda", generator=g))).bfloat16()
        x = torch.rand((n, side, side, cin), device="cuda", generator=g).bfloat16()
        dw = torch.zeros(cout, 9 * cin, device="cuda")
        db = torch.zeros(cout, device="cuda")
        assert N.lib().zb3d_pilot_conv3x3_wgrad(x.data_ptr(), dy.data_ptr(), n, side, side, cin, cout, dw.data_ptr(),
                                                db.data_ptr(), None) == 0
        torch.cuda.synchronize()
        want = dy.double().sum((0, 1, 2))
        err += float(((db.double() - want) ** 2).sum())
        ref += float((want ** 2).sum())
    assert (err / ref) ** 0.5 < 8.1e-7, (err / ref) ** 0.5
