"""Tensor-core F-engine: the split of (element, 32-spectrum group) work over the CTAs.
A call's bits do not depend on where the split falls: every element comes out as it
does in a call of its own (fewer groups than SMs, about as many, several elements to
a CTA, ragged ends)."""
import pytest
import torch

from x16util import unswizzle_x16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne,ntaps,nsp,q8", [(3, 8, 9, False), (5, 4, 1000, False), (152, 8, 32, True),
                                             (153, 4, 33, False), (19, 8, 257, True),
                                             (331, 4, 40, False)])
def test_split_does_not_show(mdt, cuda, ne, ntaps, nsp, q8):
    nch = 1024
    g = torch.Generator(device="cuda")
    g.manual_seed(ne + nsp)
    iq = torch.randint(-128, 128, (nsp + ntaps - 1, ne, nch, 2), generator=g, device="cuda",
                       dtype=torch.int32).to(torch.int8)
    win = torch.empty(nch * ntaps, dtype=torch.float32, device="cuda")
    mdt.window_hamming_sinc(nch, ntaps, win)
    qs = torch.full((nch,), 0.01, dtype=torch.float32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(x, n):
        X16 = torch.zeros(mdt.x16_bytes(n, nch, nsp), dtype=torch.uint8, device="cuda")
        if q8:
            mdt.fengine_tc_q8(n, nch, ntaps, nsp, x, win, X16, qs, err)
        else:
            mdt.fengine_tc(n, nch, ntaps, nsp, x, win, X16, err, scale=2.0 ** -6)
        return unswizzle_x16(X16.cpu().numpy(), nch, nsp, n, -(-n // 16) * 16)

    got = run(iq, ne)
    for e in sorted({0, 1, ne // 2, ne - 2, ne - 1}):
        assert (run(iq[:, e:e + 1].contiguous(), 1)[:, :, 0] == got[:, :, e]).all(), e
    assert err.item() == 0
