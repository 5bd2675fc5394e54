"""Spectrum-block F-engines (blocked FP32, f16 / bf16 and int8 operands) where one
block takes several 8-spectrum groups: more groups than the GPU holds blocks, a last
chunk that Nsp does not fill, padded rows, each transform size and the general tap
count, against the element-row FP32 F-engine."""
import numpy as np
import pytest
import torch

from x16util import unswizzle_x16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nch", [128, 256, 512, 1024, 2048])
@pytest.mark.parametrize("ntaps,ne,nsp", [(4, 37, 250), (8, 37, 250), (8, 3, 9), (5, 11, 70),
                                           (16, 37, 250), (16, 5, 11)])
def test_blocks_match_rows(mdt, cuda, nch, ntaps, ne, nsp):
    g = torch.Generator(device="cuda")
    g.manual_seed(nch + 7 * ntaps + nsp)
    iq = torch.randint(-128, 128, (nsp + ntaps - 1, ne, nch, 2), generator=g, device="cuda",
                       dtype=torch.int32).to(torch.int8)
    win = torch.empty(nch * ntaps, dtype=torch.float32, device="cuda")
    mdt.window_hamming_sinc(nch, ntaps, win)
    nan = complex(float("nan"), float("nan"))
    rows = torch.full((nch, nsp, ne), nan, dtype=torch.complex64, device="cuda")
    mdt.fengine_f32(ne, nch, ntaps, nsp, iq, win, rows)
    nsb = -(-nsp // 8)
    xb = torch.full((nsb, nch, ne, 8), nan, dtype=torch.complex64, device="cuda")
    mdt.fengine_c64b(ne, nch, ntaps, nsp, iq, win, xb)
    flat = xb.permute(1, 0, 3, 2).reshape(nch, nsb * 8, ne)
    assert torch.equal(torch.view_as_real(flat[:, :nsp]), torch.view_as_real(rows))
    assert not torch.view_as_real(flat[:, nsp:]).any()

    f = torch.view_as_real(rows).cpu().numpy()
    nep = -(-ne // 16) * 16
    for fmt, ulp in ((0, 2.0 ** -11), (1, 2.0 ** -8)):
        X16 = torch.zeros(mdt.x16_bytes(ne, nch, nsp), dtype=torch.uint8, device="cuda")
        mdt.fengine_x16(ne, nch, ntaps, nsp, iq, win, X16, ab_fmt=fmt)
        got = unswizzle_x16(X16.cpu().numpy(), nch, nsp, ne, nep, bf16=fmt == 1)
        # half an ulp of the format, and its spacing among the smallest
        assert np.all(np.abs(got - f) <= ulp * np.abs(f) + 2.0 ** -25)
    qs = (20.0 / rows.abs().square().mean(dim=(1, 2)).sqrt()).to(torch.float32)
    X16 = torch.zeros(mdt.x16_bytes(ne, nch, nsp), dtype=torch.uint8, device="cuda")
    mdt.fengine_q8(ne, nch, ntaps, nsp, iq, win, X16, qs)
    got = unswizzle_x16(X16.cpu().numpy(), nch, nsp, ne, nep)
    v = np.clip(f.astype(np.float64) * qs.cpu().numpy()[:, None, None, None], -127, 127)
    assert np.all(got == np.rint(got)) and np.all(np.abs(got - v) <= 0.5 + 1e-4)
