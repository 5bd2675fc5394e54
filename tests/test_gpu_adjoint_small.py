"""Gradient sums of small upstream gradients (a loss scaled down), whose products leave
FP32's range: the double sum's value to half a unit in the last place, down to the
smallest FP32 number; sums without a product that is not zero; infinities against zeros."""
import numpy as np
import pytest
import torch

from adjref import crandn

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def check(got, want, mag):
    """One rounding to FP32 (half a unit: 2^-24 of it, 2^-150 below its normal range), and
    the sum's own error, 2^-44 of the sum of magnitudes."""
    tol = 2.0 ** -24 * np.abs(want) + 2.0 ** -150 + 2.0 ** -44 * mag
    assert np.all(np.abs(got - want) <= tol)


@pytest.mark.parametrize("ne,nch,nsp", [(6, 40, 37), (7, 33, 19)])
@pytest.mark.parametrize("power", [0, 60, 80, 100, 110, 120, 130])
def test_gain_sums(mdt, cuda, ne, nch, nsp, power):
    rng = np.random.default_rng(power)
    dY, X = (crandn(rng, nch, nsp, ne) for _ in range(2))
    dY = (dY * 2.0 ** -power).astype(np.complex64)
    X = (X * 2.0 ** -8).astype(np.complex64)
    X[3] = 0                        # a channel without a signal
    dY[4, :, 1] = 0
    out = torch.full((nch, ne), complex(9, 9), dtype=torch.complex64, device="cuda")
    mdt.gain_adjoint(ne, nch, nsp, dev(dY), X=dev(X), dgains=out)
    z = dY.astype(np.complex128) * np.conj(X.astype(np.complex128))
    got, want, mag = out.cpu().numpy(), z.sum(axis=1), np.abs(z).sum(axis=1)
    check(got.real.astype(np.float64), want.real, mag)
    check(got.imag.astype(np.float64), want.imag, mag)
    assert np.all(got[3] == 0) and np.all(got[4, 1] == 0)


@pytest.mark.parametrize("ne,nch,ntaps,nsp", [(3, 40, 4, 37), (2, 33, 8, 21)])
@pytest.mark.parametrize("power", [0, 80, 100, 120, 135, 145])
def test_tap_sums(mdt, cuda, ne, nch, ntaps, nsp, power):
    rng = np.random.default_rng(power)
    iq = rng.integers(-128, 128, size=(nsp + ntaps - 1, ne, nch, 2)).astype(np.int8)
    iq[:, :, 5] = 0
    gP = (crandn(rng, nsp, ne, nch) * 2.0 ** -power).astype(np.complex64)
    gP[:, :, 6] = 0
    x = iq[..., 0].astype(np.float64) + 1j * iq[..., 1]
    g = gP.astype(np.complex128)
    want = np.stack([np.real(np.sum(g * np.conj(x[i:i + nsp]), axis=(0, 1))) for i in range(ntaps)])
    gW = torch.full((ntaps * nch,), 9.0, dtype=torch.float32, device="cuda")
    ws = torch.empty(ntaps * nch * 64, dtype=torch.float64, device="cuda")
    mdt.pfb_tap_grad(ne, nch, ntaps, nsp, dev(gP), dev(iq), gW, ws)
    got = gW.cpu().numpy().reshape(ntaps, nch).astype(np.float64)
    check(got, want, np.sum(np.abs(g), axis=(0, 1)) * 256)
    assert np.all(got[:, 5:7] == 0)


def test_infinity_times_zero(mdt, cuda):
    dY = np.zeros((2, 9, 4), np.complex64)
    X = np.zeros((2, 9, 4), np.complex64)
    X[1, 3, 2] = complex(np.inf, 0)
    out = torch.zeros(2, 4, dtype=torch.complex64, device="cuda")
    mdt.gain_adjoint(4, 2, 9, dev(dY), X=dev(X), dgains=out)
    got = out.cpu().numpy()
    assert np.isnan(got[1, 2].real) and np.isnan(got[1, 2].imag)
    got[1, 2] = 0
    assert np.all(got == 0)
