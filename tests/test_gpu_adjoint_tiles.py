"""Adjoint kernels at the edges of their tiles: X-engine adjoint tiles of 16, 32 and 64
elements with few and many spectra, the reorder's adjoint in tiles of 32 and 64 (an
exact transpose without gains), tap gradients over short and long runs."""
import numpy as np
import pytest
import torch

from adjref import crandn

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.parametrize("ne", [1, 15, 16, 17, 32, 33, 64, 65, 96, 129])
@pytest.mark.parametrize("nch,nsp", [(3, 1), (2, 32), (2, 33), (3, 64), (2, 65), (1, 300), (700, 35)])
def test_xengine_adjoint_tiles(mdt, cuda, ne, nch, nsp):
    if nch * ne * nsp > 2e6:
        ne = 31  # many channels: several spectrum tiles to a block
    rng = np.random.default_rng(ne * 1009 + nsp)
    G = crandn(rng, nch, ne, ne).astype(np.complex64)
    Y = crandn(rng, nch, nsp, ne).astype(np.complex64)
    dY = torch.full((nch, nsp, ne), float("nan"), dtype=torch.complex64, device="cuda")
    mdt.xengine_adjoint_f32(ne, nch, nsp, dev(G), dev(Y), dY, 0.5)
    Gm = np.transpose(G.astype(np.complex128), (0, 2, 1))
    H = Gm + np.conj(np.transpose(Gm, (0, 2, 1)))
    want = 0.5 * np.matmul(Y.astype(np.complex128), np.transpose(H, (0, 2, 1)))
    # an FP32 chain of 2 NE fmas: 2^-24 of a random walk's length, and H's rounding
    assert rel(dY.cpu().numpy(), want) < 2.0 ** -24 * (2 + 2 * np.sqrt(2 * ne))


@pytest.mark.parametrize("ne,nch,nsp", [(3, 40, 7), (5, 64, 33), (33, 300, 100), (64, 512, 65)])
def test_reorder_adjoint_tiles(mdt, cuda, ne, nch, nsp):
    dY = dev(crandn(np.random.default_rng(nch), nch, nsp, ne).astype(np.complex64))
    dF = torch.full((nsp, ne, nch), float("nan"), dtype=torch.complex64, device="cuda")
    mdt.gain_adjoint(ne, nch, nsp, dY, gains=None, dF=dF)
    assert torch.equal(torch.view_as_real(dF), torch.view_as_real(dY.permute(1, 2, 0)))


@pytest.mark.parametrize("ntaps", [4, 8])
@pytest.mark.parametrize("ne,nch,nsp", [(1, 32, 2), (3, 256, 16), (3, 255, 33), (20, 512, 70),
                                        (64, 128, 129)])
def test_tap_grad_runs(mdt, cuda, ntaps, ne, nch, nsp):
    rng = np.random.default_rng(nsp + ntaps)
    gP = crandn(rng, nsp, ne, nch).astype(np.complex64)
    iq = rng.integers(-128, 128, (nsp + ntaps - 1, ne, nch, 2)).astype(np.int8)
    gW = torch.full((ntaps, nch), float("nan"), dtype=torch.float32, device="cuda")
    ws = torch.empty(ntaps * nch * 64, dtype=torch.float64, device="cuda")
    mdt.pfb_tap_grad(ne, nch, ntaps, nsp, dev(gP), dev(iq), gW, ws)
    x = iq[..., 0] + 1j * iq[..., 1].astype(np.float64)
    want = np.stack([np.einsum("sek,sek->k", gP.astype(np.complex128), np.conj(x[i:i + nsp])).real
                     for i in range(ntaps)])
    # sums in twice the working precision, rounded once to FP32 (cancelling sums: of
    # the products' own size)
    size = np.stack([np.einsum("sek,sek->k", np.abs(gP), np.abs(x[i:i + nsp]))
                     for i in range(ntaps)])
    got = gW.cpu().numpy()
    assert np.all(np.abs(got - want) <= 2.0 ** -24 * np.abs(want) + 2.0 ** -40 * size)


@pytest.mark.parametrize("ne,nch,ntaps,nsp", [(3, 32, 4, 3), (5, 64, 8, 7), (11, 512, 4, 386),
                                              (16, 2048, 5, 40), (3, 4096, 16, 9)])
def test_fengine_with_gains(mdt, cuda, ne, nch, ntaps, nsp):
    """One pass gives the bits of the F-engine and of the gains on its output."""
    rng = np.random.default_rng(nch + ne)
    iq = dev(rng.integers(-128, 128, (nsp + ntaps - 1, ne, nch, 2)).astype(np.int8))
    win = dev(rng.standard_normal(ntaps * nch).astype(np.float32))
    g = dev(crandn(rng, nch, ne).astype(np.complex64))
    X, Y, X2, Y2, Y3 = (torch.full((nch, nsp, ne), float("nan"), dtype=torch.complex64,
                                   device="cuda") for _ in range(5))
    mdt.fengine_f32(ne, nch, ntaps, nsp, iq, win, X)
    mdt.apply_gains(ne, nch, nsp, X, g, Y)
    mdt.fengine_gains_f32(ne, nch, ntaps, nsp, iq, win, g, Y2, X=X2)
    mdt.fengine_gains_f32(ne, nch, ntaps, nsp, iq, win, g, Y3)
    for a, b in ((X, X2), (Y, Y2), (Y, Y3)):
        assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))


@pytest.mark.parametrize("ne,nch,nsp", [(1, 32, 3), (5, 64, 7), (3, 128, 5), (11, 256, 33),
                                        (64, 512, 9), (7, 1024, 10), (3, 2048, 11)])
def test_reorder_adjoint_with_ifft(mdt, cuda, ne, nch, nsp):
    """One pass gives the bits of the reorder's adjoint and the inverse FFT of it."""
    rng = np.random.default_rng(nch + ne)
    dY = dev(crandn(rng, nch, nsp, ne).astype(np.complex64))
    g = dev(crandn(rng, nch, ne).astype(np.complex64))
    dF, dP, got = (torch.full((nsp, ne, nch), float("nan"), dtype=torch.complex64, device="cuda")
                   for _ in range(3))
    mdt.gain_adjoint(ne, nch, nsp, dY, gains=g, dF=dF)
    mdt.fft_c2c(dF, dP, nsp * ne, nch, 1)
    mdt.reorder_adjoint_ifft(ne, nch, nsp, dY, g, got)
    assert torch.equal(torch.view_as_real(got), torch.view_as_real(dP))
