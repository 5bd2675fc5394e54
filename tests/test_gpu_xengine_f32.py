"""FP32 X-engine on the tensor cores (products of split samples) at the edges of its
tiles: channel slots of 16, 32 and 64 elements, channels that do not fill a
block, tiles below the diagonal, stages that Nsp does not fill (from 256 spectra
on; fewer take the SIMT kernel), both operand layouts, samples of any size,
infinities and NaN."""
import numpy as np
import pytest
import torch

from adjref import crandn

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def run(mdt, X, alpha, ld=None):
    nch, nsp, ne = X.shape
    ld = ne if ld is None else ld
    buf = torch.full((nch, nsp, ld), complex(float("nan"), 3.0), dtype=torch.complex64, device="cuda")
    buf[:, :, :ne] = dev(X)
    V = torch.full((nch, ne, ne), float("nan"), dtype=torch.complex64, device="cuda")
    mdt.xengine_f32(ne, nch, nsp, buf, ld, nsp * ld, alpha, V)
    return V.cpu().numpy()


def exact(X, alpha):
    Z = X.astype(np.complex128)
    return alpha * np.einsum("csr,csq->cqr", Z, np.conj(Z))


def scaled_error(X, V, alpha):
    """Largest |V - exact| over sqrt(V_rr V_qq), the scale of a product's rounding."""
    E = exact(X, alpha)
    p = np.sqrt(np.abs(np.diagonal(E, axis1=1, axis2=2)))
    return np.max(np.abs(V - E) / (p[:, :, None] * p[:, None, :]))


# Tolerance, of sqrt(V_rr V_qq): samples keep 22 bits below the element's
# largest component of a stage (2^-22 with the dropped rest products), the integer
# sums are exact or truncated once, and the stages' sums are added in FP32 (2^-24
# each, of the running sum, generously one per 32 spectra).
@pytest.mark.parametrize("ne", [1, 3, 8, 9, 16, 17, 31, 32, 33, 40, 63, 64, 65, 127, 128, 129, 200])
@pytest.mark.parametrize("nch,nsp,pad", [(1, 256, 0), (3, 257, 1), (5, 320, 0), (2, 383, 3),
                                         (7, 512, 0), (2, 700, 0)])
def test_shapes(mdt, cuda, ne, nch, nsp, pad):
    rng = np.random.default_rng(ne * 1000 + nsp)
    X = crandn(rng, nch, nsp, ne).astype(np.complex64)
    V = run(mdt, X, 1.0 / nsp, ld=ne + pad)
    assert scaled_error(X, V, 1.0 / nsp) < 2.0 ** -22 + nsp / 32 * 2.0 ** -24
    assert np.array_equal(V, np.conj(np.transpose(V, (0, 2, 1))))
    assert np.all(np.diagonal(V, axis1=1, axis2=2).imag == 0)


@pytest.mark.parametrize("ne", [12, 40, 70])
def test_magnitudes(mdt, cuda, ne):
    """Elements from 2^-40 to 2^40 times the others, and spikes within one."""
    rng = np.random.default_rng(ne)
    nch, nsp = 3, 352
    X = crandn(rng, nch, nsp, ne)
    X *= 2.0 ** rng.integers(-40, 41, size=(nch, 1, ne))
    X[:, 5, ::3] *= 2.0 ** 12
    X = X.astype(np.complex64)
    V = run(mdt, X, 1.0)
    assert scaled_error(X, V, 1.0) < 2.0 ** -22 + nsp / 32 * 2.0 ** -24


@pytest.mark.parametrize("ne", [12, 30, 40, 70])
def test_not_finite(mdt, cuda, ne):
    """Infinities, NaN and products that overflow: what FP32 multiply-adds in
    spectrum order give, and nothing in the other visibilities."""
    rng = np.random.default_rng(ne)
    nch, nsp = 5, 296
    X = crandn(rng, nch, nsp, ne).astype(np.complex64)
    clean = run(mdt, X, 1.0)
    X[0, 7, 2] = complex(np.inf, 1.0)
    X[1, 8, 3] = complex(np.nan, 0.0)
    X[3, 1, 4] = 3e38
    X[4, 295, ne - 1] = complex(0.0, -np.inf)
    V = run(mdt, X, 1.0)
    with np.errstate(all="ignore"):
        want = np.zeros((nch, ne, ne, 2), np.float32)
        for s in range(nsp):
            a, b = X[:, s, None, :], X[:, s, :, None]       # row r, column q: [c][q][r]
            want[..., 0] += a.real * b.real + a.imag * b.imag
            want[..., 1] += a.imag * b.real - a.real * b.imag
        # the complex alpha = 1 + 0i multiplies them
        want = np.stack([want[..., 0] - np.float32(0) * want[..., 1],
                         want[..., 1] + np.float32(0) * want[..., 0]], axis=-1)
    low = np.arange(ne)[None, :] >= np.arange(ne)[:, None]  # r >= q
    for c in range(nch):
        for part, w in ((V[c].real, want[c, ..., 0]), (V[c].imag, want[c, ..., 1])):
            off = low & ~np.eye(ne, dtype=bool) if w is not want[c, ..., 0] else low
            assert np.array_equal(np.isnan(part[off]), np.isnan(w[off])), c
            assert np.array_equal(part[off][np.isinf(part[off])], w[off][np.isinf(w[off])]), c
    hit = np.zeros((nch, ne), bool)
    hit[0, 2] = hit[1, 3] = hit[3, 4] = hit[4, ne - 1] = True
    same = ~(hit[:, :, None] | hit[:, None, :])
    assert np.array_equal(V[same], clean[same])


@pytest.mark.parametrize("ne,nch,ntaps,nsp", [(5, 64, 4, 261), (20, 32, 8, 262), (40, 128, 8, 300),
                                              (100, 32, 4, 256), (40, 32, 4, 255)])
def test_layouts_agree(mdt, cuda, ne, nch, ntaps, nsp):
    """The blocked operand (plan) and X[c][s][e] (stage entry point) of the same
    samples give the same bits."""
    rng = np.random.default_rng(ne)
    iq = dev(rng.integers(-100, 101, size=(nsp + ntaps - 1) * ne * nch * 2).astype(np.int8))
    win = torch.empty(nch * ntaps, dtype=torch.float32, device="cuda")
    mdt.window_hamming_sinc(nch, ntaps, win)
    X = torch.empty(nch * nsp * ne, dtype=torch.complex64, device="cuda")
    mdt.fengine_f32(ne, nch, ntaps, nsp, iq, win, X)
    V1 = torch.empty(nch, ne, ne, dtype=torch.complex64, device="cuda")
    V2 = torch.empty_like(V1)
    mdt.xengine_f32(ne, nch, nsp, X, ne, nsp * ne, 1.0 / nsp, V1)
    plan = mdt.FxPlan(ne, nch, ntaps, nsp)
    plan.set_window(win)
    plan.execute(iq, 1, V2)
    assert torch.equal(V1.view(torch.int64), V2.view(torch.int64))
    plan.close()
