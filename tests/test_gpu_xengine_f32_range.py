"""FP32 X-engine on the tensor cores: samples of uneven size within a stage of 64 spectra.
Every visibility is measured against sum |a||b| of its own products, so that a burst which
the other element does not share cannot hide what it costs."""
import numpy as np
import pytest
import torch

from adjref import crandn

pytestmark = pytest.mark.gpu

# Of sum |a||b|.  Uneven elements: two-level sums of FP32 multiply-adds, 32 of each sign
# and kind at the first level and Nsp / 16 sums at the second, rounding errors of random
# sign: 4 sqrt(64 + Nsp / 16) 2^-25 = 1.2e-6 in the worst of some 10^4 visibilities if every
# partial sum were as large as the last; they grow to it, a factor of 0.6.  The others:
# 2^-23 of the largest component, 32 times the least that three quarters of the samples are.
TOL = 1e-6


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def run(mdt, X, alpha=1.0):
    nch, nsp, ne = X.shape
    V = torch.full((nch, ne, ne), float("nan"), dtype=torch.complex64, device="cuda")
    mdt.xengine_f32(ne, nch, nsp, dev(X), ne, nsp * ne, alpha, V)
    return V.cpu().numpy()


def error(X, V):
    """Largest |V - exact| over sum |a||b| of the same two elements; products that are all
    zero have to be zero."""
    Z = X.astype(np.complex128)
    E = np.einsum("csr,csq->cqr", Z, np.conj(Z))
    M = np.einsum("csr,csq->cqr", np.abs(Z), np.abs(Z))
    assert np.all(V[M == 0] == 0)
    return np.max(np.abs(V - E) / np.where(M == 0, 1, M))


def changed(X, kind, k, a, b):
    """Elements a and b: a is large, by 2^k, where b is zero."""
    X = X.copy()
    nsp = X.shape[1]
    if kind == "burst":                     # one spectrum of 64
        at = np.arange(5, nsp, 64)
    elif kind == "half":
        at = np.arange(0, nsp, 2)
    elif kind == "last":                    # of a stage that Nsp does not fill
        at = np.arange(nsp - 1, nsp)
    else:                                   # "sparse": b is there in one spectrum of eight
        at = np.flatnonzero(np.arange(nsp) % 8)
    X[:, at, a] *= np.float32(2.0 ** k)
    X[:, at, b] = 0
    return X


@pytest.mark.parametrize("ne,a,b", [(3, 0, 2), (10, 0, 1), (16, 15, 2), (30, 29, 0), (40, 1, 39),
                                    (64, 63, 0), (70, 0, 69), (70, 68, 3), (130, 1, 129)])
@pytest.mark.parametrize("kind", ["burst", "half", "last", "sparse"])
def test_uneven_samples(mdt, cuda, ne, a, b, kind):
    rng = np.random.default_rng(ne + len(kind))
    nch, nsp = 3, 64 * 5 + 3
    X = (crandn(rng, nch, nsp, ne) + crandn(rng, nch, nsp, 1)).astype(np.complex64)
    clean = run(mdt, X)
    assert error(X, clean) < TOL
    others = np.ones(ne, bool)
    others[[a, b]] = False
    others = others[:, None] & others[None, :]
    for k in (1, 3, 4, 5, 8, 12, 20, 30, 40):
        Y = changed(X, kind, k, a, b)
        V = run(mdt, Y)
        assert error(Y, V) < TOL, k
        # and the visibilities of the other elements do not know of it
        assert np.array_equal(V[:, others], clean[:, others]), k
        assert np.array_equal(V, np.conj(np.transpose(V, (0, 2, 1))))


@pytest.mark.parametrize("ne", [10, 20, 40, 70])
def test_sizes_and_zeros(mdt, cuda, ne):
    """Elements of any size, an element that is zero, one that is zero but for one spectrum,
    and every element uneven in every stage."""
    rng = np.random.default_rng(ne)
    nch, nsp = 5, 700
    X = crandn(rng, nch, nsp, ne)
    X[0] *= 2.0 ** rng.integers(-75, 62, size=(1, ne))
    X[1, :, 3] = 0
    X[2, :500, 4] = 0
    X[2, 501:, 4] = 0
    X[3] *= 2.0 ** rng.integers(-30, 31, size=(nsp, ne))
    X[4, ::3] *= 2.0 ** 9
    X = X.astype(np.complex64)
    V = run(mdt, X)
    # (products below 2^-120 lose bits to FP32's range, 2^-149 each)
    Z = X.astype(np.complex128)
    E = np.einsum("csr,csq->cqr", Z, np.conj(Z))
    M = np.einsum("csr,csq->cqr", np.abs(Z), np.abs(Z))
    big = np.abs(E) > 3.4e38             # autocorrelations of 2^61 and above: past FP32
    assert np.all(np.isinf(V.real[big]))
    assert np.all(np.abs(V - E)[~big] <= TOL * M[~big] + nsp * 2.0 ** -148)
    assert np.all(V[1, 3] == 0) and np.all(V[1, :, 3] == 0)


def test_many_stages(mdt, cuda):
    """Uneven in one stage of 520."""
    rng = np.random.default_rng(1)
    nsp = 64 * 520
    X = crandn(rng, 1, nsp, 6).astype(np.complex64)
    X[0, 64 * 515 + 7, 1] *= 2.0 ** 14
    X[0, 64 * 515 + 7, 2] = 0
    X[0, 64 * 3:64 * 515, 1] = 0
    V = run(mdt, X)
    assert error(X, V) < TOL


@pytest.mark.parametrize("ne,nch,ntaps,nsp", [(5, 64, 4, 261), (20, 32, 8, 330), (40, 64, 4, 300),
                                              (100, 32, 4, 256)])
def test_layouts_agree(mdt, cuda, ne, nch, ntaps, nsp):
    """A plan's blocked operand and X[c][s][e] give the same bits with uneven elements too."""
    rng = np.random.default_rng(ne)
    iq = rng.integers(-1, 2, size=(nsp + ntaps - 1, ne, nch, 2)).astype(np.int8)
    iq[40:42, ::2] = rng.integers(-128, 128, size=(2, (ne + 1) // 2, nch, 2))
    iq[36:50, 1::2] = 0
    iq = dev(iq)
    win = torch.empty(nch * ntaps, dtype=torch.float32, device="cuda")
    mdt.window_hamming_sinc(nch, ntaps, win)
    X = torch.empty(nch * nsp * ne, dtype=torch.complex64, device="cuda")
    mdt.fengine_f32(ne, nch, ntaps, nsp, iq, win, X)
    V1 = torch.empty(nch, ne, ne, dtype=torch.complex64, device="cuda")
    V2 = torch.empty_like(V1)
    mdt.xengine_f32(ne, nch, nsp, X, ne, nsp * ne, 1.0, V1)
    plan = mdt.FxPlan(ne, nch, ntaps, nsp)
    plan.set_window(win)
    plan.execute(iq, 1, V2)
    # the plan divides by Nsp
    want = V1.cpu().numpy() * np.float32(1.0 / nsp)
    assert error(X.view(nch, nsp, ne).cpu().numpy(), V1.cpu().numpy()) < TOL
    V3 = torch.empty_like(V1)
    mdt.xengine_f32(ne, nch, nsp, X, ne, nsp * ne, 1.0 / nsp, V3)
    assert torch.equal(V3.view(torch.int64), V2.view(torch.int64))
    assert np.allclose(want, V3.cpu().numpy(), rtol=1e-6, atol=0)
    plan.close()


@pytest.mark.parametrize("ne", [10, 40, 100])
def test_previous_values(mdt, cuda, ne):
    """cublasCgemmBatched with beta: V = alpha X X^H + beta V, with and without a burst."""
    rng = np.random.default_rng(ne)
    nch, nsp, alpha, beta = 3, 300, 0.25, 0.5
    X = crandn(rng, nch, nsp, ne).astype(np.complex64)
    X[1, 7, 2] *= 2.0 ** 14
    X[1, 7, 3] = 0
    V0 = crandn(rng, nch, ne, ne).astype(np.complex64)
    V0 = (V0 + np.conj(np.transpose(V0, (0, 2, 1)))) / 2   # Hermitian, as every use of it
    dX, dV = dev(X), dev(V0)
    at = torch.arange(nch, dtype=torch.int64, device="cuda")
    xp, vp = dX.data_ptr() + at * (nsp * ne * 8), dV.data_ptr() + at * (ne * ne * 8)
    h = mdt.cublasCreate()
    mdt.cublasSetStream(h, torch.cuda.current_stream())
    mdt.cublasCgemmBatched(h, mdt.CUBLAS_OP_N, mdt.CUBLAS_OP_C, ne, ne, nsp, alpha, xp, ne, xp, ne,
                           beta, vp, ne, nch)
    Z = X.astype(np.complex128)
    E = alpha * np.einsum("csr,csq->cqr", Z, np.conj(Z)) + beta * V0
    M = alpha * np.einsum("csr,csq->cqr", np.abs(Z), np.abs(Z)) + beta * np.abs(V0)
    assert np.all(np.abs(dV.cpu().numpy() - E) <= TOL * M)
