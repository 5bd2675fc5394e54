"""FP32 (SIMT) X-engine for few spectra: K slices whose sums one thread per value adds
(up to 28 inputs), at odd channel counts and in both operand layouts."""
import numpy as np
import pytest
import torch

from adjref import crandn

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("ne", [1, 2, 4, 5, 10, 16, 17, 28, 29, 64])
@pytest.mark.parametrize("nch,nsp", [(1, 1), (3, 2), (5, 31), (2, 33), (7, 100), (1000, 20)])
def test_slices(mdt, cuda, ne, nch, nsp):
    rng = np.random.default_rng(100 * ne + nsp)
    X = crandn(rng, nch, nsp, ne + 1).astype(np.complex64)
    V = torch.full((nch, ne, ne), float("nan"), dtype=torch.complex64, device="cuda")
    mdt.xengine_f32(ne, nch, nsp, dev(X), ne + 1, nsp * (ne + 1), 0.5, V)
    Z = X[:, :, :ne].astype(np.complex128)
    want = 0.5 * np.matmul(np.transpose(np.conj(Z), (0, 2, 1)), Z)
    got = V.cpu().numpy()
    p = np.sqrt(np.abs(np.diagonal(want, axis1=1, axis2=2)))
    # two FP32 roundings a spectrum, of sums no larger than sqrt(V_rr V_qq)
    tol = 2.0 ** -24 * (2 * nsp + 18)
    assert np.all(np.abs(got - want) <= tol * p[:, :, None] * p[:, None, :])
    assert np.array_equal(got, np.conj(np.transpose(got, (0, 2, 1))))


@pytest.mark.parametrize("ne", [3, 10, 28])
def test_plan_and_stage_agree(mdt, cuda, ne):
    """The plan's blocked operand and the element-row operand give the same bits."""
    nch, ntaps, nsp = 64, 4, 45
    g = torch.Generator(device="cuda")
    g.manual_seed(ne)
    iq = torch.randint(-90, 90, (nsp + ntaps - 1, ne, nch, 2), generator=g, device="cuda",
                       dtype=torch.int32).to(torch.int8)
    win = torch.empty(nch * ntaps, dtype=torch.float32, device="cuda")
    mdt.window_hamming_sinc(nch, ntaps, win)
    plan = mdt.FxPlan(ne, nch, ntaps, nsp, precision=mdt.MDT_PREC_FP32)
    plan.set_window(win)
    vis = torch.empty(nch, ne, ne, dtype=torch.complex64, device="cuda")
    plan.execute(iq, 1, vis)
    plan.check()
    plan.close()
    X = torch.empty(nch * nsp * ne, dtype=torch.complex64, device="cuda")
    mdt.fengine_f32(ne, nch, ntaps, nsp, iq, win, X)
    V = torch.empty_like(vis)
    mdt.xengine_f32(ne, nch, nsp, X, ne, nsp * ne, 1.0 / nsp, V)
    assert torch.equal(torch.view_as_real(V), torch.view_as_real(vis))
