"""Tensor-core X-engines whose blocks take several channels of a small array: padded
rows of 16 to 64, channel counts that no group divides, the FP64 accumulator, a
channel with infinities and NaN among finite ones, and the batch against plans.
The samples are small integers and Nsp a power of two, so every result is exact."""
import numpy as np
import pytest
import torch

from conftest import rel_fro
from test_gpu_batch import gen
from x16util import swizzle_x16

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def samples(ne, nch, nsp):
    rng = np.random.default_rng(ne * 10007 + nch)
    return rng.integers(-9, 10, size=(nch, nsp, ne, 2))


def sums(X):
    Z = X[..., 0] + 1j * X[..., 1].astype(np.float64)
    return np.matmul(np.transpose(np.conj(Z), (0, 2, 1)), Z)  # [c][q][r]


@pytest.mark.parametrize("ne", [1, 10, 16, 17, 32, 33, 48, 50, 64, 65])
@pytest.mark.parametrize("nch", [307, 613, 1221])
def test_groups(mdt, cuda, ne, nch):
    nsp = 64
    X = samples(ne, nch, nsp)
    X16 = dev(swizzle_x16(X, (ne + 15) // 16 * 16))
    want = sums(X)
    vis = torch.full((nch, ne, ne), float("nan"), dtype=torch.complex64, device="cuda")
    acc = torch.ones(nch, ne, ne, dtype=torch.complex128, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    mdt.xengine_tc(ne, nch, nsp, X16, vis, vis_acc=acc, err=err)
    qs = torch.from_numpy(2.0 ** (np.arange(nch) % 5 - 2)).to(torch.float32).cuda()
    q8 = torch.full_like(vis, float("nan"))
    raw = torch.full((nch, ne, ne, 2), -1, dtype=torch.int32, device="cuda")
    mdt.xengine_q8(ne, nch, nsp, X16, qs, vis=q8, vis_i32=raw, err=err)
    torch.cuda.synchronize()
    assert err.item() == 0
    assert np.array_equal(vis.cpu().numpy(), want / nsp)
    assert np.array_equal(acc.cpu().numpy(), want / nsp + 1)
    assert np.array_equal(raw.cpu().numpy()[..., 0], want.real)
    assert np.array_equal(raw.cpu().numpy()[..., 1], want.imag)
    s2 = qs.cpu().numpy().astype(np.float64)[:, None, None] ** 2
    assert np.array_equal(q8.cpu().numpy(), want / nsp / s2)


@pytest.mark.parametrize("ne", [10, 40])
def test_not_finite_stays_in_its_channel(mdt, cuda, ne):
    nch, nsp, bad = 1221, 32, 701
    X = samples(ne, nch, nsp)
    want = sums(X) / nsp
    S = X.astype(np.float32)
    S[bad, 3, ne // 2] = np.inf
    S[bad, 5, 0] = np.nan
    X16 = dev(swizzle_x16(S, (ne + 15) // 16 * 16))
    vis = torch.empty(nch, ne, ne, dtype=torch.complex64, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    mdt.xengine_tc(ne, nch, nsp, X16, vis, err=err)
    torch.cuda.synchronize()
    v = vis.cpu().numpy()
    rest = np.arange(nch) != bad
    assert np.array_equal(v[rest], want[rest])
    assert not np.isfinite(v[bad, 0]).any() and not np.isfinite(v[bad, ne // 2]).any()


def test_batch_groups(mdt, cuda):
    jobs = [(10, 2048, 4, 40), (30, 1024, 4, 33), (17, 512, 8, 100), (60, 1024, 4, 64),
            (130, 256, 4, 32), (64, 256, 8, 7)]
    cfgs = [mdt.configs.Config("job%d" % k, ne, nch, nt, nsp, 1, seed=40 + k, sigma=(12.0, 20.0),
                               tones=[(None, 8.0)]) for k, (ne, nch, nt, nsp) in enumerate(jobs)]
    iqs = [gen(mdt, c, c.nspectra + c.ntaps - 1) for c in cfgs]
    vis = [torch.full((nch, ne, ne), float("nan"), dtype=torch.complex64, device="cuda")
           for ne, nch, nt, nsp in jobs]
    batch = mdt.FxBatch(jobs)
    batch.execute(iqs, vis)
    batch.check()
    for k, (ne, nch, nt, nsp) in enumerate(jobs):
        win = torch.empty(nch * nt, dtype=torch.float32, device="cuda")
        mdt.window_hamming_sinc(nch, nt, win)
        plan = mdt.FxPlan(ne, nch, nt, nsp, precision=mdt.MDT_PREC_FP16)
        plan.set_window(win)
        ref = torch.empty_like(vis[k])
        plan.execute(iqs[k], 1, ref)
        plan.check()
        plan.close()
        assert rel_fro(vis[k].cpu().numpy(), ref.cpu().numpy().astype(np.complex128)) < 1e-6, k
