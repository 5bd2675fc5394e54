"""FP32 X-engine on the tensor cores: samples of constant amplitude, whose sums of integer
parts are past 2^24, where the tensor core truncates."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# Relative to the power, V_rr = sum |a|^2: each of the four instructions of a stage may take
# a unit in the last place off the running sum (2^-23), two samples are rounded to 2^-23 of
# their largest component (all alike if they are constant), and the stages' sums round in
# FP32 (2^-24 each for ten or so): a one-sided error of at most 4 2^-23, 8 2^-23 in all.
@pytest.mark.parametrize("ne", [10, 40, 70])
@pytest.mark.parametrize("nsp", [256, 1000])
@pytest.mark.parametrize("amplitude", [1.0, 1.41, 1.99])  # integer parts up to 1024 .. 2047
@pytest.mark.parametrize("kind", ["tone", "constant"])
def test_constant_amplitude(mdt, cuda, ne, nsp, amplitude, kind):
    rng = np.random.default_rng(ne + nsp)
    nch = 4
    phase = rng.uniform(0, 2 * np.pi, (nch, 1, ne))
    if kind == "tone":
        phase = phase + rng.uniform(0, np.pi, (nch, 1, 1)) * np.arange(nsp)[None, :, None]
    else:
        phase = phase + np.zeros((nch, nsp, 1))
    X = (amplitude * np.exp(1j * phase)).astype(np.complex64)
    V = torch.empty(nch, ne, ne, dtype=torch.complex64, device="cuda")
    mdt.xengine_f32(ne, nch, nsp, torch.from_numpy(X).cuda(), ne, nsp * ne, 1.0, V)
    Z = X.astype(np.complex128)
    E = np.einsum("csr,csq->cqr", Z, np.conj(Z))
    M = np.einsum("csr,csq->cqr", np.abs(Z), np.abs(Z))
    err = V.cpu().numpy() - E
    assert np.all(np.abs(err) <= 8 * 2.0 ** -23 * M)
    auto = np.diagonal(err, axis1=1, axis2=2).real / np.diagonal(M, axis1=1, axis2=2)
    assert -4 * 2.0 ** -23 <= auto.mean() <= 2.0 ** -23
