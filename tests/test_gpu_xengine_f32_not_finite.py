"""FP32 X-engine on the tensor cores: what samples that are not finite cost, and that
they stay in their elements' visibilities."""
import numpy as np
import pytest
import torch

from adjref import crandn

pytestmark = pytest.mark.gpu


def run(mdt, X, V):
    nch, nsp, ne = X.shape
    mdt.xengine_f32(ne, nch, nsp, X, ne, nsp * ne, 1.0, V)


def best_ms(f):
    f()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    best = 1e9
    for _ in range(5):
        ev[0].record()
        f()
        ev[1].record()
        ev[1].synchronize()
        best = min(best, ev[0].elapsed_time(ev[1]))
    return best


# An element that is not finite costs at most what the multiply-adds of its tiles cost, for
# each tile about twice the tensor cores' time: under 4 times in all, whatever is not finite.
# (One thread per visibility, one after the other, took 11 and 22 times with one element,
# 15 and 61 with all.)
@pytest.mark.parametrize("ne,nch,nsp", [(40, 608, 2048), (256, 152, 2048)])
@pytest.mark.parametrize("which", ["one", "all"])
def test_cost(mdt, cuda, ne, nch, nsp, which):
    g = torch.Generator(device="cuda")
    g.manual_seed(ne)
    X = torch.randn(nch, nsp, ne, dtype=torch.complex64, device="cuda", generator=g)
    V = torch.empty(nch, ne, ne, dtype=torch.complex64, device="cuda")
    clean = best_ms(lambda: run(mdt, X, V))
    ref = V.clone()
    hit = torch.zeros(ne, dtype=torch.bool, device="cuda")
    hit[ne // 2 if which == "one" else slice(None)] = True
    X[:, 7, hit] = complex(float("nan"), 0.0)
    bad = best_ms(lambda: run(mdt, X, V))
    touched = hit[:, None] | hit[None, :]
    assert bool(torch.all(torch.isnan(V[:, touched].real)))
    assert torch.equal(V[:, ~touched], ref[:, ~touched])
    assert bad < 4 * clean, (clean, bad)


@pytest.mark.parametrize("ne", [3, 16, 33, 64, 70, 130])
@pytest.mark.parametrize("value", [complex(np.inf, 1), complex(0, -np.inf), complex(np.nan, 0),
                                   complex(0, np.nan)])
def test_stays_in_its_element(mdt, cuda, ne, value):
    """In a full stage, in the last one, and with spectra after it."""
    rng = np.random.default_rng(ne)
    nch, nsp = 5, 330
    X = crandn(rng, nch, nsp, ne).astype(np.complex64)
    Y = X.copy()
    hit = np.zeros((nch, ne), bool)
    for c, s, e in ((0, 0, 0), (1, 63, ne - 1), (2, 329, ne // 2), (4, 130, 1)):
        Y[c, s, e] = value
        hit[c, e] = True
    out = []
    for Z in (X, Y):
        V = torch.empty(nch, ne, ne, dtype=torch.complex64, device="cuda")
        run(mdt, torch.from_numpy(Z).cuda(), V)
        out.append(V.cpu().numpy())
    clean, V = out
    same = ~(hit[:, :, None] | hit[:, None, :])
    assert np.array_equal(V[same], clean[same])
    for c, e in np.argwhere(hit):
        # the real part of each of its products, and its power
        assert not np.any(np.isfinite(V[c, e].real) & np.isfinite(V[c, e].imag))
        assert not np.isfinite(V[c, e, e].real)
