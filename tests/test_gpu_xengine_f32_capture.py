"""FP32 X-engine on the tensor cores and the kernel after it, captured in a CUDA graph: new
samples at each replay, with and without uneven ones, equal to direct calls; two streams
at once."""
import numpy as np
import pytest
import torch

from adjref import crandn

pytestmark = pytest.mark.gpu


def samples(ne, nch, nsp, seed, burst):
    X = crandn(np.random.default_rng(seed), nch, nsp, ne).astype(np.complex64)
    if burst:
        X[1, 40, ::2] *= 2.0 ** 12
        X[1, 40, 1::2] = 0
        X[2, 200, ne - 1] = complex(np.nan, 1)
    return torch.from_numpy(X).cuda()


def call(mdt, X, V):
    nch, nsp, ne = X.shape
    mdt.xengine_f32(ne, nch, nsp, X, ne, nsp * ne, 1.0 / nsp, V)


def same(a, b):
    return torch.equal(a.view(torch.int64), b.view(torch.int64))


@pytest.mark.parametrize("ne", [10, 40, 70])
def test_replays(mdt, cuda, ne):
    nch, nsp = 4, 330
    X = samples(ne, nch, nsp, 0, False)
    V = torch.zeros(nch, ne, ne, dtype=torch.complex64, device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        call(mdt, X, V)
        with torch.cuda.graph(graph, stream=stream):
            call(mdt, X, V)
    want = torch.empty_like(V)
    for seed, burst in ((1, False), (2, True), (3, False), (4, True)):
        X.copy_(samples(ne, nch, nsp, seed, burst))
        call(mdt, X, want)
        V.fill_(complex(5, 5))
        graph.replay()
        torch.cuda.synchronize()
        assert same(V, want), seed


@pytest.mark.parametrize("ne", [10, 70])
def test_two_streams(mdt, cuda, ne):
    nch, nsp = 64, 330
    Xs = [samples(ne, nch, nsp, s, s % 2 == 1) for s in range(4)]
    want = [torch.empty(nch, ne, ne, dtype=torch.complex64, device="cuda") for _ in Xs]
    got = [torch.empty_like(v) for v in want]
    for X, V in zip(Xs, want):
        call(mdt, X, V)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(5):
        for V in got:
            V.fill_(complex(5, 5))
        torch.cuda.synchronize()
        for i, (X, V) in enumerate(zip(Xs, got)):
            with torch.cuda.stream(streams[i % 2]):
                call(mdt, X, V)
        torch.cuda.synchronize()
        assert all(same(a, b) for a, b in zip(got, want))
