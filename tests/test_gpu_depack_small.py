"""Depacketiser calls of few packets: time per call, and the same samples as one call of
all packets."""
import numpy as np
import pytest
import torch

from packets import fmt_dict, packetise
from test_gpu_depack import Depack, rand_words

pytestmark = pytest.mark.gpu


def us_per_call(mdt, sample_bits, npk):
    """Of the kernel alone: twenty launches in a graph."""
    ne, nch = 38, 1024
    fmt = mdt.packet_format(28, sample_bits=sample_bits)
    nsp = npk // 4 * 28 // nch + 1
    pk = torch.zeros(npk, fmt.packet_bytes, dtype=torch.uint8, device="cuda")
    head = pk.view(torch.int32)
    n = torch.arange(npk, dtype=torch.int32, device="cuda")
    head[:, 1] = n % 4
    head[:, 2] = n // 4
    seen = torch.zeros(mdt.depacketise_seen_words(fmt, ne, nch, 0, nsp), dtype=torch.int32,
                       device="cuda")
    stats = torch.zeros(5, dtype=torch.int64, device="cuda")
    out = torch.empty(nsp, ne, nch, dtype=torch.complex64, device="cuda")

    def call():
        mdt.depacketise(fmt, pk, npk, ne, nch, 0, nsp, out, seen, stats)

    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        call()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(20):
                call()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    best = 1e9
    for _ in range(6):
        ev[0].record()
        graph.replay()
        ev[1].record()
        ev[1].synchronize()
        best = min(best, ev[0].elapsed_time(ev[1]) * 1e3 / 20)
    return best


@pytest.mark.parametrize("sample_bits", [32, 8])
def test_few_packets_take_little_time(mdt, cuda, sample_bits):
    # a quarter of what sixty times the packets take
    assert us_per_call(mdt, sample_bits, 600) < us_per_call(mdt, sample_bits, 37200) / 4


@pytest.mark.parametrize("bits", [32, 8])
@pytest.mark.parametrize("npk", [1, 3, 4, 5, 127])
def test_calls_of_any_length(mdt, cuda, bits, npk):
    """The window's packets in calls of npk; 8000 packets at once for the other end."""
    ne, nch, sper, nsp = 38, 64, 28, 40
    rng = np.random.default_rng(npk)
    fd = fmt_dict(sper, bits=bits)
    shape = (nsp + 1, ne, nch, 2)
    words = rand_words(rng, shape) if bits == 32 else \
        rng.integers(-128, 128, shape).astype(np.int8)
    pk, _ = packetise(words, ne, nch, range(nsp * nch // sper), fd)
    at_once = Depack(mdt, fd, ne, nch, 0, nsp)
    at_once.push(np.concatenate([pk] * (8000 // len(pk) + 1)))
    at_once.finish()
    d = Depack(mdt, fd, ne, nch, 0, nsp)
    for i in range(0, len(pk), npk):
        d.push(pk[i:i + npk])
    st = d.finish()
    assert st["accepted"] == len(pk) and st["duplicate"] == 0 and st["outside"] == 0
    a, b = at_once.out.cpu().numpy(), d.out.cpu().numpy()
    assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    last = nsp * nch // sper * sper          # samples up to here came
    if bits == 8:
        flat = np.transpose(words[:nsp], (0, 2, 1, 3)).reshape(nsp * nch, ne, 2)
        got = np.transpose(b, (0, 2, 1, 3)).reshape(nsp * nch, ne, 2)
        assert np.array_equal(got[:last], flat[:last])
