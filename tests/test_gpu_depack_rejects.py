"""Depacketiser: rejected packets (no such SNAP, no such station, counters before and
after the window) among accepted ones.  A warp takes eight packets in turn through two
staging buffers, so a rejected packet's payload must not reach the packet two later.
Bit-exact against the oracle, for both copy widths and one and two runs of samples."""
import numpy as np
import pytest
import torch

from packets import fmt_dict, packetise
from test_gpu_depack import Depack, rand_words

pytestmark = pytest.mark.gpu


def rejects(rng, pk, fd, n, beyond):
    """n packets of random payload that no window takes: a third each of an unknown SNAP,
    an unknown station and a counter from `beyond` on or before the window."""
    out = pk[rng.integers(0, len(pk), n)].copy()
    hb = 4 * fd["words_header"]
    out[:, hb:] = rng.integers(0, 256, out[:, hb:].shape, dtype=np.uint8)
    head = out[:, :12].copy().view(np.uint32)
    kind = rng.integers(0, 3, n)
    head[kind == 0, 1] = len(fd["inputs_per_snap"]) + rng.integers(0, 5)
    head[kind == 1, 0] = 1000
    late = rng.integers(0, 2, n) * (beyond + 5)
    head[kind == 2, 2] = late[kind == 2]
    out[:, :12] = head.view(np.uint8)
    return out


@pytest.mark.parametrize("sper,bits,snaps,hdr", [(28, 32, (10, 10, 10, 8), 4),
                                                 (40, 32, (10, 10, 10, 8), 4),
                                                 (33, 32, (3, 16), 3), (32, 8, (64, 1), 4),
                                                 (9, 8, (5, 7, 1), 3)])
@pytest.mark.parametrize("pattern", ["mixed", "runs", "every_other"])
def test_rejected_packets(mdt, cuda, oracle, sper, bits, snaps, hdr, pattern):
    ne, nch, nsp, s0sp = sum(snaps), 64, 60, 2
    rng = np.random.default_rng(sper * 7 + len(pattern))
    fd = fmt_dict(sper, bits=bits, snaps=snaps, ips=ne, words_header=hdr)
    last = -(-(s0sp + nsp) * nch // sper)
    shape = (last * sper // nch + 2, ne, nch, 2)
    words = rand_words(rng, shape) if bits == 32 else \
        rng.integers(-128, 128, shape).astype(np.int8)
    good, _ = packetise(words, ne, nch, range(s0sp * nch // sper, last), fd)
    junk = rejects(rng, good, fd, 3 * len(good), last)
    # which packets are good: a warp's packets are four apart
    n = np.arange(4 * len(good))
    if pattern == "mixed":
        take = rng.permutation(n) < len(good)
    elif pattern == "runs":          # three of its packets rejected, the next accepted
        take = (n // 4) % 4 == 3
    else:                            # accepted, rejected, accepted, ... by warp and turn
        take = (n // 4 + n) % 2 == 0
    pk = np.empty((len(n), fd["packet_bytes"]), np.uint8)
    gi = np.cumsum(take) - 1
    take &= gi < len(good)
    pk[take] = good[gi[take]]
    pk[~take] = junk[rng.integers(0, len(junk), int((~take).sum()))]
    for _ in range(3):
        d = Depack(mdt, fd, ne, nch, s0sp * nch, nsp)
        d.push(pk)
        st = d.finish()
        want, ost = oracle.depacketise(fd, pk, len(pk), ne, nch, s0sp * nch, nsp)
        assert [st["accepted"], st["outside"], st["bad"]] == ost
        assert st["accepted"] == int(take.sum())
        got = d.out.cpu().numpy()
        assert np.array_equal(got.view(np.uint8), want.view(np.uint8))
