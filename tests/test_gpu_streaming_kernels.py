"""The memory-bound kernels at the edges of their tiles, runs and vector
widths: packet depacketiser, baseline formatter, drop-in PpS and corner turn
(all bit-exact against the oracle or a gather in numpy), and the compensated
gradient sums against FP64 with their results in infinities."""
import numpy as np
import pytest
import torch

from adjref import crandn
from packets import fmt_dict, packetise
from test_gpu_depack import Depack, rand_words
from test_gpu_dropin import bits, dev
from test_gpu_output import ref_gather

pytestmark = pytest.mark.gpu


# sper 40: two runs of a packet; 3 header words: 4-byte copies; 20 inputs of
# int32: a block per packet; 16 inputs: the staging buffer exactly full
@pytest.mark.parametrize("sper,bits_,snaps,hdr", [(28, 32, (10, 10, 10, 8), 4),
                                                  (40, 32, (10, 10, 10, 8), 4),
                                                  (33, 32, (3, 16), 3), (64, 32, (20, 2), 4),
                                                  (32, 8, (64, 1), 4), (9, 8, (5, 7, 1), 3)])
def test_depack_widths_and_runs(mdt, cuda, oracle, sper, bits_, snaps, hdr):
    ne, nch, nsp, s0sp = sum(snaps), 64, 7, 1
    rng = np.random.default_rng(sper + hdr)
    fd = fmt_dict(sper, bits=bits_, snaps=snaps, ips=ne, words_header=hdr)
    npk = -(-((s0sp + nsp + 1) * nch) // sper) + 1
    shape = (npk * sper // nch + 1, ne, nch, 2)
    words = rand_words(rng, shape) if bits_ == 32 else \
        rng.integers(-128, 128, shape).astype(np.int8)
    pk, _ = packetise(words, ne, nch, range(npk), fd)
    keep = rng.permutation(len(pk))[: len(pk) - 3]
    d = Depack(mdt, fd, ne, nch, s0sp * nch, nsp)
    d.push(pk[keep])
    st = d.finish()
    assert st["bad"] == 0 and st["duplicate"] == 0
    assert st["accepted"] + st["outside"] == len(keep)
    got = d.out.cpu().numpy()
    full = Depack(mdt, fd, ne, nch, s0sp * nch, nsp)
    full.push(pk)
    assert full.finish()["missing"] == 0
    if bits_ == 32:
        want, ost = oracle.depacketise(fd, pk[keep], len(keep), ne, nch, s0sp * nch, nsp)
        assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
        assert [st["accepted"], st["outside"], st["bad"]] == ost
    else:
        want = words[s0sp:s0sp + nsp]
        assert np.array_equal(full.out.cpu().numpy(), want)
        assert np.all((got == want) | (got == 0))


@pytest.mark.parametrize("nel,npol,nch", [(33, 2, 130), (64, 1, 64), (65, 3, 62)])
def test_format_tiles(mdt, cuda, nel, npol, nch):
    rng = np.random.default_rng(nel + nch)
    V = crandn(rng, nch, (nel * npol) ** 2).astype(np.complex64)
    out = torch.full((mdt.num_baselines(nel, npol), nch), complex(9, 9), dtype=torch.complex64,
                     device="cuda")
    mdt.format_baselines(nel, npol, nch, dev(V), out)
    want = ref_gather(V, nel, npol, nch, True)
    assert np.array_equal(out.cpu().numpy().view(np.uint64), want.view(np.uint64))


# enough blocks for runs of 16 spectra (the last of 3) and of 32 (the last of 11)
@pytest.mark.parametrize("nsp", [2563, 5003])
@pytest.mark.parametrize("ntaps", [4, 8, 16, 5])
def test_pps_runs(mdt, cuda, oracle, ntaps, nsp):
    nch, ne = 64, 8
    rng = np.random.default_rng(ntaps)
    x = crandn(rng, nsp + ntaps - 1, ne, nch).astype(np.complex64)
    w = rng.standard_normal(ntaps * nch).astype(np.float32)
    out = torch.full((nsp, ne, nch), float("nan"), dtype=torch.complex64, device="cuda")
    mdt.PpS_Batch((1, nsp, ne), (1024,), nch, ntaps, dev(w), dev(x), out)
    want = oracle.pps_f32_exact(w, x, nch, ntaps, ne, nsp)
    assert np.array_equal(bits(out).ravel(), np.asarray(want).view(np.uint32).ravel())


@pytest.mark.parametrize("ne,nch,nsp", [(5, 34, 13), (38, 64, 27), (1, 31, 2), (64, 130, 3)])
def test_reorder_tiles(mdt, cuda, oracle, ne, nch, nsp):
    rng = np.random.default_rng(ne)
    F = crandn(rng, nsp * ne * nch).astype(np.complex64)
    X = torch.full((nsp * ne * nch,), float("nan"), dtype=torch.complex64, device="cuda")
    mdt.ReorderFOutput(((ne + 31) // 32, (nch + 31) // 32, nsp), (32, 32), ne, nch, dev(F), X)
    assert np.array_equal(bits(X), oracle.reorder_c64(F, ne, nch, nsp).view(np.uint32))


def _tap_grad(mdt, gP, iq, ne, nch, ntaps, nsp):
    gW = torch.empty(ntaps * nch, dtype=torch.float32, device="cuda")
    ws = torch.empty(ntaps * nch * 64, dtype=torch.float64, device="cuda")
    mdt.pfb_tap_grad(ne, nch, ntaps, nsp, gP, iq, gW, ws)
    return gW.cpu().numpy()


# odd Nch, or buffers one value past a 16-byte boundary: one channel a thread;
# Nsp 65 and 70: a last run of one spectrum and one that is no multiple of the taps
@pytest.mark.parametrize("ne,nch,ntaps,nsp,off", [(3, 33, 4, 65, 0), (2, 64, 8, 70, 0),
                                                  (2, 64, 8, 31, 1), (1, 130, 4, 2, 0),
                                                  (3, 40, 6, 12, 0)])
def test_tap_grad_sums(mdt, cuda, ne, nch, ntaps, nsp, off):
    rng = np.random.default_rng(nsp)
    iq = rng.integers(-128, 128, size=(nsp + ntaps - 1, ne, nch, 2)).astype(np.int8)
    gP = crandn(rng, nsp, ne, nch).astype(np.complex64)
    buf = torch.empty(gP.size + off, dtype=torch.complex64, device="cuda")
    g = buf[off:]
    g.copy_(dev(gP).view(-1))
    x = iq[..., 0].astype(np.float64) + 1j * iq[..., 1]
    want = np.stack([np.real(np.sum(gP * np.conj(x[i:i + nsp]), axis=(0, 1)))
                     for i in range(ntaps)])
    got = _tap_grad(mdt, g, dev(iq), ne, nch, ntaps, nsp).reshape(ntaps, nch)
    # one FP32 rounding of each sum, which may cancel: half an ulp (6e-8) of the
    # result and 2^-44 of the sum of magnitudes
    mag = np.sum(np.abs(gP), axis=(0, 1)) * 256
    assert np.all(np.abs(got - want) <= 6e-8 * np.abs(want) + 2.0 ** -44 * mag)
    # an infinite gradient makes exactly the sums infinite or NaN that double sums give
    gP[nsp // 2, 0, 5] = complex(np.inf, 1.0)
    iq[nsp // 2:nsp // 2 + ntaps, 0, 5] = 3
    g.copy_(dev(gP).view(-1))
    got = _tap_grad(mdt, g, dev(iq), ne, nch, ntaps, nsp).reshape(ntaps, nch)
    assert np.all(np.isposinf(got[:, 5])) and np.all(np.isfinite(np.delete(got, 5, axis=1)))


@pytest.mark.parametrize("ne,nch,nsp,off", [(7, 33, 19, 0), (6, 40, 9, 0), (6, 40, 9, 1),
                                            (1, 3, 300, 0), (2, 70, 33, 0)])
def test_gain_sums_and_rows(mdt, cuda, ne, nch, nsp, off):
    rng = np.random.default_rng(ne * nsp)
    n = nch * nsp * ne

    def at(a):
        buf = torch.empty(a.size + off, dtype=torch.complex64, device="cuda")
        buf[off:].copy_(dev(a).view(-1))
        return buf[off:]

    dY, X = (crandn(rng, nch, nsp, ne).astype(np.complex64) for _ in range(2))
    g = crandn(rng, nch, ne).astype(np.complex64)
    dX, ddY, dg_ = at(X), at(dY), at(g)
    out = torch.empty(nch, ne, dtype=torch.complex64, device="cuda")
    dF = torch.empty(nsp, ne, nch, dtype=torch.complex64, device="cuda")
    mdt.gain_adjoint(ne, nch, nsp, ddY, X=dX, gains=dg_, dgains=out, dF=dF)
    Y = torch.empty(n + off, dtype=torch.complex64, device="cuda")[off:]
    mdt.apply_gains(ne, nch, nsp, dX, dg_, Y)
    z = dY.astype(np.complex128) * np.conj(X)
    err = out.cpu().numpy() - z.sum(axis=1)
    tol = 6e-8 * np.abs(z.sum(axis=1)) * 2 + 2.0 ** -44 * np.abs(z).sum(axis=1)
    assert np.all(np.abs(err.real) <= tol) and np.all(np.abs(err.imag) <= tol)
    g128 = g.astype(np.complex128)[:, None, :]
    # one complex product of three roundings: under 2^-22 of its magnitude
    wantF = np.transpose(np.conj(g128) * dY, (1, 2, 0))
    assert np.all(np.abs(dF.cpu().numpy() - wantF) <= 2.0 ** -22 * np.abs(wantF))
    wantY = g128 * X
    got = Y.cpu().numpy().reshape(nch, nsp, ne)
    assert np.all(np.abs(got - wantY) <= 2.0 ** -22 * np.abs(wantY))
    X[1, nsp // 2, 0] = complex(np.inf, 0.0)
    mdt.gain_adjoint(ne, nch, nsp, ddY, X=at(X), gains=dg_, dgains=out)
    got = out.cpu().numpy()
    assert not np.isfinite(got[1, 0]) and np.isinf(got[1, 0].real)
    got[1, 0] = 0
    assert np.all(np.isfinite(got))


# one chunk of 64 elements kept over several tiles of 64 spectra, a second block of
# tiles, and two chunks
@pytest.mark.parametrize("ne,nch,nsp", [(64, 2, 300), (65, 1, 257), (7, 3, 520)])
def test_xengine_adjoint_tiles(mdt, cuda, ne, nch, nsp):
    rng = np.random.default_rng(ne + nsp)
    G = crandn(rng, nch, ne, ne).astype(np.complex64)
    Y = crandn(rng, nch, nsp, ne).astype(np.complex64)
    dY = torch.full((nch, nsp, ne), float("nan"), dtype=torch.complex64, device="cuda")
    mdt.xengine_adjoint_f32(ne, nch, nsp, dev(G), dev(Y), dY, 0.5)
    Gm = np.transpose(G.astype(np.complex128), (0, 2, 1))
    H = Gm + np.conj(np.transpose(Gm, (0, 2, 1)))
    want = 0.5 * np.einsum("crq,csq->csr", H, Y.astype(np.complex128))
    # four multiply-adds per q: under 4 NE 2^-24 of the sum of magnitudes
    mag = 0.5 * np.einsum("crq,csq->csr", np.abs(H), np.abs(Y))
    assert np.all(np.abs(dY.cpu().numpy() - want) <= 4 * ne * 2.0 ** -24 * mag)
