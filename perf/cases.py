"""Performance cases of the FX correlator: what its users run, through the
package's public entry points.

listed() names the cases, draw(rng) gives more of the same ranges,
prepare(case, seed) makes what a user's program holds before the call (inputs
on the GPU, a plan with its window, a batch, a handle), run(state) is one
call and its outputs, work(case) the bytes and operations that the call
cannot do without, exact(case, seed) the same outputs in 64-bit arithmetic by
plain torch.

Samples are int8 I/Q of receiver noise with a per-element sigma of 8 to 24
LSB plus a weak sky source that reaches the elements with integer delays, as
in the package's own configurations; the window is a Hamming windowed sinc
(or, in the reference's own call sequence, a min. 4-term Blackman-Harris
windowed sinc) handed to the plan by the caller.
"""
import importlib
import math

import numpy as np
import torch

mdt = importlib.import_module("mdt_fpga-gpu_pipeline_gb300")
adjoint = importlib.import_module("mdt_fpga-gpu_pipeline_gb300.adjoint")

PREC = {"fp32": mdt.MDT_PREC_FP32, "f16": mdt.MDT_PREC_FP16, "bf16": mdt.MDT_PREC_BF16,
        "int8": mdt.MDT_PREC_INT8}
SNAP_INPUTS = (10, 10, 10, 8)  # the SNAP boards of one station
DEV = "cuda"


# ------------------------------------------------------------------ cases
def _fx(name, prec, ne, nch, ntaps, nsp, nint, acc=False):
    return {"name": name, "kind": "fx", "prec": prec, "ne": ne, "nch": nch, "ntaps": ntaps,
            "nsp": nsp, "nint": nint, "acc": acc}


def listed():
    return [
        # a short integration of one SNAP board's ten inputs, as a laboratory
        # bench or a test of the station runs it: launches and latency
        _fx("fp32_snap10_short", "fp32", 10, 1024, 4, 64, 1),
        # one SNAP board, one integration (configuration c1)
        _fx("fp32_snap10", "fp32", 10, 1024, 4, 1000, 1),
        # a station of 40 inputs, integrations streamed with the PFB history
        # carried (configuration c2), the default precision
        _fx("fp32_station40", "fp32", 40, 2048, 8, 4096, 2),
        # the 256-input array (configuration c3) at the default precision, a
        # quarter of its integration time
        _fx("fp32_array256", "fp32", 256, 1024, 8, 2048, 1),
        # the 256-input array at full size on the tensor-core path: the
        # headline workload, two streamed integrations
        _fx("f16_array256", "f16", 256, 1024, 8, 8192, 2),
        # a station in bf16 with the FP64 sum over integrations
        _fx("bf16_station40", "bf16", 40, 2048, 8, 4096, 2, acc=True),
        # the array with exact integer correlation
        _fx("int8_array256", "int8", 256, 1024, 8, 4096, 1),
        # independent sub-array jobs of uneven shape in one batch
        # (configuration c4's generator)
        {"name": "batch_ragged8", "kind": "batch", "njobs": 8, "jobs_seed": 404, "most": 8192},
        # the reference client's own call sequence on complex64 samples at the
        # instrument's default parameters (19 antennas x 2 polarisations)
        {"name": "dropin_station38", "kind": "dropin", "ne": 38, "nch": 1024, "ntaps": 8,
         "nsp": 1024},
        # one gradient step of a gain and tap calibration (configuration c5)
        {"name": "gaincal64", "kind": "grad", "ne": 64, "nch": 512, "ntaps": 4, "nsp": 2048},
        # one integration of int32 SNAP packets (28 samples an input) of one
        # station into the sample array, lost packets zero-filled
        {"name": "depack_station38", "kind": "depack", "nst": 1, "nch": 1024, "nsp": 1024,
         "sper": 28, "bits": 32, "lost": 0.001},
        # the array's visibilities into the reference's baseline order, as
        # each integration is written out
        {"name": "format_array256", "kind": "format", "nel": 128, "npol": 2, "nch": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fx", "fx", "fx", "fx", "fx", "batch", "dropin", "grad", "depack",
                       "format"])
    if kind == "fx":
        prec = rng.choice(["fp32", "fp32", "f16", "bf16", "int8"])
        ne = _log(rng, 3, 300)
        nch = rng.choice([32, 128, 512, 1024, 1024, 1024, 2048])
        if prec == "fp32" and rng.random() < 0.15:
            nch = rng.choice([4096, 16384])
        ne = min(ne, int(math.sqrt(2**27 / nch)))  # the visibilities' size
        ntaps = rng.choice([4, 8, 8, 16])
        nint = rng.choice([1, 1, 2])
        most = 5e8 if prec == "fp32" else 1.5e9  # antenna-samples of a call
        nsp = _log(rng, 16, max(17, min(8192, most / (ne * nch * nint))))
        return {"kind": "fx", "prec": prec, "ne": ne, "nch": nch, "ntaps": ntaps, "nsp": nsp,
                "nint": nint, "acc": rng.random() < 0.25}
    if kind == "batch":
        njobs = rng.randint(2, 8)
        return {"kind": "batch", "njobs": njobs, "jobs_seed": rng.randint(1, 10**6),
                "most": rng.choice([512, 1024, 2048 if njobs > 4 else 4096])}
    nch = rng.choice([256, 512, 1024, 2048])
    if kind == "dropin":
        ne = _log(rng, 3, 128)
        return {"kind": kind, "ne": ne, "nch": nch, "ntaps": rng.choice([4, 8, 16]),
                "nsp": _log(rng, 16, max(17, min(4096, 2e8 / (ne * nch))))}
    if kind == "grad":
        ne = _log(rng, 3, 96)
        return {"kind": kind, "ne": ne, "nch": nch, "ntaps": rng.choice([4, 8]),
                "nsp": _log(rng, 16, max(17, min(4096, 1.2e8 / (ne * nch))))}
    if kind == "depack":
        return {"kind": kind, "nst": rng.choice([1, 1, 2]), "nch": nch,
                "nsp": _log(rng, 16, 1024), "sper": rng.choice([16, 20, 28]),
                "bits": rng.choice([32, 32, 8]), "lost": rng.choice([0.0, 0.001, 0.01])}
    return {"kind": "format", "nel": _log(rng, 3, 128), "npol": rng.choice([1, 2]), "nch": nch}


# ----------------------------------------------------------------- inputs
def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) % (2**62))
    return g


def _iq(ne, nch, nspec, seed, salt=0):
    """int8 I/Q [nspec][ne][nch][2]."""
    g = _gen(seed, salt)
    rng = np.random.default_rng([int(seed) % (2**32), salt, 77])
    sigma = rng.uniform(8.0, 24.0, ne)
    delay = rng.integers(0, 80, ne)
    n = nspec * nch
    sky = torch.randn(n + 80, 2, generator=g, device=DEV, dtype=torch.float32) * 3.0
    iq = torch.empty(nspec, ne, nch, 2, dtype=torch.int8, device=DEV)
    for e in range(ne):
        x = torch.randn(n, 2, generator=g, device=DEV, dtype=torch.float32)
        x.mul_(float(sigma[e])).add_(sky[int(delay[e]):int(delay[e]) + n])
        iq[:, e] = x.round_().clamp_(-127, 127).to(torch.int8).view(nspec, nch, 2)
    return iq


def _window(nch, ntaps, kind="hamming"):
    n = torch.arange(ntaps * nch, dtype=torch.float64, device=DEV)
    w = torch.sinc((n - ntaps * nch / 2) / nch)
    t = 2 * math.pi * n / (ntaps * nch)
    if kind == "hamming":
        w = w * (0.54 - 0.46 * torch.cos(t))
    else:
        w = w * (0.35875 - 0.48829 * torch.cos(t) + 0.14128 * torch.cos(2 * t) -
                 0.01168 * torch.cos(3 * t))
    return w.to(torch.float32)


def _cnormal(shape, seed, salt):
    return torch.randn(*shape, dtype=torch.complex64, device=DEV, generator=_gen(seed, salt))


def _total(c):
    return c["nint"] * c["nsp"] + c["ntaps"] - 1


def _jobs(c):
    return [(j.nelements, j.nchannels, j.ntaps, min(j.nspectra, c["most"]))
            for j in mdt.configs.ragged_jobs(c["jobs_seed"], c["njobs"])]


def _complex_samples(c, seed):
    """complex64 samples [nsp + ntaps - 1][ne][nch], as the depacketiser leaves
    them: int32 fixed point with 19 fraction bits."""
    shape = (c["nsp"] + c["ntaps"] - 1, c["ne"], c["nch"], 2)
    x = torch.randn(*shape, generator=_gen(seed, 1), device=DEV, dtype=torch.float32)
    x = (x * (0.5 * 2**19)).round_() * 2.0**-19
    return torch.view_as_complex(x)


def _fixed_samples(c, seed):
    """Packet payload values [packets][sper][inputs][2] (int32 or int8) of all
    stations, and which (station, SNAP, packet) got lost."""
    npk = -(-(c["nsp"] * c["nch"]) // c["sper"])
    nin = c["nst"] * sum(SNAP_INPUTS)
    g = _gen(seed, 2)
    x = torch.randn(npk, c["sper"], nin, 2, generator=g, device=DEV, dtype=torch.float32)
    x = (x * (0.5 * 2**19)).round_().to(torch.int32) if c["bits"] == 32 else \
        (x * 16).round_().clamp_(-127, 127).to(torch.int8)
    lost = torch.rand(c["nst"], len(SNAP_INPUTS), npk, generator=g, device=DEV) < c["lost"]
    return x, lost


def _packets(c, fmt, seed):
    """uint8 [n][packet_bytes] in arrival order (by packet counter)."""
    x, lost = _fixed_samples(c, seed)
    npk = x.shape[0]
    per = 8 if c["bits"] == 32 else 2
    p = torch.zeros(npk, c["nst"], len(SNAP_INPUTS), fmt.packet_bytes, dtype=torch.uint8,
                    device=DEV)
    head = p.view(torch.int32)
    head[..., 0] = torch.arange(c["nst"], device=DEV, dtype=torch.int32)[None, :, None]
    head[..., 1] = torch.arange(len(SNAP_INPUTS), device=DEV, dtype=torch.int32)[None, None, :]
    head[..., 2] = torch.arange(npk, device=DEV, dtype=torch.int32)[:, None, None]
    e = 0
    for s in range(c["nst"]):
        for k, nin in enumerate(SNAP_INPUTS):
            pay = x[:, :, e:e + nin].contiguous().view(torch.uint8).view(npk, -1)
            p[:, s, k, 16:16 + c["sper"] * nin * per] = pay
            e += nin
    keep = ~lost.permute(2, 0, 1)
    return p[keep].contiguous()


def prepare(case, seed):
    c = case
    s = {"case": c}
    if c["kind"] == "fx":
        ne, nch, nsp = c["ne"], c["nch"], c["nsp"]
        s["iq"] = _iq(ne, nch, _total(c), seed)
        s["vis"] = torch.empty(c["nint"], nch, ne, ne, dtype=torch.complex64, device=DEV)
        s["plan"] = mdt.FxPlan(ne, nch, c["ntaps"], nsp, precision=PREC[c["prec"]])
        s["plan"].set_window(_window(nch, c["ntaps"]))
        if c["acc"]:
            s["acc"] = torch.zeros(nch, ne, ne, dtype=torch.complex128, device=DEV)
            s["plan"].set_accumulator(s["acc"])
    elif c["kind"] == "batch":
        jobs = _jobs(c)
        s["iqs"] = [_iq(ne, nch, nsp + nt - 1, seed, j)
                    for j, (ne, nch, nt, nsp) in enumerate(jobs)]
        s["viss"] = [torch.empty(nch, ne, ne, dtype=torch.complex64, device=DEV)
                     for ne, nch, nt, nsp in jobs]
        s["batch"] = mdt.FxBatch(jobs)
        for j, (ne, nch, nt, nsp) in enumerate(jobs):
            s["batch"].set_window(j, _window(nch, nt))
        s["batch"].autotune()
        s["stream"] = torch.cuda.ExternalStream(s["batch"].stream)
    elif c["kind"] == "dropin":
        ne, nch, nsp = c["ne"], c["nch"], c["nsp"]
        s["x"] = _complex_samples(c, seed)
        s["win"] = _window(nch, c["ntaps"], "bh4")
        s["f"] = torch.empty(nsp, ne, nch, dtype=torch.complex64, device=DEV)
        s["xin"] = torch.empty(nch, nsp, ne, dtype=torch.complex64, device=DEV)
        s["v"] = torch.empty(nch, ne, ne, dtype=torch.complex64, device=DEV)
        at = torch.arange(nch, dtype=torch.int64, device=DEV)
        s["xptr"] = s["xin"].data_ptr() + at * (nsp * ne * 8)
        s["vptr"] = s["v"].data_ptr() + at * (ne * ne * 8)
        st = torch.cuda.current_stream()
        s["fft"] = mdt.cufftPlan1d(nch, mdt.CUFFT_C2C, nsp * ne)
        mdt.cufftSetStream(s["fft"], st)
        s["blas"] = mdt.cublasCreate()
        mdt.cublasSetStream(s["blas"], st)
    elif c["kind"] == "grad":
        ne, nch = c["ne"], c["nch"]
        s["iq"] = _iq(ne, nch, c["nsp"] + c["ntaps"] - 1, seed).view(-1)
        s["taps"] = _window(nch, c["ntaps"]).requires_grad_(True)
        s["gains"] = _gains(c, seed).requires_grad_(True)
        s["up"] = _upstream(c, seed)
    elif c["kind"] == "depack":
        s["fmt"] = mdt.packet_format(c["sper"], SNAP_INPUTS, sample_bits=c["bits"])
        s["pk"] = _packets(c, s["fmt"], seed)
        ne = c["nst"] * sum(SNAP_INPUTS)
        words = mdt.depacketise_seen_words(s["fmt"], ne, c["nch"], 0, c["nsp"])
        s["seen"] = torch.zeros(words, dtype=torch.int32, device=DEV)
        s["stats"] = torch.zeros(5, dtype=torch.int64, device=DEV)
        if c["bits"] == 32:
            s["out"] = torch.empty(c["nsp"], ne, c["nch"], dtype=torch.complex64, device=DEV)
        else:
            s["out"] = torch.empty(c["nsp"], ne, c["nch"], 2, dtype=torch.int8, device=DEV)
    else:
        n = c["nel"] * c["npol"]
        s["vis"] = _cnormal((c["nch"], n, n), seed, 5)
        s["out"] = torch.empty(mdt.num_baselines(c["nel"], c["npol"]), c["nch"],
                               dtype=torch.complex64, device=DEV)
    return s


def _gains(c, seed):
    g = _gen(seed, 3)
    shape = (c["nch"], c["ne"])
    amp = 0.8 + 0.4 * torch.rand(*shape, generator=g, device=DEV)
    ph = 2 * math.pi * torch.rand(*shape, generator=g, device=DEV)
    return torch.polar(amp, ph)


def _upstream(c, seed):
    """dL/dV of a squared loss against noisy data: no symmetry to rely on."""
    return _cnormal((c["nch"], c["ne"], c["ne"]), seed, 4)


# -------------------------------------------------------------------- run
def run(state):
    s, c = state, state["case"]
    if c["kind"] == "fx":
        plan, nsp, lead = s["plan"], c["nsp"], c["ntaps"] - 1
        if c["acc"]:
            s["acc"].zero_()
        plan.stream_reset()
        plan.stream_push(s["iq"], s["vis"][0])
        for j in range(1, c["nint"]):
            plan.stream_push(s["iq"][j * nsp + lead:], s["vis"][j])
        return (s["vis"], s["acc"]) if c["acc"] else s["vis"]
    if c["kind"] == "batch":
        here = torch.cuda.current_stream()
        s["stream"].wait_stream(here)
        s["batch"].execute(s["iqs"], s["viss"])
        here.wait_stream(s["stream"])
        return s["viss"]
    if c["kind"] == "dropin":
        ne, nch, nsp = c["ne"], c["nch"], c["nsp"]
        blk = min(nch, 1024)
        mdt.PpS_Batch((nch // blk, nsp, ne), (blk,), nch, c["ntaps"], s["win"], s["x"], s["f"])
        mdt.cufftExecC2C(s["fft"], s["f"], s["f"], mdt.CUFFT_FORWARD)
        mdt.ReorderFOutput(((ne + 31) // 32, (nch + 31) // 32, nsp), (32, 32), ne, nch, s["f"],
                           s["xin"])
        mdt.cublasCgemmBatched(s["blas"], mdt.CUBLAS_OP_N, mdt.CUBLAS_OP_C, ne, ne, nsp,
                               1.0 / nsp, s["xptr"], ne, s["xptr"], ne, 0.0, s["vptr"], ne, nch)
        return s["xin"], s["v"]
    if c["kind"] == "grad":
        v = adjoint.fx_correlate(s["iq"], s["taps"], s["gains"], c["ne"], c["nch"], c["ntaps"],
                                 c["nsp"])
        dtaps, dgains = torch.autograd.grad(v, (s["taps"], s["gains"]), s["up"])
        return v.detach(), dtaps, dgains
    if c["kind"] == "depack":
        ne = c["nst"] * sum(SNAP_INPUTS)
        s["stats"].zero_()
        mdt.depacketise(s["fmt"], s["pk"], s["pk"].shape[0], ne, c["nch"], 0, c["nsp"], s["out"],
                        s["seen"], s["stats"])
        mdt.depacketise_finish(s["fmt"], ne, c["nch"], 0, c["nsp"], s["out"], s["seen"],
                               s["stats"])
        return s["out"], s["stats"]
    mdt.format_baselines(c["nel"], c["npol"], c["nch"], s["vis"], s["out"])
    return s["out"]


# ------------------------------------------------------------------- work
def _fx_work(ne, nch, ntaps, nsp, nint=1, in_bytes=2):
    n = float(ne) * nch * nsp * nint
    return {"bytes": in_bytes * float(ne) * nch * (nint * nsp + ntaps - 1) + 4.0 * ntaps * nch +
            8.0 * ne * ne * nch * nint,
            "flops": n * (4 * ntaps + 5 * math.log2(nch)) + 4.0 * (ne + 1) * n}


def work(case):
    c = case
    if c["kind"] == "fx":
        w = _fx_work(c["ne"], c["nch"], c["ntaps"], c["nsp"], c["nint"])
        if c["acc"]:
            w["bytes"] += 16.0 * c["ne"] * c["ne"] * c["nch"]
        return w
    if c["kind"] == "batch":
        ws = [_fx_work(*j) for j in _jobs(c)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    if c["kind"] == "dropin":
        w = _fx_work(c["ne"], c["nch"], c["ntaps"], c["nsp"], 1, 8)
        w["bytes"] += 8.0 * c["ne"] * c["nch"] * c["nsp"]  # the reordered F-output is an output
        return w
    if c["kind"] == "grad":
        w = _fx_work(c["ne"], c["nch"], c["ntaps"], c["nsp"])
        n = float(c["ne"]) * c["nch"] * c["nsp"]
        w["flops"] += n * (8.0 * c["ne"] + 16 + 5 * math.log2(c["nch"]) + 4 * c["ntaps"])
        w["bytes"] += 8.0 * c["nch"] * c["ne"] * (c["ne"] + 2) + 4.0 * c["ntaps"] * c["nch"]
        return w
    if c["kind"] == "depack":
        n = float(c["nst"] * sum(SNAP_INPUTS)) * c["nch"] * c["nsp"]
        return {"bytes": n * (16 if c["bits"] == 32 else 4), "flops": 0}
    nbl = c["npol"] * (c["npol"] + 1) // 2 * (c["nel"] * (c["nel"] + 1) // 2)
    return {"bytes": 16.0 * nbl * c["nch"], "flops": 0}


# ------------------------------------------------------------------ exact
def _fengine64(samples, win, nch, ntaps, nsp):
    """complex128 [nch][ne][nsp] from samples(e0, e1) -> complex128
    [nsp + ntaps - 1][e1 - e0][nch], a few elements at a time."""
    w = win.to(torch.float64).view(ntaps, 1, nch)
    ne = samples.shape[1]
    out = torch.empty(nch, ne, nsp, dtype=torch.complex128, device=DEV)
    step = max(1, int(2**27 / (nch * (nsp + ntaps))))
    for e in range(0, ne, step):
        x = samples[:, e:e + step]
        if x.dtype == torch.int8:
            x = torch.view_as_complex(x.to(torch.float64))
        x = x.to(torch.complex128)
        p = torch.zeros(nsp, x.shape[1], nch, dtype=torch.complex128, device=DEV)
        for i in range(ntaps):
            p += w[i] * x[i:i + nsp]
        out[:, e:e + step] = torch.fft.fft(p, dim=2).permute(2, 1, 0)
    return out


def _vis64(f):
    """[c][q][r] = mean over s of f[c][r][s] conj(f[c][q][s])."""
    nch, ne, nsp = f.shape
    v = torch.empty(nch, ne, ne, dtype=torch.complex128, device=DEV)
    step = max(1, int(2**28 / (ne * nsp)))
    for a in range(0, nch, step):
        x = f[a:a + step]
        v[a:a + step] = torch.matmul(x.conj(), x.transpose(1, 2)) / nsp
    return v


def exact(case, seed):
    c = case
    if c["kind"] == "fx":
        iq = _iq(c["ne"], c["nch"], _total(c), seed)
        win = _window(c["nch"], c["ntaps"])
        nsp, lead = c["nsp"], c["ntaps"] - 1
        vis = torch.empty(c["nint"], c["nch"], c["ne"], c["ne"], dtype=torch.complex128,
                          device=DEV)
        for j in range(c["nint"]):
            vis[j] = _vis64(_fengine64(iq[j * nsp:(j + 1) * nsp + lead], win, c["nch"],
                                       c["ntaps"], nsp))
        return (vis, vis.sum(0)) if c["acc"] else vis
    if c["kind"] == "batch":
        return [_vis64(_fengine64(_iq(ne, nch, nsp + nt - 1, seed, j), _window(nch, nt), nch, nt,
                                  nsp)) for j, (ne, nch, nt, nsp) in enumerate(_jobs(c))]
    if c["kind"] == "dropin":
        f = _fengine64(_complex_samples(c, seed), _window(c["nch"], c["ntaps"], "bh4"), c["nch"],
                       c["ntaps"], c["nsp"])
        return f.transpose(1, 2).contiguous(), _vis64(f)
    if c["kind"] == "grad":
        return _grad64(c, seed)
    if c["kind"] == "depack":
        if c["bits"] == 8:
            return None
        x, lost = _fixed_samples(c, seed)
        n, nch = c["nsp"] * c["nch"], c["nch"]
        each = [lost[s, k][None].expand(m, -1) for s in range(c["nst"])
                for k, m in enumerate(SNAP_INPUTS)]
        x = x.to(torch.float64) * 2.0**-19
        x[torch.cat(each).t()[:, None].expand(x.shape[:3])] = 0
        x = x.view(-1, x.shape[2], 2)[:n].view(c["nsp"], nch, -1, 2).transpose(1, 2).contiguous()
        return torch.view_as_complex(x), None
    n = c["nel"] * c["npol"]
    at = [(k * c["npol"] + q, j * c["npol"] + p) for j in range(c["nel"])
          for p in range(c["npol"]) for k in range(j, c["nel"]) for q in range(p, c["npol"])]
    at = torch.tensor(at, device=DEV)
    v = _cnormal((c["nch"], n, n), seed, 5)[:, at[:, 0], at[:, 1]].t()
    return torch.roll(v, c["nch"] // 2, 1).to(torch.complex128)


def _grad64(c, seed):
    """V, dL/dtaps and dL/dgains for dL/dV = up, by the chain rule."""
    ne, nch, nt, nsp = c["ne"], c["nch"], c["ntaps"], c["nsp"]
    iq = _iq(ne, nch, nsp + nt - 1, seed)
    win, up = _window(nch, nt), _upstream(c, seed).to(torch.complex128)
    gains = _gains(c, seed).to(torch.complex128)
    f = _fengine64(iq, win, nch, nt, nsp)        # [c][e][s]
    y = gains[:, :, None] * f
    v = _vis64(y)
    g = up.transpose(1, 2)                       # g[c][r][q] = dL/dV_rq
    dy = torch.matmul(g + g.mH, y) / nsp
    dgains = (dy * f.conj()).sum(2)
    del f, y
    df = gains.conj()[:, :, None] * dy
    del dy
    dtaps = torch.zeros(nt, nch, dtype=torch.float64, device=DEV)
    step = max(1, int(2**27 / (nch * (nsp + nt))))
    for e in range(0, ne, step):
        # the adjoint of the unnormalised forward transform
        dp = torch.fft.ifft(df[:, e:e + step].permute(2, 1, 0), dim=2) * nch
        x = torch.view_as_complex(iq[:, e:e + step].to(torch.float64))
        for i in range(nt):
            dtaps[i] += (dp * x[i:i + nsp].conj()).real.sum((0, 1))
    return v, dtaps.view(-1), dgains
