"""Workloads of the dedispersion engine for timing and comparison.

Each case is one call that a search program makes through the public Python
mirror of the C API: a time-domain plan on device or host buffers, a batch of
beams, or a Fourier-domain plan. Frequency setups are the ones of the
repository's benchmark configurations (1024 channels below 1581.8 MHz at 250
us, 4096 channels below 1500 MHz at 64 us, 1536 channels below 1670 MHz at
81.92 us) and a small 64-channel one; sample counts are cut where a full
observation would not fit the card several times.

`exact` is plain torch in 64 bits: shifted sums channel by channel, and a
64-bit FFT of them where the output is a spectrum.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import dedisp_tests_b200 as dd

# f_top (MHz), bandwidth (MHz), sampling time (s) of the setups
SETUPS = {
    "small": (1500.0, -64.0, 250e-6),
    "survey": (1581.8, -400.0, 250e-6),
    "fine": (1500.0, -320.0, 64e-6),
    "beams": (1670.0, -384.0, 81.92e-6),
}

# shifted sums above this many terms would take `exact` too long
EXACT_TERMS = 1.2e12


def _params(case):
    f0, band, dt = SETUPS[case["setup"]]
    return case["nchans"], dt, f0, band / case["nchans"]


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # Smallest call: a quick look at one short subband, host arrays in and
        # out as the C API's default; bound by launches and latency.
        {"name": "tdd_host_small_u8", "kind": "tdd", "setup": "small", "nchans": 64, "nsamps": 8192,
         "nbits": 8, "out_nbits": 32, "ndm": 32, "dm_max": 100.0, "host": True},
        # An ordinary search call: one 16 s block of a 1024-channel survey,
        # 512 trials, buffers already on the device.
        {"name": "tdd_1024ch_u8", "kind": "tdd", "setup": "survey", "nchans": 1024, "nsamps": 65536,
         "nbits": 8, "out_nbits": 32, "ndm": 512, "dm_max": 500.0, "host": False},
        # The same search fed from pinned host memory, with the input and
        # output copies inside the call.
        {"name": "tdd_host_1024ch_u8", "kind": "tdd", "setup": "survey", "nchans": 1024, "nsamps": 262144,
         "nbits": 8, "out_nbits": 32, "ndm": 512, "dm_max": 500.0, "host": True},
        # The production search: 4096 fine channels and the tolerance-spaced
        # DM list, one 17 s gulp of it.
        {"name": "tdd_4096ch_u8", "kind": "tdd", "setup": "fine", "nchans": 4096, "nsamps": 262144,
         "nbits": 8, "out_nbits": 32, "ndm": 3643, "dm_max": 2000.0, "generated": True, "host": False},
        # 4-bit recordings, an odd sample count and an odd trial count, and
        # 8-bit output for a compact archive of the trials.
        {"name": "tdd_4096ch_u4_odd", "kind": "tdd", "setup": "fine", "nchans": 4096, "nsamps": 150001,
         "nbits": 4, "out_nbits": 8, "ndm": 1801, "dm_max": 2000.0, "host": False},
        # A streaming gulp at 2 bits: 65536 new samples after the overlap
        # tail of the largest delay, 2048 trials.
        {"name": "tdd_gulp_4096ch_u2", "kind": "tdd", "setup": "fine", "nchans": 4096, "nsamps": 92160,
         "nbits": 2, "out_nbits": 32, "ndm": 2048, "dm_max": 1500.0, "host": False},
        # 16-bit samples of a coherently summed beam.
        {"name": "tdd_1024ch_u16", "kind": "tdd", "setup": "survey", "nchans": 1024, "nsamps": 65536,
         "nbits": 16, "out_nbits": 32, "ndm": 512, "dm_max": 500.0, "host": False},
        # Several beams of uneven length and DM range in one batch launch.
        {"name": "tdd_batch_1536ch_u8", "kind": "batch", "setup": "beams", "nchans": 1536, "nbits": 8,
         "beams": "131072:1024:500,170001:1500:1200,98304:777:800"},
        # Fourier domain with the plan's default precision: segmented, 32-bit
        # float samples.
        {"name": "fdd_f32_1024ch", "kind": "fdd", "setup": "survey", "nchans": 1024, "nsamps": 262144,
         "nbits": 32, "ndm": 512, "dm_max": 500.0, "segmented": 1, "precision": 0, "segment": "32768"},
        # Fourier domain with every option at its default: the whole-series
        # spectrum of 8-bit samples.
        {"name": "fdd_spectrum_1024ch_u8", "kind": "fdd", "setup": "survey", "nchans": 1024, "nsamps": 131072,
         "nbits": 8, "ndm": 512, "dm_max": 500.0, "segmented": 0, "precision": 0, "segment": "0"},
        # Fourier domain on the tensor cores: the 2048-trial search in
        # 32768-point segments.
        {"name": "fdd_tc_1024ch", "kind": "fdd", "setup": "survey", "nchans": 1024, "nsamps": 524288,
         "nbits": 32, "ndm": 2048, "dm_max": 1000.0, "segmented": 1, "precision": 1, "segment": "32768"},
        # Several uneven beams in one Fourier-domain batch.
        {"name": "fdd_batch_1536ch_u8", "kind": "fdd_batch", "setup": "beams", "nchans": 1536, "nbits": 8,
         "segment": "auto", "beams": "131072:1024:500,170001:1500:1200"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_beams(rng, max_samples, max_dms):
    beams = []
    for _ in range(rng.randint(1, 3)):
        beams.append(f"{_log_int(rng, 65536, max_samples)}:{_log_int(rng, 100, max_dms)}:{_log_int(rng, 100, 1200)}")
    return ",".join(beams)


def draw(rng):
    """One more case of the same ranges: any width, odd sample and trial
    counts, ragged channel counts."""
    kind = rng.choice(["tdd", "tdd", "tdd", "tdd", "batch", "fdd", "fdd", "fdd_batch"])
    if kind == "batch":
        return {"kind": kind, "setup": "beams", "nchans": 1536, "nbits": rng.choice([2, 4, 8, 8]),
                "beams": _draw_beams(rng, 170000, 1500)}
    if kind == "fdd_batch":
        return {"kind": kind, "setup": "beams", "nchans": 1536, "nbits": 8, "segment": rng.choice(["0", "auto"]),
                "beams": _draw_beams(rng, 131072, 1200)}
    if kind == "fdd":
        segmented = rng.randint(0, 1)
        return {"kind": kind, "setup": "survey", "nchans": 32 * rng.randint(1, 32),
                "nsamps": _log_int(rng, 16384, 262144), "nbits": rng.choice([8, 8, 32]),
                "ndm": _log_int(rng, 16, 1024), "dm_max": float(_log_int(rng, 50, 1000)), "segmented": segmented,
                "precision": rng.randint(0, 1), "segment": rng.choice(["0", "32768"]) if segmented else "0"}
    setup = rng.choice(["small", "survey", "fine", "beams"])
    nbits = rng.choice([1, 2, 4, 8, 8, 8, 16])
    most = {"small": 256, "survey": 1024, "fine": 4096, "beams": 1536}[setup]
    step = max(1, 32 // nbits)
    nchans = step * max(1, _log_int(rng, 32, most) // step)
    dm_max = float(_log_int(rng, 50, {"small": 500, "survey": 500, "fine": 1500, "beams": 1200}[setup]))
    return {"kind": "tdd", "setup": setup, "nchans": nchans, "nsamps": _log_int(rng, 4096, 131072) + 36000,
            "nbits": nbits, "out_nbits": rng.choice([8, 16, 32, 32, 32]), "ndm": _log_int(rng, 8, 2048),
            "dm_max": dm_max, "host": rng.random() < 0.25}


# ---------------------------------------------------------------------------
# Inputs, plans, passes
# ---------------------------------------------------------------------------

def _dm_list(ndm, dm_max):
    return (dm_max * np.arange(ndm) / max(ndm - 1, 1)).astype(np.float32)


def _beam_specs(case):
    return [(int(n), int(m), float(d)) for n, m, d in (b.split(":") for b in case["beams"].split(","))]


def _filterbank(nsamps, nchans, nbits, seed):
    """Time-major noise rows with a few broadband pulses, packed LSB first
    (32 bits: IEEE floats), as a uint8 CUDA tensor [nsamps][row bytes]."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    row_bytes = nchans * nbits // 8
    out = torch.empty((nsamps, row_bytes), dtype=torch.uint8, device="cuda")
    sigma = {1: 0.5, 2: 1.0, 4: 3.0, 8: 16.0, 16: 2000.0, 32: 1.0}[nbits]
    mean = 0.0 if nbits == 32 else (2 ** nbits - 1) / 2.0
    pulses = torch.randint(0, nsamps, (4,), generator=g, device="cuda")
    rows = max(1, (1 << 27) // nchans)
    for r0 in range(0, nsamps, rows):
        r1 = min(nsamps, r0 + rows)
        x = torch.randn((r1 - r0, nchans), generator=g, device="cuda")
        t = torch.arange(r0, r1, device="cuda")[:, None]
        x.add_((((t - pulses).abs() < 4).sum(1, keepdim=True)).float())
        x.mul_(sigma).add_(mean)
        if nbits == 32:
            out[r0:r1] = x.view(torch.uint8).view(r1 - r0, row_bytes)
            continue
        q = x.round_().clamp_(0, 2 ** nbits - 1).to(torch.int32)
        if nbits == 16:
            lo, hi = (q & 255).to(torch.uint8), (q >> 8).to(torch.uint8)
            out[r0:r1] = torch.stack((lo, hi), dim=2).view(r1 - r0, row_bytes)
        else:
            per = 8 // nbits
            shift = torch.arange(per, device="cuda", dtype=torch.int32) * nbits
            out[r0:r1] = (q.view(r1 - r0, row_bytes, per) << shift).sum(2).to(torch.uint8)
    return out


# 16-bit outputs are held as int16 bit patterns
OUT_DTYPE = {8: torch.uint8, 16: torch.int16, 32: torch.float32}


def _tdd_plan(case):
    p = dd.TDDPlan(*_params(case))
    if case.get("generated"):
        p.generate_dm_list(0.0, case["dm_max"], 40.0, 1.25)
    else:
        p.set_dm_list(_dm_list(case["ndm"], case["dm_max"]))
    return p


def prepare(case, seed):
    kind, nbits = case["kind"], case["nbits"]
    if kind == "tdd":
        p = _tdd_plan(case)
        x = _filterbank(case["nsamps"], case["nchans"], nbits, seed)
        shape = (p.get_dm_count(), case["nsamps"] - p.get_max_delay())
        if case["host"]:
            x = x.cpu().pin_memory()
            y = torch.zeros(shape, dtype=OUT_DTYPE[case["out_nbits"]]).pin_memory()
            flags = 0
        else:
            y = torch.zeros(shape, dtype=OUT_DTYPE[case["out_nbits"]], device="cuda")
            flags = dd.DEDISP_DEVICE_POINTERS
        torch.cuda.synchronize()
        return {"kind": kind, "plan": p, "nsamps": case["nsamps"], "in": x, "nbits": nbits, "out": y,
                "out_nbits": case["out_nbits"], "flags": flags}
    if kind == "fdd":
        p = dd.FDDGPUPlan(*_params(case))
        p.set_dm_list(_dm_list(case["ndm"], case["dm_max"]))
        p.set_options(segmented=case["segmented"], precision=case["precision"], segment_nfft=int(case["segment"]))
        x = _filterbank(case["nsamps"], case["nchans"], nbits, seed)
        y = torch.zeros((case["ndm"], p.output_row_length(case["nsamps"])), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        return {"kind": kind, "plan": p, "nsamps": case["nsamps"], "in": x, "nbits": nbits, "out": y,
                "out_nbits": 32, "flags": dd.DEDISP_DEVICE_POINTERS}
    specs = _beam_specs(case)
    if kind == "batch":
        b = dd.Batch(*_params(case), in_nbits=nbits, out_nbits=32)
    else:
        b = dd.FddBatch(*_params(case), in_nbits=nbits)
        b.set_segment_nfft("auto" if case["segment"] == "auto" else int(case["segment"]))
    probe = dd.TDDPlan(*_params(case))
    beams, outs = [], []
    for i, (nsamps, ndm, dm_max) in enumerate(specs):
        dms = _dm_list(ndm, dm_max)
        probe.set_dm_list(dms)
        x = _filterbank(nsamps, case["nchans"], nbits, seed + 1000 * i)
        y = torch.zeros((ndm, nsamps - probe.get_max_delay()), dtype=torch.float32, device="cuda")
        beams.append((x, x.shape[1], nsamps, dms, y, 4 * y.shape[1]))
        outs.append(y)
    b.set_beams(beams)
    torch.cuda.synchronize()
    return {"kind": kind, "batch": b, "out": outs}


def run(state):
    if "plan" in state:
        state["plan"].execute(state["nsamps"], state["in"], state["nbits"], state["out"], state["out_nbits"],
                              state["flags"])
    else:
        # execute only enqueues; sync waits for it and reports its errors
        state["batch"].execute()
        state["batch"].sync()
    return state["out"]


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------

def _delays(case):
    """Channel delays in samples per unit DM, float32 as the API defines them."""
    nchans, dt, f0, df = _params(case)
    f0, df = np.float32(f0), -np.abs(np.float32(df))
    a = np.float32(1.0) / (f0 + np.arange(nchans, dtype=np.float32) * df)
    b = np.float32(1.0) / f0
    return (4.15e3 / np.float64(np.float32(dt)) * (a * a - b * b).astype(np.float64)).astype(np.float32)


def _max_delay(case, dm_last):
    return int(np.float64(np.float32(dm_last) * _delays(case)[-1]) + 0.5)


def _fft_length(case, max_delay):
    if not case["segmented"]:
        return -(-(case["nsamps"] + max_delay) // 16384) * 16384
    n = int(case["segment"])
    if not n:
        n = 16384
        while n * (1.0 - float(np.float32(0.8))) < max_delay:
            n *= 2
    return n


def work(case):
    """Inputs read once, outputs written once; one addition per trial, output
    sample and channel (time domain), or the forward transforms, a complex
    multiply-add per trial, channel and bin, and the inverse transforms."""
    nchans, nbits, kind = case["nchans"], case["nbits"], case["kind"]
    if kind in ("batch", "fdd_batch"):
        series = _beam_specs(case)
    else:
        series = [(case["nsamps"], case["ndm"], case["dm_max"])]
    nbytes = flops = 0.0
    for nsamps, ndm, dm_max in series:
        nout = nsamps - _max_delay(case, dm_max)
        out_bytes = case.get("out_nbits", 32) // 8
        if kind == "fdd" and not case["segmented"]:
            n = _fft_length(case, nsamps - nout)
            nbytes += nsamps * nchans * nbits / 8 + ndm * n * 4
            flops += nchans * 2.5 * n * math.log2(n) + 8.0 * nchans * ndm * (n / 2)
        elif kind in ("fdd", "fdd_batch"):
            nbytes += nsamps * nchans * nbits / 8 + ndm * nout * 4
            flops += (nchans * nsamps + ndm * nout) * 2.5 * 15 + 8.0 * nchans * ndm * (nout / 2)
        else:
            nbytes += nsamps * nchans * nbits / 8 + ndm * nout * out_bytes
            flops += float(nchans) * ndm * nout
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------

def _channel(x, c, nbits):
    """Samples of channel c as a float64 vector."""
    if nbits == 32:
        return x[:, 4 * c:4 * c + 4].contiguous().view(torch.float32)[:, 0].double()
    if nbits == 16:
        return x[:, 2 * c].double() + 256.0 * x[:, 2 * c + 1].double()
    per = 8 // nbits
    return ((x[:, c // per] >> ((c % per) * nbits)) & (2 ** nbits - 1)).double()


def _shifted_sums(x, nbits, delay, nout, offset):
    """[ndm][nout] float64: sum over channels of (sample + offset) at
    t + delay[dm][channel], trials in chunks that bound the memory."""
    ndm, nchans = delay.shape
    out = torch.zeros((ndm, nout), dtype=torch.float64, device="cuda")
    d = torch.as_tensor(delay, device="cuda")
    step = max(1, (1 << 28) // max(nout, 1))
    for c in range(nchans):
        w = (_channel(x, c, nbits) + offset).unfold(0, nout, 1)
        for i in range(0, ndm, step):
            out[i:i + step] += w[d[i:i + step, c]]
    return out


def _fdd_exact(x, case, nsamps, ndm, dm_max, nfft):
    nchans, nbits = case["nchans"], case["nbits"]
    # integer delays: truncated float32 products
    d = np.trunc(_dm_list(ndm, dm_max)[:, None] * _delays(case)[None, :]).astype(np.int64)
    mid = 0.0 if nbits == 32 else (2 ** nbits - 1) / 2.0
    if not nfft:
        return _shifted_sums(x, nbits, d, nsamps - _max_delay(case, dm_max), -mid) / nchans
    z = torch.zeros((ndm, nfft), dtype=torch.float64, device="cuda")
    for c in range(nchans):
        v = torch.zeros(2 * nfft, dtype=torch.float64, device="cuda")
        v[:nsamps] = _channel(x, c, nbits) - mid
        v[nfft:] = v[:nfft].clone()  # circular
        z += v.unfold(0, nfft, 1)[torch.as_tensor(d[:, c] % nfft, device="cuda")]
    s = torch.view_as_real(torch.fft.rfft(z)[:, :nfft // 2] / nchans)
    return s.reshape(ndm, nfft)


def exact(case, seed):
    kind, nchans, nbits = case["kind"], case["nchans"], case["nbits"]
    if work(case)["flops"] / (8.0 if kind.startswith("fdd") else 1.0) > EXACT_TERMS:
        return None
    if kind in ("batch", "fdd_batch"):
        series = [(n, m, d, seed + 1000 * i) for i, (n, m, d) in enumerate(_beam_specs(case))]
    else:
        series = [(case["nsamps"], case["ndm"], case["dm_max"], seed)]
    outs = []
    for nsamps, ndm, dm_max, s in series:
        x = _filterbank(nsamps, nchans, nbits, s)
        if kind in ("fdd", "fdd_batch"):
            whole = kind == "fdd" and not case["segmented"]
            nfft = _fft_length(case, _max_delay(case, dm_max)) if whole else 0
            outs.append(_fdd_exact(x, case, nsamps, ndm, dm_max, nfft))
            continue
        if case.get("out_nbits", 32) != 32 or case.get("generated"):
            return None  # whole numbers, or the list is the library's own
        # delays rounded half to even; sums scaled to the output range
        d = np.rint(_dm_list(ndm, dm_max)[:, None] * _delays(case)[None, :]).astype(np.int64)
        y = _shifted_sums(x, nbits, d, nsamps - _max_delay(case, dm_max), 0.0)
        y *= 3.0 * 1024.0 / 255.0 / 16.0 / ((2 ** nbits - 1) * float(nchans))
        outs.append(y.cpu() if case.get("host") else y)
    return outs if kind in ("batch", "fdd_batch") else outs[0]
