"""Workloads of the receiver-side reduction, through its public entry points.

Each case is one call that a simulation makes once per ping: the plain form
(``Context.reduce``) on 1D and 2D sensors, the precision form from device and
from host memory, a batch of mixed sensors, and the echo-sample epilogue that
turns ray hits into samples. The sensors are those of the repository's own
configurations (``rtac_simulation_gb300/workloads.py``); samples are drawn on
the GPU from the seed.

``exact`` restates every path in 64 bits with torch alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from rtac_simulation_gb300 import _lib

F32 = np.float32
DEG = math.pi / 180.0
CELERITY = 1500.0
PHASE_CENTRE_M = 3.0e-3        # receive-array phase reference off the sensor origin: a complex directivity


# ---- the cases --------------------------------------------------------------

def listed():
    return [
        # The reference's EA400 38 kHz echosounder, one ping at a time: the
        # smallest call, where launches and latency are everything.
        dict(name="echosounder_ea400", op="plain_1d", n=20000, ranges=1049, rmin=0.1, rmax=49.999, carrier=38e3,
             pulse="sine", duration=128e-6, scene="uniform"),
        # A dense 1D ping with a pulse over 65 range bins and an odd sample count.
        dict(name="echosounder_dense", op="plain_1d", n=3000001, ranges=4096, rmin=0.5, rmax=100.0, carrier=38e3,
             pulse="burst", taps=65, scene="uniform"),
        # The reference's Oculus M1200d receiver: adaptive pulse duration (one
        # range bin), an oversampled sine table, a sinc beam over the whole fan.
        dict(name="imaging_reference", op="plain_2d", n=20000, ranges=500, rmin=0.1, rmax=6.5, bearings=256,
             carrier=1.2e6, pulse="sine", duration=0.0, beam="sinc", scene="uniform", echo=False),
        # An odd-sized imaging sensor (even pulse length, bearings and ranges
        # that fill no tile) and a small ping.
        dict(name="imaging_ragged", op="plain_2d", n=150003, ranges=777, rmin=0.5, rmax=30.0, bearings=387,
             carrier=1.2e6, pulse="burst", taps=24, beam="narrow", half=20, scene="seafloor", echo=False),
        # The imaging-sonar ping of the benchmark: 2^20 samples over a flat
        # seafloor, 512 bearings, narrow beams.
        dict(name="imaging", op="plain_2d", n=1 << 20, ranges=1024, rmin=0.3, rmax=40.0, bearings=512,
             carrier=1.2e6, pulse="burst", taps=33, beam="narrow", half=16, scene="seafloor", echo=False),
        # Side lobes over the whole fan: every sample reaches every bearing.
        # The carrier phase and the spreading loss are applied on the device.
        dict(name="imaging_wide_beam", op="plain_2d", n=1 << 22, ranges=4096, rmin=0.3, rmax=120.0, bearings=512,
             carrier=1.2e6, pulse="envelope", taps=33, beam="wide", scene="uniform", echo=True),
        # The precision form on a small sensor and ping: five short kernels.
        dict(name="precision_small", op="precision", n=65537, ranges=512, rmin=0.3, rmax=120.0, bearings=128,
             carrier=1.2e6, pulse="envelope", taps=33, beam="wide", scene="uniform", echo=True, flags=0),
        # The benchmark's headline ping: 2^24 samples, 512 bearings x 4096 ranges.
        dict(name="precision", op="precision", n=1 << 24, ranges=4096, rmin=0.3, rmax=120.0, bearings=512,
             carrier=1.2e6, pulse="envelope", taps=33, beam="wide", scene="uniform", echo=True, flags=0),
        # A wreck in view: half of the samples in 1 % of the ranges, a grid
        # larger than the L2, the hot-range option on.
        dict(name="precision_wreck", op="precision", n=1 << 26, ranges=8192, rmin=0.5, rmax=100.0, bearings=1024,
             carrier=1.2e6, pulse="envelope", taps=33, beam="narrow", half=16, scene="wreck", echo=True,
             flags=_lib.RTACX_PRECISION_HOT_RANGE),
        # A host-side caller: samples from pinned memory, the ping back to it.
        dict(name="precision_host", op="precision_host", n=1 << 22, ranges=1024, rmin=0.3, rmax=60.0, bearings=256,
             carrier=1.2e6, pulse="envelope", taps=33, beam="wide", scene="uniform", echo=True, flags=0),
        # A fleet of mixed sensors, one graph launch for all their pings.
        dict(name="batch", op="batch", pings=16, log2_min=13.0, log2_max=20.0, mix=7),
        # Ray hits to samples: carrier phase, spreading, receiver directivity.
        dict(name="echo_samples", op="echo", n=1 << 22, carrier=1.2e6, table=128),
    ]


def _log(rng, lo, hi):
    return int(round(2.0 ** rng.uniform(math.log2(lo), math.log2(hi))))


def draw(rng):
    op = rng.choice(["plain_1d", "plain_2d", "plain_2d", "plain_2d", "precision", "precision", "precision_host",
                     "batch", "echo"])
    if op == "batch":
        return dict(op=op, pings=rng.randint(4, 16), log2_min=12.0, log2_max=rng.uniform(15.0, 19.5),
                    mix=rng.randint(0, 1 << 20))
    if op == "echo":
        return dict(op=op, n=_log(rng, 1 << 14, 1 << 23), carrier=rng.uniform(3e4, 1.2e6), table=rng.randint(16, 300))
    rmin = rng.uniform(0.1, 2.0)
    case = dict(op=op, rmin=rmin, rmax=rmin + rng.uniform(5.0, 110.0), carrier=rng.choice([38e3, 200e3, 1.2e6]))
    if op == "plain_1d":
        case.update(n=_log(rng, 1 << 12, 1 << 22), ranges=_log(rng, 300, 8192), scene="uniform")
        if rng.random() < 0.25:
            case.update(pulse="sine", duration=rng.uniform(64e-6, 256e-6), carrier=38e3)
        else:
            case.update(pulse=rng.choice(["burst", "envelope"]), taps=rng.randint(9, 65))
        return case
    if op == "plain_2d":
        case.update(ranges=_log(rng, 128, 2048), bearings=_log(rng, 48, 600), echo=rng.random() < 0.4)
        if rng.random() < 0.2:
            case.update(n=_log(rng, 1 << 12, 1 << 17), pulse="sine", duration=0.0, beam="sinc", scene="uniform",
                        rmax=rmin + rng.uniform(5.0, 15.0))
        elif rng.random() < 0.2:
            case.update(n=_log(rng, 1 << 12, 1 << 20), pulse="envelope", taps=rng.randint(9, 49), beam="wide",
                        scene=rng.choice(["uniform", "wreck"]))
        else:
            case.update(n=_log(rng, 1 << 12, 1 << 21), pulse=rng.choice(["burst", "envelope"]),
                        taps=rng.randint(9, 65), beam="narrow", half=rng.randint(8, 32),
                        scene=rng.choice(["seafloor", "seafloor", "uniform", "wreck"]))
        return case
    flags = rng.choice([0, 0, _lib.RTACX_PRECISION_FP16_ROWSCALE, _lib.RTACX_PRECISION_HOT_RANGE])
    case.update(n=_log(rng, 1 << 14, 1 << (23 if op == "precision_host" else 24)), ranges=_log(rng, 256, 4096),
                bearings=_log(rng, 64, 640), pulse="envelope", taps=rng.randint(9, 65),
                beam=rng.choice(["wide", "narrow"]), half=rng.randint(8, 32),
                scene="wreck" if flags == _lib.RTACX_PRECISION_HOT_RANGE else "uniform", echo=True, flags=flags)
    return case


# ---- sensors and samples ----------------------------------------------------

def _resolution(rmin, rmax, n):
    return F32(F32(F32(rmax) - F32(rmin)) / F32(n - 1))


def _arcsin_bearings(n):
    k = np.arange(n, dtype=np.float64)
    return np.arcsin(math.sin(65.0 * DEG) * (2.0 * k / (n - 1) - 1.0)).astype(F32)


def _sensor(case):
    """Keyword arguments of Context.configure_1d / configure_2d."""
    res = float(_resolution(case["rmin"], case["rmax"], case["ranges"]))
    if case["pulse"] == "sine":
        # Waveform table at 8x oversampling; duration 0: one range bin, the reference's adaptive duration.
        duration = F32(case["duration"]) if case["duration"] else F32(F32(res) / F32(CELERITY))
        fs = F32(F32(2.0) * F32(case["carrier"]) * F32(8))
        phase = np.arange(max(1, int(fs * duration)), dtype=np.float64) * (2.0 * math.pi * case["carrier"] / float(fs))
        pulse = np.exp(1j * phase.astype(F32).astype(np.float64)).astype(np.complex64)
    else:
        # One tap per range bin: a Gaussian envelope, with the two-way carrier ("burst") or at baseband.
        taps = case["taps"]
        d = np.arange(taps, dtype=np.float64) - (taps - 1) / 2.0
        tone = 4.0 * math.pi * case["carrier"] * res / CELERITY if case["pulse"] == "burst" else 0.0
        pulse = (np.exp(-0.5 * (d * 6.0 / taps) ** 2) * np.exp(1j * tone * d)).astype(np.complex64)
        duration = F32(F32(taps * res) / F32(CELERITY))
    s = dict(range_min=float(F32(case["rmin"])), range_max=float(F32(case["rmax"])), range_count=case["ranges"],
             sound_celerity=CELERITY, pulse_duration=float(duration), margin=float(F32(F32(CELERITY) * duration)),
             pulse=pulse)
    if "bearings" not in case:
        return s
    n, null = case["bearings"], 0.6 * DEG
    if case["beam"] == "sinc":
        span = 130.0 * DEG
        taps, power, floor = 2 * int(round(4.0 * span / null)) + 1, 1, -1.0
    elif case["beam"] == "wide":
        span = 262.0 * DEG
        taps, power, floor = int(math.ceil(span / (null / 8.0))) | 1, 2, 0.01
    else:
        span = (2 * case["half"] + 1) * 130.0 * DEG / (n - 1)
        taps, power, floor = 8 * (2 * case["half"] + 1) + 1, 2, 0.0
    x = ((np.arange(taps, dtype=np.float64) + 0.5) / taps - 0.5) * span
    s.update(beam=np.maximum(np.sinc(x / null) ** power, floor).astype(F32), beam_span=float(F32(span)),
             bearings=_arcsin_bearings(n))
    return s


def _samples(case, seed):
    """SimSample1D / SimSample2D records [n][3 or 4] on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    n, two_d = case["n"], "bearings" in case
    u = lambda lo, hi, m=n: torch.rand(m, generator=g, device="cuda") * (hi - lo) + lo  # noqa: E731
    out = torch.empty((n, 4 if two_d else 3), device="cuda")
    rmin, rmax = case["rmin"], case["rmax"]
    if case["scene"] == "uniform":
        # A little beyond the range window on both sides, as rays come.
        t = u(0.99 * rmin, 1.005 * rmax)
    else:
        altitude = min(0.5 * rmax, max(1.5 * rmin, rmax / 8.0))
        t = altitude / u(altitude / rmax, 1.0)
        clutter = u(0.0, 1.0) < 0.01
        t = torch.where(clutter, u(rmin, rmax), t)
    if two_d:
        out[:, 3] = u(-65.0 * DEG, 65.0 * DEG)
    if case["scene"] == "wreck":
        hot = u(0.0, 1.0) < 0.5
        t = torch.where(hot, torch.randn(n, generator=g, device="cuda") * (0.0025 * (rmax - rmin)) +
                        (rmin + 0.4 * (rmax - rmin)), t)
        out[:, 3] = torch.where(hot, torch.randn(n, generator=g, device="cuda") * (3.0 * DEG) + 10.0 * DEG, out[:, 3])
    out[:, 2] = t
    out[:, :2].normal_(generator=g)       # Rayleigh amplitudes with uniform phases
    return out


def _precision_tables(case, s):
    """Directivity [grid][nB] and range taps [2][L] of the binned model, sampled from the sensor's tables: four grid
    bearings per output bearing, range nodes two bins apart, the receive array's phase reference off the origin."""
    bear = torch.from_numpy(s["bearings"]).double().cuda()
    cells = (4 * bear.numel() + 31) // 32 * 32
    first, last = float(s["bearings"][0]), float(s["bearings"][-1])
    step = float(F32(F32(F32(last) - F32(first)) / F32(cells - 1)))
    grid = first + torch.arange(cells, device="cuda", dtype=torch.float64) * step
    beam = torch.from_numpy(s["beam"]).double().cuda()
    kappa = 2.0 * math.pi * PHASE_CENTRE_M * case["carrier"] / CELERITY
    w = _lerp(beam, (grid[:, None] - bear[None, :]) / s["beam_span"])
    D = (w * torch.exp(1j * kappa * (torch.sin(grid)[:, None] - torch.sin(bear)[None, :]))).to(torch.complex64)
    res = float(_resolution(s["range_min"], s["range_max"], s["range_count"]))
    ext = s["pulse_duration"] * CELERITY
    reach = int(math.ceil(0.5 * ext / (2.0 * res))) + 1
    d = torch.arange(-reach, reach + 1, dtype=torch.float64)
    pulse = torch.from_numpy(s["pulse"]).to(torch.complex128)
    taps = torch.stack([_lerp(pulse, (2.0 * d - p) * res / ext) for p in range(2)]).to(torch.complex64)
    return dict(directivity=D.cpu().numpy(), range_taps=taps.numpy(), tap_center=reach, grid_count=cells,
                grid_first=first, grid_last=last)


def _batch_cases(case):
    """The pings of a batch: half 512-bearing 2D, a quarter 256-bearing 2D, a quarter 1D sensors, log-uniform sample
    counts, pulses of 17..65 range bins, beams of +/-8..32 bearings."""
    rng = np.random.default_rng(case["mix"])
    pings = []
    for i in range(case["pings"]):
        n = int(round(2.0 ** rng.uniform(case["log2_min"], case["log2_max"])))
        taps, half = int(rng.integers(17, 66)), int(rng.integers(8, 33))
        if i % 4 == 3:
            pings.append(dict(op="plain_1d", n=n, ranges=2048, rmin=0.5, rmax=100.0, carrier=38e3, pulse="burst",
                              taps=taps, scene="uniform"))
        else:
            big = i % 4 != 2
            pings.append(dict(op="plain_2d", n=n, ranges=1024 if big else 512, rmin=0.3 if big else 0.5,
                              rmax=40.0 if big else 30.0, bearings=512 if big else 256, carrier=1.2e6, pulse="burst",
                              taps=taps, beam="narrow", half=half, scene="seafloor", echo=False))
    return pings


def _hits(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    hits = torch.empty((case["n"], 6), device="cuda")
    hits[:, 0:2].normal_(generator=g)
    hits[:, 2].uniform_(0.2, 60.0, generator=g)
    hits[::97, 2] = 0.0                                   # rays that hit nothing
    az = (torch.rand(case["n"], generator=g, device="cuda") - 0.5) * (130.0 * DEG)
    el = (torch.rand(case["n"], generator=g, device="cuda") - 0.5) * (40.0 * DEG)
    hits[:, 3], hits[:, 4], hits[:, 5] = torch.cos(el) * torch.cos(az), torch.cos(el) * torch.sin(az), torch.sin(el)
    return hits


def _receiver(case):
    yaw, pitch = 0.3, -0.1
    cy, sy, cp, sp = math.cos(yaw), math.sin(yaw), math.cos(pitch), math.sin(pitch)
    rotation = np.array([[cy * cp, -sy, cy * sp], [sy * cp, cy, sy * sp], [-sp, 0.0, cp]], F32)
    w = np.arange(case["table"], dtype=np.float64) / case["table"]
    h = np.arange(case["table"] // 2, dtype=np.float64) / (case["table"] // 2)
    table = (np.sinc(3.0 * np.sin(math.pi * h))[:, None] * np.sinc(2.0 * np.sin(math.pi * w))[None, :]).astype(F32)
    return rotation, table


# ---- one pass ---------------------------------------------------------------

def _context(case, s):
    ctx = _lib.Context(0)
    (ctx.configure_2d if "bearings" in case else ctx.configure_1d)(**s)
    if case.get("echo"):
        ctx.set_echo_model(case["carrier"], _lib.RTACX_ECHO_PHASE | _lib.RTACX_ECHO_SPREADING)
    return ctx


def _ping_shape(case):
    return (case["ranges"], case["bearings"], 2) if "bearings" in case else (case["ranges"], 2)


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        pings = []
        for i, c in enumerate(_batch_cases(case)):
            ctx = _context(c, _sensor(c))
            smp = _samples(c, seed * 1000 + i)
            pings.append((ctx, smp, c["n"], torch.empty(_ping_shape(c), device="cuda")))
        torch.cuda.synchronize()
        batch = _lib.Batch(0)
        batch.plan(pings)
        return dict(op=op, batch=batch, pings=pings)
    if op == "echo":
        rotation, table = _receiver(case)
        one = dict(ranges=64, rmin=0.3, rmax=60.0, bearings=64, carrier=case["carrier"], pulse="envelope", taps=9,
                   beam="narrow", half=8)
        ctx = _context(one, _sensor(one))
        ctx.configure_receiver(rotation, table, case["carrier"], _lib.RTACX_ECHO_PHASE | _lib.RTACX_ECHO_SPREADING)
        return dict(op=op, ctx=ctx, hits=_hits(case, seed), n=case["n"], out=torch.empty((case["n"], 4), device="cuda"))
    s = _sensor(case)
    ctx = _context(case, s)
    smp = _samples(case, seed)
    out = torch.empty(_ping_shape(case), device="cuda")
    if op in ("plain_1d", "plain_2d"):
        ctx.reserve(case["n"])
    else:
        ctx.configure_precision(**_precision_tables(case, s), flags=case["flags"])
    if op == "precision_host":
        smp, out = smp.cpu().pin_memory(), out.cpu().pin_memory()
    return dict(op=op, ctx=ctx, smp=smp, n=case["n"], out=out)


def run(state):
    op, stream = state["op"], torch.cuda.current_stream()
    if op == "batch":
        state["batch"].run(stream)
        return [p[3] for p in state["pings"]]
    if op == "echo":
        state["ctx"].make_samples(state["hits"], state["n"], state["out"], stream=stream)
    elif op == "precision":
        state["ctx"].reduce_precision(state["smp"], state["n"], state["out"], stream=stream)
    elif op == "precision_host":
        state["ctx"].reduce_precision_host(state["smp"], state["n"], state["out"], stream=stream)
    else:
        state["ctx"].reduce(state["smp"], state["n"], state["out"], stream=stream)
    return state["out"]


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    op = case["op"]
    if op == "batch":
        each = [work(c) for c in _batch_cases(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if op == "echo":
        return {"bytes": case["n"] * (24 + 16), "flops": case["n"] * 60}
    s = _sensor(case)
    n, nR = case["n"], case["ranges"]
    res = float(_resolution(s["range_min"], s["range_max"], nR))
    rows = max(1.0, s["pulse_duration"] * CELERITY / res)             # output rows that a sample reaches
    if op == "plain_1d":
        return {"bytes": 12 * n + 8 * nR, "flops": 8 * n * rows}
    nB = case["bearings"]
    reached = min(nB, s["beam_span"] / (130.0 * DEG) * nB)            # output bearings that a sample reaches
    if op == "plain_2d":
        # A value per (sample, bearing), then over the pulse's rows either per sample or per output cell.
        return {"bytes": 16 * n + 8 * nR * nB, "flops": 4 * n * reached + min(8 * n * reached, 8 * nR * nB) * rows}
    cells, nodes = (4 * nB + 31) // 32 * 32, nR // 2 + 1
    return {"bytes": 16 * n + 8 * nR * nB + 8 * cells * nB,
            "flops": 40 * n + 8 * nodes * cells * nB + 8 * nR * nB * rows / 2}


# ---- the same in 64 bits ----------------------------------------------------

def _lerp(table, u):
    """Linear interpolation of a table spanning [-0.5, 0.5] at u, texel centres, zero outside."""
    n = table.numel()
    x = u * n + (0.5 * n - 0.5)
    fl = torch.floor(x)
    inside = (fl >= -1) & (fl <= n - 1)
    i = torch.where(inside, fl, torch.zeros_like(fl)).long()
    pad = torch.cat([table.new_zeros(1), table, table.new_zeros(1)])
    a = x - fl
    return torch.where(inside, pad[i + 1] * (1.0 - a) + pad[(i + 2).clamp(max=n + 1)] * a, table.new_zeros(()))


def _range_keys(s, t):
    """Range bin of each travel (float32 arithmetic, as the bins are defined), -1 out of range, and the window's
    half width in bins."""
    n, lo, hi, margin = s["range_count"], F32(s["range_min"]), F32(s["range_max"]), F32(s["margin"])
    res = F32(F32(hi - lo) / F32(n))
    m, M = F32(lo - F32(F32(0.5) * res)), F32(hi + F32(F32(0.5) * res))
    a = F32(F32(n - 1) / F32(M - m))
    b = F32(F32(F32(-m) * a) + F32(0.5))
    key = torch.trunc((t.double() * float(a) + float(b)).float())     # fused multiply-add, then truncation
    low = torch.where(key >= float(F32(m - margin)), 0.0, -1.0)
    high = torch.where(key <= float(F32(M + margin)), float(n - 1), -1.0)
    key = torch.where(key < 0, low, torch.where(key >= n, high, key)).long()
    return key, int(F32(margin / F32(F32(hi - lo) / F32(n - 1))))


def _rows_on(s, key, overlap):
    """Rows whose window of bins holds at least two that are not empty."""
    n = s["range_count"]
    full = torch.zeros(n + 1, dtype=torch.long, device=key.device)
    full[1:][torch.bincount(key, minlength=n) > 0] = 1
    full = torch.cumsum(full, 0)
    r = torch.arange(n, device=key.device)
    return full[(r + overlap + 1).clamp(max=n)] - full[(r - overlap).clamp(min=0)] >= 2


def _echo(case, smp):
    v = torch.complex(smp[:, 0].double(), smp[:, 1].double())
    if case.get("echo"):
        t = smp[:, 2].double()
        cycles = t * (2.0 * case["carrier"] / CELERITY)
        v = v * torch.exp(2j * math.pi * (cycles - torch.round(cycles))) / t ** 2
    return v


def _exact_plain(case, s, smp):
    two_d = "bearings" in case
    smp = smp[torch.argsort(smp[:, 2])]
    key, overlap = _range_keys(s, smp[:, 2])
    smp, key = smp[key >= 0], key[key >= 0]
    v, t = _echo(case, smp), smp[:, 2].contiguous()
    n = s["range_count"]
    # Output ranges as float32 holds them; the distance to them is a float32 difference by definition.
    R = torch.from_numpy((F32(s["range_min"]) + np.arange(n, dtype=F32) * _resolution(s["range_min"], s["range_max"], n))
                         .astype(F32)).cuda()
    ext = F32(F32(s["pulse_duration"]) * F32(CELERITY))
    pscale = float(F32(F32(1.0) / ext))
    reach = 0.51 * float(ext) * (1.0 + 1.0 / len(s["pulse"])) + 1e-5 * s["range_max"]
    pulse = torch.from_numpy(s["pulse"]).to(torch.complex128).cuda()
    out = torch.zeros((n, case.get("bearings", 1)), dtype=torch.complex128, device="cuda")
    if two_d:
        beam = torch.from_numpy(s["beam"]).double().cuda()
        bscale = float(F32(F32(1.0) / F32(s["beam_span"])))
        bear = torch.from_numpy(s["bearings"]).cuda()
    for r0 in range(0, n, 64):
        r = torch.arange(r0, min(n, r0 + 64), device="cuda")
        ends = torch.stack([R[r0] - reach, R[r[-1]] + reach])
        k0, k1 = (int(x) for x in torch.searchsorted(t, ends))
        for a in range(k0, k1, 1 << 16):
            z = min(k1, a + (1 << 16))
            U = v[None, a:z] * _lerp(pulse, (t[None, a:z] - R[r][:, None]).double() * pscale)
            U = torch.where((key[None, a:z] - r[:, None]).abs() <= overlap, U, torch.zeros_like(U))
            if two_d:
                B = _lerp(beam, (smp[a:z, 3][:, None] - bear[None, :]).double() * bscale)
                out[r] += torch.complex(U.real @ B, U.imag @ B)
            else:
                out[r, 0] += U.sum(1)
    out = torch.where(_rows_on(s, key, overlap)[:, None], out, torch.zeros_like(out))
    return torch.view_as_real(out if two_d else out[:, 0])


def _exact_precision(case, s, smp):
    tab = _precision_tables(case, s)
    key, overlap = _range_keys(s, smp[:, 2])
    smp, key = smp[key >= 0], key[key >= 0]
    nR, cells, taps, center = s["range_count"], tab["grid_count"], tab["range_taps"].shape[1], tab["tap_center"]
    h = 2.0 * float(_resolution(s["range_min"], s["range_max"], nR))
    first = F32(tab["grid_first"])
    step = float(F32(F32(F32(tab["grid_last"]) - first) / F32(cells - 1)))
    nodes = (nR - 1) // 2 + 1
    shift = center + 1
    G = torch.zeros((nodes + taps + 1) * cells, 2, dtype=torch.float64, device="cuda")
    for a in range(0, smp.shape[0], 1 << 24):
        part = smp[a:a + (1 << 24)]
        v = _echo(case, part)
        x = (part[:, 2].double() - s["range_min"]) / h
        j = torch.floor(x)
        y = (part[:, 3].double() - float(first)) / step
        q = torch.floor(y).clamp(0, cells - 2)
        ok = (j >= -shift) & (j <= nodes + taps - center - 2)
        v, j, q, x, y = v[ok], j[ok], q[ok], x[ok], y[ok]
        alpha, w = x - j, (y - q).clamp(0.0, 1.0)
        cell = (j.long() + shift) * cells + q.long()
        for dj, wj in ((0, 1.0 - alpha), (1, alpha)):
            for dq, wq in ((0, 1.0 - w), (1, w)):
                G.index_add_(0, cell + dj * cells + dq, torch.view_as_real(v * (wj * wq)))
    G = torch.view_as_complex(G).view(-1, cells)
    C = G @ torch.from_numpy(tab["directivity"]).to(torch.complex128).cuda()
    coef = torch.from_numpy(tab["range_taps"]).to(torch.complex128).cuda()
    r = torch.arange(nR, device="cuda")
    out = torch.zeros((nR, case["bearings"]), dtype=torch.complex128, device="cuda")
    for k in range(taps):
        out += coef[r % 2, k][:, None] * C[r // 2 + k + 1]
    return torch.view_as_real(torch.where(_rows_on(s, key, overlap)[:, None], out, torch.zeros_like(out)))


def _exact_echo(case, hits):
    rotation, table = _receiver(case)
    e, R = hits.double(), torch.from_numpy(rotation).double().cuda()
    tab = torch.from_numpy(table).double().cuda()
    d = e[:, 2]
    live = hits[:, 2] >= 1.0e-4
    cycles = d * (2.0 * case["carrier"] / CELERITY)
    v = torch.complex(e[:, 0], e[:, 1]) * torch.exp(2j * math.pi * (cycles - torch.round(cycles)))
    v = v / torch.where(live, d, torch.ones_like(d)) ** 2
    loc = e[:, 3:6] @ R
    az, el = torch.atan2(loc[:, 1], loc[:, 0]), torch.atan2(loc[:, 2], loc[:, 0])

    def axis(u, n):                                       # mirror addressing, texel centres
        u = torch.remainder(u, 2.0)
        x = torch.where(u <= 1.0, u, 2.0 - u) * n - 0.5
        i = torch.floor(x)
        fold = lambda k: torch.where(k < 0, -k - 1, torch.where(k >= n, 2 * n - k - 1, k)).clamp(0, n - 1)  # noqa: E731
        return x - i, fold(i.long()), fold(i.long() + 1)

    ax, x0, x1 = axis(az / math.pi, tab.shape[1])
    ay, y0, y1 = axis(el / math.pi, tab.shape[0])
    top = tab[y0, x0] * (1.0 - ax) + tab[y0, x1] * ax
    bot = tab[y1, x0] * (1.0 - ax) + tab[y1, x1] * ax
    v = v * (top * (1.0 - ay) + bot * ay)
    rec = torch.stack([v.real, v.imag, d, -az], 1)
    null = torch.tensor([0.0, 0.0, -1.0, 0.0], dtype=torch.float64, device="cuda")
    return torch.where(live[:, None], rec, null[None, :])


def exact(case, seed):
    if case["op"] == "batch":
        return [_exact_plain(c, _sensor(c), _samples(c, seed * 1000 + i)) for i, c in enumerate(_batch_cases(case))]
    if case["op"] == "echo":
        return _exact_echo(case, _hits(case, seed))
    s, smp = _sensor(case), _samples(case, seed)
    if case["op"] in ("plain_1d", "plain_2d"):
        return _exact_plain(case, s, smp)
    out = _exact_precision(case, s, smp)
    return out.cpu() if case["op"] == "precision_host" else out
