"""Plain 2D form over range cells (pulse taps one output range apart) at the
edges of its tiles: bearing counts around the 64- and 128-bearing segments,
range counts around the filter's 8 and 32 rows, the shortest pulses, even and
odd tables, pings of one unit of samples or a few, samples next to and beyond
the range window. Each ping against the FP64 oracle at the plain form's
tolerance, 1e-5 relative L2."""
import numpy as np
import pytest

from rtac_simulation_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

from helpers_gpu import gpu_reduce, make_context, rel_l2  # noqa: E402

TOL = 1e-5


def ping(n, nR, nB, taps, wide, beam_taps=0, seed=3, rmin=0.4, rmax=30.0):
    res = float(wl.linspace_resolution(rmin, rmax, nR))
    bearings = wl.arcsin_bearings(nB, 130.0) if nB > 1 else np.zeros(1, np.float32)
    spacing = 130.0 * wl.DEG / max(nB - 1, 1)
    if wide:
        span = 262.0 * wl.DEG
        beam = wl.beam_sinc2(beam_taps or 701, span, 2.0 * wl.DEG, floor=0.01)
    else:
        span = 9 * spacing
        beam = wl.beam_sinc2(beam_taps or 73, span, 2.0 * spacing)
    pulse = wl.pulse_at_bin_spacing(taps, res, 1.2e6, 1500.0)
    rng = np.random.default_rng(seed)
    t = rng.uniform(rmin - 2 * taps * res, rmax + 2 * taps * res, n)
    if n > 64:
        R = wl.linspace(rmin, rmax, nR)
        t[:64] = R[rng.integers(0, nR, 64)]              # exactly on output ranges
        t[64 - min(8, n // 8):64] = rmin
    th = rng.uniform(-70.0 * wl.DEG, 70.0 * wl.DEG, n)
    re, im = rng.normal(size=(2, n))
    s = wl.sensor_2d(rmin, rmax, nR, 1500.0, pulse, taps * res, beam, span, bearings)
    return wl.Workload("cells", 2, s, wl._pack(re, im, t, th))


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("n,nR,nB,taps,beam_taps", [
    (2, 2, 1, 2, 0), (31, 7, 3, 1, 0), (128, 8, 31, 2, 0), (129, 9, 33, 3, 72), (1000, 31, 63, 4, 0),
    (1024, 33, 64, 5, 700), (1025, 64, 65, 8, 0), (3000, 65, 127, 9, 0), (5000, 100, 128, 16, 71),
    (20000, 257, 129, 33, 0), (40000, 300, 200, 64, 0), (200003, 130, 257, 33, 0),
])
def test_cells_match_fp64_oracle(oracle, n, nR, nB, taps, beam_taps, wide):
    wk = ping(n, nR, nB, taps, wide, beam_taps)
    got = gpu_reduce(make_context(wk), wk.samples, wk.out_shape)
    want = oracle.reduce(wk.samples, wk.sensor)
    assert np.isfinite(got).all()
    assert rel_l2(got, want) <= TOL, rel_l2(got, want)


@pytest.mark.parametrize("nB,beam_taps,roll,level", [
    (129, 701, 0, 0.01), (129, 700, 0, 0.01), (200, 701, 90, 0.01), (200, 700, -141, -0.02), (600, 1501, 0, 0.3),
])
def test_lobes_on_a_flat_floor(oracle, nB, beam_taps, roll, level):
    """Wide beams that are one level outside a lobe, in the middle of the table
    or not, on both sides of the sample count from which the lobe is taken
    apart; samples whose bearings leave the table, or are not numbers."""
    for n in ((1 << 24) // nB, (1 << 24) // nB + 1):
        wk = ping(n, 90, nB, 9, True, beam_taps)
        beam = np.roll(wk.sensor["beam"], roll)
        wk.sensor["beam"] = np.where(beam == np.float32(0.01), np.float32(level), beam).astype(np.float32)
        wk.samples[100:200, 3] *= 3.0
        wk.samples[200:210, 3] = np.nan
        good = wk.samples.copy()
        good[200:210, :2] = 0.0
        good[200:210, 3] = 0.0
        got = gpu_reduce(make_context(wk), wk.samples, wk.out_shape)
        assert rel_l2(got, oracle.reduce(good, wk.sensor)) <= TOL


@pytest.mark.parametrize("nB,wide", [(65, False), (640, False), (65, True), (200, True)])
@pytest.mark.parametrize("n", [1, 33, 5000, 90000])
def test_pings_of_samples_next_to_knots_alone(oracle, n, nB, wide):
    """Every travel on a knot (an odd pulse's knots lie on the output ranges):
    units without a sample for the cell rows, in windows of 64 and 128 bearings,
    shared-out windows and the lobe form."""
    wk = ping(n, 90, nB, 9, wide)
    wk.samples[:, 2] = wl.linspace(0.4, 30.0, 90)[np.arange(n) % 90]
    got = gpu_reduce(make_context(wk), wk.samples, wk.out_shape)
    assert rel_l2(got, oracle.reduce(wk.samples, wk.sensor)) <= TOL


@pytest.mark.parametrize("n", [20001, (1 << 21) + 1])
def test_cells_far_from_the_sensor(oracle, n):
    """Ranges 1e5 of their spacings away, where a cell coordinate's float
    rounding is 4e-3 of a cell: the cells' fractions keep the coordinate's
    residual (1e-3 relative without, or with it twice), and the two sorts' count
    and scatter agree on every sample's cell block."""
    wk = ping(n, 1024, 33, 8, False, rmin=100.0, rmax=101.023)
    got = gpu_reduce(make_context(wk), wk.samples, wk.out_shape)
    assert rel_l2(got, oracle.reduce(wk.samples, wk.sensor)) <= TOL


@pytest.mark.parametrize("n", [1023, 1025, 1 << 21, (1 << 21) + 1])
def test_pings_around_the_ranked_sort_limits(oracle, n):
    """One count CTA and two, the most samples that are ranked and one more;
    all samples of a wall in few bins."""
    for wall in (False, True):
        wk = ping(n, 41, 33, 3, False)
        if wall:
            wk.samples[n // 4:, 2] = 7.03
            wk.samples[n // 4:, 3] = 0.11
        got = gpu_reduce(make_context(wk), wk.samples, wk.out_shape)
        assert rel_l2(got, oracle.reduce(wk.samples, wk.sensor)) <= TOL


@pytest.mark.parametrize("n", [(1 << 21) + 1, (1 << 22) + 1])
def test_many_bins_around_their_ranked_limit(oracle, n):
    """More bins than the tile sort reserves in one batch: ranked up to 2^22."""
    wk = ping(n, 2600, 129, 2, False)
    got = gpu_reduce(make_context(wk), wk.samples, wk.out_shape)
    assert rel_l2(got, oracle.reduce(wk.samples, wk.sensor)) <= TOL


@pytest.mark.parametrize("nB,beam_taps", [(65, 605), (65, 606), (65, 607), (3, 1), (3, 2), (640, 1006), (640, 1007)])
def test_tables_around_the_replicated_limit(oracle, nB, beam_taps):
    """Beam tables on both sides of the largest that is kept in 16 copies (for
    64- and 128-bearing windows), and the smallest, samples of all warps."""
    wk = ping(70001, 90, nB, 9, False, beam_taps)
    got = gpu_reduce(make_context(wk), wk.samples, wk.out_shape)
    assert rel_l2(got, oracle.reduce(wk.samples, wk.sensor)) <= TOL


@pytest.mark.parametrize("spread,span", [(0.01, 0.5), (0.0, 0.1), (0.0, 0.02)])
def test_clustered_bearings(oracle, spread, span):
    """Bearings that no windows of 128 can hold (most of them in one direction,
    narrow beams): right, and configured in a fraction of the 0.1 s that a
    search through all windows took."""
    import time
    wk = ping(5000, 100, 512, 9, False)
    s = wk.sensor
    s["bearings"] = np.concatenate([[-1.1], np.linspace(0.0, spread * wl.DEG, 510), [1.1]]).astype(np.float32)
    s["beam_span"] = span * wl.DEG
    wk.samples[::2, 3] = np.linspace(-span, span, len(wk.samples[::2])) * wl.DEG
    wk.samples[1::8, 3] = np.float32(1.1)
    ctx = make_context(wk)
    took = []
    for _ in range(3):
        t0 = time.perf_counter()
        ctx.configure_2d(**s)
        took.append(time.perf_counter() - t0)
    got = gpu_reduce(ctx, wk.samples, wk.out_shape)
    assert rel_l2(got, oracle.reduce(wk.samples, s)) <= TOL
    assert min(took) < 0.02, took


@pytest.mark.parametrize("change", ["half_margin", "half_tap", "long_pulse"])
def test_sensors_off_the_cell_rule_match_fp64_oracle(oracle, change):
    """A margin that cuts the pulse's window, taps that are not one range
    apart: the per-row gathers, as before."""
    wk = ping(4000, 100, 65, 17, False)
    s = wk.sensor
    if change == "half_margin":
        s["margin"] = 0.25 * s["margin"]
    elif change == "half_tap":
        s["pulse_duration"] = 0.5 * s["pulse_duration"]
    else:
        s["pulse_duration"] = 1.01 * s["pulse_duration"]
    got = gpu_reduce(make_context(wk), wk.samples, wk.out_shape)
    want = oracle.reduce(wk.samples, wk.sensor)
    assert rel_l2(got, want) <= TOL


def test_cells_drop_samples_without_a_bearing_or_travel():
    """NaN and far-away bearings and NaN travels carry no weight."""
    wk = ping(3000, 100, 65, 9, False)
    bad = wk.samples.copy()
    bad[::50, 3] = np.nan
    bad[1::50, 3] = 1e30
    bad[2::50, 3] = -np.inf
    clean = bad.copy()
    clean[~np.isfinite(bad[:, 3]) | (np.abs(bad[:, 3]) > 1e3), :2] = 0.0
    ctx = make_context(wk)
    a = gpu_reduce(ctx, bad, wk.out_shape)
    b = gpu_reduce(ctx, clean, wk.out_shape)
    assert np.isfinite(a).all()
    assert rel_l2(a, b) <= 1e-6


def test_sorted_scratch_after_a_ping_keeps_its_order(oracle):
    """rtacx_reduce sorts a cell-form ping in its own order; the diagnostic
    copy of the sorted scratch still has every in-range sample once, grouped
    by ascending (range bin, bearing sub-bin), and pings after it are right."""
    from test_gpu_sorted import KEY_OOR, composite_keys, record_hash
    wk = ping(20001, 257, 200, 17, False)
    ctx = make_context(wk)
    first = gpu_reduce(ctx, wk.samples, wk.out_shape)
    buf = torch.zeros((wk.n, 4), device="cuda")
    ctx.diag_sorted(buf, wk.n, stream=torch.cuda.current_stream())
    recs = buf.cpu().numpy()
    key = composite_keys(oracle, wk, wk.samples)
    inside = wk.samples[key != KEY_OOR]
    got = recs[:len(inside)]
    assert np.all(np.diff(composite_keys(oracle, wk, got).astype(np.int64)) >= 0)
    assert np.array_equal(np.sort(record_hash(got)), np.sort(record_hash(inside)))
    assert rel_l2(gpu_reduce(ctx, wk.samples, wk.out_shape), first) <= 1e-6


@pytest.mark.parametrize("dims", [1, 2])
def test_sorted_scratch_after_replayed_pings(oracle, dims):
    """A captured ping replayed between other calls on its context: the
    diagnostic copy is in its order after each of them, also when the scratch
    was put in order (or filled by rtacx_bin) since the capture."""
    from test_gpu_sorted import KEY_OOR, composite_keys, record_hash
    wk = ping(20001, 257, 200, 17, False) if dims == 2 else ping_1d(20001, 257, 17)
    n = wk.n
    ctx = make_context(wk)
    ctx.reserve(n + 500)
    dev = torch.from_numpy(wk.samples).cuda()
    out = torch.zeros(wk.out_shape + (2,), device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.reduce(dev, n, out, stream=torch.cuda.current_stream())

    def check(samples, count):
        buf = torch.zeros((n, 4), device="cuda")
        ctx.diag_sorted(buf, n, stream=torch.cuda.current_stream())
        recs = np.zeros((count, 4), np.float32)
        recs[:, :samples.shape[1]] = samples[:count]
        inside = recs[composite_keys(oracle, wk, recs) != KEY_OOR]
        got = buf.cpu().numpy()[:len(inside)]
        assert np.all(np.diff(composite_keys(oracle, wk, got).astype(np.int64)) >= 0)
        assert np.array_equal(np.sort(record_hash(got)), np.sort(record_hash(inside)))

    stream = torch.cuda.current_stream()
    for scale in (1.0, 0.9, 0.8):
        samples = wk.samples.copy()
        samples[:, 2] *= np.float32(scale)
        dev.copy_(torch.from_numpy(samples))
        graph.replay()
        check(samples, n)
        check(samples, n)
        ctx.bin(dev, n // 3, dims, stream=stream)
        check(samples, n // 3)


@pytest.mark.parametrize("margin", [1.0, 0.999, 3.0])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("n,nR,nB,H", [(1, 2, 1, 3), (33, 5, 33, 2), (1000, 64, 65, 17), (30000, 300, 129, 164)])
def test_row_pairs_match_fp64_oracle(oracle, n, nR, nB, H, wide, margin):
    """Pulses one output range long (the adaptive duration): every sample
    reaches at most two rows; a margin under one bin switches every row off."""
    wk = ping(n, nR, nB, 5, wide)
    s = wk.sensor
    res = float(wl.linspace_resolution(s["range_min"], s["range_max"], nR))
    s["pulse"] = np.exp(1j * np.linspace(0.0, 40.0, H)).astype(np.complex64)
    s["pulse_duration"] = float(np.float32(np.float32(res) / np.float32(1500.0)))
    s["margin"] = margin * float(np.float32(1500.0) * np.float32(s["pulse_duration"]))
    got = gpu_reduce(make_context(wk), wk.samples, wk.out_shape)
    want = oracle.reduce(wk.samples, s)
    assert np.isfinite(got).all()
    assert rel_l2(got, want) <= TOL, rel_l2(got, want)


def by_rows(ctx):
    """Whether the context's last (traced) ping went through the per-row
    gathers, which alone have windows."""
    return ctx.stage_times()["windows"] > 0.0


def row_pairs(wk):
    """The ping's sensor with a pulse one output range long."""
    s = wk.sensor
    res = float(wl.linspace_resolution(s["range_min"], s["range_max"], s["range_count"]))
    s["pulse"] = np.exp(1j * np.linspace(0.0, 9.0, 20)).astype(np.complex64)
    s["pulse_duration"] = float(np.float32(np.float32(res) / np.float32(1500.0)))
    s["margin"] = float(np.float32(1500.0) * np.float32(s["pulse_duration"]))
    return wk


@pytest.mark.parametrize("nB,nR,wide,pairs,few,many", [
    (512, 4096, False, False, 201, 3001), (512, 6000, True, False, 1000, 20000), (600, 8000, False, True, 33, 3000),
])
def test_small_pings_of_large_sensors_gather_per_row(oracle, nB, nR, wide, pairs, few, many):
    """A few samples against cell rows of a size: the gathers; more of them, or
    none, the cell form, on one context in turn."""
    wk = ping(many, nR, nB, 33, wide)
    if pairs:
        row_pairs(wk)
    ctx = make_context(wk)
    ctx.set_tracing(True)
    for n in (few, many, 0, 1, few):
        got = gpu_reduce(ctx, wk.samples[:n], wk.out_shape)
        assert by_rows(ctx) == (0 < n <= few), n
        assert rel_l2(got, oracle.reduce(wk.samples[:n], wk.sensor)) <= TOL, n


def test_cell_rows_come_with_the_scratch_of_samples(oracle):
    """A configured sensor holds no cell rows (135 MB here) until a ping or
    rtacx_reserve sizes the scratch; a sensor configured on a context that has
    scratch can be captured at once."""
    wk = ping(60000, 8192, 1024, 9, False)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    ctx = make_context(wk)
    assert free0 - torch.cuda.mem_get_info()[0] < 64 << 20
    ctx.reserve(wk.n)
    assert free0 - torch.cuda.mem_get_info()[0] > 120 << 20
    small = ping(60000, 300, 64, 9, False)
    ctx.configure_2d(**small.sensor)
    d = torch.from_numpy(small.samples).cuda()
    out = torch.zeros(small.out_shape + (2,), device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.reduce(d, small.n, out, stream=torch.cuda.current_stream())
    graph.replay()
    torch.cuda.synchronize()
    got = out.cpu().numpy()[..., 0] + 1j * out.cpu().numpy()[..., 1]
    assert rel_l2(got, oracle.reduce(small.samples, small.sensor)) <= TOL


@pytest.mark.parametrize("large", [0, 150000])
def test_batches_of_small_pings(oracle, large):
    """Small pings of every form alone, which the per-row gathers take, and
    next to a large one, with which the cell form does."""
    from rtac_simulation_gb300 import _lib
    pings = [ping(300, 1024, 512, 33, False), ping(900, 512, 130, 17, True), row_pairs(ping(50, 400, 200, 5, True)),
             ping(100, 4096, 512, 33, False), ping_1d(999, 64, 17), ping_1d(999, 64, 2, 40, 2.0)]
    if large:
        pings.append(ping(large, 257, 129, 33, False))
    ctxs = [make_context(wk) for wk in pings]
    devs = [torch.from_numpy(wk.samples.reshape(-1)).cuda() for wk in pings]
    outs = [torch.full(wk.out_shape + (2,), float("nan"), device="cuda") for wk in pings]
    batch = _lib.Batch(0)
    batch.plan([(c, d, wk.n, o) for wk, c, d, o in zip(pings, ctxs, devs, outs)], autotune=False)
    for _ in range(2):
        batch.run(torch.cuda.current_stream())
    batch.status(torch.cuda.current_stream())
    for wk, o in zip(pings, outs):
        got = o.cpu().numpy()[..., 0] + 1j * o.cpu().numpy()[..., 1]
        assert rel_l2(got, oracle.reduce(wk.samples, wk.sensor)) <= TOL, (wk.name, wk.n)
    batch.close()


def ping_1d(n, nR, taps, H=0, ext_bins=0.0, seed=5):
    rmin, rmax = 0.4, 30.0
    res = float(wl.linspace_resolution(rmin, rmax, nR))
    pulse = wl.pulse_at_bin_spacing(H or taps, res, 38e3, 1500.0)
    rng = np.random.default_rng(seed)
    t = rng.uniform(rmin - 2 * taps * res, rmax + 2 * taps * res, n)
    if n > 64:
        t[:32] = wl.linspace(rmin, rmax, nR)[rng.integers(0, nR, 32)]
    re, im = rng.normal(size=(2, n))
    return wl.Workload("cells_1d", 1, wl.sensor_1d(rmin, rmax, nR, 1500.0, pulse, (ext_bins or taps) * res),
                       wl._pack(re, im, t))


@pytest.mark.parametrize("n,nR,taps,H,ext", [
    (1, 2, 1, 0, 0), (2, 31, 2, 0, 0), (33, 32, 3, 0, 0), (255, 33, 8, 0, 0), (1025, 100, 65, 0, 0),
    (70001, 1025, 33, 0, 0), (1 << 20, 300, 9, 0, 0),                       # taps one range apart
    (33, 31, 1, 7, 0.9), (1000, 64, 2, 40, 2.0), (5000, 257, 4, 77, 4.03),   # row by row
    (200000, 500, 30, 77, 29.7), (2000, 3000, 200, 77, 150.2),               # the sorted gather again
])
def test_1d_pings_match_fp64_oracle(oracle, n, nR, taps, H, ext):
    wk = ping_1d(n, nR, taps, H, ext)
    for offset in (0, 1):
        got = gpu_reduce(make_context(wk), wk.samples, wk.out_shape, offset_floats=offset)
        want = oracle.reduce(wk.samples, wk.sensor)
        assert np.isfinite(got).all()
        assert rel_l2(got, want) <= TOL, rel_l2(got, want)


def test_row_sums_of_1d_pings_keep_their_digits(oracle):
    """About 95 reductions per output row, in one word one after the other
    2e-7 off: the rms of a rounded sum of n terms of either sign is 2^-24 /
    sqrt(3) sqrt(n / 2), 2.4e-7 for 95 and 8e-8 for the 12 of a copy, with three
    roundings per product and eight copies together under 1.4e-7."""
    wk = wl.ea400_reference_1d(n_samples=20000)
    got = gpu_reduce(make_context(wk), wk.samples, wk.out_shape)
    assert rel_l2(got, oracle.reduce(wk.samples, wk.sensor)) <= 1.4e-7


def test_1d_sorted_scratch_after_a_ping(oracle):
    from test_gpu_sorted import KEY_OOR, composite_keys, record_hash
    wk = ping_1d(5000, 257, 17)
    ctx = make_context(wk)
    gpu_reduce(ctx, wk.samples, wk.out_shape)
    buf = torch.zeros((wk.n, 4), device="cuda")
    ctx.diag_sorted(buf, wk.n, stream=torch.cuda.current_stream())
    recs = np.zeros((wk.n, 4), np.float32)
    recs[:, :3] = wk.samples
    inside = recs[composite_keys(oracle, wk, recs) != KEY_OOR]
    got = buf.cpu().numpy()[:len(inside)]
    assert np.all(np.diff(composite_keys(oracle, wk, got).astype(np.int64)) >= 0)
    assert np.array_equal(np.sort(record_hash(got)), np.sort(record_hash(inside)))


@pytest.mark.parametrize("autotune", [False, True])
def test_batch_of_every_form_matches_fp64_oracle(oracle, autotune):
    """One batch with a ping of every form (narrow and wide cells, row pairs,
    a 2D sensor off the rule, 1D cells, row by row and sorted), run twice."""
    from rtac_simulation_gb300 import _lib
    pair = ping(3000, 100, 65, 5, True)
    res = float(wl.linspace_resolution(0.4, 30.0, 100))
    pair.sensor["pulse"] = np.exp(1j * np.linspace(0.0, 9.0, 20)).astype(np.complex64)
    pair.sensor["pulse_duration"] = float(np.float32(res) / np.float32(1500.0))
    off = ping(2000, 64, 40, 9, False)
    off.sensor["pulse_duration"] *= 0.5
    pings = [ping(70001, 257, 129, 33, False), ping(9000, 200, 200, 17, True), pair, off,
             ping_1d(300000, 300, 33), ping_1d(999, 64, 2, 40, 2.0), ping_1d(200000, 500, 30, 77, 29.7),
             ping(1, 9, 33, 3, False)]
    ctxs = [make_context(wk) for wk in pings]
    devs = [torch.from_numpy(wk.samples.reshape(-1)).cuda() for wk in pings]
    outs = [torch.full(wk.out_shape + (2,), float("nan"), device="cuda") for wk in pings]
    batch = _lib.Batch(0)
    batch.plan([(c, d, wk.n, o) for wk, c, d, o in zip(pings, ctxs, devs, outs)], autotune=autotune)
    assert batch.graph_kernels() == 1
    for _ in range(2):
        batch.run(torch.cuda.current_stream())
        batch.status(torch.cuda.current_stream())
        for wk, o in zip(pings, outs):
            got = o.cpu().numpy()
            got = got[..., 0].astype(np.float64) + 1j * got[..., 1]
            want = oracle.reduce(wk.samples, wk.sensor)
            assert rel_l2(got, want) <= TOL, (wk.name, wk.n, rel_l2(got, want))
    # A single ping on a context that the batch used, and the batch again.
    one = gpu_reduce(ctxs[0], pings[0].samples, pings[0].out_shape)
    assert rel_l2(one, oracle.reduce(pings[0].samples, pings[0].sensor)) <= TOL
    batch.close()


@pytest.mark.parametrize("maker", [
    lambda: ping(20001, 257, 200, 17, False), lambda: ping(5000, 300, 128, 9, True),
    lambda: ping_1d(5000, 257, 17), lambda: ping_1d(1000, 64, 2, 40, 2.0),
])
def test_chained_pings_read_what_the_kernel_ahead_wrote(maker):
    """Samples written by a kernel right before the ping, two different ones in
    turn through the same context, sample buffer and ping, without a pause."""
    wk = maker()
    ctx = make_context(wk)
    stream = torch.cuda.current_stream()
    a = torch.from_numpy(wk.samples).cuda()
    b = a.flip(0).contiguous()
    b[:, :2] *= -0.5
    b[:, 2] = b[:, 2] * 0.75 + 0.5
    buf = torch.empty_like(a)
    out = torch.empty(wk.out_shape + (2,), device="cuda")
    want = []
    for src in (a, b):
        torch.mul(src, 1.0, out=buf)
        torch.cuda.synchronize()
        ctx.reduce(buf, wk.n, out, stream=stream)
        torch.cuda.synchronize()
        want.append(out.clone())
    got = []
    for _ in range(40):
        for src in (a, b):
            torch.mul(src, 1.0, out=buf)
            ctx.reduce(buf, wk.n, out, stream=stream)
            got.append(out.clone())
    torch.cuda.synchronize()
    for i, g in enumerate(got):
        assert float((g - want[i % 2]).norm() / want[i % 2].norm()) <= 2e-6, i


@pytest.mark.parametrize("n", [1, 4095, 4097, 12289, (1 << 21) + 1])
def test_batches_around_the_ranked_chunks(oracle, n):
    """A ping of n samples next to a small one: one chunk of the batch's ranked
    count and more, and more samples than are ranked."""
    from rtac_simulation_gb300 import _lib
    pings = [ping(n, 41, 33, 3, False), ping(500, 64, 130, 40, False, seed=4)]
    ctxs = [make_context(wk) for wk in pings]
    devs = [torch.from_numpy(wk.samples.reshape(-1)).cuda() for wk in pings]
    outs = [torch.full(wk.out_shape + (2,), float("nan"), device="cuda") for wk in pings]
    batch = _lib.Batch(0)
    batch.plan([(c, d, wk.n, o) for wk, c, d, o in zip(pings, ctxs, devs, outs)], autotune=False)
    for _ in range(2):
        batch.run(stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    for wk, o in zip(pings, outs):
        got = o.cpu().numpy()[..., 0] + 1j * o.cpu().numpy()[..., 1]
        assert rel_l2(got, oracle.reduce(wk.samples, wk.sensor)) <= TOL


def test_sorted_scratch_after_a_batch(oracle):
    """The documented order from the scratch that a batch left, of sensors whose
    single pings sort into other bins (a lobe on a floor) or into the same."""
    from rtac_simulation_gb300 import _lib
    from test_gpu_sorted import KEY_OOR, composite_keys, record_hash
    pings = [ping(20000, 257, 129, 9, False), ping(90000, 100, 200, 9, True)]
    ctxs = [make_context(wk) for wk in pings]
    gpu_reduce(ctxs[1], pings[1].samples, pings[1].out_shape)
    devs = [torch.from_numpy(wk.samples.reshape(-1)).cuda() for wk in pings]
    outs = [torch.empty(wk.out_shape + (2,), device="cuda") for wk in pings]
    batch = _lib.Batch(0)
    batch.plan([(c, d, wk.n, o) for wk, c, d, o in zip(pings, ctxs, devs, outs)], autotune=False)
    batch.run(torch.cuda.current_stream())
    for wk, ctx in zip(pings, ctxs):
        buf = torch.zeros((wk.n, 4), device="cuda")
        ctx.diag_sorted(buf, wk.n, stream=torch.cuda.current_stream())
        inside = wk.samples[composite_keys(oracle, wk, wk.samples) != KEY_OOR]
        got = buf.cpu().numpy()[:len(inside)]
        assert np.all(np.diff(composite_keys(oracle, wk, got).astype(np.int64)) >= 0)
        assert np.array_equal(np.sort(record_hash(got)), np.sort(record_hash(inside)))
    batch.close()
