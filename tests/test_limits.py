"""Calls at the limits of their inputs: delays outside the simulator's window,
trace lengths at the demodulator's grid limit, delays that are not numbers, and
RF plans with every launch shape."""

from __future__ import annotations

import numpy as np
import pytest

from gold import rel_l2
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture()
def gpu():
    import torch
    from usx import capi
    ctx = capi.Context(0, stream=torch.cuda.current_stream().cuda_stream)
    yield torch, capi, ctx
    ctx.close()


def pulse_echo(capi, torch, ctx, delays, apod):
    n_ev, n_el = delays.shape
    rng = np.random.default_rng(5)
    scat = np.zeros((40, 8), np.float32)
    scat[:, 0], scat[:, 2] = rng.uniform(-3e-3, 3e-3, 40), rng.uniform(3e-3, 0.016, 40)
    scat[:, 3] = rng.normal(size=40)
    tx = [dict(type=1, angle=0.0, delays=d, apodization=w) for d, w in zip(delays, apod)]
    ch = capi.Channel(capi.Probe(n_el, 3e-4, 2.7e-4, 5e-3, 5e6, 0.6), capi.Medium(1540.0, 0.5, 1000.0),
                      capi.Acquisition(2e7, 500, 0.0, 5e3), tx)
    d = torch.from_numpy(scat).cuda()
    rf = torch.full((n_ev, n_el, 500), 7.0, device="cuda")
    ctx.simulate(ch, capi.sim_config(noise_db=-200.0), d.data_ptr(), len(scat), None, rf.data_ptr())
    return rf.cpu().numpy()


@pytest.mark.parametrize("late", [1e-3, 100.0, 1e30, np.inf])
def test_an_element_fired_outside_the_window_adds_nothing(gpu, late):
    """A pulse placed milliseconds to for ever after the first arrival is past
    the 30 us window: the RF is that of the aperture without the element. (The
    sums' fixed-point step follows the total apodization: 1e-6.)"""
    torch, capi, ctx = gpu
    delays, apod = np.zeros((2, 16), np.float32), np.ones((2, 16), np.float32)
    delays[:, 5] = late
    got = pulse_echo(capi, torch, ctx, delays, apod)
    apod[:, 5] = 0.0
    want = pulse_echo(capi, torch, ctx, np.zeros_like(delays), apod)
    assert np.isfinite(got).all() and np.abs(want).max() > 0
    assert rel_l2(got, want) < 1e-6


@pytest.mark.parametrize("full", [0, 1])
@pytest.mark.parametrize("n_el,first", [(16, 0), (33, 32), (75, 40), (130, 65)])
def test_records_that_end_before_the_echoes(gpu, oracle, full, n_el, first):
    """A record of 130 samples (5 mm) of scatterers 2 to 16 mm deep, elements
    before `first` not firing: against the oracle (FP32 sums in another order,
    1e-5), and the samples and echo counts of a longer record's start."""
    torch, capi, ctx = gpu
    rng = np.random.default_rng(n_el)
    scat = np.zeros((60, 8), np.float32)
    scat[:, 0], scat[:, 2] = rng.uniform(-8e-3, 8e-3, 60), rng.uniform(2e-3, 0.016, 60)
    scat[:, 3] = rng.normal(size=60)
    z, w = np.zeros((2, n_el), np.float32), np.ones((2, n_el), np.float32)
    w[1, :first] = 0.0
    tx = [dict(type=1, angle=0.0, delays=z[e], apodization=w[e]) for e in range(2)]
    cfg = dict(noise_db=-200.0, full_transmit_diffraction=full)
    d = torch.from_numpy(scat).cuda()

    def record(n_smp):
        ch = capi.Channel(capi.Probe(n_el, 3e-4, 2.7e-4, 5e-3, 5e6, 0.6), capi.Medium(1540.0, 0.5, 1000.0),
                          capi.Acquisition(2e7, n_smp, 0.0, 5e3), tx)
        rf = torch.full((2, n_el, n_smp), 7.0, device="cuda")
        count, _ = ctx.simulate(ch, capi.sim_config(**cfg), d.data_ptr(), len(scat), None, rf.data_ptr(), True)
        return rf, count

    got, count = record(130)
    longer, more = record(600)
    assert torch.equal(got, longer[:, :, :130]) and 0 < count < more
    cd = O.channel_desc(O.probe(n_elements=n_el, pitch=3e-4, element_width=2.7e-4, center_frequency=5e6, bandwidth=0.6),
                        O.medium(), O.acquisition(fs=2e7, n_samples=130, prf=5e3),
                        O.TxSet(np.full(2, 1, np.int32), np.zeros(2, np.float32), np.zeros((2, 3), np.float32),
                                np.zeros((2, 3), np.float32), z, w))
    want = oracle.simulate(cd, O.sim_config(**cfg), scat)
    assert np.abs(want).max() > 0 and rel_l2(got.cpu().numpy(), want) < 1e-5


@pytest.mark.parametrize("n_smp,taps", [(14679840, 33), (14680064, 33), (14680064, 21)])
def test_demodulation_of_the_longest_traces(gpu, oracle, n_smp, taps):
    """65,535 segments of 224 outputs, and one more: against the oracle, tap by
    tap in the same order (1e-5 of the largest output, as at other sizes)."""
    torch, capi, ctx = gpu
    rf = np.random.default_rng(6).standard_normal((1, 1, n_smp)).astype(np.float32)
    z, w = np.zeros((1, 1), np.float32), np.ones((1, 1), np.float32)
    ch = capi.Channel(capi.Probe(1, 3e-4, 2.7e-4, 5e-3, 5e6, 0.6), capi.Medium(1540.0, 0.5, 1000.0),
                      capi.Acquisition(2e7, n_smp, 0.0, 5e3), [dict(type=1, angle=0.0, delays=z[0], apodization=w[0])])
    cd = O.channel_desc(O.probe(n_elements=1, pitch=3e-4, element_width=2.7e-4, center_frequency=5e6, bandwidth=0.6),
                        O.medium(), O.acquisition(fs=2e7, n_samples=n_smp, prf=5e3),
                        O.TxSet(np.full(1, 1, np.int32), np.zeros(1, np.float32), np.zeros((1, 3), np.float32),
                                np.zeros((1, 3), np.float32), z, w))
    want = oracle.demodulate(cd, O.demod_config(filter_taps=taps), rf)
    d = torch.from_numpy(rf).cuda()
    iq = torch.full(want.shape, float("nan"), dtype=torch.complex64, device="cuda")
    ctx.demodulate(ch, capi.demod_config(filter_taps=taps), d.data_ptr(), iq.data_ptr())
    assert np.abs(iq.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("n_smp,cfg", [(30, dict(filter_taps=65)), (300, dict(filter_taps=47)),
                                       (1100, dict(decimation=4)), (700, dict(filter_taps=127, decimation=13))])
def test_demodulation_of_few_traces(gpu, n_smp, cfg):
    """Blocks of one, two, four and eight traces: each trace as among nine, bit for bit."""
    torch, capi, ctx = gpu
    rf = torch.from_numpy(np.random.default_rng(8).standard_normal((9, n_smp)).astype(np.float32)).cuda()

    def demodulated(n):
        tx = [dict(type=1, angle=0.0, delays=np.zeros(n, np.float32), apodization=np.ones(n, np.float32))]
        ch = capi.Channel(capi.Probe(n, 3e-4, 2.7e-4, 5e-3, 5e6, 0.6), capi.Medium(1540.0, 0.5, 1000.0),
                          capi.Acquisition(2e7, n_smp, 1e-6, 5e3), tx)
        iq = torch.full((n + 1, -(-n_smp // cfg.get("decimation", 1))), 7.0, dtype=torch.complex64, device="cuda")
        ctx.demodulate(ch, capi.demod_config(**cfg), rf.data_ptr(), iq.data_ptr())
        assert (iq[n] == 7.0).all()   # nothing past the last trace
        return iq[:n]

    want = demodulated(9)
    assert torch.isfinite(torch.view_as_real(want)).all() and want.abs().max() > 0
    for n in (1, 2, 3, 4, 5, 8):
        assert torch.equal(demodulated(n), want[:n])


def probe_channel(capi, n_ev, n_el=40, n_smp=260, kind=1, t0=0.0, iq=True):
    tx = [dict(type=kind, angle=0.1 * e - 0.1, focus=(0.0, 0.0, -0.01 - 1e-3 * e), delays=np.zeros(n_el, np.float32),
               apodization=np.ones(n_el, np.float32)) for e in range(n_ev)]
    return tx, lambda: capi.Channel(capi.Probe(n_el, 3e-4, 2.7e-4, 5e-3, 5e6, 0.6), capi.Medium(1540.0, 0.5, 1000.0),
                                    capi.Acquisition(2e7, n_smp, t0, 5e3), tx, iq, 5e6 if iq else 0.0)


def image_points(n0=9, n1=20):
    ax0 = np.linspace(-5e-3, 5e-3, n0).astype(np.float32)
    ax1 = np.linspace(0.0, 9e-3, n1).astype(np.float32)
    pts = np.stack(np.broadcast_arrays(ax0[:, None], 0.0, ax1[None]), -1).astype(np.float32)
    return ax0, ax1, pts.reshape(-1, 3).copy()


def frames_of(capi, torch, ctx, ch, grid, data, variants, mv=False, **cfg):
    d = torch.from_numpy(data).cuda()
    out, got = torch.empty(grid.shape, dtype=torch.complex64, device="cuda"), []
    for v in variants:
        plan = ctx.plan(ch, grid, capi.bf_config(f_number=1.0, combiner=2 if mv else 0, **cfg))
        if mv:
            plan.set_mv_mode(3)
        if v is not None:
            plan.set_variant(v)
        out.fill_(7.0)
        plan.execute(d.data_ptr(), out.data_ptr())
        got.append(out.cpu().numpy())
        plan.close()
    return got


@pytest.mark.parametrize("mv", [False, True])
@pytest.mark.parametrize("what", ["angle", "focus", "t0", "late t0", "points"])
@pytest.mark.parametrize("weighting", [0, 1])
def test_delays_that_are_no_numbers_reach_the_frame(gpu, what, weighting, mv):
    """A NaN in an event's steering, in the time origin or in a point is not
    dropped: each channel-warp shape gives the pixels of the thread-per-pixel
    kernel, NaN where its are."""
    torch, capi, ctx = gpu
    t0 = np.nan if what == "t0" else np.inf if what == "late t0" else 0.0
    tx, channel = probe_channel(capi, 3, kind=2 if what == "focus" else 1, t0=t0)
    if what == "angle":
        tx[1]["angle"] = np.nan
    if what == "focus":
        tx[2]["focus"] = (0.0, np.nan, -0.01)
    ax0, ax1, pts = image_points()
    if what == "points":
        for k, c in ((30, 0), (75, 1), (120, 2), (50, 0), (95, 1), (140, 2)):
            pts[k, c] = np.nan if k in (30, 75, 120) else np.inf
        pts[170] = (0.5 * 3e-4, 0.0, np.nan)   # over an element
    rng = np.random.default_rng(8)
    iq = (rng.normal(size=(3, 40, 260)) + 1j * rng.normal(size=(3, 40, 260))).astype(np.complex64)
    got = frames_of(capi, torch, ctx, channel(), capi.Grid(0, ax0, ax1, pts), iq, (0, None, 1, 2, 3, 22, 23), mv=mv,
                    transmit_weighting=weighting, rx_window=0)
    if not mv and what not in ("late t0",):
        assert np.isnan(got[0]).any()
    for g in got[1:]:
        assert np.array_equal(g, got[0], equal_nan=True)


@pytest.mark.parametrize("cfg", [{}, dict(compounding=1), dict(compounding=2)])
def test_rf_frames_are_the_same_in_every_shape(gpu, cfg):
    """RF data run one launch shape whichever is set, and tuning picks one."""
    torch, capi, ctx = gpu
    _, channel = probe_channel(capi, 3, iq=False)
    grid = capi.Grid(0, *image_points())
    rf = np.random.default_rng(9).normal(size=(3, 40, 260)).astype(np.float32)
    n = len(capi.das_variants())
    got = frames_of(capi, torch, ctx, channel(), grid, rf, (None, *range(n)), **cfg)
    assert np.abs(got[0]).max() > 0 and not (got[0] == 7.0).any()
    for v, g in enumerate(got[1:]):
        assert np.array_equal(g, got[0]), v
    plan = ctx.plan(channel(), grid, capi.bf_config(f_number=1.0, **cfg))
    d, out = torch.from_numpy(rf).cuda(), torch.full(grid.shape, 7.0, dtype=torch.complex64, device="cuda")
    best, ms = plan.autotune(d.data_ptr(), out.data_ptr(), 1)
    assert 0 <= best < n and all(m > 0 for m in ms)
    assert np.array_equal(out.cpu().numpy(), got[0])
    plan.close()


def test_a_first_large_rf_frame_is_tuned(gpu):
    """The host class times the shapes on a plan's first frame of 1e9 pixel x
    event x channel terms or more: RF as IQ, the frame that of the next call."""
    import usx
    probe = usx.presets.linear_5mhz()
    probe.n_elements = 32
    acq = usx.presets.acquisition(probe, depth=0.02, medium=usx.Medium(), samples_per_wavelength=4.0)
    cfg = usx.SimulatorConfig()
    cfg.noise_db = -200.0
    sim = usx.Simulator(probe, usx.Medium(), acq, cfg)
    raw = sim.simulate(sim.make_plane_waves(usx.angles_deg(-6, 6, 31)), usx.Phantom.speckle_box(-0.004, 0.004, 0.004, 0.018,
                                                                                               0.0, 100, 5))
    grid = usx.ScanGrid.cartesian(-0.004, 0.004, 800, 0.004, 0.018, 1300)
    bf = usx.Beamformer(usx.BeamformerConfig())
    first, second = (np.asarray(bf.beamform(raw, grid).data) for _ in range(2))
    assert np.abs(first).max() > 0 and np.array_equal(first, second)


@pytest.mark.parametrize("n_ev,n_el", [(1, 40), (2, 9), (5, 64), (40, 24), (90, 40)])
@pytest.mark.parametrize("mv", [False, True])
def test_selected_events_are_the_first_of_the_largest_weight(gpu, n_ev, n_el, mv):
    """Beams in pairs of equal illumination: the pixels take the first of a
    pair, in every shape as in the thread-per-pixel kernel, in a queue too."""
    torch, capi, ctx = gpu
    pitch, n_smp = 3e-4, 260
    pos = (np.arange(n_el) - 0.5 * (n_el - 1)) * pitch
    tx = []
    for e in range(n_ev):
        x = 0.8 * pos[-1] * (2.0 * (e // 2) / max(1, (n_ev + 1) // 2 - 1) - 1.0) if n_ev > 2 else 0.0
        apod = (np.abs(pos - x) <= 6 * pitch).astype(np.float32)
        tx.append(dict(type=0, angle=0.0, focus=(x, 0.0, 0.006), origin=(x, 0.0, 0.0),
                       delays=np.zeros(n_el, np.float32), apodization=apod))
    ch = capi.Channel(capi.Probe(n_el, pitch, 2.7e-4, 5e-3, 5e6, 0.6), capi.Medium(1540.0, 0.5, 1000.0),
                      capi.Acquisition(2e7, n_smp, 0.0, 5e3), tx, True, 5e6)
    grid = capi.Grid(0, *image_points(13, 37))
    rng = np.random.default_rng(n_ev)
    iq = (rng.normal(size=(n_ev, n_el, n_smp)) + 1j * rng.normal(size=(n_ev, n_el, n_smp))).astype(np.complex64)
    got = frames_of(capi, torch, ctx, ch, grid, iq, (0, None, 1, 2, 3, 22, 23), mv=mv, compounding=2)
    assert np.abs(got[0]).max() > 0
    for g in got[1:]:
        assert np.array_equal(g, got[0])
    if not mv:
        plans = [ctx.plan(ch, grid, capi.bf_config(f_number=1.0, compounding=c)) for c in (2, 0, 2)]
        d = torch.from_numpy(iq).cuda()
        out = torch.full((3, *grid.shape), 7.0, dtype=torch.complex64, device="cuda")
        ctx.execute_queue(plans, [d.data_ptr()] * 3, [o.data_ptr() for o in out])
        want = frames_of(capi, torch, ctx, ch, grid, iq, (0,))[0]
        for o, w in zip(out.cpu().numpy(), (got[0], want, got[0])):
            assert np.array_equal(o, w)
        for p in plans:
            p.close()


@pytest.mark.parametrize("n0,n1,n_ev", [(4, 8, 3), (40, 90, 3), (300, 400, 3), (300, 400, 20), (200, 300, 70)])
def test_a_plan_reports_the_shape_it_runs(gpu, n0, n1, n_ev):
    """Neither set nor tuned: the shape of one acquisition, so that what is
    read from a plan and set on another leaves its speed as it was."""
    torch, capi, ctx = gpu
    _, channel = probe_channel(capi, n_ev)
    grid = capi.Grid(0, *image_points(n0, n1))
    kinds = [v[5] for v in capi.das_variants()]
    for cfg, iq, want in ((dict(), True, 4), (dict(compounding=2), True, 4), (dict(compounding=1), True, 0)):
        plan = ctx.plan(channel(), grid, capi.bf_config(f_number=1.0, **cfg))
        assert kinds[plan.variant()] == want
        plan.set_variant(0)
        assert plan.variant() == 0
        plan.close()
    _, rf = probe_channel(capi, n_ev, iq=False)
    plan = ctx.plan(rf(), grid, capi.bf_config(f_number=1.0))
    assert plan.variant() == 0
    plan.close()


def test_tuning_that_fails_leaves_the_plan_as_it_was(gpu):
    """A learned plan without its network cannot be tuned: it keeps the rule's
    shape, and a shape that was set stays set."""
    torch, capi, ctx = gpu
    _, channel = probe_channel(capi, 3)
    grid = capi.Grid(0, *image_points())
    d = torch.zeros((3, 40, 260), dtype=torch.complex64, device="cuda")
    out = torch.zeros(grid.shape, dtype=torch.complex64, device="cuda")
    plan = ctx.plan(channel(), grid, capi.bf_config(f_number=1.0, combiner=3))
    before = plan.variant()
    assert before != 0
    for v in (before, 6):
        with pytest.raises(Exception, match="no network"):
            plan.autotune(d.data_ptr(), out.data_ptr(), 1)
        assert plan.variant() == v
        plan.set_variant(6)
    plan.close()


@pytest.mark.parametrize("n_el,n0,n1,n_ev,cfg,kind", [
    (2, 512, 1024, 1, {}, 0), (4, 512, 1024, 75, {}, 0), (8, 512, 1024, 1, {}, 0), (6, 512, 1024, 11, dict(compounding=2), 0),
    (32, 1, 200000, 11, {}, 0), (64, 2, 100000, 40, {}, 0),
    (8, 512, 1024, 20, {}, 4), (2, 16, 40, 3, {}, 4), (9, 512, 1024, 1, {}, 4), (128, 1, 200000, 11, {}, 4)])
def test_the_shape_of_few_channels_and_thin_grids(gpu, n_el, n0, n1, n_ev, cfg, kind):
    """Where channel warps or tiles would stay empty, a thread per pixel."""
    torch, capi, ctx = gpu
    _, channel = probe_channel(capi, n_ev, n_el=n_el)
    ax0, ax1 = np.linspace(-5e-3, 5e-3, n0).astype(np.float32), np.linspace(1e-3, 9e-3, n1).astype(np.float32)
    pts = np.stack(np.broadcast_arrays(ax0[:, None], 0.0, ax1[None]), -1).astype(np.float32)
    plan = ctx.plan(channel(), capi.Grid(0, ax0, ax1, pts.reshape(-1, 3)), capi.bf_config(f_number=1.0, **cfg))
    assert capi.das_variants()[plan.variant()][5] == kind
    plan.close()


@pytest.mark.parametrize("n,wall", [(5, 0), (12, 1), (33, 2), (9, 2)])
def test_wall_filter_in_place(gpu, n, wall):
    torch, capi, ctx = gpu
    rng = np.random.default_rng(n)
    z = torch.from_numpy((rng.normal(size=(n, 1000)) + 1j * rng.normal(size=(n, 1000))).astype(np.complex64)).cuda()
    out = torch.empty_like(z)
    ctx.wall_filter(z.data_ptr(), n, 1000, wall, 2, out.data_ptr())
    ctx.wall_filter(z.data_ptr(), n, 1000, wall, 2, z.data_ptr())
    assert torch.equal(z, out)


@pytest.mark.parametrize("n0,n1", [(1, 3), (2, 9), (7, 5), (16, 40)])
def test_scan_extent_keeps_the_first_zero_s_sign(gpu, n0, n1):
    """Extents of zero: as one pass over the points keeps the first of equal
    values, whichever zeros follow it."""
    torch, capi, ctx = gpu
    rng = np.random.default_rng(n0)
    img, px = torch.zeros((n0, n1), device="cuda"), torch.empty((4, 4), device="cuda")
    for side in (1.0, -1.0):
        pts = (side * rng.random((n0 * n1, 3))).astype(np.float32)
        pts[rng.random(pts.shape) < 0.2] = 0.0
        pts[rng.random(pts.shape) < 0.2] = -0.0
        pts[n0 * n1 // 3] = 0.0
        got = ctx.scan_convert(img.data_ptr(), capi.Grid(0, np.linspace(-1, 1, n0), np.linspace(0, 1, n1), pts), 4, 4,
                               0.0, px.data_ptr())
        want = []
        for c in (0, 2):
            lo, hi = np.float32(np.finfo(np.float32).max), np.float32(-np.finfo(np.float32).max)
            for v in pts[:, c]:
                lo, hi = (v if v < lo else lo), (v if hi < v else hi)
            want += [lo, hi]
        assert np.asarray(got, np.float32).tobytes() == np.asarray(want, np.float32).tobytes()


def test_queues_of_few_channels_and_thin_grids(gpu):
    """Both tiles of the queue, by its entries' work: each frame as alone."""
    torch, capi, ctx = gpu
    rng = np.random.default_rng(12)

    def entry(n_el, n_ev, n0, n1, **cfg):
        _, channel = probe_channel(capi, n_ev, n_el=n_el)
        iq = (rng.normal(size=(n_ev, n_el, 260)) + 1j * rng.normal(size=(n_ev, n_el, 260))).astype(np.complex64)
        grid = capi.Grid(0, *image_points(n0, n1))
        want = frames_of(capi, torch, ctx, channel(), grid, iq, (0,), **cfg)[0]
        return ctx.plan(channel(), grid, capi.bf_config(f_number=1.0, **cfg)), torch.from_numpy(iq).cuda(), want

    few = [entry(3, 40, 30, 70), entry(24, 2, 9, 33, compounding=2), entry(1, 1, 1, 1)]
    thin = [entry(64, 3, 2, 700), entry(40, 35, 1, 900)]
    full = [entry(128, 5, 40, 50), entry(128, 83, 17, 20, compounding=2)]
    for queue in (few, thin, full, few + thin + full, full[:1] + few):
        out = [torch.full(w.shape, 7.0, dtype=torch.complex64, device="cuda") for _, _, w in queue]
        ctx.execute_queue([p for p, _, _ in queue], [d.data_ptr() for _, d, _ in queue], [o.data_ptr() for o in out])
        for o, (_, _, w) in zip(out, queue):
            assert np.array_equal(o.cpu().numpy(), w)
    for p, _, _ in few + thin + full:
        p.close()


def test_a_plane_wave_s_unused_focus_does_not_matter(gpu):
    """Its delays are numbers: the rule's shape, and the frame."""
    torch, capi, ctx = gpu
    tx, channel = probe_channel(capi, 3)
    grid = capi.Grid(0, *image_points())
    rng = np.random.default_rng(2)
    iq = (rng.normal(size=(3, 40, 260)) + 1j * rng.normal(size=(3, 40, 260))).astype(np.complex64)
    want = frames_of(capi, torch, ctx, channel(), grid, iq, (0,))[0]
    for t in tx:
        t["focus"] = (0.0, np.nan, np.inf)
    plan = ctx.plan(channel(), grid, capi.bf_config(f_number=1.0))
    assert plan.variant() != 0
    plan.close()
    assert np.array_equal(frames_of(capi, torch, ctx, channel(), grid, iq, (None,))[0], want)
