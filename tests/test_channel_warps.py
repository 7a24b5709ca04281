"""The channel-warp delay-and-sum shapes and the rule that picks one of them for
a plan whose shape was neither set nor tuned: every frame equals the
thread-per-pixel kernel's (shape 0) bit for bit, at the edges of the tiles, of
the channel groups, of the transmit table and of the traces."""

from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLANE, DIVERGING, FOCUSED = 1, 2, 0
SHAPES = (1, 2, 3, 22, 23)

# name: elements, samples, events, transmit, n0, n1, t0, config
CASES = {
    "tiny": (32, 300, 1, PLANE, 1, 1, 0.0, {}),
    "ragged channels": (30, 200, 7, PLANE, 9, 33, 0.0, dict(f_number=1.0)),
    "one channel": (1, 120, 2, PLANE, 5, 40, 0.0, dict(rx_window=0)),
    "more events than the table": (18, 160, 83, PLANE, 6, 31, 0.0, {}),
    "time offset, short traces": (33, 70, 5, PLANE, 8, 65, 2.5e-6, dict(f_number=1.2, rx_window=0)),
    "two-sample traces": (16, 2, 3, PLANE, 4, 24, 2e-6, dict(rx_window=0)),
    "one-sample traces": (16, 1, 3, PLANE, 4, 24, 2e-6, dict(rx_window=0)),
    "diverging DMAS with coherence factor": (64, 400, 9, DIVERGING, 12, 50, 0.0,
                                             dict(combiner=1, coherence_factor=1)),
    "focused select": (32, 300, 11, FOCUSED, 16, 40, 0.0, dict(compounding=2)),
    "select past the table": (20, 200, 90, FOCUSED, 5, 20, 0.0, dict(compounding=2, combiner=1)),
    "unweighted": (128, 500, 4, PLANE, 20, 70, 0.0, dict(transmit_weighting=0, f_number=0.8)),
    "wide": (128, 500, 3, PLANE, 200, 300, 0.0, {}),
}


def build(capi, n_el, n_smp, n_ev, kind, n0, n1, t0):
    tx = []
    for e in range(n_ev):
        s = 0.0 if n_ev == 1 else -1.0 + 2.0 * e / (n_ev - 1)
        a = 0.2 * s
        focus = (0.0, 0.0, 0.03) if kind == PLANE else (-0.01 * math.sin(a), 0.0, -0.01 * math.cos(a)) \
            if kind == DIVERGING else (0.004 * s, 0.0, 0.012)
        tx.append(dict(type=kind, angle=a, focus=focus, origin=(0.004 * s if kind == FOCUSED else 0.0, 0, 0),
                       delays=np.zeros(n_el, np.float32), apodization=np.ones(n_el, np.float32)))
    ch = capi.Channel(capi.Probe(n_el, 3e-4, 2.7e-4, 5e-3, 5e6, 0.6), capi.Medium(1540.0, 0.5, 1000.0),
                      capi.Acquisition(2e7, n_smp, t0, 5e3), tx, True, 5e6)
    half = 0.5 * n_el * 3e-4
    ax0 = np.linspace(-half, half, n0).astype(np.float32)
    ax1 = np.linspace(0.0, 0.016, n1).astype(np.float32)   # the first depth has no aperture
    pts = np.stack(np.broadcast_arrays(ax0[:, None], 0.0, ax1[None]), -1).astype(np.float32)
    return ch, capi.Grid(0, ax0, ax1, pts.reshape(-1, 3))


@pytest.mark.parametrize("name", CASES)
def test_frames_equal_the_thread_per_pixel_kernel(name):
    import torch
    from usx import capi
    n_el, n_smp, n_ev, kind, n0, n1, t0, cfg = CASES[name]
    ctx = capi.Context(0, stream=torch.cuda.current_stream().cuda_stream)
    ch, grid = build(capi, n_el, n_smp, n_ev, kind, n0, n1, t0)
    rng = np.random.default_rng(3)
    iq = (rng.normal(size=(n_ev, n_el, n_smp)) + 1j * rng.normal(size=(n_ev, n_el, n_smp))).astype(np.complex64)
    if n_smp > 100:   # a broken sample stays where it is read
        iq[0, 0, 50], iq[-1, -1, 60] = np.nan, np.inf
    d = torch.from_numpy(iq).cuda()
    out = torch.empty(grid.shape, dtype=torch.complex64, device="cuda")

    def frame(variant):
        plan = ctx.plan(ch, grid, capi.bf_config(**{"f_number": 1.5, **cfg}))
        if variant is not None:
            plan.set_variant(variant)
        out.fill_(7.0)
        plan.execute(d.data_ptr(), out.data_ptr())
        r = out.cpu().numpy()
        plan.close()
        return r

    want = frame(0)
    assert np.abs(np.nan_to_num(want)).max() > 0 or n_smp < 3 or n1 == 1   # (the first depth has no aperture)
    for v in (None, *SHAPES):
        assert np.array_equal(frame(v), want, equal_nan=True), v
    plan = ctx.plan(ch, grid, capi.bf_config(**{"f_number": 1.5, **cfg}))
    out.fill_(7.0)
    ctx.execute_queue([plan], [d.data_ptr()], [out.data_ptr()])
    assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)
    plan.close()
    ctx.close()


@pytest.mark.parametrize("epf,n0,n1", [(1, 3, 17), (4, 40, 90)])
def test_sequences_take_each_frame_s_events(epf, n0, n1):
    import torch
    from usx import capi
    n_f, n_el, n_smp = 5, 22, 260
    ctx = capi.Context(0, stream=torch.cuda.current_stream().cuda_stream)
    ch, grid = build(capi, n_el, n_smp, epf * n_f, PLANE, n0, n1, 0.0)
    rng = np.random.default_rng(4)
    shape = (epf * n_f, n_el, n_smp)
    d = torch.from_numpy((rng.normal(size=shape) + 1j * rng.normal(size=shape)).astype(np.complex64)).cuda()
    got = []
    for v in (0, None, *SHAPES):
        plan = ctx.plan(ch, grid, capi.bf_config(f_number=1.5))
        if v is not None:
            plan.set_variant(v)
        out = torch.full((n_f, n0, n1), 7.0, dtype=torch.complex64, device="cuda")
        plan.execute_sequence(epf, n_f, d.data_ptr(), out.data_ptr(), n0 * n1)
        got.append(out.cpu().numpy())
        plan.close()
    assert np.abs(got[0]).max() > 0
    for g in got[1:]:
        assert np.array_equal(g, got[0])
    ctx.close()
