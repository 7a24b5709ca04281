"""The FP32 minimum variance (factor with the right-hand sides as rows, panels of
four or eight columns) at every subarray length where a panel, a row slot or a class
ends, against the kernel in the reference's operation order."""

from __future__ import annotations

import numpy as np
import pytest

from gold import rel_l2

pytestmark = pytest.mark.gpu

# FP32 Cholesky of a covariance loaded by 1%: condition number at most ~100 L,
# so the two orders of summation differ by a few 1e-6; the bar of the FP32
# solver's other tests.
TOL = 1e-4


def setup(capi, torch, n_el, n0, n1, ev=1, seed=0):
    tx = [dict(type=1, angle=0.05 * e, delays=np.zeros(n_el, np.float32), apodization=np.ones(n_el, np.float32))
          for e in range(ev)]
    ch = capi.Channel(capi.Probe(n_el, 3e-4, 2.7e-4, 5e-3, 5e6, 0.6), capi.Medium(1540.0, 0.5, 1000.0),
                      capi.Acquisition(2e7, 1500, 0.0, 5e3), tx, True, 5e6)
    ax0 = np.linspace(-0.3, 0.3, n0).astype(np.float32) * n_el * 3e-4
    ax1 = np.linspace(1e-4, 0.04, n1).astype(np.float32)   # from no active channel to all of them
    pts = np.stack(np.broadcast_arrays(ax0[:, None], 0.0, ax1[None]), -1).astype(np.float32)
    rng = np.random.default_rng(seed)
    iq = (rng.normal(size=(ev, n_el, 1500)) + 1j * rng.normal(size=(ev, n_el, 1500))).astype(np.complex64)
    iq[:, :, 600:640] = 0   # some pixels without any signal
    return ch, capi.Grid(0, ax0, ax1, pts.reshape(-1, 3)), torch.from_numpy(iq).cuda()


def frames(capi, torch, n_el, n0, n1, ev=1, **cfg):
    ctx = capi.Context(0, stream=torch.cuda.current_stream().cuda_stream)
    ch, grid, iq = setup(capi, torch, n_el, n0, n1, ev)
    out = []
    for mode in (0, 3):
        plan = ctx.plan(ch, grid, capi.bf_config(combiner=2, f_number=1.0, **cfg))
        plan.set_mv_mode(mode)
        f = torch.full(grid.shape, float("nan"), dtype=torch.complex64, device="cuda")
        plan.execute(iq.data_ptr(), f.data_ptr())
        out.append(f.cpu().numpy())
        plan.close()
    ctx.close()
    return out


@pytest.mark.parametrize("L", [2, 3, 4, 5, 8, 15, 16, 17, 30, 31, 32, 33, 47, 48, 61, 62, 63, 64])
def test_every_subarray_length(L):
    import torch
    from usx import capi
    want, got = frames(capi, torch, 128, 3, 60, mv_subarray=L, mv_range_average=2)
    assert np.isfinite(got).all() and np.abs(want).max() > 0
    assert rel_l2(got, want) < TOL


@pytest.mark.parametrize("n_el,ra,cfg", [
    (4, 2, {}), (9, 0, {}), (31, 1, dict(coherence_factor=1)), (64, 4, {}), (127, 3, dict(rx_window=0)),
    (40, 2, dict(mv_diagonal_loading=0.2)), (33, 2, dict(compounding=1)), (128, 4, dict(coherence_factor=1)),
])
def test_rows_windows_and_options(n_el, ra, cfg):
    import torch
    from usx import capi
    want, got = frames(capi, torch, n_el, 4, 50, ev=2, mv_subarray=64, mv_range_average=ra, **cfg)
    assert np.isfinite(got).all() and np.abs(want).max() > 0
    assert rel_l2(got, want) < TOL


def test_training_export_still_returns_the_weights():
    """The export needs the weights themselves: its frames agree with the plain solver's."""
    import torch
    from usx import capi
    ctx = capi.Context(0, stream=torch.cuda.current_stream().cuda_stream)
    ch, grid, iq = setup(capi, torch, 128, 3, 60)
    out = []
    for export in (False, True):
        plan = ctx.plan(ch, grid, capi.bf_config(combiner=2, f_number=1.0, mv_subarray=64))
        plan.set_mv_mode(3)
        f = torch.empty(grid.shape, dtype=torch.complex64, device="cuda")
        if export:
            feat, w = torch.zeros((180, 256), device="cuda"), torch.zeros((180, 128), device="cuda")
            valid = torch.zeros(180, dtype=torch.uint8, device="cuda")
            plan.set_training_export(feat.data_ptr(), w.data_ptr(), valid.data_ptr())
        plan.execute(iq.data_ptr(), f.data_ptr())
        out.append(f.cpu().numpy())
        plan.close()
    ok = valid.cpu().numpy().astype(bool)
    s = w.view(-1, 64, 2)[..., 0].sum(1).cpu().numpy()
    assert ok.sum() > 100 and (s[ok] > 0).all()
    assert rel_l2(out[0], out[1]) < 1e-5
    ctx.close()
