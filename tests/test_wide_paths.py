"""Paths chosen by size: the simulator's pulse and time-table variants, the
four-line displacement kernel against the oracle at ragged sizes and at the
columns its windows clip, and the scan converter's extent of the points."""

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


# FP32 sums of at most a few hundred terms, the oracle's expressions in the same
# order: the bar of the simulator's and the tracker's other tests, 1e-5.
@pytest.mark.parametrize("n_el,n_smp,cfg", [
    (33, 500, dict(oversampling=8)),                      # pulse of more than 64 slots
    (17, 8192, {}), (17, 8193, {}),                       # the time table's last size, and past it
    (64, 600, dict(oversampling=1, incident_trim_db=-20.0)),
    (5, 700, dict(full_transmit_diffraction=0)),
])
def test_simulator_variants(gpu, oracle, n_el, n_smp, cfg):
    torch, capi, ctx = gpu
    rng = np.random.default_rng(n_el)
    half = 0.5 * n_el * 3e-4
    scat = np.zeros((60, 8), np.float32)
    scat[:, 0], scat[:, 2] = rng.uniform(-half, half, 60), rng.uniform(3e-3, 0.016, 60)
    scat[:, 3], scat[:, 6] = rng.normal(size=60), 0.01
    ang = np.array([-0.15, 0.1], np.float32)
    ex = ((np.arange(n_el) - 0.5 * (n_el - 1)) * 3e-4).astype(np.float32)
    delays = (ex[None] * np.sin(ang)[:, None] / 1540.0).astype(np.float32)
    apod = np.ones((2, n_el), np.float32)
    tx = [dict(type=1, angle=float(a), delays=d, apodization=w) for a, d, w in zip(ang, delays, apod)]
    args = dict(noise_db=-200.0, **cfg)
    ch = capi.Channel(capi.Probe(n_el, 3e-4, 2.7e-4, 5e-3, 5e6, 0.6), capi.Medium(1540.0, 0.5, 1000.0),
                      capi.Acquisition(2e7, n_smp, 0.0, 5e3), tx)
    d = torch.from_numpy(scat).cuda()
    rf = torch.full((2, n_el, n_smp), 7.0, device="cuda")
    ctx.simulate(ch, capi.sim_config(**args), d.data_ptr(), len(scat), None, rf.data_ptr())
    txs = O.TxSet(np.full(2, 1, np.int32), ang, np.tile(np.array([0, 0, 0.03], np.float32), (2, 1)),
                  np.zeros((2, 3), np.float32), delays, apod)
    cd = O.channel_desc(O.probe(n_elements=n_el, pitch=3e-4, element_width=2.7e-4, center_frequency=5e6,
                                bandwidth=0.6), O.medium(), O.acquisition(fs=2e7, n_samples=n_smp, prf=5e3), txs)
    want = oracle.simulate(cd, O.sim_config(**args), scat)
    assert np.abs(want).max() > 0
    assert rel_l2(rf.cpu().numpy(), want) < 1e-5


@pytest.mark.parametrize("n0,n1,ka,kl,lag", [
    (9, 70, 12, 2, 9),       # ragged lines, few interior columns
    (5, 44, 12, 2, 9),       # one interior column more than the clipped ones
    (4, 42, 12, 2, 9),       # none
    (33, 300, 8, 1, 20), (130, 140, 4, 0, 45), (200, 400, 4, 0, 6), (150, 300, 6, 2, 0),
    (12, 60, 3, 3, 4),       # wider than the four-line kernel takes
])
def test_displacement_at_every_edge(gpu, oracle, n0, n1, ka, kl, lag):
    torch, capi, ctx = gpu
    rng = np.random.default_rng(n1)
    z = rng.normal(size=(2, n0, n1 + 8))
    a = (z[0] + 1j * z[1])
    a = sum(a[:, j:j + n1] for j in range(6))
    b = (np.roll(a, 3, axis=1) * np.exp(-0.4j) + 0.05 * rng.normal(size=(n0, n1))).astype(np.complex64)
    a = a.astype(np.complex64)
    axis = (0.02 + 3.5e-5 * np.arange(n1)).astype(np.float32)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    ax, cr = torch.full((n0, n1), 7.0, device="cuda"), torch.full((n0, n1), 7.0, device="cuda")
    ctx.axial_displacement(da.data_ptr(), db.data_ptr(), n0, n1, axis, 5e6, 1540.0, ka, kl, lag, ax.data_ptr(),
                           cr.data_ptr())
    want_ax, want_cr = oracle.displacement(a, b, axis, 5e6, 1540.0, ka, kl, lag)
    assert rel_l2(cr.cpu().numpy(), want_cr) < 1e-5
    # A tie between two lags within the rounding of hypot may break either way.
    dz = float(axis[1] - axis[0])
    off = np.abs(ax.cpu().numpy() - want_ax) > 1e-3 * dz
    assert off.mean() <= 1e-3


@pytest.mark.parametrize("n0,n1", [(1, 1), (1, 7), (3, 5), (2, 8), (5, 13), (64, 33)])
def test_scan_extent_is_the_points_extent(gpu, n0, n1):
    torch, capi, ctx = gpu
    rng = np.random.default_rng(n0 * 100 + n1)
    pts = rng.normal(size=(n0 * n1, 3)).astype(np.float32)
    pts[rng.random(pts.shape) < 0.1] = np.nan     # passed over, as std::min passes it over
    pts[0] = (0.5, np.nan, 0.25)
    grid = capi.Grid(0, np.linspace(-1, 1, n0), np.linspace(0, 1, n1), pts)
    img = torch.zeros((n0, n1), device="cuda")
    px = torch.empty((4, 4), device="cuda")
    got = ctx.scan_convert(img.data_ptr(), grid, 4, 4, 0.0, px.data_ptr())
    want = [np.nanmin(pts[:, 0]), np.nanmax(pts[:, 0]), np.nanmin(pts[:, 2]), np.nanmax(pts[:, 2])]
    assert np.array_equal(got, np.array(want, np.float32))


@pytest.mark.parametrize("n,n0,n1,ka,kl,order", [
    (8, 241, 515, 4, 1, 1),     # four lines per thread: ragged lines and depths
    (33, 83, 500, 6, 2, 2),     # more than one row block of the wall filter
    (9, 300, 140, 0, 2, 1),     # a window of one depth
    (64, 65, 700, 3, 2, 0),     # the longest ensemble
    (5, 20, 33, 4, 1, 1), (12, 40, 60, 2, 3, 1),   # a pixel per thread
])
def test_colour_flow_at_every_window(gpu, oracle, n, n0, n1, ka, kl, order):
    """Maps against the oracle, whose sums run in the same order: power and
    variance to 1e-5, gates equal but for pixels within rounding of one."""
    torch, capi, ctx = gpu
    rng = np.random.default_rng(n * n1)
    ph = np.exp(1j * 0.5 * np.arange(n))[:, None, None] * np.exp(2j * np.arange(n1))[None, None]
    ens = ph + 3.0 + 0.5 * (rng.normal(size=(n, n0, n1)) + 1j * rng.normal(size=(n, n0, n1)))
    ens = ens.astype(np.complex64)
    axis = (0.02 + 4.9e-5 * np.arange(n1)).astype(np.float32)
    kw = dict(polynomial_order=order, kernel_axial=ka, kernel_lateral=kl)
    d = torch.from_numpy(ens).cuda()
    out = [torch.full((n0, n1), 7.0, device="cuda") for _ in range(3)] + \
          [torch.full((n0, n1), 9, dtype=torch.uint8, device="cuda")]
    ctx.color_flow(d.data_ptr(), n, n0, n1, axis, 5e6, 5e3, 1540.0, capi.doppler_config(**kw),
                   *[o.data_ptr() for o in out])
    vel, power, var, valid = (o.cpu().numpy() for o in out)
    w = oracle.color_flow(ens, axis, 5e6, 5e3, 1540.0, O.doppler_config(**kw))
    assert rel_l2(power, w[1]) < 1e-5 and rel_l2(var, w[2]) < 1e-5
    assert (valid != w[3]).mean() <= 1e-3
    both = (valid == 1) & (np.asarray(w[3]) == 1)
    if both.any():   # (8 frames: the wall filter leaves no pixel coherent enough)
        assert np.abs(vel - w[0])[both].max() <= 1e-4 * np.abs(w[0]).max()
    batch = [torch.empty((2, n0, n1), dtype=o.dtype, device="cuda") for o in out]
    ctx.color_flow_batch(d.data_ptr(), [n, n - 1], [0, 1], n0, n1, axis, 5e6, 5e3, 1540.0, capi.doppler_config(**kw),
                         *[o.data_ptr() for o in batch])
    for o, b in zip(out, batch):
        assert torch.equal(o, b[0])
