"""Calls at the limits of their inputs: delays outside the simulator's window,
trace lengths at the demodulator's grid limit, delays that are not numbers, and
RF plans with every launch shape."""

from __future__ import annotations

import numpy as np
import pytest

from gold import rel_l2

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
