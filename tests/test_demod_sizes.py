"""The demodulator at the sizes where its kernels change: outputs per lane
(7, 11 or 13) by padding and number of traces, traces short of a block, traces
shorter than the filter, and the runtime-tap kernel with partial trace groups."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture()
def gpu():
    import torch
    from usx import capi
    ctx = capi.Context(0, stream=torch.cuda.current_stream().cuda_stream)
    yield torch, capi, ctx
    ctx.close()


@pytest.mark.parametrize("n_tx,n_el,n_smp,cfg", [
    (1, 3, 20, {}), (1, 9, 224, {}), (2, 7, 225, {}),                      # 7 outputs per lane
    (13, 127, 833, {}), (13, 127, 700, {}), (13, 127, 832, {}),            # 7, 11 and 13, several traces per warp
    (13, 127, 705, dict(filter_taps=21)), (1, 5, 16, dict(filter_taps=21)),
    (1, 11, 300, dict(filter_taps=47)), (2, 5, 129, dict(filter_taps=33, decimation=4)),
    (1, 9, 30, dict(filter_taps=65)),
])
def test_demodulation_at_every_split(gpu, oracle, n_tx, n_el, n_smp, cfg):
    """Against the oracle, tap by tap in the same order: FP32 rounding of the
    sums and of the mixing phase's sine, 1e-5 of the largest output, every
    sample written."""
    torch, capi, ctx = gpu
    rng = np.random.default_rng(n_smp)
    rf = rng.standard_normal((n_tx, n_el, n_smp)).astype(np.float32)
    z, w = np.zeros((n_tx, n_el), np.float32), np.ones((n_tx, n_el), np.float32)
    tx = [dict(type=1, angle=0.0, delays=z[e], apodization=w[e]) for e in range(n_tx)]
    ch = capi.Channel(capi.Probe(n_el, 3e-4, 2.7e-4, 5e-3, 5e6, 0.6), capi.Medium(1540.0, 0.5, 1000.0),
                      capi.Acquisition(2e7, n_smp, 1e-6, 5e3), tx)
    cd = O.channel_desc(O.probe(n_elements=n_el, pitch=3e-4, element_width=2.7e-4, center_frequency=5e6,
                                bandwidth=0.6), O.medium(), O.acquisition(fs=2e7, n_samples=n_smp, t0=1e-6, prf=5e3),
                        O.TxSet(np.full(n_tx, 1, np.int32), np.zeros(n_tx, np.float32),
                                np.zeros((n_tx, 3), np.float32), np.zeros((n_tx, 3), np.float32), z, w))
    want = oracle.demodulate(cd, O.demod_config(**cfg), rf)
    d = torch.from_numpy(rf).cuda()
    iq = torch.full(want.shape, float("nan"), dtype=torch.complex64, device="cuda")
    ctx.demodulate(ch, capi.demod_config(**cfg), d.data_ptr(), iq.data_ptr())
    assert np.abs(iq.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()
