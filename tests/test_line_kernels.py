"""The four-line kernels of the colour flow and the displacement: which sizes
take them, by the name that the profiler gives, and their maps against the
pixel-per-thread kernels', bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def gpu():
    import torch
    from usx import capi
    ctx = capi.Context(0, stream=torch.cuda.current_stream().cuda_stream)
    yield torch, capi, ctx
    ctx.close()


def kernels(capi, torch, ctx, call):
    """Names of the kernels of one call."""
    capi.profile(ctx, True)
    capi.profile_reset(ctx)
    call()
    torch.cuda.synchronize()
    names = set(capi.profile_read(ctx))
    capi.profile(ctx, False)
    return names


def axis(n1):
    return (0.02 + 4.9e-5 * np.arange(n1)).astype(np.float32)


def speckle(torch, shape, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, dtype=torch.complex64, device="cuda", generator=g) + 2.0


def flow_maps(torch, shape):
    return [torch.full(shape, 7.0, device="cuda") for _ in range(3)] + \
           [torch.full(shape, 9, dtype=torch.uint8, device="cuda")]


def flow(ctx, capi, ens, maps, **cfg):
    n, n0, n1 = ens.shape
    ctx.color_flow(ens.data_ptr(), n, n0, n1, axis(n1), 5e6, 5e3, 1540.0, capi.doppler_config(**cfg),
                   *[m.data_ptr() for m in maps])


def flow_kernels(capi, torch, ctx, n, n0, n1, ka, kl):
    ens, maps = speckle(torch, (n, n0, n1)), flow_maps(torch, (n0, n1))
    return kernels(capi, torch, ctx, lambda: flow(ctx, capi, ens, maps, kernel_axial=ka, kernel_lateral=kl))


def disp_kernels(capi, torch, ctx, n0, n1, ka, kl, lag):
    a, b = speckle(torch, (n0, n1)), speckle(torch, (n0, n1), 1)
    ax, cr = torch.empty((n0, n1), device="cuda"), torch.empty((n0, n1), device="cuda")
    return kernels(capi, torch, ctx, lambda: ctx.axial_displacement(
        a.data_ptr(), b.data_ptr(), n0, n1, axis(n1), 5e6, 1540.0, ka, kl, lag, ax.data_ptr(), cr.data_ptr()))


def test_the_profiler_names_the_kernel_that_ran(gpu):
    torch, capi, ctx = gpu
    assert "flow_lines_kernel" in flow_kernels(capi, torch, ctx, 16, 256, 512, 4, 1)
    assert "flow_kernel" in flow_kernels(capi, torch, ctx, 16, 16, 40, 4, 1)
    assert "displacement_lines_kernel" in disp_kernels(capi, torch, ctx, 256, 1024, 8, 2, 8)
    assert "displacement_kernel" in disp_kernels(capi, torch, ctx, 16, 64, 4, 1, 4)
    ens, maps = speckle(torch, (24, 256, 512)), flow_maps(torch, (2, 256, 512))
    got = kernels(capi, torch, ctx, lambda: ctx.color_flow_batch(
        ens.data_ptr(), [16, 8], [0, 16], 256, 512, axis(512), 5e6, 5e3, 1540.0, capi.doppler_config(),
        *[m.data_ptr() for m in maps]))
    assert "flow_lines_batch_kernel" in got and "flow_batch_kernel" not in got
