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


@pytest.mark.parametrize("n,n0,n1,ka,kl,lines", [
    (16, 256, 512, 4, 1, True), (12, 200, 512, 6, 2, True), (8, 500, 1000, 1, 1, True), (32, 60, 700, 4, 2, True),
    (32, 3000, 40, 4, 1, False), (16, 1000, 130, 4, 1, False),    # blocks mostly empty in depth
    (32, 256, 512, 0, 1, False), (32, 256, 512, 1, 1, False),     # windows that do not pay for the staging
    (32, 400, 128, 6, 2, True), (12, 400, 128, 6, 2, False),      # one block in depth
    (12, 60, 700, 2, 2, False), (16, 1, 150000, 4, 2, False),     # too few blocks, no second line
    (5, 500, 1000, 4, 1, False), (16, 256, 512, 4, 3, False)])
def test_colour_flow_kernel_by_size(gpu, n, n0, n1, ka, kl, lines):
    torch, capi, ctx = gpu
    assert ("flow_lines_kernel" in flow_kernels(capi, torch, ctx, n, n0, n1, ka, kl)) == lines


@pytest.mark.parametrize("n,n0,n1,ka,kl", [(8, 261, 640, 4, 1), (33, 183, 500, 6, 2), (9, 500, 999, 1, 2),
                                           (64, 255, 512, 3, 1)])
def test_colour_flow_lines_equal_a_pixel_per_thread(gpu, n, n0, n1, ka, kl):
    """A hundred columns of the same ensemble run a pixel per thread; away from
    their cut edges every sum is over the same terms in the same order. (The
    valid bytes pass the power gate, which depends on the frame's maximum.)"""
    torch, capi, ctx = gpu
    ens = speckle(torch, (n, n0, n1), n)
    ens[:, 7, 300:340] = 0
    ens[1, 20, 330] = float("nan")
    ens[2, 40, 310] = float("inf")
    cfg = dict(kernel_axial=ka, kernel_lateral=kl, power_threshold_db=-300.0, coherence_threshold=0.05, polynomial_order=0)
    whole, part = flow_maps(torch, (n0, n1)), flow_maps(torch, (n0, 100))
    assert "flow_lines_kernel" in kernels(capi, torch, ctx, lambda: flow(ctx, capi, ens, whole, **cfg))
    for j0 in (0, 128 - 50, 300, n1 - 100):
        cut = ens[:, :, j0:j0 + 100].contiguous()
        assert "flow_kernel" in kernels(capi, torch, ctx, lambda: flow(ctx, capi, cut, part, **cfg))
        lo, hi = (0 if j0 == 0 else ka + 1), (100 if j0 == n1 - 100 else 100 - ka - 1)
        for w, p in zip(whole[:3], part):
            w, p = w[:, j0 + lo:j0 + hi].cpu().numpy(), p[:, lo:hi].cpu().numpy()
            assert np.array_equal(w, p, equal_nan=True)
    assert (whole[0] != 0).sum() > 1000   # coherent pixels have a velocity


@pytest.mark.parametrize("ka,kl", [(4, 1), (3, 2)])
def test_uneven_batches_equal_one_ensemble_at_a_time(gpu, ka, kl):
    """Ensembles of 32, 2, 7 and 9 frames in one four-line launch; alone, those
    below eight frames run a pixel per thread."""
    torch, capi, ctx = gpu
    frames, n0, n1 = [32, 2, 7, 9], 256, 512
    ens = speckle(torch, (sum(frames), n0, n1), 3)
    cfg = dict(kernel_axial=ka, kernel_lateral=kl, coherence_threshold=0.05, polynomial_order=0)
    off = [0, 32, 34, 41]
    maps = flow_maps(torch, (4, n0, n1))
    got = kernels(capi, torch, ctx, lambda: ctx.color_flow_batch(
        ens.data_ptr(), frames, off, n0, n1, axis(n1), 5e6, 5e3, 1540.0, capi.doppler_config(**cfg),
        *[m.data_ptr() for m in maps]))
    assert "flow_lines_batch_kernel" in got
    for e, (n, o) in enumerate(zip(frames, off)):
        one = flow_maps(torch, (n0, n1))
        names = kernels(capi, torch, ctx, lambda: flow(ctx, capi, ens[o:o + n].contiguous(), one, **cfg))
        assert ("flow_kernel" in names) == (n < 8)
        for m, w in zip(maps, one):
            assert torch.equal(m[e], w)
        assert (one[3] == 1).any()


@pytest.mark.parametrize("n0,n1,ka,kl,lag,lines", [
    (256, 1024, 8, 2, 8, True), (256, 300, 4, 2, 4, True), (128, 512, 12, 0, 8, True), (2000, 80, 4, 2, 8, True),
    (20000, 12, 1, 2, 2, False), (5000, 30, 4, 1, 4, False), (2000, 50, 2, 0, 12, False),   # few interior columns
    (128, 512, 1, 0, 30, False), (64, 256, 4, 0, 4, False), (1, 100000, 2, 2, 12, False), (1, 100000, 8, 2, 8, True),
    (12, 64, 8, 2, 8, False),
    (256, 1024, 4, 3, 8, False)])
def test_displacement_kernel_by_size(gpu, n0, n1, ka, kl, lag, lines):
    torch, capi, ctx = gpu
    assert ("displacement_lines_kernel" in disp_kernels(capi, torch, ctx, n0, n1, ka, kl, lag)) == lines


@pytest.mark.parametrize("n0,n1,ka,kl,lag", [(130, 700, 8, 2, 8), (257, 640, 3, 1, 5), (515, 400, 6, 0, 12)])
def test_displacement_lines_equal_a_pixel_per_thread(gpu, n0, n1, ka, kl, lag):
    """Six lines of the same frames run a pixel per thread; away from their cut
    edges every sum is over the same terms in the same order."""
    torch, capi, ctx = gpu
    a = speckle(torch, (n0, n1), n0)
    b = torch.roll(a, 3, 1) * np.exp(-0.4j) + 0.05 * speckle(torch, (n0, n1), 1)
    a[7, 300:340] = 0
    b[9, 200] = float("nan")
    ax, cr = torch.full((n0, n1), 7.0, device="cuda"), torch.full((n0, n1), 7.0, device="cuda")

    def run(x, y, m, c):
        return kernels(capi, torch, ctx, lambda: ctx.axial_displacement(
            x.data_ptr(), y.data_ptr(), x.shape[0], n1, axis(n1), 5e6, 1540.0, ka, kl, lag, m.data_ptr(), c.data_ptr()))

    assert "displacement_lines_kernel" in run(a, b, ax, cr)
    for i0 in (0, 61, n0 - 6):
        m, c = torch.empty((6, n1), device="cuda"), torch.empty((6, n1), device="cuda")
        assert "displacement_kernel" in run(a[i0:i0 + 6].contiguous(), b[i0:i0 + 6].contiguous(), m, c)
        lo, hi = (0 if i0 == 0 else kl), (6 if i0 == n0 - 6 else 6 - kl)
        for w, part in ((ax, m), (cr, c)):
            assert np.array_equal(w[i0 + lo:i0 + hi].cpu().numpy(), part[lo:hi].cpu().numpy(), equal_nan=True)
    assert (cr > 0).float().mean() > 0.5
