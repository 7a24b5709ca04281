"""The network's kernels at the sizes where their splits change: the forward
GEMM's columns over CTAs (few row tiles), the backward launch's three parts
(input gradient, weight gradient split along the rows, bias sums), the loss,
and the transposed weights of a network with more layers
than one launch takes. Oracle: oracle/mlp_oracle.py (same BF16 roundings,
float64 sums)."""

import numpy as np
import pytest

from gold import rel_l2
from oracle import mlp_oracle as MO


@pytest.fixture(scope="module")
def gpu():
    torch = pytest.importorskip("torch")
    from usx import capi
    ctx = capi.Context(0, stream=0)
    yield torch, capi, ctx
    ctx.close()


def _net(capi, ctx, dims, seed):
    rng = np.random.default_rng(seed)
    mlp = capi.Mlp(ctx, dims, seed=seed)
    p = mlp.get_params()
    for _, b in mlp.layers(p):
        b[:] = rng.standard_normal(b.size).astype(np.float32) * 0.1
    mlp.set_params(p)
    return mlp, p, rng


@pytest.mark.gpu
@pytest.mark.parametrize("dims,rows", [
    ((256, 256), 38 * 128), ((256, 256), 39 * 128), ((128, 256), 76 * 128), ((256, 256), 77 * 128),
    ((256, 128), 76 * 128), ((256, 128), 77 * 128), ((64 * 2, 256), 128)])
def test_forward_at_every_column_split(gpu, dims, rows):
    """256 columns as 4 x 64, 2 x 128 and whole, 128 as 2 x 64 and whole: FP32
    sums of at most 256 products (1e-5 of the largest, as between two GEMMs)."""
    torch, capi, ctx = gpu
    mlp, p, rng = _net(capi, ctx, dims, rows)
    x = rng.standard_normal((rows, dims[0])).astype(np.float32)
    dx, dy = torch.from_numpy(x).cuda(), torch.full((rows, dims[-1]), float("nan"), device="cuda")
    mlp.forward(dx.data_ptr(), rows, dy.data_ptr())
    ctx.synchronize()
    want, _ = MO.forward(p, dims, x, quantize=True)
    assert np.abs(dy.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("dims,rows", [((128, 128), 128), ((256, 128), 5 * 128), ((256, 384), 11 * 128),
                                       ((128, 128), 320 * 128), ((256, 128, 256), 3 * 128)])
def test_training_step_at_every_row_split(gpu, dims, rows):
    """Loss and gradients. One layer: the loss is an FP32 sum (1e-5); the output
    gradient's BF16 rounding goes the other way for the few in 10^4 outputs
    within FP32 rounding of a tie, 2^-8 each (3e-4). Two layers: hidden
    activations round too (3e-3)."""
    torch, capi, ctx = gpu
    mlp, p, rng = _net(capi, ctx, dims, rows + 1)
    x = rng.standard_normal((rows, dims[0])).astype(np.float32)
    t = rng.standard_normal((rows, dims[-1])).astype(np.float32)
    dx, dt = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    loss, grad = mlp.train_step(dx.data_ptr(), dt.data_ptr(), None, rows, 0.0, True, True)
    want_loss, want = MO.backward(p, dims, x, t, None, quantize=True)
    tol = 3e-4 if len(dims) == 2 else 3e-3
    assert abs(loss - want_loss) <= (1e-5 if len(dims) == 2 else 1e-3) * want_loss
    for (w, b), (ww, wb) in zip(MO.layers(grad, dims), MO.layers(want, dims)):
        assert rel_l2(w, ww) < tol and rel_l2(b, wb) < tol


@pytest.mark.gpu
def test_weights_of_a_deep_network_are_all_transposed(gpu):
    """Eighteen layers, two of the transposing launches: against the path that
    reads the weights as stored (activations round to BF16 at each layer: 1e-2)."""
    torch, capi, ctx = gpu
    dims = (128,) * 19
    mlp, _, rng = _net(capi, ctx, dims, 9)
    dx = torch.from_numpy(rng.standard_normal((256, 128)).astype(np.float32)).cuda()
    out = []
    for path in (capi.Mlp.GEMM_AUTO, capi.Mlp.GEMM_MMA_SYNC):
        mlp.set_gemm_path(path)
        dy = torch.full((256, 128), float("nan"), device="cuda")
        mlp.forward(dx.data_ptr(), 256, dy.data_ptr())
        ctx.synchronize()
        out.append(dy.cpu().numpy())
    assert rel_l2(out[0], out[1]) < 1e-2
