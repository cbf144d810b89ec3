"""Sizes where the network kernels change shape.  The tensor-core inference
takes one tile of 128 points per SM, then two: a point's value may not depend
on the others, so any batch must give, bit for bit, what small batches of the
same points give.  The training GEMMs change tiles with the batch: the gradient
against the float64 oracle at batches around their edges (the tolerance of
the existing gradient test, derived from fp32 accumulation)."""
import numpy as np
import pytest

from oracle import mlp_ref
from isosurface_gb300.surrogate import Surrogate

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("tiles,extra", [(1, -1), (1, 1), (2, 0), ("sms", 0), ("sms", 1), ("2sms", 5), ("5sms", 77)])
def test_values_do_not_depend_on_the_batch(ctx, tiles, extra):
    sms = _sms()
    n = 128 * {"sms": sms, "2sms": 2 * sms, "5sms": 5 * sms}.get(tiles, tiles) + extra
    net = Surrogate(ctx, seed=8)
    x = np.random.default_rng(n).uniform(-1, 1, (n, 3)).astype(np.float32)
    whole = net.forward(x, bf16=True)
    for lo in range(0, n, 4096):
        if lo % 20480 == 0 or lo + 4096 >= n:
            part = net.forward(x[lo:lo + 4096], bf16=True)
            assert np.array_equal(part.view(np.uint32), whole[lo:lo + 4096].view(np.uint32)), lo
    net.close()


@pytest.mark.parametrize("n", [1, 63, 65, 129, 1000, 9729])
def test_gradient_at_tile_edges(ctx, n):
    net = Surrogate(ctx, seed=9)
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    y0, _, _ = mlp_ref.forward(net.params, x)
    t = (y0 + rng.choice([-0.05, 0.05], n)).astype(np.float32)  # no residual near zero: the L1 sign is not in doubt
    loss, g = net.loss_grad(x, t, clamp_d=10.0)
    wl, wg = mlp_ref.loss_grad(net.params, x, t, 10.0)
    assert abs(loss - wl) <= 1e-5 + 1e-4 * abs(wl)
    assert np.linalg.norm(g - wg) <= 1e-4 * np.linalg.norm(wg)
    net.close()
