"""The fused training forward pass (CTA pairs, 256-row tiles) at the edges of its tiles: batches of one CTA's rows, an odd
number of them, one tile for every pair of SMs and one more, and evaluations of ragged row counts.

Tolerance: the loss parts are FP32 sums of per-row values that the inference kernel gives bit for bit; summation order and
the hardware exponential of the loss (2^-21) leave 1e-5, and two sums of the same values 2e-6."""
import numpy as np
import pytest

from sirius_b200 import abi

pytestmark = pytest.mark.gpu


def rows(torch, n, seed=2):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.rand(n, 5, device="cuda", generator=g) * 2 - 1
    hit = (torch.hypot(x[:, 2], x[:, 3]) > 0.35).float()
    t = torch.stack([hit, hit * 0.5 * x[:, 2], hit * (0.6 + 0.3 * x[:, 3]), 0.1 * x[:, 4]], 1).contiguous()
    return x.contiguous(), t, torch.ones(n, device="cuda")


@pytest.mark.parametrize("batch", [128, 384, 74 * 256, 74 * 256 + 128])
def test_batches_and_ragged_evaluations(engine, batch):
    import torch

    from sirius_b200.surrogate_train import init_params
    engine.configure(abi.default_config())
    p = init_params(np.random.default_rng(3))
    engine.train_init(p, abi.train_config(batch=batch))
    x, t, w = rows(torch, batch)
    whole = engine.train_evaluate(x.data_ptr(), t.data_ptr(), w.data_ptr(), batch)
    parts, grad = engine.train_gradient(x.data_ptr(), t.data_ptr(), w.data_ptr(), batch)
    np.testing.assert_allclose(parts, whole, rtol=2e-6)
    assert np.isfinite(grad).all() and np.count_nonzero(grad) > 0.9 * grad.size
    # the network's own inference kernel on the same rows gives the same binary cross-entropy
    engine.surrogate_load(p)
    for n in (1, 127, 129, batch):
        n = min(n, batch)
        y = torch.empty(n, 4, device="cuda")
        engine.surrogate_infer(x.data_ptr(), n, y.data_ptr())
        bce = torch.nn.functional.binary_cross_entropy_with_logits(y[:, 0], t[:n, 0]).item()
        higher = ((y[:, 3] - t[:n, 3]) ** 2).mean().item()
        ev = engine.train_evaluate(x.data_ptr(), t.data_ptr(), w.data_ptr(), n)
        np.testing.assert_allclose([ev[0], ev[3]], [bce, higher], rtol=1e-5, atol=1e-9)
