"""The MLP kernel on CTA pairs (256-row tiles, 128 rows per CTA) at the edges of its tiles: one row, one CTA's rows, one
pair's and one more of each, every pair of SMs busy once and once more, a row list through the gated renderer.

Tolerance: as in test_gpu_surrogate.py, a PyTorch forward with the same BF16 roundings; hardware tanh (2^-11) and FP32
summation order flip single BF16 roundings, 2 % of the output scale at most and 0.2 % in the mean. A row's outputs do not
depend on where it lies in the launch, so every size is also compared bit for bit with one large launch."""
import os

import numpy as np
import pytest

from sirius_b200 import abi

pytestmark = pytest.mark.gpu
WEIGHTS = os.path.join(os.path.dirname(abi.__file__), "data", "surrogate_kerr.npy")


def reference(torch, p, x):
    bf = lambda t: t.to(torch.bfloat16).float()  # noqa: E731
    p = torch.from_numpy(p).cuda()
    hi = bf(x)
    off, h = 0, None
    for k, (o, i) in enumerate(((256, 5), (256, 256), (256, 256), (256, 256), (4, 256))):
        w, b = bf(p[off:off + o * i].reshape(o, i)), p[off + o * i:off + o * i + o]
        off += o * i + o
        h = hi @ w.T + bf(x - hi) @ w.T + b if k == 0 else h @ w.T + b
        if k < 4:
            h = bf(h * torch.sigmoid(h))
    return h


@pytest.fixture(scope="module")
def full(engine):
    import torch
    p = np.load(WEIGHTS).astype(np.float32).ravel()
    engine.surrogate_load(p)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    n = 148 * 256 + 129
    x = (torch.rand(n, 5, device="cuda", generator=g) * 2 - 1).contiguous()
    y = torch.full((n, 4), float("nan"), device="cuda")
    engine.surrogate_infer(x.data_ptr(), n, y.data_ptr())
    return torch, p, x, y


def test_forward_against_reference(full):
    torch, p, x, y = full
    torch.backends.cuda.matmul.allow_tf32 = False
    ref = reference(torch, p, x)
    err = (y - ref).abs().amax(0) / ref.abs().amax(0)
    mean = (y - ref).abs().mean(0) / ref.abs().amax(0)
    assert torch.isfinite(y).all() and (err < 2e-2).all() and (mean < 2e-3).all(), (err, mean)


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 255, 256, 257, 511, 513, 74 * 256 - 1, 74 * 256 + 1, 148 * 256])
def test_sizes_equal_one_launch(engine, full, n):
    torch, _, x, y = full
    out = torch.full((n + 2, 4), float("nan"), device="cuda")
    for first in (0, 100):
        part = x[first:first + n].contiguous()
        engine.surrogate_infer(part.data_ptr(), n, out.data_ptr())
        assert torch.equal(out[:n], y[first:first + n])
        assert torch.isnan(out[n:]).all()


def test_launches_of_any_size_in_turn(engine, full):
    """The tile counter, which the kernel itself leaves at zero, serves launches of other sizes in any order."""
    torch, _, x, y = full
    for n in (300, 148 * 256, 1, 4000, 257):
        out = torch.empty(n, 4, device="cuda")
        engine.surrogate_infer(x.data_ptr(), n, out.data_ptr())
        assert torch.equal(out, y[:n])
