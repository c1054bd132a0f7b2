"""Training on a driver that encodes no tensor maps (the library linked with that query failing): the forward kernel's
weights and every GEMM operand go through registers.

Tolerance: both forms give the tensor core the same operands in the same order, so the network's outputs and the loss are
those of the form with tensor maps up to the order of FP32 atomic sums (2e-6), and a weight's gradient up to that of its 64
partial sums (1e-5 of the layer's largest)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import fake_cuda  # noqa: E402

from sirius_b200 import abi  # noqa: E402
from sirius_b200.engine import Engine, load_library  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plain(tmp_path_factory):
    lib = fake_cuda.link_without_tensor_maps(str(tmp_path_factory.mktemp("no_maps")))
    if lib is None:
        pytest.skip("the library's objects are not here")
    e = Engine(0, lib=load_library(lib))
    yield e
    e.close()


@pytest.mark.parametrize("batch", [128, 640, 74 * 256 + 128])
def test_forward_and_gradient_equal_the_mapped_form(engine, plain, batch):
    import torch

    from sirius_b200.surrogate_train import init_params
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    x = torch.rand(batch, 5, device="cuda", generator=g) * 2 - 1
    hit = (torch.hypot(x[:, 2], x[:, 3]) > 0.35).float()
    t = torch.stack([hit, hit * 0.5 * x[:, 2], hit * (0.6 + 0.3 * x[:, 3]), 0.1 * x[:, 4]], 1).contiguous()
    w = torch.ones(batch, device="cuda")
    p = init_params(np.random.default_rng(7))
    got = []
    for e in (engine, plain):
        e.train_init(p, abi.train_config(batch=batch))
        parts, grad = e.train_gradient(x.data_ptr(), t.data_ptr(), w.data_ptr(), batch)
        ragged = e.train_evaluate(x.data_ptr(), t.data_ptr(), w.data_ptr(), batch - 1)
        e.train_steps(x.data_ptr(), t.data_ptr(), w.data_ptr(), batch, 2)
        got.append((parts, grad, ragged, e.train_params()[1]))
    np.testing.assert_allclose(got[1][0], got[0][0], rtol=2e-6)
    np.testing.assert_allclose(got[1][2], got[0][2], rtol=2e-6)
    assert got[0][3] == got[1][3] == 2
    off = 0
    for o, i in ((256, 5), (256, 256), (256, 256), (256, 256), (4, 256)):
        for n in (o * i, o):
            a, b = (v[1][off:off + n] for v in got)
            assert np.abs(b - a).max() <= 1e-5 * np.abs(a).max()
            off += n
