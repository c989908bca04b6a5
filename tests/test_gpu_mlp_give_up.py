"""Completion waits that give up, without a fault: with a limit of no polls every wait of the network's kernels
gives up at once, raises the error flag, and then waits for the product in flight, so the kernels end in order.
An inference then writes no output, a training step changes neither weights nor gradients nor loss scale;
with the limit restored the same network goes on as one that never saw it."""
import numpy as np
import pytest
import torch

from render_engine_gb300 import mlp

pytestmark = pytest.mark.gpu


def _inputs(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    P = torch.rand(n, 4, device="cuda", generator=g) * torch.tensor([8.0, 4.0, 3.0, 0.0], device="cuda")
    N = torch.nn.functional.normalize(torch.randn(n, 4, device="cuda", generator=g), dim=1)
    return P.contiguous(), N.contiguous(), torch.rand(n, 4, device="cuda", generator=g)


@pytest.mark.parametrize("n", [1, 128, 700, 128 * 153 + 1, 128 * 700])
def test_inference_that_gives_up_writes_nothing(n):
    P, N, aux = _inputs(n, n)
    net, ref = mlp.Mlp(n_out=3, seed=6), mlp.Mlp(n_out=3, seed=6)
    out, want = torch.full((n, 4), -7.0, device="cuda"), torch.full((n, 4), -7.0, device="cuda")
    torch.cuda.synchronize()
    net.wait_limit(0)
    net.infer_raw(P, N, aux, n, out.data_ptr(), 4)
    assert net.error_flags() == 1
    assert (out == -7).all()
    net.wait_limit(1 << 24)
    net.infer_raw(P, N, aux, n, out.data_ptr(), 4)
    ref.infer_raw(P, N, aux, n, want.data_ptr(), 4)
    assert net.error_flags() == 1 and ref.error_flags() == 0   # the flag stays
    assert torch.equal(out, want) and (out[:, :3] != -7).any()
    net.close()
    ref.close()


@pytest.mark.parametrize("tiles", [1, 3, 152, 160, 500])
def test_training_that_gives_up_changes_nothing(tiles):
    n = 128 * tiles
    P, N, aux = _inputs(n, tiles)
    target = torch.rand(n, 4, device="cuda")
    net, ref = mlp.Mlp(n_out=3, seed=8, lr=1e-2, max_batch=n), mlp.Mlp(n_out=3, seed=8, lr=1e-2, max_batch=n)
    torch.cuda.synchronize()
    for m in (net, ref):
        m.train(P, N, aux, target)
    before = net.weights(), net.gradients(), net.loss_scale()
    net.wait_limit(0)
    net.train(P, N, aux, target)
    net.train(P, N, aux, target)
    assert net.error_flags() == 1
    assert np.array_equal(net.weights(), before[0]) and np.array_equal(net.gradients(), before[1]) and net.loss_scale() == before[2]
    net.wait_limit(1 << 24)
    for m in (net, ref):
        m.train(P, N, aux, target)
    assert ref.error_flags() == 0
    assert np.array_equal(net.weights(), ref.weights()) and np.array_equal(net.gradients(), ref.gradients())
    assert net.loss_scale() == ref.loss_scale()
    net.close()
    ref.close()


def test_wait_limit_range():
    net = mlp.Mlp(n_out=1)
    with pytest.raises(Exception):
        net.wait_limit((1 << 24) + 1)
    net.close()
