"""The training step's and the inference's persistent tiles.  Training: the gradient of n samples equals the sum of the gradients of
its parts, whatever the number of 128-sample tiles per CTA (none to four, whole and partial rounds)
and of outputs.  With the learning rate at zero the weights stay put; the loss gradient is scaled by
1 / (n n_out), so a part of n / k samples weighs 1 / k.  Both sides are FP32 sums of the same bf16
products in other orders: at most 2^-23 x (terms per sum, in order) of the sum of magnitudes, and the
scaling by a power of two is exact (parts are a power of two of each other)."""
import numpy as np
import pytest
import torch

from render_engine_gb300 import mlp

pytestmark = pytest.mark.gpu


def _inputs(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    P = torch.rand(n, 4, device="cuda", generator=g) * torch.tensor([8.0, 4.0, 3.0, 0.0], device="cuda")
    N = torch.nn.functional.normalize(torch.randn(n, 3, device="cuda", generator=g), dim=1)
    N = torch.cat([N, torch.zeros(n, 1, device="cuda")], 1).contiguous()
    return P.contiguous(), N, torch.rand(n, 4, device="cuda", generator=g)


@pytest.mark.parametrize("tiles,n_out", [(2, 1), (2, 5), (4, 16), (16, 4), (152, 3), (154, 3), (304, 3), (306, 2), (608, 3), (610, 3)])
def test_gradient_is_the_sum_of_its_halves(tiles, n_out):
    n = 128 * tiles
    P, N, aux = _inputs(n, tiles)
    target = torch.rand(n, n_out, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    net = mlp.Mlp(n_out=n_out, seed=9, lr=0.0, max_batch=n)
    idx = torch.arange(n, dtype=torch.int32, device="cuda")
    got = []
    for part in (idx, idx[: n // 2].contiguous(), idx[n // 2:].contiguous()):
        net.train(P, N, aux, target, idx=part)
        got.append(net.gradients().astype(np.float64))
    assert net.error_flags() == 0
    whole, halves = got[0], 0.5 * (got[1] + got[2])
    scale = np.sqrt((got[1] ** 2 + got[2] ** 2).mean())
    assert scale > 0
    # bf16 rounding of the scaled gradients is the same for both (a power of two apart), so what is left
    # is FP32 summation: n terms, errors growing as their square root
    assert np.abs(whole - halves).max() <= 64 * 2.0 ** -24 * np.sqrt(n) * max(scale, np.abs(whole).max())
    net.close()


@pytest.mark.parametrize("n", [1, 127, 129, 128 * 152, 128 * 153 + 1, 128 * 305, 128 * 608 - 5, 128 * 611 + 77, 128 * 1000])
@pytest.mark.parametrize("n_out", [1, 3, 16])
def test_outputs_do_not_depend_on_the_batch(n, n_out):
    """A query's outputs are its own: the same bits in a batch of one tile and in one of many
    tiles per CTA, and nothing beyond the batch or its outputs is written."""
    P, N, aux = _inputs(n, n)
    net = mlp.Mlp(n_out=n_out, seed=4)
    whole = torch.full((n + 1, n_out + 1), -7.0, device="cuda")
    torch.cuda.synchronize()
    net.infer_raw(P, N, aux, n, whole.data_ptr(), n_out + 1)
    assert net.error_flags() == 0
    assert (whole[n] == -7).all() and (whole[:, n_out] == -7).all()
    for at in sorted({0, max(0, n - 128), 128 * (n // 256)}):
        m = min(128, n - at)
        part = torch.zeros(m, n_out, device="cuda")
        p, q, x = P[at:at + m].contiguous(), N[at:at + m].contiguous(), aux[at:at + m].contiguous()
        torch.cuda.synchronize()
        net.infer(p, q, x, part)
        assert net.error_flags() == 0
        assert torch.equal(part, whole[at:at + m, :n_out])
    net.close()
