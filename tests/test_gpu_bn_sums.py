"""Sums of the normalisation's passes: blocks of one row of channels and of many, rows that do not share out evenly."""
import pytest
import torch

from nectarml_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,c", [(131072, 256), (131079, 256), (524288 + 3, 64), (16385, 2048), (131071, 256), (70001, 24), (9001, 2040), (5000, 128), (40003, 8)])
def test_statistics_and_gradients(rows, c):
    gen = torch.Generator(device="cuda").manual_seed(rows + c)
    x = (torch.randn(rows, c, device="cuda", generator=gen) + 0.5).half()
    dy = torch.randn(rows, c, device="cuda", generator=gen).half()
    x[-1], dy[-1] = 100.0, 100.0  # (the last row, of a ragged share or not, is seen in every sum: 1.9e-4 of the mean and 100 of a gradient at least)
    gamma, beta = torch.rand(c, device="cuda", generator=gen) + 0.5, torch.randn(c, device="cuda", generator=gen)
    ws, n = ops.Workspace(), ops._native
    y, _, mean, rstd, _ = n.bn_forward(x, None, gamma, beta, 1, 0.0, 1e-5, None, False, ws)
    mu, var = x.double().mean(0), x.double().var(0, unbiased=False)
    # fp32 sums of at most a few thousand terms a thread, rounded at random: errors of sqrt(terms) * 2^-24 of the terms' size and well below 1e-5
    assert ((mean.double() - mu).abs() <= 1e-5).all()
    assert ((rstd.double() * (var + 1e-5).sqrt() - 1).abs() <= 1e-5).all()
    dgamma, dbeta = torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    n.bn_backward(dy, None, False, None, x, gamma, beta, mean, rstd, 1, 0.0, False, dgamma, dbeta, ws)
    dz = dy.double() * (y > 0)
    xhat = (x.double() - mean.double()) * rstd.double()
    bound = 1e-5 * rows ** 0.5 * 10  # (the sums are of the size of sqrt(rows))
    assert ((dbeta.double() - dz.sum(0)).abs() <= bound).all()
    assert ((dgamma.double() - (dz * xhat).sum(0)).abs() <= bound).all()
