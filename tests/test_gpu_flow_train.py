"""The coupling flow's training step on batches that end inside a tile, at dimension counts that use every
slot and part of the dims: the same loss and gradient as a batch of whole tiles whose extra points weigh
nothing. Both divide by their own point count, so each back-propagated number is rounded to bf16 (relative
2^-9) at another scale: at most 2 * 2^-9 per product's operands and three layers of products, 1.2 % of
a matrix's norm; the losses, fp32 sums of the same terms, differ by less than 2^-24 per addition of
the terms' magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,count", [(2, 129), (3, 127), (5, 300), (7, 130), (8, 257)])
def test_ragged_batch_equals_zero_weight_padding(ctx, dim, count):
    g = np.random.default_rng(100 + dim)
    fl = ctx.flow(dim, seed=dim)
    fl.set_params(fl.params() + 0.05 * g.standard_normal(fl.params().shape).astype(np.float32))
    whole = -(-count // 128) * 128 + 128
    x, w = g.random((whole, dim)), g.random(whole) * 2.0
    w[count:] = 0.0
    loss, grad = fl.gradient(x[:count], w[:count])
    loss_p, grad_p = fl.gradient(x, w)
    terms = (w * np.abs(fl.density(x)[1])).sum()
    assert abs(loss * count - loss_p * whole) <= whole * 2.0 ** -24 * terms + 1e-6
    a, b = grad.reshape(-1, grad.shape[-1] ** 2) * count, grad_p.reshape(-1, grad.shape[-1] ** 2) * whole
    for m, (u, v) in enumerate(zip(a, b)):
        assert np.linalg.norm(u - v) <= 0.012 * np.linalg.norm(v) + 1e-12, m
