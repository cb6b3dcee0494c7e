"""The two row tiles of the colloid far field's own kernel add in the same order: a
suspension's product is the same bit for bit whether its context takes the narrow or the
wide tiles, which depends on the blocks of the whole launch.  Alone, twice, and beside small
ones, at the edges of the tiles and at the sizes where a context changes over (929 colloids
alone, 768 by the batch, 1025 back again)."""
import numpy as np
import pytest

from polystokes_brownian_b200 import configs

pytestmark = pytest.mark.gpu

PARAMS = configs.suspension(n=2, phi=0.01, seed=0).params


def _suspension(n, seed=0):
    k = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 3.0
    x = g + np.random.default_rng([seed, n]).uniform(-0.4, 0.4, size=g.shape)
    return configs.System("bb", dict(PARAMS, Nc=n), x)


def _apply(systems, inputs):
    import torch
    from polystokes_brownian_b200.engine import Batch
    b = Batch(systems)
    b.stage()
    y = b.mobility_apply(torch.cat(inputs))
    out = [b.seg(y, r, "top").clone() for r in range(len(systems))]
    b.close()
    return out


def _input(n, seed):
    import torch
    return torch.randn(11 * n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))


@pytest.mark.parametrize("n", [2, 31, 33, 300, 768, 896, 897, 928, 929, 960, 1024, 1025])
def test_alone_and_in_batches(n):
    import torch
    s, u = _suspension(n), _input(n, n)
    alone = _apply([s], [u])[0]
    twice = _apply([s, s], [u, u])
    mixed = _apply([_suspension(60), s] + [_suspension(2)] * 3, [_input(60, 1), u] + [_input(2, 2)] * 3)
    assert torch.isfinite(alone).all()
    assert torch.equal(alone, twice[0]) and torch.equal(alone, twice[1]) and torch.equal(alone, mixed[1])
