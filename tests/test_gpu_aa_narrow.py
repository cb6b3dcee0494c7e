"""Monomer tile pairs of edge 64 in launches of many (two warps per tile pair, bands one after
the other, padding left out) against the same replica alone (a block of all bands, checked
against 64-bit sums elsewhere): products and square roots bit for bit, with replicas of one to
several tiles at the edges of warps, tiles and the step rotation, FP64 and FP32, both pair
scalar families, chains that skip their own pairs, and probes beside them."""
import numpy as np
import pytest

from polystokes_brownian_b200 import _capi, configs

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 15, 16, 17, 31, 32, 33, 34, 63, 64, 65, 66, 97, 128, 129, 200]


def _system(n, mode, per_chain, Nc):
    rng = np.random.default_rng([n, Nc])
    x = rng.uniform(-1.5, 1.5, size=(n, 3)) * n ** (1.0 / 3.0)
    c = rng.uniform(-2.0, 2.0, size=(Nc, 3)) + np.array([[40.0, 0.0, 0.0], [0.0, 40.0, 0.0]])[:Nc]
    p = configs.make_params(Nm=n, Nc=Nc, Npoly=-(-n // per_chain), Nmono_per_chain=per_chain, beta=0.5, mm_HI=1,
                            chain_HI=int(per_chain > 1), aa_mode=mode, ab_mode=mode)
    return configs.System("narrow", p, np.vstack([x, c]))


def _input(s, k):
    import torch
    n = 3 * s.params["Nm"] + 11 * s.params["Nc"]
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(k))


def _batch(systems, inputs, precision):
    import torch
    from polystokes_brownian_b200.engine import Batch
    b = Batch(systems, precision=precision)
    b.stage()
    u = torch.cat(inputs)
    y = b.mobility_apply(u)
    w, _ = b.sqrtm(u, kmax=9, tol=1e-15)
    out = [(b.seg(y, r, "top").clone(), b.seg(w, r, "top").clone()) for r in range(len(systems))]
    b.close()
    return out


@pytest.mark.parametrize("precision", [_capi.PS_PREC_FP64, _capi.PS_PREC_MIXED])
@pytest.mark.parametrize("mode,per_chain,Nc", [(1, 1, 0), (0, 1, 0), (1, 7, 0), (1, 1, 2)])
def test_alone_and_in_a_launch_of_many(precision, mode, per_chain, Nc):
    import torch
    sizes = SIZES if per_chain == 1 else [per_chain * k for k in (1, 2, 4, 5, 9, 10, 18, 19, 28)]
    systems = [_system(n, mode, per_chain, Nc) for n in sizes]
    inputs = [_input(s, k) for k, s in enumerate(systems)]
    tiles = sum((t := -(-n // 64)) * (t + 1) // 2 for n in sizes)
    copies = (2400 if Nc else 600) // tiles + 1              # above the line of either precision
    many = _batch(systems * copies, inputs * copies, precision)
    for k, s in enumerate(systems):
        y, w = _batch([s], [inputs[k]], precision)[0]
        assert torch.isfinite(y).all() and torch.isfinite(w).all()
        for r in (k, k + len(systems) * (copies - 1)):
            assert torch.equal(many[r][0], y), (s.params["Nm"], r)
            assert torch.equal(many[r][1], w), (s.params["Nm"], r)
