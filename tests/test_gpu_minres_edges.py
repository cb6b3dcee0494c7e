"""MINRES with its scalars recomputed from sub-block sums: saddle vectors around
the sub-blocks of 256 and table blocks of 1024 entries.  Monomer systems, where
the saddle system has the closed solution F = -b_bot, U = M F - b_top: at rtol
1e-13 the error is bounded by rtol times the condition of the preconditioned
system (below 1e3 for these dilute clouds), so 1e-10.  A ragged batch solves each
replica exactly as alone, and an iteration cap is reported as -3."""
import numpy as np
import pytest

from polystokes_brownian_b200 import configs

pytestmark = pytest.mark.gpu


def _system(n):
    x = np.random.default_rng(n).uniform(-3.0, 3.0, size=(n, 3)) * n ** (1.0 / 3.0)
    p = configs.make_params(Nm=n, Nc=0, Npoly=n, Nmono_per_chain=1, beta=0.5, mm_HI=1, aa_mode=1, ab_mode=1)
    return configs.System("minres", p, x)


def _rhs(n, seed):
    import torch
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))


@pytest.mark.parametrize("n", [1, 42, 43, 85, 86, 170, 171, 683])
def test_solution(n):
    import torch
    from polystokes_brownian_b200.engine import Batch
    b = Batch([_system(n)])
    b.stage()
    r = _rhs(b.nvec, n)
    x, res = b.solve(r, rtol=1e-13, maxit=5000)
    F = -r[b.ntop:]
    want = torch.cat([F, b.mobility_apply(F.contiguous()) - r[:b.ntop]])
    assert res.reason == 2
    assert (torch.linalg.norm(x - want) / torch.linalg.norm(want)).item() < 1e-10
    b.close()


def test_batch_alone_and_cap():
    import torch
    from polystokes_brownian_b200.engine import Batch
    systems = [_system(n) for n in (1, 43, 171, 400)]
    big = Batch(systems)
    big.stage()
    r = _rhs(big.nvec, 3)
    x, res = big.solve(r, rtol=1e-10)
    assert res.reason == 2
    for k, s in enumerate(systems):
        one = Batch([s])
        one.stage()
        xo, _ = one.solve(big.seg(r, k, "vec").contiguous(), rtol=1e-10)
        assert torch.equal(xo, big.seg(x, k, "vec")), k
        one.close()
    for cap in (1, 8, 9):
        _, res = big.solve(r, rtol=1e-14, maxit=cap)
        assert res.reason == -3 and res.iters_max == cap
    _, res = big.solve(r, rtol=1e-10)
    assert res.reason == 2
    big.close()
