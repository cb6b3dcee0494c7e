"""Replicas that stop by themselves inside a launch of many blocks: the Lanczos root on an
invariant subspace (beads so far apart that M is beta^-1 times the identity to 1e-12: the
root is known, sqrt(1/beta) z, within the breakdown threshold of 1e-12), and the pair-space
CG on colloids in near contact, whose far field is not positive definite, which MINRES then
finishes.  Repeats agree bit for bit, and an ordinary replica beside them is the same as alone."""
import numpy as np
import pytest

from polystokes_brownian_b200 import configs

pytestmark = pytest.mark.gpu


def _params(n, **kw):
    return configs.make_params(Nm=n, Nc=0, Npoly=n, Nmono_per_chain=1, beta=0.5, mm_HI=1, aa_mode=1, ab_mode=1, **kw)


@pytest.mark.parametrize("n", [2, 86, 700])
def test_lanczos_stops_on_an_invariant_subspace(n):
    import torch
    from polystokes_brownian_b200.engine import Batch
    x = np.random.default_rng(0).uniform(-3.0, 3.0, size=(300, 3)) * 7.0
    plain = configs.System("plain", _params(300), x)
    k = int(np.ceil(n ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 1e16
    b = Batch([plain, configs.System("apart", _params(n), grid)])
    b.stage()
    z = torch.randn(b.ntop, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    w, _ = b.sqrtm(z, kmax=40, tol=1e-12)
    zs, ws = b.seg(z, 1, "top"), b.seg(w, 1, "top")
    assert (torch.linalg.norm(ws - 2.0 ** 0.5 * zs) / torch.linalg.norm(ws)).item() <= 1e-12
    for _ in range(20):
        assert torch.equal(b.sqrtm(z, kmax=40, tol=1e-12)[0], w)
    one = Batch([plain])
    one.stage()
    assert torch.equal(one.sqrtm(b.seg(z, 0, "top").contiguous(), kmax=40, tol=1e-12)[0], b.seg(w, 0, "top"))
    b.close()
    one.close()


@pytest.mark.parametrize("gap", [0.001, 0.05])
def test_cg_stops_on_an_indefinite_far_field(gap):
    import torch
    from polystokes_brownian_b200.engine import Batch
    c = np.stack(np.meshgrid(np.arange(3), np.arange(2), np.arange(2), indexing="ij"), -1).reshape(-1, 3) * (2.0 + gap)
    p = configs.make_params(Nm=40, Nc=12, Npoly=40, Nmono_per_chain=1, beta=0.3, kT=1.0, dt=1e-4, mm_HI=1, aa_mode=1,
                            ab_mode=1, lub_on=1, lub_gap=0.5)
    m = np.random.default_rng(2).uniform(-4.0, 4.0, size=(40, 3)) + 14.0
    b = Batch([configs.System("contact", p, np.vstack([m, c]))])
    b.stage()
    r = torch.randn(b.nvec, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(7))
    x, res = b.solve(r, rtol=1e-9, maxit=5000, method=1)
    assert res.reason == 2
    d = b.diagonal()
    # both solvers' tests are rtol in a preconditioned norm; 1e-6 allows for its condition near contact
    assert (torch.linalg.norm((r - b.matmult(x)) / d) / torch.linalg.norm(r / d)).item() <= 1e-6
    print("gap", gap, "iterations", res.iters_max)
    for _ in range(5):
        y, again = b.solve(r, rtol=1e-9, maxit=5000, method=1)
        assert again.iters_max == res.iters_max and torch.equal(x, y)
    b.close()
