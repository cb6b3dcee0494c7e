"""The pair-space solves and the lists and forces beside them at the edges of their work split:
CG on lubricated polymer replicas (blocks of 32 beads; a lone colloid, several colloids whose
lists hold more than eight pairs, replicas without a near pair), MINRES on suspensions (blocks of
two beads, the wide and the narrow row tiles of the colloid product).  The saddle residual
D^-1 (b - A x) through the operator itself is bounded by the solver's own test, rtol times
|D^-1 b|, with a factor of 10 for the difference of the two residual norms; a replica's
solution alone equals the one in a ragged batch, bit for bit."""
import numpy as np
import pytest

from polystokes_brownian_b200 import configs

pytestmark = pytest.mark.gpu


def _crowd(n_mono, n_coll, seed):
    """Monomers in a dense slab beside a close-packed row of colloids with many near neighbours."""
    rng = np.random.default_rng(seed)
    beta = 0.3
    k = int(np.ceil(n_mono ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n_mono] * (2.2 * beta)
    xm = g + rng.uniform(-0.02, 0.02, size=g.shape) + 6.0
    m = int(np.ceil(n_coll ** (1 / 3)))
    xc = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n_coll] * 2.2 - 8.0
    p = configs.make_params(Nm=n_mono, Nc=n_coll, Npoly=n_mono, Nmono_per_chain=1, beta=beta, kT=1.0, dt=1e-4, mm_HI=1,
                            aa_mode=1, ab_mode=1, lub_on=1, lub_gap=0.5)
    return configs.System("crowd", p, np.vstack([xm, xc])[: n_mono + n_coll])


SYSTEMS = {
    "one_pair": lambda: _crowd(2, 0, 0), "no_pair": lambda: _crowd(1, 1, 1), "block31": lambda: _crowd(31, 0, 2),
    "block33": lambda: _crowd(31, 2, 3), "colloid8": lambda: _crowd(64, 8, 4), "colloid12": lambda: _crowd(95, 12, 5),
}


def _solve(systems, rtol=1e-9):
    import torch
    from polystokes_brownian_b200.engine import Batch
    b = Batch(systems)
    b.stage()
    r = torch.randn(b.nvec, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    x, res = b.solve(r, rtol=rtol, maxit=5000, method=1)
    return b, r, x, res


def _residual_ok(b, r, x, rtol):
    import torch
    d = b.diagonal()
    return (torch.linalg.norm((r - b.matmult(x)) / d) / torch.linalg.norm(r / d)).item() <= 10 * rtol


@pytest.mark.parametrize("name", list(SYSTEMS))
def test_cg(name):
    b, r, x, res = _solve([SYSTEMS[name]()])
    assert res.reason == 2
    assert _residual_ok(b, r, x, 1e-9)
    b.close()


@pytest.mark.parametrize("n", [13, 32, 33, 64, 65, 897])
def test_minres_suspension(n):
    s = configs.suspension(n=n, phi=0.1, seed=n, gap=0.1)
    b, r, x, res = _solve([configs.System(s.name, dict(s.params, lub_on=1), s.x)])
    assert res.reason == 2
    assert _residual_ok(b, r, x, 1e-6)      # PETSc's estimate of the preconditioned residual, another norm
    b.close()


def test_batch_alone():
    import torch
    systems = [SYSTEMS[k]() for k in ("one_pair", "colloid8", "no_pair", "block33", "block31")]
    from polystokes_brownian_b200.engine import Batch
    b, r, x, _ = _solve(systems)
    for k, s in enumerate(systems):
        one = Batch([s])
        one.stage()
        xo, _ = one.solve(b.seg(r, k, "vec").contiguous(), rtol=1e-9, maxit=5000, method=1)
        assert torch.equal(xo, b.seg(x, k, "vec")), k
        one.close()
    b.close()


@pytest.mark.parametrize("which", [0, 2])
@pytest.mark.parametrize("n_mono,n_coll,spacing", [(27, 0, 0.2), (125, 3, 0.05), (300, 0, 0.02)])
def test_lists_ascending_and_complete(which, n_mono, n_coll, spacing):
    """Pair lists against all pairs in numpy, down to piles of more than 32 partners per bead."""
    from polystokes_brownian_b200.engine import Batch
    s = _crowd(n_mono, n_coll, 1)
    s.x[:n_mono] = (s.x[:n_mono] - 6.0) * (spacing / 0.66) + 6.0
    b = Batch([s])
    b.stage()
    pi, pj = (t.cpu().numpy() for t in b.pair_list(which))
    x, beta = s.x, s.params["beta"]
    dr = np.sqrt((x[:, None, 0] - x[None, :, 0]) ** 2 + (x[:, None, 1] - x[None, :, 1]) ** 2
                 + (x[:, None, 2] - x[None, :, 2]) ** 2)
    mono = np.arange(len(x)) < n_mono
    if which == 0:
        rv = [np.float64(np.float32(v)) for v in (0.05 + 2 * beta, 1.5 + beta, 2.5)]
        lim = np.where(mono[:, None] & mono[None], rv[0], np.where(mono[:, None] | mono[None], rv[1], rv[2]))
        hit = dr < lim
    else:
        a = np.where(mono, beta, 1.0)
        hit = (mono[:, None] == mono[None]) & (dr - 2 * a[:, None] < s.params["lub_gap"] * a[:, None])
    i, j = np.nonzero(np.triu(hit, 1))
    assert list(zip(pi.tolist(), pj.tolist())) == list(zip(i.tolist(), j.tolist()))
    b.close()
