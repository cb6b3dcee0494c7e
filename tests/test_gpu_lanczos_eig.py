"""The eigensolver of the Lanczos root (Sturm bisection and twisted factorisations,
QL where eigenvalues are too close): M^(1/2) z on systems whose Krylov space is
exhausted within the basis cap, so that the root is exact, against the dense
root.  Orders at the edges of the solver's teams and warps (3 to 63), repeated
eigenvalues (far-apart copies of one dimer, nearly equal to 1e-4 ... 1e-9) and a
single bead.  The projected root is backward stable: the error is bounded by
some eps |M| / sqrt(lambda_min), below 1e-10 here."""
import numpy as np
import pytest

from oracle import psoracle as po
from polystokes_brownian_b200 import configs

pytestmark = pytest.mark.gpu


def _system(x):
    n = len(x)
    p = configs.make_params(Nm=n, Nc=0, Npoly=n, Nmono_per_chain=1, beta=0.5, mm_HI=1, aa_mode=1, ab_mode=1)
    return configs.System("eig", p, np.asarray(x, dtype=float))


def _cloud(n):
    return np.random.default_rng(n).uniform(-1.5, 1.5, size=(n, 3)) * n ** (1.0 / 3.0)


def _dimers(k, gap):
    return np.concatenate([[[i * gap, 0.0, 0.0], [i * gap, 1.2, 0.3]] for i in range(k)])


@pytest.mark.parametrize("x", [_cloud(n) for n in (1, 2, 3, 8, 10, 11, 13, 21)] + [_dimers(2, 1e4), _dimers(3, 1e6),
                                                                                     _dimers(4, 1e9)],
                         ids=[f"cloud{n}" for n in (1, 2, 3, 8, 10, 11, 13, 21)] + ["dimers4", "dimers6", "dimers9"])
def test_exhausted_krylov_root(x):
    import torch
    from polystokes_brownian_b200.engine import Batch
    s = _system(x)
    o = po.OracleSim(po.default_params(**s.params), s.x.ravel())
    o.stage()
    M = o.dense_mobility()
    z = np.random.default_rng(1).normal(size=M.shape[0])
    b = Batch([s])
    b.stage()
    w, _ = b.sqrtm(torch.from_numpy(z).cuda(), kmax=64, tol=1e-15)
    ref = po.sqrtm_eig(M, z)
    assert np.linalg.norm(w.cpu().numpy() - ref) <= 1e-10 * np.linalg.norm(ref)
    b.close()


@pytest.mark.parametrize("n", [85, 86, 171, 341, 342, 683])
def test_root_at_sub_block_edges(n):
    """Vector lengths around the sub-blocks of 256 and table blocks of 1024 entries.  A dilute
    cloud is well conditioned (eigenvalues within a factor of a few), so 64 vectors reach
    rounding: 1e-11 allows for the growth of the basis's rounding errors."""
    import torch
    from polystokes_brownian_b200.engine import Batch
    s = _system(np.random.default_rng(n).uniform(-1.0, 1.0, size=(n, 3)) * 40.0 * n ** (1.0 / 3.0))
    o = po.OracleSim(po.default_params(**s.params), s.x.ravel())
    o.stage()
    M = o.dense_mobility()
    z = np.random.default_rng(1).normal(size=M.shape[0])
    lam, Q = np.linalg.eigh(M)
    ref = (Q * np.sqrt(lam)) @ (Q.T @ z)
    b = Batch([s])
    b.stage()
    w, _ = b.sqrtm(torch.from_numpy(z).cuda(), kmax=64, tol=1e-15)
    assert np.linalg.norm(w.cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)
    b.close()
