"""The arrowhead Schur floor (parallel-ordered Jacobi, Gram over chunks of
monomers) against the oracle: odd and even orders n = 11 Nc up to the dense
limit, monomer counts around the chunk of the largest order (74 monomers at
n = 55), both monomer-colloid scalar families, with and without floored
eigenvalues.  Block-Cholesky noise and saddle diagonal to 1e-12."""
import numpy as np
import pytest

from oracle import psoracle as po
from polystokes_brownian_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nc,chains,ab_mode,spread", [
    (1, (1, 2), 0, 6.0), (1, (11, 20), 1, 9.0), (2, (5, 37), 1, 9.0), (3, (4, 9), 0, 8.0), (4, (1, 93), 1, 10.0),
    (5, (1, 74), 1, 10.0), (5, (3, 25), 0, 10.0), (5, (30, 10), 1, 12.0)])
def test_schur_noise_and_diagonal(Nc, chains, ab_mode, spread):
    import torch
    from polystokes_brownian_b200.engine import Batch
    s = configs.small_mixed(seed=Nc, Nm_chain=chains, Nc=Nc, mm_HI=0, spread=spread, ab_mode=ab_mode)
    o = po.OracleSim(po.default_params(**s.params), s.x.ravel())
    o.stage()
    z = np.random.default_rng(4).normal(size=o.nm3nc11)
    b = Batch([s])
    b.stage()
    w, _ = b.sqrtm(torch.from_numpy(z).cuda())
    wo = o.slip_noise(z)
    assert np.linalg.norm(w.cpu().numpy() - wo) <= 1e-12 * np.linalg.norm(wo)
    do = o.saddle_diag()
    assert np.linalg.norm(b.diagonal().cpu().numpy() - do) <= 1e-12 * np.linalg.norm(do)
    b.close()


# n = 11 .. 55, (chains, spread) so that each order is met with the floor inactive (the iterated
# root, no correction) and active (eigenvectors).  The root's error is at most about
# n eps sqrt(condition) = 55 x 2.2e-16 x sqrt(1000) = 4e-13 of its norm.
@pytest.mark.parametrize("Nc", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("chains,spread,ab_mode,floored", [((2, 3), 60.0, 0, False), ((6, 30), 6.0, 1, True)])
def test_schur_root_with_and_without_floor(Nc, chains, spread, ab_mode, floored):
    import torch
    from polystokes_brownian_b200.engine import Batch
    s = configs.small_mixed(seed=20 + Nc, Nm_chain=chains, Nc=Nc, mm_HI=0, spread=spread, ab_mode=ab_mode)
    o = po.OracleSim(po.default_params(**s.params), s.x.ravel())
    o.stage()
    do = o.saddle_diag()
    n3, n = 3 * (chains[0] * chains[1]), 11 * Nc
    base = np.r_[np.ones(3 * Nc), np.full(3 * Nc, 0.75), np.full(5 * Nc, 1.8)]
    assert (np.abs(do[n3:n3 + n] - base).max() > 0) == floored
    b = Batch([s, s])
    b.stage()
    z = np.random.default_rng(Nc).normal(size=(2, o.nm3nc11))
    w, _ = b.sqrtm(torch.from_numpy(z).cuda().reshape(-1))
    w = w.cpu().numpy().reshape(2, -1)
    for r in range(2):
        wo = o.slip_noise(z[r])
        assert np.linalg.norm(w[r] - wo) <= 1e-12 * np.linalg.norm(wo)
    d = b.diagonal().cpu().numpy().reshape(2, -1)
    assert np.abs(d - do).max() <= 1e-12 * np.abs(do).max()
    b.close()
