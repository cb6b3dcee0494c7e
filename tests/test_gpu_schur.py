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
