"""The Gram matrix of the arrowhead Schur floor over more than one chunk of monomers: a chunk
holds 283 monomers for one and two colloids, 169 for three, 120 for four and five (rows of
schur_ld(11 Nc) doubles in a buffer of 20480).  One less, as many and one more than a chunk,
and more than two, against the oracle's block-Cholesky noise and saddle diagonal to 1e-12, the
bound of the single chunk."""
import numpy as np
import pytest

from oracle import psoracle as po
from polystokes_brownian_b200 import configs

pytestmark = pytest.mark.gpu

CHUNK = {1: 283, 2: 283, 3: 169, 4: 120, 5: 120}


@pytest.mark.parametrize("Nc", sorted(CHUNK))
@pytest.mark.parametrize("extra", ["less", "as many", "more", "three"])
def test_chunk_edges(Nc, extra):
    import torch
    from polystokes_brownian_b200.engine import Batch
    n = {"less": CHUNK[Nc] - 1, "as many": CHUNK[Nc], "more": CHUNK[Nc] + 1, "three": 2 * CHUNK[Nc] + 2}[extra]
    s = configs.small_mixed(seed=Nc, Nm_chain=(n, 1), Nc=Nc, mm_HI=0, spread=14.0, ab_mode=1)
    assert s.params["Nm"] == n
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
