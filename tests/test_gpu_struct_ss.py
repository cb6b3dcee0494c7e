"""The dense stresslet solve of the structured path (Gauss-Jordan in place, pivot rows found by
every warp) against the oracle's direct solve: orders 5 Nc from one colloid to the dense
limit of twelve (more than one row per lane, more entries than threads), a batch of them."""
import numpy as np
import pytest

from oracle import psoracle as po
from polystokes_brownian_b200 import _capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nc", [1, 2, 3, 6, 7, 12])
@pytest.mark.parametrize("mm_HI", [0, 1])
def test_structured_solve_residual(Nc, mm_HI):
    import torch
    from polystokes_brownian_b200.engine import Batch
    s = configs.small_mixed(seed=40 + Nc, Nm_chain=(2, 4), Nc=Nc, mm_HI=mm_HI, spread=14.0)
    o = po.OracleSim(po.default_params(**s.params), s.x.ravel())
    o.stage()
    rhs = np.random.default_rng(Nc).normal(size=o.n)
    b = Batch([s, s])
    b.stage()
    x, res = b.solve(torch.from_numpy(np.r_[rhs, 2.0 * rhs]).cuda(), rtol=1e-12, method=_capi.PS_SOLVE_STRUCTURED)
    y = b.matmult(x).cpu().numpy().reshape(2, -1)
    x = x.cpu().numpy().reshape(2, -1)
    # backward stability: n^2 eps |A| |x| with n = 60 unknowns eliminated, |A| of order ten
    for r in range(2):
        t = (1.0 + r) * rhs
        assert np.linalg.norm(y[r] - t) <= 1e-11 * (np.linalg.norm(t) + np.linalg.norm(x[r]))
    b.close()
