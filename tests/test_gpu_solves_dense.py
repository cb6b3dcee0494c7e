"""Structured solves against dense solutions in numpy.  Without lubrication the saddle system
has the closed solution F_t = -b_bot, M_SS F_S = b_S - M_St F_t, U = (M F)_t - b_t, taken here
from the oracle's dense mobility: the dense stresslet block by elimination, one to twelve
colloids (condition of M_SS below 1e2, so 1e-12).  Lubricated suspensions beyond that go by
pair-space MINRES, against a dense solve of the operator itself, column by column: at rtol
1e-13 the error is at most that times the condition of the preconditioned system, which is
below 1e4 at gaps of 0.1, so 1e-9; a lost pair or a stop far too early shows at 1e-6."""
import numpy as np
import pytest

from oracle import psoracle as po
from polystokes_brownian_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nc,chains", [(1, (1, 1)), (1, (2, 9)), (2, (3, 7)), (5, (2, 20)), (12, (4, 10))])
def test_stresslet_block_by_elimination(Nc, chains):
    import torch
    from polystokes_brownian_b200.engine import Batch
    s = configs.small_mixed(seed=Nc, Nm_chain=chains, Nc=Nc, mm_HI=1, spread=9.0, aa_mode=1, ab_mode=1)
    o = po.OracleSim(po.default_params(**s.params), s.x.ravel())
    o.stage()
    M = o.dense_mobility()
    n6, top = 3 * s.params["Nm"] + 6 * Nc, M.shape[0]
    r = np.random.default_rng(Nc).normal(size=top + n6)
    F = np.zeros(top)
    F[:n6] = -r[top:]
    F[n6:] = np.linalg.solve(M[n6:, n6:], r[n6:top] - M[n6:, :n6] @ F[:n6])
    want = np.r_[F, M[:n6] @ F - r[:n6]]
    b = Batch([s])
    b.stage()
    x, res = b.solve(torch.from_numpy(r).cuda(), method=1)
    assert res.reason == 2
    assert np.linalg.norm(x.cpu().numpy() - want) <= 1e-12 * np.linalg.norm(want)
    b.close()


@pytest.mark.parametrize("n", [13, 32, 33, 64])
def test_lubricated_suspension(n):
    import torch
    from polystokes_brownian_b200.engine import Batch
    s = configs.suspension(n=n, phi=0.1, seed=n, gap=0.1)
    b = Batch([configs.System(s.name, dict(s.params, lub_on=1), s.x)])
    b.stage()
    eye = torch.eye(b.nvec, dtype=torch.float64, device="cuda")
    A = torch.stack([b.matmult(eye[k].contiguous()) for k in range(b.nvec)], 1)
    r = torch.randn(b.nvec, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    want = torch.linalg.solve(A, r)
    x, res = b.solve(r, rtol=1e-13, maxit=20000, method=1)
    assert res.reason == 2
    assert (torch.linalg.norm(x - want) / torch.linalg.norm(want)).item() <= 1e-9
    b.close()
