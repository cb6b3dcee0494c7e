"""A solve on a side stream does not depend on what the default stream has queued: the
first pair-space MINRES solve of a fresh suspension context (which allocates and clears
its workspace on the way) beside a default stream that stays busy for 20 us to 2 ms, so
that anything left on it would land in the middle of the solve, against the same solve
on the default stream, bit for bit."""
import pytest

from polystokes_brownian_b200 import configs

pytestmark = pytest.mark.gpu


def _solve(system, r, busy_cycles):
    import torch
    from polystokes_brownian_b200.engine import Batch
    b = Batch([system])
    b.stage()
    torch.cuda.synchronize()
    if busy_cycles:
        side = torch.cuda.Stream()
        torch.cuda._sleep(busy_cycles)
        with torch.cuda.stream(side):
            x, res = b.solve(r, rtol=1e-9, maxit=5000, method=1)
        side.synchronize()
    else:
        x, res = b.solve(r, rtol=1e-9, maxit=5000, method=1)
    x = x.clone()
    torch.cuda.synchronize()
    b.close()
    return x, (res.reason, res.iters_max)


@pytest.mark.parametrize("lub", [0, 1])
def test_first_solve_on_a_side_stream(lub):
    import torch
    s = configs.suspension(n=33, phi=0.1, seed=3, gap=0.1)
    s = configs.System(s.name, dict(s.params, lub_on=lub), s.x)
    r = torch.randn(17 * 33, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    want, how = _solve(s, r, 0)
    assert how[0] == 2 and how[1] > 0
    for us in (20, 60, 150, 400, 800, 2000):
        x, got = _solve(s, r, 1900 * us)
        assert got == how and torch.equal(x, want), us
