"""A product that is not a number reaches the result of the Lanczos root: two monomers at
one place in a mixed context give a pair block 0 times infinity, so M z has no value and
M^(1/2) z must not come back as a finite vector.  Replicas in one sub-block and in several,
basis caps before and after the first convergence check; the other replica of the batch is
untouched, bit for bit."""
import numpy as np
import pytest

from polystokes_brownian_b200 import _capi, configs

pytestmark = pytest.mark.gpu


def _system(n, coincide):
    x = np.random.default_rng(n).uniform(-3.0, 3.0, size=(n, 3)) * n ** (1.0 / 3.0)
    if coincide:
        x[n // 2] = x[n - 1]
    p = configs.make_params(Nm=n, Nc=0, Npoly=n, Nmono_per_chain=1, beta=0.5, mm_HI=1, aa_mode=1, ab_mode=1)
    return configs.System("nonfinite", p, x)


@pytest.mark.parametrize("kmax", [1, 2, 12, 40])
@pytest.mark.parametrize("n", [3, 86, 700])
def test_root_of_a_product_without_a_value(n, kmax):
    import torch
    from polystokes_brownian_b200.engine import Batch
    good, bad = _system(200, False), _system(n, True)
    b = Batch([bad, good], precision=_capi.PS_PREC_MIXED)
    b.stage()
    z = torch.randn(b.ntop, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    assert not torch.isfinite(b.seg(b.mobility_apply(z), 0, "top")).all()
    w, _ = b.sqrtm(z, kmax=kmax, tol=1e-15)
    assert not torch.isfinite(b.seg(w, 0, "top")).any()
    one = Batch([good], precision=_capi.PS_PREC_MIXED)
    one.stage()
    want, _ = one.sqrtm(b.seg(z, 1, "top").contiguous(), kmax=kmax, tol=1e-15)
    assert torch.isfinite(want).all() and torch.equal(b.seg(w, 1, "top"), want)
    b.close()
    one.close()
