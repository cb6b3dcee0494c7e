"""The monomer far field, each unordered pair once in square tiles, against the
pair formulas in plain torch (64 bits): sizes at the edges of cells (32, 64),
tiles and tile rules, both pair-scalar families, chain_HI on and off, FP64 and
the mixed form; and a replica's apply alone equal to the same replica in a
ragged batch, bit for bit.

Tolerances: FP64 sums of at most 12289 terms per row stay below 1e-13 of the
result's norm; the FP32 far field is held to the mixed form's bound of 1e-6."""
import numpy as np
import pytest

from polystokes_brownian_b200 import configs

pytestmark = pytest.mark.gpu

BETA = 0.3


def _system(n, nper, aa_mode, chain_HI, seed=0):
    """n monomers (chains of nper) at random in a cube at volume fraction 0.15: overlapping pairs included."""
    rng = np.random.default_rng([seed, n])
    edge = (n * 4.19 * BETA ** 3 / 0.15) ** (1.0 / 3.0)
    x = rng.uniform(-edge / 2, edge / 2, size=(n, 3))
    p = configs.make_params(Nm=n, Nc=0, Npoly=n // nper, Nmono_per_chain=nper, beta=BETA, mm_HI=1, chain_HI=chain_HI,
                            aa_mode=aa_mode, ab_mode=aa_mode)
    return configs.System("tiles", p, x)


def _apply(s, u):
    """M u by row blocks in 64 bits."""
    import torch
    x = torch.tensor(s.x, dtype=torch.float64, device="cuda")
    n, b = x.shape[0], s.params["beta"]
    chain = torch.arange(n, device="cuda") // s.params["Nmono_per_chain"]
    F = u.view(n, 3)
    out = torch.empty_like(F)
    for i0 in range(0, n, 1024):
        i1 = min(n, i0 + 1024)
        own = torch.arange(i0, i1, device="cuda")
        d = x[i0:i1, None] - x[None]
        r = (d * d).sum(2).sqrt()
        r[own - i0, own] = 1.0
        far = r > 2 * b
        if s.params["aa_mode"]:
            fx = torch.where(far, 1.5 / r - b * b / r ** 3, (1 - 0.1875 * r / b) / b)
            fy = torch.where(far, 0.75 / r + 0.5 * b * b / r ** 3, (1 - 0.28125 * r / b) / b)
        else:
            fx = torch.where(far, 0.375 / r - 2.0 / r ** 3, 0.375 * r - 1.0)
            fy = torch.where(far, 0.75 / r - 0.5 / r ** 3, 1.0 - 0.28125 * r)
        skip = own[:, None] == torch.arange(n, device="cuda")[None]
        if s.params["chain_HI"]:
            skip = skip | (chain[i0:i1, None] == chain[None])
        fx, fy = fx.masked_fill(skip, 0.0), fy.masked_fill(skip, 0.0)
        e = d / r[..., None]
        eu = (e * F[None]).sum(2)
        out[i0:i1] = fy @ F + (((fx - fy) * eu)[..., None] * e).sum(1) + F[i0:i1] / b
    return out.reshape(-1)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,nper,aa_mode,chain_HI", [
    (2, 1, 1, 0), (31, 31, 1, 0), (33, 1, 0, 0), (64, 8, 1, 1), (65, 5, 1, 0), (127, 1, 0, 1), (129, 3, 1, 0),
    (1535, 5, 1, 1), (1536, 6, 0, 0), (1537, 1, 1, 0), (1665, 9, 0, 1), (12288, 16, 1, 0), (12289, 1, 1, 0)])
def test_apply_matches_pair_formulas(n, nper, aa_mode, chain_HI, precision):
    import torch
    from polystokes_brownian_b200.engine import Batch
    s = _system(n, nper, aa_mode, chain_HI)
    b = Batch([s], precision=precision)
    b.stage()
    u = torch.randn(b.ntop, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    y, ref = b.mobility_apply(u), _apply(s, u)
    err = (torch.linalg.norm(y - ref) / torch.linalg.norm(ref)).item()
    assert err < (1e-6 if precision else 1e-13), err
    b.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_alone_equals_batch(precision):
    import torch
    from polystokes_brownian_b200.engine import Batch
    systems = [_system(n, 1, 1, 0, seed=7) for n in (1, 2, 63, 64, 200, 1536, 1600)]
    systems.insert(2, configs.suspension(n=3, phi=0.1, seed=1))
    systems.insert(5, configs.ensemble_member(np.random.default_rng([0, 8]), 300))
    big = Batch(systems, precision=precision)
    big.stage()
    u = torch.randn(big.ntop, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    y = big.mobility_apply(u)
    for r, s in enumerate(systems):
        one = Batch([s], precision=precision)
        one.stage()
        assert torch.equal(one.mobility_apply(big.seg(u, r, "top").contiguous()), big.seg(y, r, "top")), r
        one.close()
    big.close()
