"""The two forms of the Lanczos orthogonalisation that keep the order of their sums (far
fields that may be indefinite): a cluster per replica in small batches, sweeps over the
reduction table in batches of more than 28 such replicas and beside a replica of more
than sixteen table blocks.  A replica's root is the same bit for bit in either, at vector
lengths around the table's blocks of 1024 entries and its threads' 256, with basis caps
around a convergence check, and beside replicas that take neither form."""
import numpy as np
import pytest

from polystokes_brownian_b200 import configs

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 85, 86, 341, 342, 683, 1000]


def _monomers(n, ref=True):
    x = np.random.default_rng(n).uniform(-3.0, 3.0, size=(n, 3)) * n ** (1.0 / 3.0)
    m = 0 if ref else 1
    p = configs.make_params(Nm=n, Nc=0, Npoly=n, Nmono_per_chain=1, beta=0.3, mm_HI=1, aa_mode=m, ab_mode=m)
    return configs.System("ordered", p, x)


def _roots(systems, seeds, kmax, tol=1e-15):
    import torch
    from polystokes_brownian_b200.engine import Batch
    b = Batch(systems)
    b.stage()
    z = torch.cat([torch.randn(3 * s.params["Nm"] + 11 * s.params["Nc"], dtype=torch.float64, device="cuda",
                               generator=torch.Generator("cuda").manual_seed(k)) for s, k in zip(systems, seeds)])
    w, _ = b.sqrtm(z, kmax=kmax, tol=tol)
    out = [b.seg(w, r, "top").clone() for r in range(len(systems))]
    b.close()
    return out


@pytest.mark.parametrize("kmax,tol", [(1, 1e-15), (9, 1e-15), (64, 1e-15), (40, 1e-3)])
def test_alone_and_in_a_large_batch(kmax, tol):
    import torch
    systems = [_monomers(n) for n in SIZES] * 4 + [_monomers(n, ref=False) for n in (86, 400)]
    seeds = list(range(len(systems)))
    batch = _roots(systems, seeds, kmax, tol)
    for k in list(range(len(SIZES))) + [len(systems) - 2, len(systems) - 1]:
        alone = _roots([systems[k]], [seeds[k]], kmax, tol)[0]
        assert torch.isfinite(alone).all() and torch.equal(alone, batch[k]), k


def test_beside_a_replica_of_many_table_blocks():
    import torch
    s = configs.suspension(n=40, phi=0.1, seed=1, gap=0.1)
    systems = [_monomers(342), _monomers(5462), s]          # 16386 entries: 17 table blocks
    batch = _roots(systems, [3, 4, 5], 12)
    for k in (0, 2):
        assert torch.equal(_roots([systems[k]], [3 + k], 12)[0], batch[k]), k


def test_table_blocks_at_the_clusters_limit():
    import torch
    systems = [_monomers(5461), _monomers(30)]              # 16383 entries: 16 table blocks
    alone = _roots(systems[:1], [7], 12)[0]
    pair = _roots(systems, [7, 8], 12)
    many = _roots(systems[:1] + systems[1:] * 30, [7] + [8] * 30, 12)
    assert torch.equal(alone, pair[0]) and torch.equal(alone, many[0]) and torch.equal(pair[1], many[9])
