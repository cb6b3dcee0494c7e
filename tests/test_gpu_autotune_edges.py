"""What the far-field tuner may change: a context whose replicas every candidate cuts alike
leaves the process's edge as it is (and reports one time for all of them), a context above
12288 monomers times two, and a replica's product after it is the one before it to
rounding.  In a child process, since the edge outlives the test."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.join(os.path.dirname(__file__), "..")

CHILD = r"""
import numpy as np, torch
from polystokes_brownian_b200 import configs
from polystokes_brownian_b200.engine import Batch

def batch(*sizes):
    out = []
    for n in sizes:
        p = configs.make_params(Nm=n, Nc=0, Npoly=n, Nmono_per_chain=1, beta=0.3, mm_HI=1, aa_mode=1, ab_mode=1)
        out.append(configs.System("tune", p, np.random.default_rng(n).uniform(-1, 1, size=(n, 3)) * 2 * n ** (1 / 3)))
    b = Batch(out)
    b.stage()
    return b

for sizes in ((2,), (64, 1536), (1537, 300), (12288,)):
    b = batch(*sizes)
    for _ in range(3):
        best, ms = b.autotune(2)
        assert best == 256 and len(set(ms.values())) == 1 and min(ms.values()) > 0, (sizes, best, ms)
    b.close()
b = batch(12289, 50)
u = torch.randn(b.ntop, dtype=torch.float64, device="cuda")
y = b.mobility_apply(u)
best, ms = b.autotune(2)
assert best in (128, 256) and ms[256] == ms[512] == ms[1024] and ms[best] == min(ms.values()), (best, ms)
assert (torch.linalg.norm(b.mobility_apply(u) - y) <= 1e-13 * torch.linalg.norm(y)).item()
c = batch(700)
assert c.autotune(2)[0] == best          # the edge in force stays
c.close()
b.close()
print("tuned")
"""


def test_only_a_context_that_distinguishes_edges_changes_the_edge():
    p = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "tuned" in p.stdout, p.stdout + p.stderr
