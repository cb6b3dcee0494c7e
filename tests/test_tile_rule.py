"""The serving loop's footprint follows the far field's tile rule (no GPU needed): its table of
edges is the rule in the CUDA sources, and a narrower edge in force means more partial slots."""
import os
import re

from polystokes_brownian_b200 import configs, serve

CSRC = os.path.join(os.path.dirname(__file__), "..", "polystokes_brownian_b200", "csrc")


def test_edges_are_the_kernels():
    with open(os.path.join(CSRC, "ps_internal.h")) as f:
        rule = re.search(r"constexpr int aa_tile_edge\(int Nm\) \{ return (.*?); \}", f.read()).group(1)
    got = [(int(n), int(e)) for n, e in re.findall(r"Nm <= (\d+) \? (\d+)", rule)]
    assert got == [tuple(v) for v in serve.AA_TILE_EDGES[:-1]]
    assert int(re.search(r": (\d+)\)*$", rule).group(1)) == serve.AA_TILE_EDGES[-1][1]


def test_footprint_follows_the_edge_in_force():
    def of(n, edge):
        p = configs.make_params(Nm=n, Nc=0, Npoly=n, Nmono_per_chain=1, beta=0.3, mm_HI=1)
        return serve.footprint_bytes(configs.System("foot", p, None), widest_edge=edge)
    assert of(12288, 256) == of(12288, 128)
    # one slot of 3 Nm doubles per tile of 128 instead of one per tile of 256
    assert of(16384, 128) - of(16384, 256) == 8 * 3 * 16384 * (128 - 64)
