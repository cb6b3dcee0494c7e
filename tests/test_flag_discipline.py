"""Source check of the solvers' stop flags (no GPU needed).

Blocks that share a replica's scalars run in no order: where a launch reads a replica's
done or stop flag and also writes it, warps of one block may disagree about leaving, and
those that stay add shared words that the others never wrote.  So a kernel of several
blocks per replica reads a flag of the launch before and writes another one."""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "polystokes_brownian_b200", "csrc")
# one block (or one thread) per replica: a barrier or program order stands between read and write
ONE_BLOCK = {"k_lz_check", "k_lz_check_ql", "k_lz_spec_apply", "k_sl_iter", "k_sl_load"}
FLAG = r"((?:\w+\[[^\]]*\]|\w+)\.(?:done|stop)(?:\[[^\]]*\])?)"


def test_no_kernel_writes_a_flag_that_its_launch_reads():
    seen, bad = 0, []
    for f in ("krylov.cu", "solve.cu", "rpy.cu", "ps_reduce.cuh"):
        with open(os.path.join(CSRC, f)) as fh:
            src = fh.read()
        for part in re.split(r"(?m)^(?=template|__global__|__device__|static|int |namespace|struct)", src):
            if "__global__" not in part:
                continue
            name = [n for n in re.findall(r"(\w+)\s*\(", part) if n not in ("__launch_bounds__", "__cluster_dims__")][0]
            body = part[part.index("{"):]
            shared = re.compile(r"(?:st\d?|lz|mr|pc|sc)\[")          # per-replica scalars in device memory
            writes = {m.group(1) for m in re.finditer(FLAG + r"\s*=(?!=)", body) if shared.match(m.group(1))}
            reads = {m.group(1) for m in re.finditer(FLAG + r"(?!\s*=[^=])", body) if shared.match(m.group(1))}
            seen += bool(reads)
            if writes & reads and name not in ONE_BLOCK:
                bad.append((f, name, sorted(writes & reads)))
    assert seen >= 8
    assert not bad, bad
