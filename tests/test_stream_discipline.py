"""Source check of the streams that clears run on (no GPU needed).

Every entry point works on the caller's stream, which need not wait for the legacy
default stream (PyTorch's side streams do not).  A plain cudaMemset runs on the default
stream and returns before it has run, so inside a call it may clear a buffer after the
call's kernels have written it.  Plain clears are left to the functions that run when a
context is built, or that wait for the device before they return."""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "polystokes_brownian_b200", "csrc")
# building a context: a blocking copy on the default stream follows the last clear (ps_set_seed)
AT_BUILD = {("capi.cu", "#define TRY_ALLOC"), ("krylov.cu", "build_red_table")}
SYNCED = {("observe.cu", "obs_reset")}


def _functions(src):
    """(name, text) of what starts at the left margin: macros, and functions up to the next start."""
    starts = [(m.start(), m.group(1) or m.group(2)) for m in re.finditer(r"^(?:(#define \w+)|[A-Za-z_][^;\n(]*?(\w+)\()", src, re.M)]
    for (a, name), (b, _) in zip(starts, starts[1:] + [(len(src), "")]):
        yield name, src[a:b]


def test_clears_inside_a_call_run_on_its_stream():
    found = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(CSRC, f)) as fh:
                for name, body in _functions(fh.read()):
                    if re.search(r"\bcudaMemset(?:2D|3D)?\(", body):
                        found[f, name] = body
    assert set(found) == AT_BUILD | SYNCED
    for key in SYNCED:
        last = found[key].rindex("cudaMemset(")
        assert "cudaDeviceSynchronize()" in found[key][last:], key
