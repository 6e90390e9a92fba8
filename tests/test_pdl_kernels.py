"""Kernels launched programmatically begin before their predecessor has ended (csrc/topo_common.cuh).

Each has to wait for it (TOPO_PDL_ENTRY or TOPO_PDL_WAIT), and may not take what the chain of a
solve writes through __restrict__ pointers: the compiler could load it before the wait.
"""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "topomax_gb300", "csrc")
# fixed from the end of set-up to the end of a solve: the fluid's tables and assembled rows
FIXED = {("k_fluid_apply", "S"), ("k_fluid_apply", "rows")}


def _sources():
    return "\n".join(re.sub(r"//[^\n]*", "", open(f).read()) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))))


def _definition(text, name):
    """(parameters, body) of a kernel."""
    m = re.search(r"__global__[^;{}]*?\b%s\(" % name, text)
    assert m, name
    depth, i = 1, m.end()
    while depth:
        depth += {"(": 1, ")": -1}.get(text[i], 0)
        i += 1
    start = text.index("{", i)
    end, depth = start + 1, 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[m.end():i - 1], text[start:end]


def test_programmatic_kernels_wait_and_read_the_chain_after_it():
    text = _sources()
    names = set(re.findall(r"\blaunch_pdl\(\s*(k_\w+)", text))
    assert {"k_pcg_r", "k_pcg_p", "k_dot", "k_level_down", "k_p2_rows", "k_krylov_next"} <= names
    for name in sorted(names):
        params, body = _definition(text, name)
        if name == "k_p2_rows":  # its row function waits
            body = text[text.index("void p2_rows_run("):text.index("k_p2_rows(")]
        assert "TOPO_PDL_ENTRY()" in body or "TOPO_PDL_WAIT()" in body, f"{name} does not wait"
        for p in re.findall(r"__restrict__\s+(\w+)", params):
            assert (name, p) in FIXED, f"{name}: {p} is read or written through __restrict__"
