"""The fluid solve holds and computes everything in FP64, as the package's interface says: its entry
points have no precision to choose."""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "topomax_gb300", "csrc")


def test_no_single_precision_in_the_fluid_solve():
    for name in ("topo_fluid.cu", "topo_fluid.cuh", "topo_fluid_setup.h", "topo_krylov.cuh"):
        code = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        assert not re.search(r"\bfloat\b|\b\d+\.?\d*f\b", code), name
