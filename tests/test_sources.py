"""Properties of the CUDA sources that one GPU cannot show at run time, read from the text."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mpc_gb300", "csrc")


def _code(name):
    """A source file without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"/\*.*?\*/|//[^\n]*", "", f.read(), flags=re.S)


def test_launch_grids_are_not_process_wide():
    """Grids follow the SM count of a context's device: no variable of static storage keeps them, or a
    context on a second device would change the launches of the first one's."""
    for m in re.finditer(r"\bstatic\s+(?:inline\s+)?(?!constexpr|const\b|cudaError_t|int max|int pencil)([\w:<>]+)\s+(\w+)\s*[=;]",
                         _code("mpc_shapes.cuh")):
        assert m.group(2) in ("fn", "once"), m.group(0)   # the driver's tensor-map encoder: one per process
