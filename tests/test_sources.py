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


def _functions(code):
    """(header, body) of every function definition at namespace scope: text up to a brace, and the braces' contents."""
    depth, start, head, out = 0, 0, 0, []
    code = re.sub(r"namespace\s*\w*\s*\{", " ", code)
    for i, ch in enumerate(code):
        if ch == "{":
            if depth == 0:
                start = i
            depth += 1
        elif ch == "}":
            depth -= 1
            if depth == 0:
                out.append((code[head:start], code[start:i + 1]))
                head = i + 1
    return out


def test_overlapped_kernels_use_no_read_only_loads():
    """A kernel that is launched while the kernel before still runs may read, after pdl_wait, what was written
    during its own life: no __ldg and no const __restrict__ pointer (which the compiler may turn into one)
    in it or in what it reads the field and the linear step's tables with."""
    helpers = ("plane_move", "struct YFactors", "struct XFactors", "struct XFactorsAny", "struct YSmemFactors", "struct PlaneTables",
               "struct PlaneArgs", "struct PencilArgs", "step_load_block", "xwarp_linear", "plane_line", "inner32")
    found = set()
    kernels = 0
    for name in ("mpc_kernels.cuh", "mpc_step.cuh"):
        for head, body in _functions(_code(name)):
            overlapped = "__global__" in head and "pdl_wait" in body
            helper = [h for h in helpers if re.search(re.escape(h) + r"\b(?!\w)", head)]
            if not overlapped and not helper:
                continue
            kernels += overlapped
            found.update(helper)
            after = body.split("pdl_wait", 1)[1] if overlapped else body
            assert "__ldg" not in after, head.strip()[-120:]
            if "struct" in head or overlapped or "plane_move" in head:
                assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", (head if overlapped or "plane_move" in head else "") + body), head.strip()[-120:]
    assert kernels == 8 and found == set(helpers), (kernels, found)


def test_a_timed_out_wait_waits_for_its_own_copies():
    """A kernel that gives up a wait leaves a bulk copy on its way into its shared memory, which the next CTA
    would be given: before it returns it waits again (bounded) for the late copy as well as for later ones."""
    late = r"mbar_wait\(&bars\[2 \* warp \+ \(k & 1\)\], \(uint32_t\)\(\(k >> 1\) & 1\)\)"
    sites = 0
    for name in ("mpc_kernels.cuh", "mpc_step.cuh"):
        code = _code(name)
        for part in re.split(r"atomicExch\([^;]*KERR_TMA_TIMEOUT\);", code)[1:]:
            leaving = re.split(r"\b(?:return|break);", part, maxsplit=1)[0]
            sites += 1
            if name == "mpc_kernels.cuh":
                assert re.search(r"for \(int (\w) = k;[^{]*mbar_wait\(&bars\[\1 % NBUF\]|mbar_wait\(bar, \(uint32_t\)\(k & 1\)\)",
                                 leaving), leaving
        if name == "mpc_step.cuh":   # where the first wait gives up, before the CTA's barrier
            assert len(re.findall(r"if \(!" + late + r"\) \{\s*\*dead = 1;\s*" + late + ";", code)) == 2
    assert sites == 6
