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


# tables that the host copied (twiddles, omega) or whose kernels have ended when a sweep that reads them starts
TABLES = r"&(?:a\.t[12]\.Rx\[|a\.lens[xy]\[|RyDT\[|Rx\[x0|f\[\(size_t\)q \* Nt\]|f2\[|args\.wpos\[)"


def test_overlapped_kernels_use_no_read_only_loads_of_the_field():
    """A kernel that is launched while the kernel before still runs reads a field that is written during its
    own life: no __ldg of it and no const __restrict__ pointer to it (which the compiler may turn into one),
    in the kernels and in what they move it with."""
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
            for load in re.findall(r"__ldg\((.{0,40})", body):
                assert re.match(TABLES, load), (head.strip()[-120:], load)
            if "struct" in head or overlapped or "plane_move" in head:
                assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", (head if overlapped or "plane_move" in head else "") + body), head.strip()[-120:]
    assert kernels == 8 and found == set(helpers), (kernels, found)


def test_sweeps_after_new_tables_are_launched_when_those_have_ended():
    """The tables are read with __ldg: a plane sweep overlaps the kernel before it only if no table kernel was
    queued since the last one, and only its first kernel needs that."""
    capi, shapes = _code("mpc_capi.cu"), _code("mpc_shapes.cuh")
    assert re.search(r"a\.overlap = !c->tables_fresh;\s*c->tables_fresh = 0;", capi)
    for kernel in ("k_split", "k_lens"):
        calls = [m.end() for m in re.finditer(kernel + "<<<", capi)]
        created = capi.index("int mpc_create(")
        done = capi.index('"context setup")')
        for at in calls:   # mpc_create waits for its own
            assert created < at < done or "tables_fresh = 1" in capi[at:at + 420], capi[at:at + 120]
    launches = re.findall(r"launch_sweep\((\w+)_kernel<[^;]*?, st, (?:1|CL),\s*([\w.]+),", shapes)
    assert sorted(set(launches)) == sorted((k, "1" if k == "step" else "a.overlap") for k in
                                           ("plane", "plane_smem", "plane_x", "plane_x_warp", "plane_y", "plane_y512_tma", "plane_y_tma", "step"))
    assert shapes.count("b.overlap = 1;") == 3 == shapes.count("b.in = a.out;")


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
