"""Read off the sources (no GPU needed).  Kernels launched with programmatic
dependence live beside their predecessor's last stores: what a step computes
must not reach them through read-only loads or __restrict__ pointers, which
the compiler may take across the wait at their start.  And the C entries
launch on their solver's device."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "dgcuda_gb300", "csrc")
MESH = {"nbr"}  # written when a solver is created, read-only in every launch


def sources():
    out = {}
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(f).read())
        out[os.path.basename(f)] = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return out


def restrict_params(params):
    return {m.group(1) for m in re.finditer(r"__restrict__\s*(\w+)", params)}


def test_dependent_kernels_wait_first_and_take_no_restrict_pointer():
    src = sources()
    text = "\n".join(src.values())
    names = set(re.findall(r"\blaunch\(\s*(k_\w+)<", text))
    assert {"k_face", "k_means", "k_lambda", "k_element_fx", "k_trace_fx", "k_limit_tr"} <= names
    for k in sorted(names):
        m = re.search(r"\b%s\(([^{;]*?)\)\s*\{(.*?)\n\}" % k, text, re.S)
        assert m, k
        assert restrict_params(m.group(1)) <= MESH, k
        first = [s for s in m.group(2).split(";") if "__shared__" not in s and "constexpr" not in s
                 and not s.strip().startswith("using")]
        assert first[0].strip() == "pdl_begin()", k


def test_their_device_functions_take_no_restrict_pointer_and_no_read_only_load():
    src = sources()
    for f in ("dg_kernels.cuh", "dg_fixed.cuh"):
        for m in re.finditer(r"__device__ __forceinline__ [\w:]+ \*?(\w+)\(([^{;]*?)\)\s*\{",
                             src[f], re.S):
            # (a batch's block map is read by ordinary launches)
            assert restrict_params(m.group(2)) <= MESH | {"blk2prob", "blk0"}, m.group(1)
    for f, text in src.items():
        for m in re.finditer(r"__ldg\((.{0,12})", text):
            assert m.group(1).startswith("a.vtx"), (f, m.group(0))


def test_entry_points_that_launch_set_their_device_first():
    """A solver's work runs on its own GPU whichever the thread's current one
    is: the C entries make it current before their first launch."""
    work = re.compile(r"->ops->|dg::launch_|set_bed_slopes\(|\brun\(s|run_steps\(|put_rows\(")
    text = open(os.path.join(CSRC, "dg_solver.cpp")).read()
    seen = 0
    for m in re.finditer(r'extern "C" [\w ]+\*?\b(dg_\w+)\([^{;]*\)\s*\{\n(.*?)\n\}', text, re.S):
        w = work.search(m.group(2))
        if w:
            seen += 1
            assert "cudaSetDevice" in m.group(2)[:w.start()], m.group(1)
    assert seen >= 10
