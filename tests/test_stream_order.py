"""Reads the sources: work on a context's stream that is not a kernel goes through the functions of
ctx.cuh that make the next kernel of the step a plain launch (a dependent launch waits for kernels
only), and every kernel that the step launches waits for its predecessor before anything else."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "suli-openmp_b200" / "csrc"


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def test_no_bare_copies_on_the_stream():
    bare = re.compile(r"cuda(?:Memcpy|Memset|GraphLaunch|StreamWaitEvent)\w*\([^;]*\bc->stream\b[^;]*;")
    for path in sorted(CSRC.glob("*.cu*")):
        found = [m.group(0) for m in bare.finditer(_code(path))]
        # the four functions themselves
        assert len(found) == (4 if path.name == "ctx.cuh" else 0), (path.name, found)


def test_step_kernels_wait_first():
    code = _code(CSRC / "k_fp64.cu")
    names = set(re.findall(r"step_launch\(c, \(?(k_\w+)", code)) | set(re.findall(r"LAUNCH_R\((k_\w+)", code))
    names |= set(re.findall(r"\? (k_\w+)<true> : k_\w+<false>;", code))
    assert len(names) > 25
    for name in sorted(names):
        body = re.search(r"__global__ void (?:__launch_bounds__\([^{;]*?\)\s+)?" + name + r"\([^{;]*\)\s*\{\s*([^;]*;)", code)
        assert body and body.group(1) == "pdl_wait();", name
