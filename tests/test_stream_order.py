"""Fills and uploads of device memory go through a slot's stream, held on the source: whether an unordered one is overtaken is a matter
of microseconds, so no run shows it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "rew_b200", "csrc")


def test_device_memory_is_filled_and_uploaded_on_the_slots_stream():
    """A slot's stream does not wait for the legacy default stream, and cudaMemset, or cudaMemcpy from pageable memory, may return before the
    device memory is written: a kernel of the slot could be overtaken by them."""
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        assert not re.search(r"\bcudaMemset(2D|3D)?\s*\(", text), f
        for call in re.findall(r"\bcudaMemcpy(?:2D)?\s*\((.*?)\);", text, re.S):
            assert "cudaMemcpyDeviceToHost" in call, (f, call)
        for call in re.findall(r"\bcudaMem(?:set|cpy)(?:2D)?Async\s*\((.*?)\)\s*[;)!]", text, re.S):
            assert re.search(r"stream|side", call), (f, call)


def _kernels(f):
    """(name, body) of every __global__ function of a source file."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
    for m in re.finditer(r"__global__[^;{]*?(\w+_kernel)\(", text):
        start = text.index("{", m.end())
        depth = 0
        for i in range(start, len(text)):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            if depth == 0:
                break
        yield m.group(1), text[start:i + 1]


def test_a_launch_beside_its_neighbour_learns_of_earlier_writes_from_memory():
    """The walk over portions does not wait for the launch of single tokens ahead of it, but reads what launches ahead of both wrote.  That
    the neighbour passed its wait orders nothing for another grid: it is told in memory (release, acquire), or waits itself."""
    ptx = open(os.path.join(CSRC, "ptx.cuh")).read()
    body = lambda name: ptx[ptx.index("void " + name + "("):ptx.index("\n}\n", ptx.index("void " + name + "("))]
    start, wait = body("pdl_launch_beside"), body("pdl_wait_beside")
    assert start.index("st.release.gpu") < start.index("pdl_launch_dependents();")
    assert "ld.acquire.gpu" in wait and re.search(r"if \(!__syncthreads_or\(seen\)\) pdl_wait\(\);", wait)
    for family in ("gla", "delta"):
        singles = dict(_kernels(family + ".cu"))
        beside = {n: b for n, b in singles.items() if "beside" in b}
        assert len(beside) == 2, singles.keys()
        for name, b in beside.items():
            assert re.search(r"if \(!a\.beside\) pdl_launch_dependents\(\);", b), name
            calls = [m.start() for m in re.finditer(r"pdl_launch_\w+\(", b)]
            assert len(calls) == 2 and b.rindex("pdl_wait();") < b.index("if (a.beside) pdl_launch_beside(a.passed, a.beside);"), name
        scan = dict(_kernels(family + "_chunk.cu"))[family + "_scan_kernel"]
        first = min(scan.index(x) for x in ("a.list", "a.work", "a.state", "a.partial"))
        assert re.search(r"if \(a\.beside\) pdl_wait_beside\(a\.passed, a\.beside\);\s+else pdl_wait\(\);", scan[:first]), family
        assert re.search(r"if \(a\.beside\) pdl_wait\(\);\s*\}$", scan), family
