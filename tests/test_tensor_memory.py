"""Rules of the kernels that take tensor memory, held on their source: what breaks them can stop a GPU, so no run shows it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "rew_b200", "csrc")


def _source(f):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())


FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def _kernels():
    """(name, body) of every __global__ function."""
    for f in FILES:
        text = _source(f)
        for m in re.finditer(r"__global__\s+(?:void\s+|__\w+__\s*\([^)]*\)\s*)+(\w+)\s*\(", text):
            start = text.index("{", m.end())
            depth = 0
            for i in range(start, len(text)):
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                if depth == 0:
                    break
            yield f + ":" + m.group(1), text[start:i + 1]


def test_tensor_memory_is_taken_before_later_launches_may_start():
    """A CTA that let the next launch start before it had its columns could wait for columns which that launch holds while it
    waits for this one to end.  One helper does both in the safe order; nothing else may do either."""
    bodies = dict(_kernels())
    takers = {k for k, b in bodies.items() if "alloc_then_launch_dependents" in b}
    assert len(takers) >= 8 and any("linear_tc_pair" in k for k in takers) and any("flash_tc" in k for k in takers), takers
    for k in takers:
        assert "pdl_launch_dependents" not in bodies[k], k
    for k, b in bodies.items():
        assert "tcgen05.alloc" not in b, k
    helper = _source("tc.cuh")
    at = helper.index("void alloc_then_launch_dependents")
    body = helper[at:helper.index("\n}\n", at)]
    assert body.rindex("tcgen05.alloc") < body.index("pdl_launch_dependents();")
    for f in FILES:
        assert f == "tc.cuh" or "tcgen05.alloc" not in _source(f), f


def test_kernels_with_all_tensor_memory_of_an_sm_take_its_shared_memory_too():
    """The persistent and the pair Linear hold 512 columns for a whole launch: no CTA that starts early may sit beside them."""
    text = _source("linear_tc.cu")
    assert re.search(r"kAllSmem = 227 \* 1024;", text)
    cfgs = re.findall(r"struct (\w+Cfg) \{(.*?)\n\};", text, re.S)
    wide = {n for n, body in cfgs if re.search(r"TMEM_COLS = 512;", body)}
    assert wide == {"PersistCfg", "PairCfg"}
    for n, body in cfgs:
        if n in wide:
            assert re.search(r"int SMEM = kAllSmem;", body), n
    for call in re.findall(r"launch_k\((linear_tc_(?:persist|pair)_kernel.*?)\)\);", text, re.S):
        assert re.search(r"\(size_t\)P\w+Cfg::SMEM,", call), call


def test_accumulators_are_waited_for_by_whole_warps():
    """The way out of an accumulator reads tensor memory and trades values between lanes, both collective over the warp: its wait
    ends with a vote, so that lanes which gave up cannot leave the others in there."""
    text = _source("linear_tc.cu")
    waits = re.findall(r"(\w+)\(&?tmem_full\b", text)
    assert [w for w in waits if w.startswith("mbar_wait")] == ["mbar_wait_warp"] * 3, waits
    assert re.search(r"bool mbar_wait_warp\([^)]*\) \{\s*return __all_sync\(0xffffffffu, mbar_wait\(", _source("ptx.cuh"))
