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
