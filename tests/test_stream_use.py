"""Every device operation of the library names a stream: the library's streams do
not wait for the legacy stream, so what runs there is not ordered with them."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jfem_b200", "csrc")


def sources():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as h:
                yield f, re.sub(r"//[^\n]*", "", h.read())


def test_no_operation_on_the_legacy_stream():
    bad = []
    for f, text in sources():
        bad += [(f, m.group(0)) for m in re.finditer(r"\bcudaMemset\s*\(", text)]
        # <<<grid, block, shared memory, stream>>>
        for m in re.finditer(r"<<<(.*?)>>>", text, flags=re.S):
            depth, commas = 0, 0
            for ch in m.group(1):
                depth += ch in "([{"
                depth -= ch in ")]}"
                commas += ch == "," and depth == 0
            if commas < 3:
                bad.append((f, m.group(0)))
    assert not bad, bad


def test_no_wait_for_the_whole_device():
    """cudaDeviceSynchronize is an error, and breaks the capture, while any stream of
    the device is being captured by anyone in the process."""
    assert [f for f, text in sources() if "cudaDeviceSynchronize" in text] == []
