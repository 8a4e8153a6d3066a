"""Chained launches: a kernel given to launch_chained may be scheduled while the
kernel before it in the stream is still running, so each of them has to begin
with the wait (chain_enter).  Checked in the sources: a missing wait is a race,
which a run on the GPU need not show."""
import os
import re

import funlbm_b200

CSRC = os.path.join(os.path.dirname(funlbm_b200.__file__), "csrc")


def _sources():
    text = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as fh:
                text[name] = re.sub(r"//[^\n]*", "", fh.read())
    return text


def _first_statement(text, kernel):
    """First statement of the __global__ function `kernel`, or None."""
    m = re.search(r"__global__[^{;]*?\b%s\s*\(" % kernel, text)
    if m is None:
        return None
    body = text.index("{", m.end())
    return text[body + 1:text.index(";", body)].strip()


def test_chained_kernels_wait_first():
    text = _sources()
    launched = set()
    for t in text.values():
        launched |= set(re.findall(r"launch_chained\(\s*(\w+)", t))
    launched = {k for k in launched if k.startswith("k_")}
    assert len(launched) > 10
    first = {}
    for kernel in sorted(launched):
        found = [s for s in (_first_statement(t, kernel) for t in text.values()) if s is not None]
        assert len(found) == 1, (kernel, found)
        first[kernel] = found[0]
    missing = [k for k, s in first.items() if s != "chain_enter()"]
    assert not missing, missing
