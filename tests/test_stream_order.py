"""What the engine copies to the device or clears goes through the stream of the kernels that read it.

A host-to-device cudaMemcpy from pageable memory may return before its last piece has arrived, a cudaMemset is
asynchronous, and the engine's own streams do not wait for the default one: a kernel launched next could read
what was there before (mesh indices among it).
"""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "libclsph_gb300" / "csrc"


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.iterdir()))
def test_copies_and_clears_are_stream_ordered(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    calls = re.findall(r"\b(cudaMemset|cudaMemcpy)\s*\(([^;|]*)", text)
    assert not [c for c in calls if c[0] == "cudaMemset" or "DeviceToHost" not in c[1]]
