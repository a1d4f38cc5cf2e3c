"""A handle's work runs on a stream that does not wait for the default stream, so what its kernels read
has to be written on that stream too: a plain cudaMemcpy to the device (from pageable memory it may return
once the data is staged) or cudaMemset is not in order with them."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "vocalsim-2p5d-fdtd_b200" / "csrc"
SOURCES = sorted(p for p in CSRC.iterdir() if p.suffix in (".cpp", ".cu", ".cuh", ".h"))


def calls(text, name):
    """Argument texts of every call of `name`."""
    for m in re.finditer(rf"\b{name}\s*\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_device_memory_is_written_on_the_handles_stream(path):
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)
    for name in ("cudaMemcpy", "cudaMemcpy2D", "cudaMemcpyToSymbol"):
        assert [a for a in calls(text, name) if "DeviceToHost" not in a] == []
    for name in ("cudaMemset", "cudaMemset2D"):
        assert list(calls(text, name)) == []
