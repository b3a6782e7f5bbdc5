"""Settings of a kernel hold for one device: no launch may take them from a process-wide flag.
Read from the sources, as a second device is needed to see it happen."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "gammcor_gb300" / "csrc"


def test_shared_memory_limits_are_not_set_once_per_process():
    for src in CSRC.glob("*.cu*"):
        text = src.read_text()
        for m in re.finditer(r"call_once\(.*?\}\);", text, re.S):
            assert "cudaFuncSetAttribute" not in m.group(0), (src.name, m.group(0))
        assert not re.search(r"static\s+cudaError_t", text), src.name
