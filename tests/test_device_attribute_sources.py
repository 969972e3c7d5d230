"""A kernel's attributes belong to a device: a process may hold contexts on several, so
none is set once per process (and no failure of the first device is kept for the rest)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "mymoonmd_gb300" / "csrc"


def test_no_kernel_attribute_is_set_once_per_process():
    found = 0
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        found += text.count("cudaFuncSetAttribute(")
        assert "call_once" not in text and "once_flag" not in text, path.name
        assert not re.search(r"static\s+(?:const\s+)?(?:bool|cudaError_t)\s+\w+\s*=[^;]*", text), path.name
    assert found
