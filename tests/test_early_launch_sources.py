"""Kernels that start before the previous kernel of their stream has ended (programmatic
stream serialization). What that kernel writes is not constant while they run: they
read it after the wait, through plain pointers (ld.global.nc, which __ldg and const
__restrict__ pointers give, is for data that stays constant over a kernel's lifetime),
or from L2 (__ldcg). One that reads through the L1 triggers its successor after its own wait."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "mymoonmd_gb300" / "csrc"
# kernel or its body -> the arguments that earlier kernels of the stream write
WRITTEN = {
    "csr_body": ("x", "y", "b", "xold"),
    "csr_kernel": ("x", "y", "b", "xold"),
    "csr_batch_kernel": ("x", "y", "b"),
    "sell_body": ("x", "y", "b"),
    "sell_kernel": ("x", "y", "b"),
    "sell_batch_kernel": ("x", "y", "b"),
    "k_gj_panel": ("M", "D", "steps", "prm", "rowsrc"),
    "k_gj_apply": ("src", "D", "steps", "prm", "cols"),
}


def definition(name):
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        m = re.search(r"\b" + name + r"\(((?:const )?int\b[^{;]*?)\)\s*\{", text)
        if m:
            end = text.index("\n}\n", m.end())
            return m.group(1), text[m.end():end]
    raise AssertionError(f"{name} not found")


@pytest.mark.parametrize("name", WRITTEN)
def test_written_data_is_read_through_plain_pointers(name):
    args, body = definition(name)
    for a in WRITTEN[name]:
        assert not re.search(r"__restrict__ " + a + r"\b", args), a
        assert not re.search(r"__ldg\(" + a + r"\b", body), a


@pytest.mark.parametrize("name", ["csr_body", "sell_body", "k_gj_panel", "k_gj_apply"])
def test_the_trigger_follows_the_wait(name):
    _, body = definition(name)
    assert "pdl_enter" not in body
    assert body.index("pdl_wait()") < body.index("pdl_trigger()")


def test_the_iterate_of_a_nodal_sweep_comes_from_l2():
    """k_nodal_patch triggers first: up to three colours' kernels are in flight"""
    _, body = definition("k_nodal_patch")
    reads = re.findall(r"\bxs \+|\bxs\[|\bb \+|\bb\[", body[body.index("pdl_wait()"):])
    cg = re.findall(r"__ldcg\((?:xs|b) \+", body)
    assert reads and len(reads) == len(cg)
