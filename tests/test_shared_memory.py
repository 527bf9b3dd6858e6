"""The attribute that allows a kernel more than 48 KB of dynamic shared memory."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "autograph_b200" / "csrc"


def test_attribute_is_one_constant():
    """The attribute belongs to the (kernel, GPU) pair and calls are serialised per device object only: set to a call's own
    size, or to the largest so far, it can be lowered by a thread with another device of the GPU (a recorded size above the
    real one then fails every larger call).  allow_smem, which sets one constant, is the only place that sets it."""
    setters = {p.name: p.read_text().count("cudaFuncSetAttribute") for p in CSRC.rglob("*.cu*")}
    assert {n: c for n, c in setters.items() if c} == {"common.cuh": 1}
    body = (CSRC / "common.cuh").read_text().split("int allow_smem(")[1].split("\n}\n")[0]
    assert re.search(r"cudaFuncAttributeMaxDynamicSharedMemorySize, MOST\)", body)   # a template argument
