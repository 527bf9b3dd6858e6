"""The attribute that allows a kernel more than 48 KB of dynamic shared memory."""
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "autograph_b200" / "csrc"


@pytest.mark.parametrize("name", ["nhwc_ops.cu", "conv_halo_f32.cu", "conv_halo_wgrad_f32.cu"])
def test_attribute_is_one_constant(name):
    """The attribute belongs to the (kernel, GPU) pair and calls are serialised per device object only: set to a call's own
    size, or to the largest so far, it can be lowered by a thread with another device of the GPU (a recorded size above the
    real one then fails every larger call).  allow_smem sets one constant."""
    text = (CSRC / name).read_text()
    assert "allow_smem(" in text
    assert "cudaFuncSetAttribute" not in text
