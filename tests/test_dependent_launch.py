"""Kernels that start before their predecessor in the stream has ended."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "autograph_b200" / "csrc"


def _kernels():
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        for body in re.split(r"\b__global__\b", path.read_text())[1:]:
            body = re.sub(r"//[^\n]*", "", body.split("\n}\n")[0])
            yield path.name, re.search(r"(\w+)\(", re.sub(r"__launch_bounds__\([^)]*\)", "", body)).group(1), body


def test_tensor_memory_comes_before_dependents():
    """A dependent that came first could hold columns that this kernel still waits for: every kernel with tensor
    memory allocates it, and meets at a barrier, before one of its threads lets dependents launch."""
    seen = 0
    for file, name, body in _kernels():
        trigger = re.search(r"let_dependents_launch\(|griddepcontrol\.launch_dependents", body)
        alloc = body.find("tmem_alloc(")
        if trigger is None or alloc < 0:
            continue
        seen += 1
        assert alloc < trigger.start(), f"{file}: {name} lets dependents launch before it allocates tensor memory"
        assert "__syncthreads()" in body[alloc:trigger.start()], f"{file}: {name}: no barrier between the two"
    assert seen >= 5
