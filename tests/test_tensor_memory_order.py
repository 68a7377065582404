"""Blocks of a kernel that was launched behind another one may be on an SM as soon as that one has let its dependents go, and
allocate tensor memory before they wait for it.  A kernel that allocated afterwards could find none left, in a wait that has no
end: so every kernel allocates first.  Read from the sources, since the order cannot be watched from outside."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parents[1] / "xllm_b200" / "csrc" / "kernels"


def _bodies(text):
    """(name, body) of every __global__ function."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__", text):
        head = text.index("{", text.index(")", text.index("(", re.search(r"\b\w+_kernel\s*\(", text[m.end():]).end() + m.end() - 1)))
        name = re.search(r"\b(\w+_kernel)\s*\(", text[m.end():]).group(1)
        depth, at = 0, head
        while True:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
            if depth == 0:
                break
        yield name, text[head:at]


def _late(body):
    """Whether dependents are let go before the tensor memory is there."""
    alloc, go = body.find("tcgen05.alloc"), body.find("pdl_launch_dependents()")
    return alloc >= 0 and 0 <= go < alloc


SOURCES = sorted(p for p in KERNELS.glob("*.cu") if "tcgen05.alloc" in p.read_text())


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_tensor_memory_before_dependents(path):
    bodies = list(_bodies(path.read_text()))
    assert sum("tcgen05.alloc" in b for _, b in bodies) == path.read_text().count("tcgen05.alloc")
    assert [n for n, b in bodies if _late(b)] == []


def test_the_order_is_seen():
    good = "{ if (warp == 1) { asm(\"tcgen05.alloc\"); } pdl_wait(); pdl_launch_dependents(); }"
    bad = "{ pdl_wait(); pdl_launch_dependents(); asm(\"tcgen05.alloc\"); }"
    assert not _late(good) and _late(bad)
