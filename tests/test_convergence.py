"""The `.sync.aligned` instructions of the tensor memory need all 32 lanes of a
warp at once, and a branch or a loop that lanes leave one by one does not promise
that they meet again. So each of them comes after a barrier of its warp or block in the same
function, with nothing between that only some lanes run. Read from the sources:
a warp that is apart there has no defined outcome to test for."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "onion_gen_b200", "csrc")
# what splits a warp: a branch on the thread (whole warps apart), a loop that waits, a return
SPLITS = re.compile(r"\bif \((?!threadIdx\.x < 32\))[^)]*threadIdx|\bfor \((?!int )|\bwhile \(|\breturn\b|bounded_wait|fetch_constants")


def collectives():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        functions = re.split(r"(?m)^(?=(?:template|static|__device__|__global__))", text)
        for body in functions:
            for m in re.finditer(r'"(tcgen05\.[\w:.]*\.sync\.aligned)', body):
                yield os.path.basename(path), m.group(1), body[: m.start()]


@pytest.mark.parametrize("path,what,before", [pytest.param(*c, id=f"{c[0]}-{c[1]}") for c in collectives()])
def test_a_warp_is_together_at_its_collectives(path, what, before):
    barrier = [m.end() for m in re.finditer(r"__sync(?:warp|threads)\(\);", before)]
    assert barrier, "no barrier before it in its function"
    assert not SPLITS.search(before[barrier[-1]:])


def test_the_sources_hold_such_instructions():
    assert {"alloc", "dealloc", "ld", "wait::ld"} <= {what.split(".")[1] for _, what, _ in collectives()}
