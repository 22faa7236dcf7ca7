"""Resident blocks of the k-space pass where its dynamic shared memory fills an SM's share to the last bytes: it has
no static shared memory, which would cost a block of each."""
import os
import re

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "cuda-plasticity_b200", "csrc")
SM, BLOCK = 233472, 1024   # shared memory of an SM, and what each block reserves of it


def static_bytes():
    s = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "green.cu")).read())
    sizes = {"double": 8, "float": 4, "int": 4}
    found = re.findall(r"(?<!extern )__shared__\s+(\w+)\s+\w+(?:\[(\d+)\])?", s)
    return sum(sizes[t] * int(n or 1) for t, n in found)


def need(n, radices, slots, cols=4, velt=8):
    """FP32: component slots of n + 1 rows of `cols` values, and the twiddle rows (csrc/cdd_internal.cuh)."""
    rows, span = 0, 1
    for r in radices:
        rows += rows & 1
        pitch = r + (r & 1)
        rows += span * (pitch if r < 8 else 2 * ((pitch // 2) | 1))
        span *= r
    return (slots * (n + 1) * cols + rows) * velt


def test_blocks_that_only_just_fit():
    # axis-0 length, radices, slots (6 or 9 components and 3 of scratch) -> blocks per SM
    for n, radices, slots, blocks in [(256, (8, 8, 4), 9, 3), (256, (4, 4, 4, 4), 9, 3), (288, (8, 4, 3, 3), 12, 2)]:
        assert SM // (need(n, radices, slots) + static_bytes() + BLOCK) == blocks, (n, radices)
