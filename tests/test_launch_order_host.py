"""Kernels that start before their predecessor has ended (programmatic dependent launches, csrc/cdd_internal.cuh)
may read what that predecessor writes only after their wait, through coherent loads. A __restrict__ pointer or
__ldg would allow non-coherent loads and loads moved ahead of the wait, so in the sources only the tables that no
kernel writes are read that way, in every kernel and in every function that waits."""
import glob
import os
import re

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "cuda-plasticity_b200", "csrc")
TABLES = {"insts", "pre", "pre_v", "pre_g", "tw", "ktab"}   # instance table, prefix sums, twiddles, k tables


def _close(s, i, left, right):
    """Index of the bracket that closes the one at s[i]."""
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == left) - (s[j] == right)
        if depth == 0:
            return j
    raise AssertionError("unbalanced source")


def functions():
    """(file, name, parameter list, body, is a kernel) of every function definition of the device sources."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        s = re.sub(r"//[^\n]*", "", open(path).read())
        for m in reversed(list(re.finditer(r"__(launch_bounds|cluster_dims|align)__\(", s))):   # attributes
            s = s[:m.start()] + s[_close(s, m.end() - 1, "(", ")") + 1:]
        for m in re.finditer(r"(__global__|__device__)[^;{}=]*?\b(\w+)\((?=[^()]*[*&,)])", s):
            end = _close(s, m.end() - 1, "(", ")")
            body = re.match(r"\s*(const\s*)?\{", s[end + 1:])
            if not body:
                continue
            start = end + 1 + body.end() - 1
            yield os.path.basename(path), m.group(2), s[m.end():end], s[start:_close(s, start, "{", "}")], m.group(1) == "__global__"


def test_only_tables_are_read_ahead_of_the_wait():
    kernels, waiting = 0, 0
    for path, name, params, body, kernel in functions():
        waits = "pdl_wait(" in body
        kernels += kernel and path != "io.cu"
        waiting += waits
        if path != "io.cu" and (kernel or waits):   # io.cu: plain launches
            restricted = set(re.findall(r"__restrict__\s+(\w+)", params))
            assert restricted <= TABLES, (path, name, restricted - TABLES)
    assert kernels >= 15 and waiting >= 15


def test_read_only_loads_touch_tables_only():
    uses = []
    for path, name, params, body, kernel in functions():
        uses += [(path, name, a) for a in re.findall(r"__ldg\(([^;]*?)\)\s*[;<]", body)]
    assert sorted((n, a) for _, n, a in uses) == [("find_instance", "&pre[mid]"), ("stage_tw_to_smem", "src + i")], uses


def test_every_kernel_of_the_plan_streams_waits():
    """No block of a programmatically launched kernel ends without its wait (a kernel that did would let its
    successor past its predecessor): each such kernel waits itself or through the function that does its work."""
    src = "".join(open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu")))
    launched = set(re.findall(r"launch_pdl\((\w+)", src))
    bodies = {n: b for _, n, _, b, k in functions()}
    for name in launched:
        body = bodies[name]
        called = [f for f in ("march", "mean_block") if f + "<" in body or f + "(" in body]
        assert "pdl_wait(" in body or any("pdl_wait(" in bodies[f] for f in called), name
    assert len(launched) >= 15
