"""Properties of the kernels' sources that no run shows until a compiler makes use of their absence."""
import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = sorted(glob.glob(os.path.join(ROOT, "cyclosubfield-dbfv_gb300", "csrc", "*.cu*")))


def source(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("path", CSRC, ids=os.path.basename)
def test_copies_and_waits_order_memory(path):
    """Asynchronous copies, waits and barriers written as inline assembly clobber memory: otherwise the compiler may move
    a thread's reads of a staged slot across the wait in front of them or the next copy into the slot."""
    for stmt in re.findall(r"asm\s+volatile\s*\((.*?)\);", source(path), re.S):
        if re.search(r"cp\.async|bar\.sync|barrier|mbarrier|griddepcontrol", stmt):
            assert '"memory"' in stmt, stmt


def test_side_branches_join_before_their_tensors_go():
    """A function's tensors filled on a side stream are declared before its SideBranch: when an exception leaves the
    function, the branch's destructor joins the streams first and the tensors are freed on the caller's stream behind it."""
    text = source(os.path.join(ROOT, "cyclosubfield-dbfv_gb300", "csrc", "ring.cu"))
    bodies = re.findall(r"\bSideBranch (\w+)\(R\);(.*?)\b\1\.join\(\);", text, re.S)
    assert len(bodies) >= 4
    for name, body in bodies:
        assert not re.search(r"\n        Tensor \w+ *=", body), (name, body)


@pytest.mark.parametrize("path", CSRC, ids=os.path.basename)
def test_dynamic_shared_memory_is_aligned_for_its_widest_access(path):
    """Tiles of words hold twiddles and position pairs that are read 16 bytes at a time; a static variable may lie in front."""
    for decl in re.findall(r"extern __shared__ ([^;]*);", source(path)):
        assert "int64_t" not in decl or "__align__(16)" in decl, decl
