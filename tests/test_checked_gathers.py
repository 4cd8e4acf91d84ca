"""The index-checked build guards every gather of k_node: what is read ahead of the
check of the node's corner range (before the wait for the kernel before) goes through
LULESH_IDX."""
import os
import re

from conftest import ROOT


def test_corner_list_reads_are_guarded():
    with open(os.path.join(ROOT, "lulesh.jl_gb300", "csrc", "lulesh_kernels.cu")) as f:
        src = f.read()
    body = src[src.index("k_node(DevDomain d, Params prm)"):src.index("// k_kinematics\n")]
    before, after = body.split("#ifdef LULESH_CHECK", 1)
    reads = re.findall(r"cornerList\[(.*?)\]\)", before)
    assert reads and all(r.startswith("LULESH_IDX(") for r in reads), reads
    # the range check closes over the loop's reads
    assert "t > d.nCornerList" in after and re.findall(r"cornerList\[(\w+)\]", after) == ["j"]
