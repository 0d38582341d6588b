"""Hierarchy nodes are 128 B and are indexed by an int, so a node's byte offset needs more than 32 bits
from 2^25 nodes (4 GB) on: the traversal must form addresses from the node pointer, not from a 32-bit
byte offset.  (Such a hierarchy is too large to build in a test; the address arithmetic is checked in the
source.)"""
import os
import re

from tests.conftest import ROOT


def test_node_addresses_are_64_bit():
    src = open(os.path.join(ROOT, "opticks_b200", "csrc", "phx_kernels.cuh")).read()
    src = re.sub(r"//[^\n]*", "", src)
    visit = re.search(r"PHX_D void phx_visit_node\(.*?\n}", src, flags=re.S).group(0)
    assert "reinterpret_cast<const char*>(S.bvh + ni)" in visit
    assert not re.search(r"\bni\s*(<<|\*)", visit)
