"""Cluster barriers in the kernels' sources. The .aligned forms want every lane of the warp at the instruction
together; a branch before one (a lane's write to another block, say) does not promise that, so no kernel
uses them."""
import re
from pathlib import Path

import pytest

from blitzen_gb300 import build

SOURCES = sorted(p for p in Path(build.__file__).with_name("csrc").iterdir() if p.suffix in (".cu", ".cuh"))


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_barrier_needs_a_converged_warp(path):
    assert re.findall(r"barrier\.cluster\.[a-z.]*aligned", path.read_text()) == []
