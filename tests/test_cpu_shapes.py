"""Each single-view launch shape the library accepts has a decide kernel of its own in every pass: the shape asked for
is the one that runs. Read from the built library's symbol names."""
import re
import shutil
import subprocess

import pytest

from blitzen_gb300 import build

SHAPES = [(256, 1), (256, 2), (256, 4), (128, 2), (128, 4), (512, 1)]


@pytest.fixture(scope="module")
def kernels():
    if shutil.which("nm") is None:
        pytest.skip("no nm")
    names = subprocess.run(["nm", "-C", str(build.build())], capture_output=True, text=True, check=True).stdout
    return {tuple(int(x) for x in m) for m in re.findall(r"cull_decide_kernel<(-?\d+), true, (\d+), (\d+)>", names)}


@pytest.mark.parametrize("threads,opt", SHAPES)
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_every_pass_has_the_shape(kernels, mode, threads, opt):
    assert (mode, threads, opt) in kernels
