"""Rules of the kernels that no result shows reliably, read from their sources."""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "cutedsl-fully-opensourced_b200", "csrc")
KERNELS = sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*kernel.cuh")))


@pytest.mark.parametrize("name", KERNELS)
def test_one_instruction_width_per_kernel(name):
    """tcgen05.mma instructions are executed in the order of their issue only where they have one shape and one accumulator.
    A tile whose K steps came in two widths would rest on an order that nothing promises, and still add up right on most
    days: every instruction descriptor of a kernel is therefore made from one width."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    widths = set(re.findall(r"idesc_mxf\w+\(\s*([^,()]+?)\s*[,)]", text))
    assert len(widths) == 1, widths
