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


@pytest.mark.parametrize("name", [k for k in KERNELS if "MmaAcct acct" in open(os.path.join(CSRC, k)).read()])
def test_cycle_accounting_sees_every_wait_and_issue(name):
    """Builds with -DB200FP4_ACCT split the issuing warp's cycles: every wait for an accumulator is booked as one, and every
    path through a K step books its MMAs before it goes on to the next stage."""
    text = open(os.path.join(CSRC, name)).read()
    issuer = text[text.index("MmaAcct acct; acct.start()"):text.index("acct cta" if "acct cta" in text else "acct pair")]
    assert len(re.findall(r"wait_bounded\(acc_empty_bar", issuer)) == len(re.findall(r"mark\(acct\.acc\)", issuer))
    steps = issuer.split("st.advance(")[:-1]
    assert steps and all("mark(acct.issue)" in s for s in steps)
