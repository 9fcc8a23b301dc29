"""An mbarrier arrival that frees shared memory or tensor memory for someone else to write must order the reads before it: no arrival in the kernels is relaxed but those that
announce bytes (expect_tx), which free nothing."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zgml_b200", "csrc")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_no_relaxed_arrival(path):
    with open(path) as f:
        arrivals = re.findall(r"mbarrier\.arrive[.\w:]*", f.read())
    assert not [a for a in arrivals if ".relaxed" in a and ".expect_tx" not in a]
