"""What an expired wait must not lead to: a stored tile. Every epilogue asks the status word of the call before it stores, and a loader whose
wait ran out does not announce its stage. No test can make a wait of these kernels run out (nothing may be taken out of them), so this
reads the sources."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "phoenix_core_b200", "csrc")
KERNELS = ["conv_tc.cu", "conv_tf32.cu", "narrow_tc.cu", "pointwise_tc.cu", "pointwise2_tc.cu", "qgemm_tc.cu"]


@pytest.mark.parametrize("name", KERNELS)
def test_epilogues_read_the_status_word(name):
    lines = open(os.path.join(CSRC, name)).read().split("\n")
    waits = [i for i, line in enumerate(lines) if re.search(r"mbar_wait_bounded\(.*_EPILOGUE\)", line) and "epi_bar" not in line and "if (!" not in line]
    assert waits
    for i in waits:
        assert any("warp_may_store(ok, " in line for line in lines[i:i + 4]), "%s:%d" % (name, i + 1)
    # one tile loop may do without the read (its warps would all ask at every tile); the others ask in front of their wait
    asked = sum("warp_may_store(ok, seen)" in line for line in lines)
    assert asked == sum("seen = read_status(status)" in line for line in lines) and asked >= len(waits) - (1 if name == "narrow_tc.cu" else 0)


def test_a_loader_does_not_announce_an_unfilled_stage():
    text = open(os.path.join(CSRC, "qgemm_tc.cu")).read()
    arrivals = re.findall(r"^.*mbar_arrive\(full_bar.*$", text, re.M)
    assert arrivals and all("if (ok && lane == 0)" in line for line in arrivals)
