"""What an expired wait must not lead to: a tile stored from what it left unfinished. The epilogues of the convolution kernels ask the status word of
the call before they store. The dense kernel's CTAs keep a word of their own, which the call's only gets when they end: an epilogue asks its own, and
behind the exchange of partial tiles those of every CTA of the tile; other tiles are stored. A loader whose wait ran out does not announce its stage. No
test can make a wait of these kernels run out (nothing may be taken out of them), so this reads the sources."""
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


def test_dense_tiles_ask_every_cta_that_worked_on_them():
    text = open(os.path.join(CSRC, "qgemm_tc.cu")).read()
    # the tile function is given the CTA's own word, never the call's, which is only ORed into
    calls = re.findall(r"q_tile<[^>]*>\(p\.prob.*\);", text)
    assert len(calls) == 2 and all(c.endswith(", own_status);") for c in calls)
    assert re.findall(r"^.*\bstatus\b.*$", text[text.index("const int block = blockIdx.x;"):text.index("int q_launch(")], re.M)[-1].strip().startswith(
        "if (t == 0 && *own_status != 0) atomicOr(status, *own_status);")
    # behind the exchange: the words of all CTAs of the tile, in front of the stores
    tail = text[text.index("if (split > 1 && t < Q_LOADERS) {"):]
    asked, stored = tail.index("ld_cluster_u32(smem_u32(status), peer0 + r) == 0u"), tail.index("q_store(")
    assert asked < stored and "for (int r = 0; r < split; ++r) good = good &&" in tail[:stored] and "if (good && m < p.M)" in tail[asked:stored]
