"""Grids beside an SM margin (csrc/sm_share.h), compiled for the host: every cluster of two finds a TPC with both SMs free wherever the kernels lie that
the margin is for."""
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "phoenix_core_b200", "csrc")
SOURCE = r"""
#include "sm_share.h"
#include <cstdio>
int main() {
    for (int sms = 2; sms <= 160; sms += 2)
        for (int margin = 0; margin <= 64; ++margin) {
            const int pairs = pcb::pairs_beside(sms, margin), singles = pcb::sms_beside(sms, margin);
            const int whole = sms / 2 - margin;                 // TPCs that are whole with every SM of the margin in one of its own
            if (pairs < 1 || singles < 2 || (whole >= 1 && pairs != whole) || (sms - margin >= 2 && singles != sms - margin)) {
                std::printf("%d SMs, margin %d: %d pairs, %d singles\n", sms, margin, pairs, singles);
                return 1;
            }
        }
    return 0;
}
"""


def test_pairs_beside_a_margin(tmp_path):
    source, program = tmp_path / "share.cpp", tmp_path / "share"
    source.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-I" + CSRC, "-o", str(program), str(source)])
    result = subprocess.run([str(program)], capture_output=True, text=True)
    assert result.returncode == 0, result.stdout


def test_pair_grids_are_sized_in_pairs():
    for name in ("conv_tc.cu", "conv_tf32.cu"):
        text = open(os.path.join(CSRC, name)).read()
        assert not re.search(r"pair \? sm_count\(\)", text) and len(re.findall(r"pair \? sm_pairs\(\) : sm_count\(\)", text)) == 2, name
