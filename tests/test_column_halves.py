"""The columns that either half of the fp32 epilogue's warps stores (csrc/column_halves.h), compiled for the host: each column of a tile once."""
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "phoenix_core_b200", "csrc")
SOURCE = r"""
#include "column_halves.h"
#include <cstdio>
int main() {
    for (int cols = 16; cols <= 256; cols += 16) {
        int stored[256] = {0};
        const int half = pcb::columns_per_half(cols);
        for (int h = 0; h < 2; ++h)
            for (int cb = 0; cb < 4; ++cb) {
                const int col0 = h * half + cb * 32;
                if (cb * 32 >= half || col0 >= cols) break;
                for (int j = col0; j < col0 + 32 && j < cols; ++j) ++stored[j];
            }
        for (int j = 0; j < cols; ++j)
            if (stored[j] != 1) { std::printf("column %d of %d: stored %d times\n", j, cols, stored[j]); return 1; }
    }
    return 0;
}
"""


def test_each_column_once(tmp_path):
    source, program = tmp_path / "halves.cpp", tmp_path / "halves"
    source.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-I" + CSRC, "-o", str(program), str(source)])
    result = subprocess.run([str(program)], capture_output=True, text=True)
    assert result.returncode == 0, result.stdout
    assert re.search(r"const int half = columns_per_half\(p\.n_cols\);", open(os.path.join(CSRC, "conv_tf32.cu")).read())
