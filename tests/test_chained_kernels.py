"""Kernels that are resident while the kernel in front of them still writes (launch_chained) may not read through the non-coherent path:
no __ldg and no const __restrict__ parameter in them or in the device functions they share. Checked in the sources."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "phoenix_core_b200", "csrc")
FILES = ["conv_tc.cu", "conv_tf32.cu", "narrow_tc.cu", "qgemm_tc.cu"]


def _functions(text):
    """(name, text) of every function definition with a body that ends at a brace in the first column."""
    for m in re.finditer(r"^(?:static |template |__global__|__device__)[^;{}]*?(\w+)\s*\([^;{}]*\)\s*\{\n.*?^\}", text, re.S | re.M):
        yield m.group(1), m.group(0)


@pytest.mark.parametrize("name", FILES)
def test_no_noncoherent_loads(name):
    text = open(os.path.join(CSRC, name)).read()
    functions = list(_functions(text))
    assert any("chain_wait();" in body for _, body in functions)
    for fn, body in functions:
        waits = "chain_wait();" in body
        # a kernel of its own, launched without chaining, may; helpers and chained kernels may not
        alone = body.lstrip().find("__global__") >= 0 and not waits
        if alone:
            assert not re.search(r"launch_chained(_if)?\([^;]*\b%s\b" % fn, text), fn
            continue
        assert "__ldg(" not in body, fn
        if waits:
            head = body[:body.index("{\n")]
            assert not re.search(r"const \w+\*\s*__restrict__", head), fn
