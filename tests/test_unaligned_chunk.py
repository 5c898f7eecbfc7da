"""Bounds of the dense kernels' unaligned 16-byte chunks (csrc/unaligned_chunk.h), compiled for the host with overflow checks: no vector
past the end of the tensor, none missing, up to the largest tensor the library takes."""
import os
import subprocess


from conftest import ROOT

SOURCE = r"""
#include "unaligned_chunk.h"
#include <cstdio>
#include <cstdlib>
static void check(long long at, long long total) {
    const int n = pcb::chunk_vectors((int)at, (int)total);
    const long long first = at & ~3ll;
    const long long last_needed = at + 7 < total ? at + 7 : total - 1;      // the last element of the chunk that exists
    if (n < 1 || n > 3 || first + 4 * n > total || (first + 4 * n <= last_needed)) { std::printf("at %lld total %lld: %d vectors\n", at, total, n); std::exit(1); }
}
int main() {
    for (long long total = 4; total <= 64; total += 4)
        for (long long at = 0; at < total; ++at) check(at, total);
    const long long most = 2147483644ll;                                    // four components of 536870911 elements
    for (long long at = most - 64; at < most; ++at) check(at, most);
    return 0;
}
"""


def test_chunk_vectors(tmp_path):
    source, program = tmp_path / "chunk.cpp", tmp_path / "chunk"
    source.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fsanitize=signed-integer-overflow", "-fno-sanitize-recover=all",
                           "-I" + os.path.join(ROOT, "phoenix_core_b200", "csrc"), "-o", str(program), str(source)])
    result = subprocess.run([str(program)], capture_output=True, text=True)
    assert result.returncode == 0, result.stdout + result.stderr
