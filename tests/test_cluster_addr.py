"""The marked shared-memory addresses of the clustered FP64 CG (gale_b200/csrc/
gg_cluster_addr.h), compiled for the host: the mark is told from the address for every
8-byte aligned value, wherever the cluster window lies, and survives word offsets."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gale_b200", "csrc")

MAIN = r"""
#include "gg_cluster_addr.h"
#include <cstdio>
#include <initializer_list>
using namespace gg;
int main() {
    long bad = 0;
    for (unsigned long k = 0; k < (1ul << 29); k += 7) {
        const unsigned a = (unsigned)(8 * k), m = mark_remote(a);
        bad += is_remote(a) || unmarked(a) != a || !is_remote(m) || unmarked(m) != a || m == kNoAddr || a == kNoAddr;
        const unsigned o = m + 8u * 1000u;
        bad += !is_remote(o) || unmarked(o) != a + 8000u;
    }
    for (unsigned a : {0x80000000u, 0xfffffff8u, 0x7ffffff8u, 0u})
        bad += is_remote(a) || !is_remote(mark_remote(a)) || unmarked(mark_remote(a)) != a;
    std::printf("%ld\n", bad);
    return bad != 0;
}
"""


def test_mark_is_independent_of_the_address(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    src = tmp_path / "t.cpp"
    src.write_text(MAIN)
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", CSRC, str(src), "-o", str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
