"""share_begin (csrc/shares.h), which gives each block of raw_screen_kernel its
patterns: the shares of any 32-bit total follow each other from 0 to the total
without a gap or an overlap, also where total x shares passes 2^32.  The header
is compiled for the host; no GPU is involved."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "cas-offinder-rust-old_b200", "csrc")
MAIN = """
#include <cstdio>
#include <cstdlib>
#include "shares.h"
int main(int argc, char **argv) {
    const uint32_t total = strtoul(argv[1], 0, 10), n = strtoul(argv[2], 0, 10);
    for (uint32_t i = 0; i <= n; ++i) printf("%u\\n", cof::share_begin(total, i, n));
}
"""


@pytest.fixture(scope="module")
def shares(tmp_path_factory):
    d = tmp_path_factory.mktemp("shares")
    src, exe = d / "shares.cpp", d / "shares"
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, str(src), "-o", str(exe)], check=True)

    def run(total, n):
        return [int(x) for x in subprocess.check_output([str(exe), str(total), str(n)]).split()]
    return run


@pytest.mark.parametrize("total,n", [(1, 1), (2, 2), (7, 3), (12, 12), (5, 8), (1000, 1184),
                                     (3_627_506, 1184), (3_627_507, 1184), (3_700_000, 1184),
                                     (2**32 - 1, 1184), (2**32 - 1, 1)])
def test_shares_partition_the_whole(shares, total, n):
    b = shares(total, n)
    assert b[0] == 0 and b[-1] == total
    size = [y - x for x, y in zip(b, b[1:])]
    assert min(size) >= 0 and max(size) - min(size) <= 1


def test_raw_screen_takes_its_patterns_from_it():
    text = open(os.path.join(CSRC, "raw.cu")).read()
    assert "share_begin(P.npat, blockIdx.y, gridDim.y)" in text
    assert "share_begin(P.npat, blockIdx.y + 1, gridDim.y)" in text
