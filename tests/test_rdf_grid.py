"""The g(r) kernel's grid rule, compiled for the host."""
import os
import subprocess

import pytest

from conftest import ROOT

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "fg_rdf_grid.h"
int main(int, char **v) { std::printf("%lld\n", (long long)fg::rdf_blocks(std::atoll(v[1]), 152)); }
"""


@pytest.mark.parametrize("n", [2, 128, 129, 8192, 100000, 3300000, 5000000, 2 ** 24 - 1])
def test_a_blocks_pairs_fit_its_counters(tmp_path, n):
    """The most pairs of one block (tiles b, b + blocks, ... of 128 x 128) stay
    below 2^32, up to the largest system; ordinary ones fill the SMs."""
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "beofaunus_gb300", "csrc"), "-o", exe, str(tmp_path / "main.cpp")], check=True)
    blocks = int(subprocess.run([exe, str(n)], capture_output=True, text=True, check=True).stdout)
    tiles = (-(-n // 128)) ** 2
    assert -(-tiles // blocks) * 128 * 128 < 2 ** 32 and blocks < 2 ** 31
    if n <= 100000:
        assert blocks == min(tiles, 8 * 152)
