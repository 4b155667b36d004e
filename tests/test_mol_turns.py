"""The molecule sweep's launch rule for more systems than the device runs at
once, compiled for the host."""
import os
import subprocess

import pytest

from conftest import ROOT

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "fg_mol_turns.h"
int main(int, char **v) {
    const fgm::MolTurns t = fgm::mol_turns(std::atoll(v[1]), std::atoi(v[2]), std::atoi(v[3]), 16, std::atoi(v[4]), 65536);
    std::printf("%d %lld\n", t.slots, (long long)t.quantum);
}
"""


@pytest.fixture(scope="module")
def turns(tmp_path_factory):
    d = tmp_path_factory.mktemp("turns")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover=all",
                    "-I" + os.path.join(ROOT, "beofaunus_gb300", "csrc"), "-o", str(d / "main"), str(d / "main.cpp")], check=True)

    def run(maxn, n, fit, molecules=1000):
        r = subprocess.run([str(d / "main"), str(maxn), str(n), str(fit), str(molecules)], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        return tuple(int(x) for x in r.stdout.split())
    return run


@pytest.mark.parametrize("n,fit", [(1, 36), (38, 36), (41, 36), (73, 36), (38, 0)])
def test_empty_streams_launch_nothing(turns, n, fit):
    """More systems than fit, none with a trial: all in one set, no turns."""
    assert turns(0, n, fit) == (n, 65536)


@pytest.mark.parametrize("maxn", [1, 15, 16, 17, 256, 1000, 10 ** 6, 2 ** 40])
@pytest.mark.parametrize("n", [1, 36, 37, 38, 41, 71, 72, 73, 608])
def test_every_system_gets_all_its_turns(turns, n, maxn):
    """Whole groups within a launch's limit; the rotation (launch r runs the
    systems (r slots + i) mod n) reaches every system often enough."""
    slots, quantum = turns(maxn, n, 36)
    assert quantum % 16 == 0 and 0 < quantum <= 65536 and (slots == n or slots == 36)
    if slots < n:
        per = -(-maxn // quantum)
        rounds = -(-per * n // slots)
        assert rounds * slots >= per * n


@pytest.mark.parametrize("molecules,trials,take", [(1000, 64, False), (1000, 256, True), (200, 64, False), (200, 256, True),
                                                   (200, 1024, True), (60, 64, False), (60, 1024, True), (24, 256, True),
                                                   (2, 16, False)])
def test_turns_where_they_were_faster(turns, molecules, trials, take):
    """38 systems on 36 slots, as measured (mol_turns); never for one group."""
    assert (turns(trials, 38, 36, molecules)[0] == 36) == take
