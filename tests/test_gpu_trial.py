"""The plain trial and its commit where their split changes: systems of one and
of several CTAs, particles and k-vectors around the thread count, cells, the
positive-octant k-vectors; against the FP64 oracle, accepted and rejected
trials in turn, and the exact Q(k) of the commits against a rebuild."""
import numpy as np
import pytest

from beofaunus_gb300 import workloads
from beofaunus_gb300.gpu import System
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu

CASES = {
    "rpm 2": lambda: workloads.rpm_ewald(2, 12.0, 3, 5, cutoff=5.0, start="scatter"),
    "rpm 240": lambda: workloads.rpm_ewald(240, 40.0, 5, 5, cutoff=19.0, start="scatter"),
    "rpm 1026": lambda: workloads.rpm_ewald(1026, 65.0, 7, 5, start="scatter"),      # two CTAs
    "rpm 3000 cells": lambda: workloads.rpm_ewald(3000, 93.0, 10, 5, start="scatter", use_cell_list=1),   # four
    "salt 512": lambda: workloads.dh_lj_salt(512, 6, start="scatter"),
    "salt 1030": lambda: workloads.dh_lj_salt(1030, 6, start="scatter"),
    "salt 5000": lambda: workloads.dh_lj_salt(5000, 6, start="scatter"),             # eight
}


def iso():
    p, x, q, ids = workloads.rpm_ewald(240, 40.0, 5, 5, cutoff=19.0, start="scatter")
    p.ewald_isotropic_pbc = 1
    return p, x, q, ids


@pytest.mark.parametrize("name", list(CASES) + ["octant"])
def test_trials_and_commits(name):
    data = iso() if name == "octant" else CASES[name]()
    s, o = System(*data), OracleSystem(*data)
    L, n = data[0].box[0], len(data[1])
    rng = np.random.default_rng(n)
    x = s.positions()
    for t in range(40):
        i = int(rng.integers(n))
        new = x[i] + (2.0 if t % 4 else 0.6 * L) * (rng.random(3) - 0.5)   # now and then far away, through a side
        new -= L * np.floor(new / L + 0.5)
        du, ref = s.trial_du(i, new), o.trial_du(i, new)
        # 1e-6 kT for steps of a sweep's length; close contacts by their double-float core within
        # 1e-10 of their size (dU of a far move is the difference of unrelated FP32 sums)
        assert t % 4 == 0 or abs(du - ref) < 1e-6 + 1e-10 * abs(ref), (t, du, ref)
        acc = t % 3 != 0 and du < 50.0
        s.commit(acc)
        o.commit(acc)
        if acc:
            x[i] = new
    d = s.positions() - o.positions()
    assert np.abs(d - L * np.round(d / L)).max() < 1e-9
    if not name.startswith("salt"):
        assert s.rebuild_qk() == 0.0   # exact: the rebuild finds what the commits kept
