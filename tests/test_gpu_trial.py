"""The plain trial and its commit where their split changes: systems of one and
of several CTAs, particles and k-vectors around the thread count, cells, the
positive-octant k-vectors; against the FP64 oracle, accepted and rejected
trials in turn, and the exact Q(k) of the commits against a rebuild."""
import numpy as np
import pytest

from beofaunus_gb300 import workloads
from beofaunus_gb300.gpu import Batch, System
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


@pytest.mark.parametrize("name,vacuum", [("rpm 240", False), ("rpm 240", True), ("rpm 3000 cells", False), ("salt 1030", False)])
def test_commit_after_a_batch_run_moved_the_particle(name, vacuum):
    """The commit takes the particle from where it is, not from where it was
    when the trial was evaluated: positions, exact Q(k), cell lists and the
    surface dipole (its energy counts in vacuum) hold."""
    data = CASES[name]()
    if vacuum:
        data[0].ewald_eps_surf = 1.0
    s, o = System(*data), OracleSystem(*data)
    L, n = data[0].box[0], len(data[1])
    rng = np.random.default_rng(n + 1)
    i = n // 2
    idx = rng.integers(0, n, 200).astype(np.int32)
    idx[::4] = i
    disp = 2.0 * (rng.random((200, 3)) - 0.5)
    disp[::4, 0] = 2.5                      # through several cells
    st = (idx, disp, np.full(200, 1e-3))
    batch = Batch([s])
    batch.stream_upload(0, *st)
    new = s.positions()[i] + 0.3
    new -= L * np.floor(new / L + 0.5)
    s.trial_du(i, new)
    batch.run()
    s.commit(True)
    o.mc_run_stream(*st)
    o.trial_du(i, new)
    o.commit(True)
    d = s.positions() - o.positions()
    assert np.abs(d - L * np.round(d / L)).max() < 1e-9
    if not name.startswith("salt"):
        assert s.rebuild_qk() == 0.0
    st = (rng.integers(0, n, 300).astype(np.int32), 2.0 * (rng.random((300, 3)) - 0.5), rng.random(300))
    r, ro = s.sweep(*st), o.mc_run_stream(*st)
    np.testing.assert_array_equal(r["acc"], ro["acc"])
    # up to 60 near terms of 2 kT, three FP32 roundings each (3e-6), and the reciprocal sum (1e-6)
    assert np.all(np.abs(r["du"] - ro["du"]) < 5e-6 + 1e-9 * np.abs(ro["du"]))


@pytest.mark.parametrize("name", list(CASES) + ["octant"])
def test_far_trials(name):
    """Particles moved by up to half the box along each axis, a corner's distance
    among them: the two positions share no partners. Ewald: up to 60 near terms
    of 2 kT, three FP32 roundings each (3e-6), and the reciprocal sum (1e-6). Salt:
    the difference form of some four ions within 2 sigma, 1 kT each, off by
    2e-7 r_o / r_n < 4e-6. Overlaps within 1e-9 of their size."""
    data = iso() if name == "octant" else CASES[name]()
    s, o = System(*data), OracleSystem(*data)
    L, n = data[0].box[0], len(data[1])
    rng = np.random.default_rng(n + 2)
    x = s.positions()
    for t in range(40):
        i = int(rng.integers(n))
        step = L * (rng.random(3) - 0.5) if t % 2 else 0.5 * L * (1.0 - 0.05 * rng.random(3))
        new = x[i] + step
        new -= L * np.floor(new / L + 0.5)
        du, ref = s.trial_du(i, new), o.trial_du(i, new)
        s.commit(False)
        o.commit(False)
        assert abs(du - ref) < (1.5e-5 if name.startswith("salt") else 5e-6) + 1e-9 * abs(ref), (t, du, ref)
