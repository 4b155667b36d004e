"""Groups of trials in the molecule sweep: the shapes where the grouped path can
go wrong (molecules met twice in a group, one site per molecule, the largest
molecule, molecules longer than the cutoff, dipoles on every site, non-uniform
LJ tables, boxes with unequal sides), and systems that take turns because
their clusters do not all fit the GPU."""
import numpy as np
import pytest

from beofaunus_gb300 import workloads
from beofaunus_gb300.gpu import MolSystem, mol_draw_stream, mol_run_many
from oracle.oracle import OracleMol

pytestmark = pytest.mark.gpu


def molecules(case):
    kw = dict(n_mol=case["m"], seed=70 + case["m"], molsize=case["gs"], box=case.get("box"), cutoff=case.get("rc", 12.0))
    if "radius" in case:
        kw["mol_radius"] = case["radius"]
    p, x, mu, mus, ids = workloads.dipolar_molecules(**kw)
    if case.get("tables"):
        for t, (s, e) in enumerate(((3.5, 0.2), (3.0, 0.35), (4.0, 0.1))):
            p.type_sigma[t], p.type_eps[t] = s, e
    if case.get("skew"):   # the same coordinates in a longer, unequal box
        p.box[1] *= 1.07
        p.box[2] *= 1.21
    if case.get("dipoles"):
        rng = np.random.default_rng(5)
        mu = rng.normal(size=x.shape)
        mu /= np.linalg.norm(mu, axis=1, keepdims=True)
        mus = np.where(np.arange(len(mus)) % 3 < 2, 0.3, 0.0)
    return p, x, mu, mus, ids


CASES = [dict(m=3, gs=20, box=50.0), dict(m=17, gs=1, box=48.0), dict(m=40, gs=31, box=70.0), dict(m=33, gs=5, box=45.0, tables=True),
         dict(m=33, gs=6, box=45.0, skew=True), dict(m=20, gs=7, box=45.0, dipoles=True), dict(m=9, gs=4, box=80.0, rc=6.0, radius=14.0),
         dict(m=130, gs=9, box=75.0, tables=True, skew=True, dipoles=True)]


@pytest.mark.parametrize("cluster", [1, 4])
@pytest.mark.parametrize("case", CASES, ids=[str(i) for i in range(len(CASES))])
def test_grouped_sweep_matches_oracle(case, cluster):
    """FP32 pair terms: a few roundings (6e-8) of each near term and of the
    larger dU of a close contact: 1e-6 kT + 4e-7 |dU|."""
    p, x, mu, mus, ids = molecules(case)
    s = MolSystem(p, x, mu, mus, ids, case["gs"], cluster=cluster)
    o = OracleMol(p, x, mu, mus, ids, case["gs"])
    st = mol_draw_stream(12, case["m"], 150, 1.0, 0.3, True)
    r, ro = s.sweep(st), o.run_stream(st)
    np.testing.assert_array_equal(r["acc"], ro["acc"])
    assert np.all(np.abs(r["du"] - ro["du"]) < 1e-6 + 4e-7 * np.abs(ro["du"]))
    xyz, mu1, _ = s.state()
    xo, mo = o.state()[:2]
    L = np.array(p.box[:3])
    d = xyz - xo
    assert np.abs(d - L * np.round(d / L)).max() < 1e-9
    assert np.abs(mu1 - mo).max() < 1e-12


def test_systems_in_turns_equal_alone():
    """More clusters than the GPU holds at once, uneven streams: every system
    ends exactly where it ends alone."""
    data = [workloads.dipolar_molecules(20 + k % 3, seed=k, molsize=6) for k in range(41)]
    streams = [mol_draw_stream(900 + k, 20 + k % 3, 40 + 7 * (k % 5), 1.0, 0.3, True) for k in range(41)]
    many = [MolSystem(p, x, mu, mus, ids, 6, cluster=4) for (p, x, mu, mus, ids) in data]
    for s, st in zip(many, streams):
        s.stream_upload(st)
    per, _ = mol_run_many(many)
    for k in (0, 7, 35, 36, 40):
        p, x, mu, mus, ids = data[k]
        alone = MolSystem(p, x, mu, mus, ids, 6, cluster=4)
        r = alone.sweep(streams[k])
        assert per[k]["trials"] == len(streams[k]["u"]) and per[k]["accepted"] == r["acc"].sum()
        for a, b in zip(many[k].state(), alone.state()):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("skew", [False, True])
def test_molecule_across_the_box(skew):
    """A molecule moved half the box along every axis: what it leaves and what it
    meets are a box diagonal's half apart. FP32 terms of the near pairs."""
    case = dict(m=40, gs=5, box=70.0, dipoles=True, skew=skew)
    p, x, mu, mus, ids = molecules(case)
    s, o = MolSystem(p, x, mu, mus, ids, 5), OracleMol(p, x, mu, mus, ids, 5)
    L = np.array(p.box[:3])
    rng = np.random.default_rng(6)
    for g in range(0, 40, 2):
        new = x.reshape(-1, 5, 3)[g] + L * (0.5 - 0.04 * rng.random(3))
        new -= L * np.round(new / L)
        du, ref = s.trial_du(g, new), o.trial_du(g, new)
        s.commit(False)
        o.commit(False)
        assert abs(du - ref) < 4e-6 + 2e-6 * abs(ref), (g, du, ref)


@pytest.mark.parametrize("cluster", [1, 4])
@pytest.mark.parametrize("off", [0.0, 1e-4, 0.05, 0.3])
def test_molecule_takes_the_place_of_one_that_left(off, cluster):
    """A molecule moves onto the sites (or within `off` Angstrom of them) that
    another left a trial before: nothing of the overlap that the group saw may
    stay in its dU. A few FP32 roundings of near terms, as above."""
    gs, m, L = 4, 12, 60.0
    p, x, mu, mus, ids = workloads.dipolar_molecules(m, seed=3, molsize=gs, box=L)
    x = x.reshape(m, gs, 3)
    x[1] = x[0] - x[0, 0] + x[1, 0]   # the same conformation
    n = 8
    trans = np.zeros((n, 3))
    group = np.array([5, 0, 1, 6, 7, 8, 9, 10], np.int32)
    trans[0] = 0.3, 0.2, 0.1
    trans[1] = 14.0, 3.0, 2.0
    trans[2] = x[0, 0] - x[1, 0] + off
    trans[2] -= L * np.round(trans[2] / L)
    trans[3:] = 0.1 * np.arange(3, n)[:, None] * np.array([1.0, -1.0, 1.0])
    st = dict(group=group, axis=np.tile([0.0, 0.0, 1.0], (n, 1)), center=np.zeros(n, np.int32), angle=np.zeros(n),
              trans=trans, u=np.full(n, 1e-30))
    x = x.reshape(-1, 3)
    s = MolSystem(p, x, mu, mus, ids, gs, cluster=cluster)
    r, ro = s.sweep(st, rotate=False), OracleMol(p, x, mu, mus, ids, gs).run_stream(st, rotate=False)
    np.testing.assert_array_equal(r["acc"], ro["acc"])
    assert np.all(np.abs(r["du"] - ro["du"]) < 1e-6 + 4e-7 * np.abs(ro["du"]))


def test_empty_streams_of_more_systems_than_fit():
    p, x, mu, mus, ids = workloads.dipolar_molecules(20, seed=1, molsize=6)
    many = [MolSystem(p, x, mu, mus, ids, 6, cluster=4) for _ in range(41)]
    for s in many[::2]:   # staged with no trial, or never staged
        s.stream_upload(mol_draw_stream(1, 20, 0))
    per, tot = mol_run_many(many)
    assert tot["trials"] == 0 and all(q["trials"] == 0 and q["accepted"] == 0 for q in per)


@pytest.mark.parametrize("m", [176, 192, 208])   # 5456, 5952 and 6448 sites with a dipole on one CTA
def test_dipole_slices_up_to_the_shared_memory(m):
    p, x, mu, mus, ids = molecules(dict(m=m // 8, gs=31, box=57.5, dipoles=True))
    cells = np.array([[a, b, c] for a in (0, 1) for b in (0, 1) for c in (0, 1)]) * 57.5 - 28.75
    x, mu, mus, ids = (x[None] + cells[:, None]).reshape(-1, 3), np.tile(mu, (8, 1)), np.full(31 * m, 0.3), np.tile(ids, 8)
    for a in range(3):
        p.box[a] = 115.0
    s, o = MolSystem(p, x, mu, mus, ids, 31, cluster=1), OracleMol(p, x, mu, mus, ids, 31)
    st = mol_draw_stream(5, m, 40, 1.0, 0.3, True)
    r, ro = s.sweep(st), o.run_stream(st)
    np.testing.assert_array_equal(r["acc"], ro["acc"])
    # 31 x 31 dipole pairs with a close molecule instead of a few: four times the bound of the grouped sweeps;
    # overlaps (up to 1e10 kT): six times r^2's rounding (1.5e-7) in r^-12, twice
    assert np.all(np.abs(r["du"] - ro["du"]) < 4e-6 + 2e-6 * np.abs(ro["du"]))
    new = s.state()[0].reshape(m, 31, 3)[3] + 0.4
    assert abs(s.trial_du(3, new) - o.trial_du(3, new)) < 4e-6
    s.commit(False)


def test_a_staged_stream_runs_on_the_state_set_after_it():
    p, x, mu, mus, ids = molecules(CASES[0])
    st = mol_draw_stream(3, 3, 60, 1.0, 0.3, True)
    s = MolSystem(p, x, mu, mus, ids, 20, cluster=1)
    s.stream_upload(st)
    y = x + 1.25                       # the same molecules, shifted
    s.set_state(y, mu, mus, ids)
    per, _ = mol_run_many([s])
    ro = OracleMol(p, y, mu, mus, ids, 20).run_stream(st)
    assert per[0]["trials"] == 60 and per[0]["accepted"] == ro["acc"].sum()
    assert abs(per[0]["energy_change"] - ro["usum"]) < 60e-6
