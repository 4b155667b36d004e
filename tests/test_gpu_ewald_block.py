"""The Ewald block sweep where its real-space branches change: more near pairs
than their queue holds, more pairs in reach than the list holds, more cell
batches than are listed at a time, steps past the short form of the
reciprocal increments, screened Ewald (kappa > 0), non-uniform type tables, a
rebuild due inside a block; on one CTA and on a cluster, against the FP64
oracle, trial by trial."""
import numpy as np
import pytest

from beofaunus_gb300 import workloads
from beofaunus_gb300.gpu import System
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu

# Up to 60 near terms of at most 2 kT, three FP32 roundings (6e-8) each, add
# 6e-8 * 2 * 3 * sqrt(60) = 3e-6; the reciprocal sum stays within 1e-6. Core
# pairs (double-float) within 1e-9 of their size. With kappa > 0 there is no
# core table: pairs of up to 10 kT in FP32, some 30 roundings each.
TOL, TOL_KAPPA = 5e-6, 2e-5

CASES = {
    "two": dict(n=2, box=12.0, kc=4),
    "crowd": dict(n=64, box=14.0, kc=4, start_sigma=2.0),
    "list": dict(n=800, box=36.0, kc=5, start_sigma=2.0),
    "odd": dict(n=1026, box=65.0, kc=6, cutoff=9.0),
    "long steps": dict(n=200, box=40.0, kc=7, dp=30.0),
    "tables": dict(n=300, box=30.0, kc=5, start_sigma=2.0, tables=True),
    "kappa": dict(n=300, box=45.0, kc=5, kappa=True, start="rsa"),
    "rebuild each": dict(n=120, box=30.0, kc=4, update_frequency=1),
    "rebuild": dict(n=120, box=30.0, kc=4, update_frequency=7),
    "cells": dict(n=3000, box=93.0, kc=6, use_cell_list=1),
    "full cells": dict(n=6000, box=84.0, kc=5, start_sigma=2.0, use_cell_list=1),
}


@pytest.mark.parametrize("ctas", [1, 4])
@pytest.mark.parametrize("name", list(CASES))
def test_block_sweep_matches_oracle(name, ctas):
    c = dict(CASES[name])
    n, box, kc, dp = c.pop("n"), c.pop("box"), c.pop("kc"), c.pop("dp", 2.0)
    tables, kappa = c.pop("tables", False), c.pop("kappa", False)
    c.setdefault("cutoff", min(20.0, 0.49 * box))
    c.setdefault("start", "scatter")
    p, x, q, ids = workloads.rpm_ewald(n, box, kc, 11 + n, sigma=c.pop("start_sigma", 4.0), **c)
    p.type_sigma[0] = p.type_sigma[1] = 4.0
    if tables:
        p.type_sigma[0], p.type_eps[0] = 3.0, 0.35
        p.type_sigma[1], p.type_eps[1] = 4.5, 0.15
    if kappa:
        p.ewald_debye_length = 15.0
    rng = np.random.default_rng(n)
    st = (rng.integers(0, n, 200).astype(np.int32), dp * (rng.random((200, 3)) - 0.5), rng.random(200))
    s, o = System(p, x, q, ids), OracleSystem(p, x, q, ids)
    s.cluster = ctas
    r, ro = s.sweep(*st), o.mc_run_stream(*st)
    np.testing.assert_array_equal(r["acc"], ro["acc"])
    bound = (TOL_KAPPA if kappa else TOL) + 1e-9 * np.abs(ro["du"])
    judged = np.abs(ro["du"]) < 10.0 if kappa else slice(None)   # TOL_KAPPA's pairs of up to 10 kT
    assert np.all((np.abs(r["du"] - ro["du"]) < bound)[judged])
    d = s.positions() - o.positions()
    assert np.abs(d - box * np.round(d / box)).max() < 1e-9


@pytest.mark.parametrize("ctas", [1, 4])
@pytest.mark.parametrize("kappa", [False, True])
def test_place_of_an_ion_that_left(ctas, kappa):
    """Ions that move onto the place that another left a trial before: nothing
    of the overlap that the block saw may stay in their dU."""
    n, box = 200, 40.0
    p, x, q, ids = workloads.rpm_ewald(n, box, 5, 8, cutoff=19.0, start="scatter")
    if kappa:
        p.ewald_debye_length = 15.0
    rng = np.random.default_rng(9)
    trials = []
    for k, r in enumerate([1.0, 0.5, 0.2, 0.1, 0.03, 0.01, 1e-3, 1e-5, 0.0]):
        onto = x[10 + k] + r - x[30 + k]
        trials += [(10 + k, np.array([11.0, 9.0, -8.0]), 1e-30), (30 + k, onto - box * np.round(onto / box), 0.5)]
        trials += [(50 + 4 * k + m, 2.0 * (rng.random(3) - 0.5), rng.random()) for m in range(4)]
    st = np.array([t[0] for t in trials], np.int32), np.array([t[1] for t in trials]), np.array([t[2] for t in trials])
    s, o = System(p, x, q, ids), OracleSystem(p, x, q, ids)
    s.cluster = ctas
    r, ro = s.sweep(*st), o.mc_run_stream(*st)
    np.testing.assert_array_equal(r["acc"], ro["acc"])
    bound = (TOL_KAPPA if kappa else TOL) + 1e-9 * np.abs(ro["du"])
    judged = np.abs(ro["du"]) < 10.0 if kappa else slice(None)   # as above
    assert np.all((np.abs(r["du"] - ro["du"]) < bound)[judged])
