"""The Debye-Hueckel + LJ block sweep where its branches change: slices of one
particle to several warps on 1..16 CTAs, screening short enough for the
general expm1 form, image changes, non-uniform type tables, systems of uneven
size sharing the GPU; against the FP64 oracle, trial by trial."""
import numpy as np
import pytest

from beofaunus_gb300 import workloads
from beofaunus_gb300.gpu import Batch, System
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu


def salt(n, debye=10.0, tables=False):
    p, x, q, ids = workloads.dh_lj_salt(n, 40 + n, debye_length=debye, start="scatter")
    if tables:
        p.type_sigma[0], p.type_eps[0] = 3.0, 0.35
        p.type_sigma[1], p.type_eps[1] = 4.5, 0.15
    return p, x, q, ids


def stream(n, trials, seed, dp=2.0):
    rng = np.random.default_rng(seed)
    return rng.integers(0, n, trials).astype(np.int32), dp * (rng.random((trials, 3)) - 0.5), rng.random(trials)


def check(du, acc, ro):
    """dU within 1e-6 kT (FP32 difference forms); close contacts by their
    double-float core within 1e-10 of their size."""
    np.testing.assert_array_equal(acc, ro["acc"])
    assert np.all(np.abs(du - ro["du"]) < 1e-6 + 1e-10 * np.abs(ro["du"]))


@pytest.mark.parametrize("n,debye,tables", [(2, 10.0, False), (31, 10.0, False), (33, 10.0, True), (64, 3.0, False), (129, 10.0, False),
                                            (300, 3.0, True), (521, 10.0, True), (1030, 10.0, False), (1030, 3.0, False)])
def test_block_sweep_matches_oracle(n, debye, tables):
    p, x, q, ids = salt(n, debye, tables)
    s, o = System(p, x, q, ids), OracleSystem(p, x, q, ids)
    st = stream(n, 400, n)
    r, ro = s.sweep(*st), o.mc_run_stream(*st)
    check(r["du"], r["acc"], ro)
    L = p.box[0]
    d = s.positions() - o.positions()
    assert np.abs(d - L * np.round(d / L)).max() < 1e-9


def test_uneven_batch_matches_oracle():
    """Members on 1..16 CTAs each in one run, every member's trials logged."""
    sizes = [40, 90, 130, 260, 410, 900, 1500, 2600]
    data = [salt(n, tables=n % 20 == 0) for n in sizes]
    batch = Batch([System(*d) for d in data])
    streams = [stream(n, 200, 7 + n) for n in sizes]
    for m, st in enumerate(streams):
        batch.stream_upload(m, *st)
        batch.set_log(m)
    batch.run()
    for s, d, st in zip(batch.systems, data, streams):
        du, acc = s.log_get(0, 200)
        check(du, acc, OracleSystem(*d).mc_run_stream(*st))
