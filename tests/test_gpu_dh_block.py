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


def overlaps(n):
    """A stream with trials on top of an ion that stays (0 - 9), of one that left
    a trial before (20 - 29 follow 10 - 19) and of one of two that overlap from
    the start (30), among ordinary ones."""
    p, x, q, ids = salt(n, tables=True)
    L = p.box[0]
    rng = np.random.default_rng(n)
    v = np.array([0.6, -0.5, 0.62])
    offs = [1.8, 1.2, 0.9, 0.6, 0.4, 0.3, 0.2, 0.1, 0.05, 0.02]
    x[n - 12] = x[n - 11] + 0.3 * v
    trials = []   # particle, displacement, uniform
    for k, r in enumerate(offs):
        def onto(i, j):
            d = x[j] + r * v - x[i]
            return i, d - L * np.round(d / L), 0.5
        trials += [onto(k, n - 1 - k), (10 + k, np.array([11.0, 9.0, -8.0]), 1e-30), onto(20 + k, 10 + k)]
        trials += [(32 + 4 * k + m, 2.0 * (rng.random(3) - 0.5), rng.random()) for m in range(4)]
    trials.append((30, x[n - 11] + 0.25 * v - x[30] - L * np.round((x[n - 11] + 0.25 * v - x[30]) / L), 0.5))
    trials.append((n - 11, np.array([5.0, 6.0, -7.0]), 0.5))
    st = np.array([t[0] for t in trials], np.int32), np.array([t[1] for t in trials]), np.array([t[2] for t in trials])
    return (p, x, q, ids), st


@pytest.mark.parametrize("n", [120, 600])   # one CTA and eight
def test_overlaps(n):
    """Energies of an overlap are held to 9e15 kT and decide as they should;
    nothing stays behind of one that is gone. Long steps (1e-6 rms) to
    six times their rms; coordinates of 48 bits: L / 2^48 of r >= 0.2 Angstrom,
    times 12, is 1e-11 of the energy."""
    data, st = overlaps(n)
    r, ro = System(*data).sweep(*st), OracleSystem(*data).mc_run_stream(*st)
    np.testing.assert_array_equal(r["acc"], ro["acc"])
    held = np.abs(ro["du"]) < 9.0e15
    assert np.all(np.abs(r["du"] - ro["du"])[held] < 6e-6 + 1e-9 * np.abs(ro["du"][held]))
    assert np.all(r["du"][~held] * np.sign(ro["du"][~held]) > 8.0e15)


@pytest.mark.parametrize("n,dp,rms", [(500, 40.0, 1.0e-6), (2001, 40.0, 1.0e-6), (500, 1e9, 1.6e-6), (2001, 1e9, 2.5e-6), (16384, 1e9, 5.0e-6)])
def test_long_steps(n, dp, rms):
    """Steps of up to 40 Angstrom and of any length. Some four near pairs (within
    2 sigma) of 0.75 kT, in difference form, are off by 1.2e-7 r_o / r_n each: with
    r_o / r_n = 18 over the box of 16384 ions 3.4e-6 together, in proportion less
    in smaller boxes; far pairs, each energy by itself, add 3e-7 (6e-6 where r_n
    came from r_o). Trials on top of another ion are left to test_overlaps."""
    p, x, q, ids = salt(n)
    dp = min(dp, p.box[0])
    st = stream(n, 900, 3 * n, dp)
    keep = OracleSystem(p, x, q, ids).mc_run_stream(*st)["du"] < 10.0   # rejected trials leave the chain as it is
    st = tuple(np.ascontiguousarray(a[keep]) for a in st)
    s, o = System(p, x, q, ids), OracleSystem(p, x, q, ids)
    r, ro = s.sweep(*st), o.mc_run_stream(*st)
    np.testing.assert_array_equal(r["acc"], ro["acc"])
    assert np.sqrt(np.mean((r["du"] - ro["du"]) ** 2)) < rms
