"""FP64 system energy and g(r) sampling at the edges of their 128 x 128 pair
tiles, of the Q(k) chunks (32 particles) and of the FP32 screens, against the
FP64 oracle."""
import numpy as np
import pytest

from beofaunus_gb300 import workloads
from oracle.oracle import OracleSystem, atom_rdf_counts

pytestmark = pytest.mark.gpu


def system(model, n, box=None):
    if model == "salt":
        return workloads.dh_lj_salt(n, 7 + n, start="scatter")
    if model == "iso":
        p, x, q, ids = system("ewald", n)
        p.ewald_isotropic_pbc = 1
        return p, x, q, ids
    L = box or (n / 0.0037) ** (1.0 / 3.0)
    return workloads.rpm_ewald(n, L, 5, 3 + n, cutoff=0.45 * min(np.atleast_1d(L)), start="scatter")


@pytest.mark.parametrize("model,n,box", [("ewald", 31, None), ("ewald", 127, None), ("ewald", 128, None), ("ewald", 129, None),
                                         ("ewald", 385, None), ("ewald", 300, (41.0, 44.5, 47.0)), ("iso", 129, None),
                                         ("salt", 2, None), ("salt", 128, None), ("salt", 257, None)])
def test_fp64_energy_and_rdf_at_tile_edges(model, n, box):
    """Sums of at most n^2/2 FP64 terms of order 1 kT and below, a few
    roundings each: 1e-9 kT is 1e3 times their bound. Counts are exact."""
    from beofaunus_gb300.gpu import System
    p, x, q, ids = system(model, n, box)
    s, o = System(p, x, q, ids), OracleSystem(p, x, q, ids)
    e, eo = s.total_energy_fp64(), o.total_energy()
    for k in ("pairs", "reciprocal", "self", "surface", "total"):
        assert abs(e[k] - eo[k]) < 1e-9, k
    pos = s.positions()
    for t1, t2, dr, bins in ((0, 0, 0.25, 90), (0, 1, 0.25, 90), (1, 0, 1e-3, 8192), (1, 1, 7.0, 3)):
        h, t = s.rdf_sample(t1, t2, dr, bins)
        ho, to = atom_rdf_counts(pos, ids, list(p.box), t1, t2, dr, bins)
        assert t == to
        np.testing.assert_array_equal(h, ho)


def test_energy_workspace_is_bounded():
    """What a system keeps for its FP64 energy and g(r): at most 4 MB, also with
    512 chunks' worth of particles and 2242 k-vectors."""
    from beofaunus_gb300.gpu import System
    p, x, q, ids = workloads.rpm_ewald(16384, 164.0, 10, 1, start="scatter")
    s = System(p, x, q, ids)
    before = s.device_bytes
    e = s.total_energy_fp64()
    s.rdf_sample(0, 1, 0.25, 90)
    assert s.device_bytes - before <= 4 << 20
    assert s.total_energy_fp64() == e


@pytest.mark.parametrize("dr", [1e-20, 1e-35, 1e-39, 1e-45, 1e-300])
def test_rdf_bins_far_below_single_precision(dr):
    """Two ions in one place count in bin 0 at any bin width, the others nowhere."""
    from beofaunus_gb300.gpu import System
    p, x, q, ids = system("salt", 257)
    x[2] = x[0]   # both of type 0
    ids[0] = ids[2] = 0
    s = System(p, x, q, ids)
    h, t = s.rdf_sample(0, 0, dr, 4)
    n = int((ids == 0).sum())
    assert t == n * (n - 1) // 2 and list(h) == [1, 0, 0, 0]
