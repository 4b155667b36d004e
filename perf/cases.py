"""What a Monte Carlo program has this library do: the cases that its speed is judged by.

Each case is one pass of such a program through the public Python front end (beofaunus_gb300.gpu), on seeded synthetic
systems with the shapes of beofaunus_gb300.workloads: the restricted primitive model under Ewald + WCA, the
Debye-Hueckel + Lennard-Jones salt, rigid dipolar molecules, and point dipoles under the dipolar Ewald sum.

dU of the ion and molecule paths is a sum of FP32 pair terms (1e-6 kT), so those values are handed on as float32;
coordinates, FP64 energies and the point-dipole path stay in float64."""
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from beofaunus_gb300 import gpu, workloads
from beofaunus_gb300.params import FG_EWALD_DIPOLE_DIPOLE, FG_MODEL_MULTIPOLE_RF, make_params

RPM_DENSITY = 800 / 60.0 ** 3   # ions per cubic Angstrom of the 800-ion workload
SALT_DENSITY = 0.002
DP = 2.0


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the drop-in inside somebody's own move loop: one energy change and one commit per call, latency only
        {"name": "trial_rpm800", "kind": "trial", "model": "ewald", "n": 800, "kc": 7, "trials": 32},
        # a small system run alone: one sweep from the host's own random stream, dU and decisions read back
        {"name": "sweep_rpm800", "kind": "sweep", "model": "ewald", "n": 800, "kc": 7, "trials": 800},
        # a large system run alone (cell list, 2242 k-vectors): the time to equilibrate one box
        {"name": "sweep_rpm16k", "kind": "sweep", "model": "ewald", "n": 16384, "kc": 10, "trials": 2048},
        # a screened salt run alone, all pairs
        {"name": "sweep_salt2001", "kind": "sweep", "model": "salt", "n": 2001, "kc": 0, "trials": 2001},
        # many independent small boxes, one sweep each: throughput of short chains
        {"name": "batch_rpm800", "kind": "batch", "model": "ewald", "n": 800, "kc": 7, "systems": 152, "trials": 800},
        # many independent large boxes: the headline workload, a slice of a sweep with its Q(k) rebuilds
        {"name": "batch_rpm16k", "kind": "batch", "model": "ewald", "n": 16384, "kc": 10, "systems": 152, "trials": 1024},
        # a parallel-tempering ladder of replicas of uneven size, one round
        {"name": "tempering64", "kind": "tempering", "replicas": 64, "n_min": 500, "n_max": 4000, "sweeps": 2},
        # the job server: jobs of uneven size submitted, run to the end, results fetched
        {"name": "serve24", "kind": "serve", "jobs": 24, "n_min": 256, "n_max": 16384},
        # rigid molecules, one box
        {"name": "mol_1000x20", "kind": "mol", "molecules": 1000, "sites": 20, "systems": 1, "cluster": 0, "trials": 128},
        # rigid molecules, the GPU filled with independent boxes
        {"name": "mol_batch38", "kind": "mol", "molecules": 1000, "sites": 20, "systems": 38, "cluster": 4, "trials": 128},
        # point dipoles, the GPU filled with independent boxes
        {"name": "dip_batch608", "kind": "dip", "n": 100, "ions": 0, "kc": 7, "systems": 608, "trials": 1024},
        # between sweeps of an NPT run: the FP64 energy, g(r) and a volume move
        {"name": "npt_rpm8k", "kind": "npt", "model": "ewald", "n": 8192, "kc": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trial", "sweep", "sweep", "batch", "batch", "tempering", "serve", "mol", "mol", "dip", "dip", "npt"])
    model = rng.choice(["ewald", "salt"])
    c = {"kind": kind}
    if kind in ("trial", "sweep", "batch"):
        n = _log_int(rng, 100, 16384)
        c.update(model=model, n=n, kc=rng.randint(5, 10) if model == "ewald" else 0)
        c["trials"] = rng.randint(8, 48) if kind == "trial" else _log_int(rng, 100, 2048)
        if kind == "batch":
            c["systems"] = _log_int(rng, 8, 152)
            per = n * n / 5e7 if model == "salt" else 1.0   # a salt trial sums all N partners
            c["trials"] = max(33, min(c["trials"], int(1024 / max(1.0, 4 * per))))
    elif kind == "tempering":
        c.update(replicas=rng.randint(8, 64), n_min=rng.randint(200, 700), n_max=rng.randint(900, 4000), sweeps=rng.randint(1, 2))
    elif kind == "serve":
        c.update(jobs=rng.randint(6, 24), n_min=rng.randint(200, 400), n_max=rng.randint(1000, 16384))
    elif kind == "mol":
        c.update(molecules=_log_int(rng, 60, 1000), sites=rng.randint(3, 24), cluster=0, systems=1, trials=rng.randint(16, 160))
        if rng.random() < 0.5:
            c.update(systems=rng.randint(4, 38), cluster=4, trials=rng.randint(32, 128))
    elif kind == "dip":
        c.update(n=rng.randint(40, 160), kc=rng.randint(5, 7), ions=rng.choice([0, 0, 10, 20]), trials=rng.randint(64, 1024))
        c["systems"] = rng.choice([1, _log_int(rng, 16, 608)])
    else:
        c.update(model=model, n=_log_int(rng, 500, 8192), kc=rng.randint(5, 8) if model == "ewald" else 0)
    return c


# ------------------------------------------------------------------ inputs
def _rng(seed, *more):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, *more])


def _box(model, n):
    return (n / (RPM_DENSITY if model == "ewald" else SALT_DENSITY)) ** (1.0 / 3.0)


def _ions(case, seed, n=None, model=None, kT=1.0, start=None):
    """(params, xyz, charges, type ids) of one salt of n ions."""
    n, model = n or case["n"], model or case["model"]
    L = _box(model, n)
    if start is None:
        start = workloads.scatter_positions(n, L, 4.0, int(_rng(seed, 1).integers(1 << 31)))
    if model == "ewald":
        return workloads.rpm_ewald(n, L, case["kc"], 0, cutoff=min(20.0, 0.49 * L), start=start)
    return workloads.dh_lj_salt(n, 0, kT_scale=kT, start=start)


def _image(xyz, L, rng):
    """Another box with the same structure: axes permuted, reflected and shifted, ions in the same order."""
    x = xyz[:, rng.permutation(3)] * rng.choice([-1.0, 1.0], 3) + rng.uniform(-0.5, 0.5, 3) * L
    return x - L * np.round(x / L)


def _stream(rng, n, trials):
    return rng.integers(0, n, trials).astype(np.int32), DP * (rng.random((trials, 3)) - 0.5), rng.random(trials)


def _sizes(case, count):
    """Even and odd particle counts, log-uniform; the smallest and the largest of the range are always there."""
    n = np.exp(_rng(case["n_min"] + case["n_max"], 2).uniform(math.log(case["n_min"]), math.log(case["n_max"]), count)).astype(int)
    n[0], n[-1] = case["n_min"], case["n_max"]
    return [int(v) for v in n]


def _temperatures(case):
    return workloads.pt_temperatures(case["replicas"])


def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def _rotate(v, axis, angle):
    """v rotated about the unit vector axis (Rodrigues)."""
    c, s = np.cos(angle), np.sin(angle)
    return v * c + np.cross(axis, v) * s + axis * (v @ axis)[..., None] * (1.0 - c)


def _molecules(case, seed):
    """(params, mass centres [M, 3], offsets [M, gs, 3], dipoles [M, 3], types [M, gs]): rigid molecules of gs sites in
    a ball of 4 Angstrom, charges -1/0/+1 with net 0, one point dipole of 1.5 e Angstrom on the first site."""
    M, gs = case["molecules"], case["sites"]
    rng = _rng(seed, 3)
    L = 150.0 * (M / 1000.0) ** (1.0 / 3.0)
    shapes = np.stack([workloads.molecule_conformation(rng, gs, 4.0, 2.0) for _ in range(16)])
    off = shapes[rng.integers(0, len(shapes), M)]
    a, w = _unit(rng.normal(size=(M, 3))), rng.uniform(0, 2 * math.pi, M)
    off = np.stack([_rotate(off[m], a[m], w[m]) for m in range(M)])
    q = rng.integers(-1, 2, (M, gs // 2))
    q = np.concatenate([q, -q, np.zeros((M, gs - 2 * (gs // 2)), dtype=q.dtype)], axis=1)
    types = rng.permuted(q, axis=1).astype(np.int32) + 1
    centres = workloads.scatter_positions(M, L, 11.5, int(rng.integers(1 << 31)))
    kinds = [dict(q=float(v), sigma=3.5, eps=0.2) for v in (-1, 0, 1)]
    p = make_params(FG_MODEL_MULTIPOLE_RF, L, 7.1, kinds, rf_cutoff=min(15.0, 0.45 * L), rf_eps_rf=1e11,
                    rf_eps_r=workloads.bjerrum_unit(298.0) / 7.1)
    return p, centres, off, _unit(rng.normal(size=(M, 3))), types


def _mol_box(case, seed, b):
    p, cm, off, mu, types = _molecules(case, seed)
    if b:
        rng, L = _rng(seed, 4, b), p.box[0]
        turn, sign, shift = rng.permutation(3), rng.choice([-1.0, 1.0], 3), rng.uniform(-0.5, 0.5, 3) * L
        cm, off, mu = cm[:, turn] * sign + shift, off[:, :, turn] * sign, mu[:, turn] * sign
        cm = cm - L * np.round(cm / L)
    return p, cm, off, mu, types


def _mol_stream(case, seed, b):
    rng, T = _rng(seed, 5, b), case["trials"]
    return dict(group=rng.integers(0, case["molecules"], T).astype(np.int32), axis=_unit(rng.normal(size=(T, 3))),
                center=np.zeros(T, np.int32), angle=0.3 * (rng.random(T) - 0.5), trans=rng.random((T, 3)) - 0.5, u=rng.random(T))


def _mol_system(case, seed, b):
    p, cm, off, mu, types = _mol_box(case, seed, b)
    M, gs, L = case["molecules"], case["sites"], p.box[0]
    x = (cm[:, None, :] + off).reshape(-1, 3)
    x = x - L * np.round(x / L)
    mu_u, mu_s = np.zeros((M * gs, 3)), np.zeros(M * gs)
    mu_u[::gs], mu_s[::gs] = mu, 1.5
    return gpu.MolSystem(p, x, mu_u, mu_s, types.reshape(-1), gs, mass_centers=cm, cluster=case["cluster"])


def _dipoles(case, seed, b):
    terms = 7 if case["ions"] else FG_EWALD_DIPOLE_DIPOLE
    p, x, mu, mus, ids, q = workloads.dipolar_fluid(n=case["n"], seed=int(_rng(seed, 6).integers(1 << 31)), kc=float(case["kc"]),
                                                    n_ions=case["ions"], terms=terms)
    if b:
        rng, L = _rng(seed, 7, b), p.box[0]
        x, mu = _image(x, L, rng), _unit(rng.normal(size=mu.shape))
    return p, x, mu, mus, ids, q


def _dip_stream(case, seed, b):
    rng, T, n = _rng(seed, 8, b), case["trials"], case["n"]
    return dict(kind=rng.integers(1, 3, T).astype(np.int32), idx=rng.integers(0, n, T).astype(np.int32),
                axis=_unit(rng.normal(size=(T, 3))), angle=1.5 * math.pi * (rng.random(T) - 0.5),
                disp=0.7 * (rng.random((T, 3)) - 0.5), u=rng.random(T))


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, s.seed, s.passes = case, int(seed), 0
    kind = case["kind"]
    if kind in ("trial", "sweep", "npt"):
        s.params, s.xyz, q, ids = _ions(case, seed)
        s.system = gpu.System(s.params, s.xyz, q, ids)
        if kind != "npt":
            s.stream = _stream(_rng(seed, 9), case["n"], case["trials"])
    elif kind == "batch":
        p, xyz, q, ids = _ions(case, seed)
        s.systems = [gpu.System(p, xyz if b == 0 else _image(xyz, p.box[0], _rng(seed, 10, b)), q, ids) for b in range(case["systems"])]
        s.batch = gpu.Batch(s.systems)
        s.batch.set_log(0)
        s.batch.set_log(case["systems"] - 1)
    elif kind == "tempering":
        s.systems = [gpu.System(*_ions(case, seed + 7919 * r, n=n, model="salt")) for r, n in enumerate(_sizes(case, case["replicas"]))]
        s.batch = gpu.Batch(s.systems)
        s.batch.pt_setup(_temperatures(case), s.seed & 0x7FFFFFFF)
    elif kind == "serve":
        s.jobs = [_ions(case, seed + 7919 * j, n=n, model="salt", kT=float(t))
                  for j, (n, t) in enumerate(zip(_sizes(case, case["jobs"]), workloads.pt_temperatures(case["jobs"])))]
        s.server = gpu.Server(8 << 30)
    elif kind == "mol":
        s.systems = [_mol_system(case, seed, b) for b in range(case["systems"])]
        s.streams = [_mol_stream(case, seed, b) for b in range(case["systems"])]
    else:
        s.systems = []
        for b in range(case["systems"]):
            p, x, mu, mus, ids, q = _dipoles(case, seed, b)
            s.systems.append(gpu.DipoleSystem(p, x, mu, mus, ids, charges=q))
        s.streams = [_dip_stream(case, seed, b) for b in range(case["systems"])]
    if kind in ("mol", "dip") and case["systems"] > 1:
        s.pool = ThreadPoolExecutor(16)   # streams of many boxes are staged from several host threads
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    out = globals()["_run_" + s.case["kind"]](s)
    s.passes += 1
    return out


def _wrap(x, L):
    return x - L * np.floor(x / L + 0.5)


def _run_trial(s):
    """A host move loop: propose, ask for dU, decide, commit."""
    idx, disp, u = s.stream
    L, dus, accs = s.params.box[0], [], []
    for t in range(len(idx)):
        i = int(idx[t])
        new = _wrap(s.xyz[i] + disp[t], L)
        du = s.system.trial_du(i, new)
        acc = not u[t] > math.exp(min(0.0, -du))
        s.system.commit(acc)
        if acc:
            s.xyz[i] = new
        dus.append(du)
        accs.append(acc)
    return {"du": np.array(dus, np.float32), "acc": np.array(accs, np.int32), "xyz": s.system.positions()}


def _run_sweep(s):
    r = s.system.sweep(*s.stream)
    return {"du": r["du"].astype(np.float32), "acc": r["acc"].astype(np.int32), "xyz": s.system.positions()}


def _stats(per):
    return (np.array([p["accepted"] for p in per]), np.array([p["energy_change"] for p in per]))


def _run_batch(s):
    T = s.case["trials"]
    s.batch.stream_philox([T] * len(s.systems), (s.seed + s.passes) & 0x7FFFFFFF)
    per, _ = s.batch.run()
    acc, de = _stats(per)
    du0, acc0 = s.systems[0].log_get(0, T)
    du1, acc1 = s.systems[-1].log_get(0, T)
    return {"accepted": acc, "energy_change": de.astype(np.float32), "du0": du0.astype(np.float32), "acc0": acc0.astype(np.int32),
            "xyz0": s.systems[0].positions(), "du1": du1.astype(np.float32), "acc1": acc1.astype(np.int32), "xyz1": s.systems[-1].positions()}


def _run_tempering(s):
    tot = s.batch.pt_run(1, s.case["sweeps"])
    st = s.batch.pt_state()
    return {"accepted": tot["accepted"], "perm": st["perm"], "energies": st["energies"].astype(np.float32), "attempts": st["attempts"],
            "accepts": st["accepts"], "xyz0": s.systems[0].positions(), "xyz1": s.systems[-1].positions()}


def _run_serve(s):
    ids = []
    for j, (p, xyz, q, types) in enumerate(s.jobs):
        ids.append(s.server.submit(p, xyz, q, types, (s.seed + 1000 * s.passes + j) & 0x7FFFFFFF, len(xyz)))
    left = len(ids)
    while left:
        left -= s.server.step()[1]
    res = [s.server.poll(i, positions=True) for i in ids]
    for i in ids:
        s.server.release(i)
    return {"accepted": np.array([r["accepted"] for r in res]), "energy": np.array([r["energy"] for r in res], np.float32),
            "xyz": np.concatenate([r["xyz"] for r in res[1:]]), "xyz0": res[0]["xyz"]}


def _run_mol(s):
    if len(s.systems) == 1:
        r = s.systems[0].sweep(s.streams[0])
        xyz, mu, cm = s.systems[0].state()
        return {"du": r["du"].astype(np.float32), "acc": r["acc"].astype(np.int32), "xyz": xyz, "mu": mu, "cm": cm}
    list(s.pool.map(lambda m, st: m.stream_upload(st), s.systems, s.streams))
    per, _ = gpu.mol_run_many(s.systems)
    acc, de = _stats(per)
    xyz, mu, cm = s.systems[0].state()
    return {"accepted": acc, "energy_change": de.astype(np.float32), "xyz": xyz, "mu": mu, "cm": cm}


def _run_dip(s):
    if len(s.systems) == 1:
        r = s.systems[0].sweep(s.streams[0])
        xyz, mu = s.systems[0].state()
        return {"du": r["du"], "acc": r["acc"].astype(np.int32), "xyz": xyz, "mu": mu}
    list(s.pool.map(lambda d, st: d.stream_upload(st), s.systems, s.streams))
    per, _ = gpu.dip_run_many(s.systems)
    acc, de = _stats(per)
    xyz, mu = s.systems[0].state()
    return {"accepted": acc, "energy_change": de, "xyz": xyz, "mu": mu}


def _rdf_bins(L):
    return int(0.5 * L / 0.25)


def _npt_move(s_seed, passes):
    rng = _rng(s_seed, 11, passes)
    return float(rng.uniform(-0.5, 0.5)), float(rng.random())


def _pressure(case):
    return 1.2 * (RPM_DENSITY if case["model"] == "ewald" else SALT_DENSITY)


def _run_npt(s):
    e = s.system.total_energy_fp64()
    bins = _rdf_bins(_box(s.case["model"], s.case["n"]))
    like, n_like = s.system.rdf_sample(0, 0, 0.25, bins)
    unlike, n_unlike = s.system.rdf_sample(0, 1, 0.25, bins)
    half, u = _npt_move(s.seed, s.passes)
    du, acc = s.system.volume_move(half, 0.004, _pressure(s.case), u)
    return {"energy": np.array([e["pairs"], e["reciprocal"], e["self"], e["surface"], e["total"], du]), "like": like, "unlike": unlike,
            "pairs": np.array([n_like, n_unlike]), "accepted": int(acc), "xyz": s.system.positions()}


# ------------------------------------------------------------------ work
def _kvectors(kc, iso=False):
    r = np.arange(-kc, kc + 1)
    x, y, z = np.meshgrid(np.arange(0, kc + 1), r, r, indexing="ij")
    n2 = x * x + y * y + z * z
    keep = (n2 > 0) & (n2 <= kc * kc)
    return np.stack([x[keep], y[keep], z[keep]], axis=1)


def _trial_flops(model, n, kc):
    """One single-particle trial: the pair terms at both positions, and under Ewald every k-vector's increment."""
    if model == "salt":
        return 60.0 * (n - 1)
    L = _box("ewald", n)
    near = min(n - 1, 4.0 / 3.0 * math.pi * min(20.0, 0.49 * L) ** 3 * RPM_DENSITY)
    return 80.0 * near + (65.0 + 0.75 * 23.0) * len(_kvectors(kc))


def _state_bytes(model, n, kc):
    return 40.0 * n + (36.0 * len(_kvectors(kc)) if model == "ewald" else 0.0)


def work(case):
    kind = case["kind"]
    if kind in ("trial", "sweep", "batch"):
        T, B = case["trials"], case.get("systems", 1)
        return {"bytes": B * (_state_bytes(case["model"], case["n"], case["kc"]) + 45.0 * T), "flops": B * T * _trial_flops(case["model"], case["n"], case["kc"])}
    if kind in ("tempering", "serve"):
        count = case["replicas"] if kind == "tempering" else case["jobs"]
        sizes = _sizes(case, count)
        per = case["sweeps"] if kind == "tempering" else 1
        return {"bytes": sum(_state_bytes("salt", n, 0) + 45.0 * n * per for n in sizes), "flops": sum(n * per * _trial_flops("salt", n, 0) for n in sizes)}
    if kind == "mol":
        M, gs = case["molecules"], case["sites"]
        N, B, T = M * gs, case["systems"], case["trials"]
        near = min(N - gs, 4.0 / 3.0 * math.pi * 15.0 ** 3 * N / (150.0 ** 3 * M / 1000.0))
        flops = 2.0 * gs * (N - gs) * 15 + 2.0 * ((N - gs) + gs * (M - 1)) * 20 + 2.0 * gs * near * 40
        return {"bytes": B * (N * 96.0 + T * 85.0), "flops": B * T * flops}
    if kind == "dip":
        n, B, T = case["n"], case["systems"], case["trials"]
        K = len(_kvectors(case["kc"]))
        return {"bytes": B * (n * 68.0 + K * 44.0 + T * 77.0), "flops": B * T * (2.0 * (n - 1) * (15 + 0.45 * 80) + 56.0 * K)}
    n, L = case["n"], _box(case["model"], case["n"])
    near = n * n / 2 * (min(1.0, 4.0 / 3.0 * math.pi * min(20.0, 0.49 * L) ** 3 / L ** 3) if case["model"] == "ewald" else 1.0)
    K = len(_kvectors(case["kc"])) if case["model"] == "ewald" else 0
    return {"bytes": 4 * 40.0 * n, "flops": 3 * near * 40.0 + 0.75 * n * n / 2 * 10.0 + 3.0 * n * K * 10.0}


# ------------------------------------------------------------------ the same in 64 bits
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(x):
    return torch.as_tensor(np.asarray(x, dtype=np.float64), device=_dev())


def _philox(seed, stream, first, count, word):
    """Philox4x32-10 (Salmon et al., SC'11): counters (first .. first + count, 0, word, 0), key (seed, stream)."""
    g = np.arange(first, first + count, dtype=np.uint64)
    m32 = np.uint64(0xFFFFFFFF)
    c = [g & m32, g >> np.uint64(32), np.full(count, word, np.uint64), np.zeros(count, np.uint64)]
    k0, k1 = int(seed) & 0xFFFFFFFF, int(stream) & 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _device_stream(seed, stream, n, L, trials):
    """The library's device-generated trials: particle, displacement, Metropolis uniform."""
    r, r2 = _philox(seed, stream, 0, trials, 0), _philox(seed, stream, 0, trials, 1)
    idx = ((r[0] * np.uint64(n)) >> np.uint64(32)).astype(np.int64)
    step = round(DP / L * 2.0 ** 32)
    d = np.stack([(r[a].astype(np.float64) - 2.0 ** 31) * step for a in (1, 2, 3)], axis=1) * (L / 2.0 ** 64)
    return idx, d, (r2[0].astype(np.float64) + 0.5) / 2.0 ** 32


class _Chain:
    """One box of ions in 64 bits: Ewald + WCA or Debye-Hueckel + LJ, one translation at a time."""

    def __init__(self, model, n, xyz, kc, L):
        self.model, self.L, self.lB = model, L, 7.1
        self.x = _t(xyz)
        self.q = _t(np.where(np.arange(n) < n // 2, 1.0, -1.0))
        if model == "ewald":
            self.alpha, self.rc = 0.2, min(20.0, 0.49 * L)
            k = 2 * math.pi * _kvectors(kc) / L
            k2 = (k * k).sum(axis=1)
            self.k = _t(k)
            self.A = _t(np.where(_kvectors(kc)[:, 0] > 0, 2.0, 1.0) * np.exp(-k2 / (4 * self.alpha ** 2)) / k2) * (2 * math.pi * self.lB / L ** 3)
            self.Q = torch.zeros(len(k), dtype=torch.complex128, device=_dev())
            for a in range(0, n, 2048):
                ph = self.x[a:a + 2048] @ self.k.T
                self.Q += (self.q[a:a + 2048, None] * torch.complex(torch.cos(ph), torch.sin(ph))).sum(dim=0)
            self.surf = 2 * math.pi * self.lB / ((2e11 + 1) * L ** 3)

    def pair(self, r2, qq):
        r = torch.sqrt(r2)
        if self.model == "ewald":
            u = torch.where(r2 <= self.rc ** 2, qq * self.lB * torch.special.erfc(self.alpha * r) / r, 0.0)
            y = (16.0 / r2) ** 3
            return u + torch.where(r2 <= 16.0 * 2 ** (1 / 3), 0.4 * (y * y - y + 0.25), 0.0)
        y = (16.0 / r2) ** 3
        return qq * self.lB / r * torch.exp(-r / 10.0) + 0.8 * (y * y - y)

    def near(self, i, at):
        d = self.x - at
        d = d - self.L * torch.round(d / self.L)
        r2 = (d * d).sum(dim=1)
        r2[i] = 1e12
        return self.pair(r2, self.q[i] * self.q).sum()

    def trial(self, i, d):
        old = self.x[i].clone()
        new = old + d
        new = new - self.L * torch.floor(new / self.L + 0.5)
        du, D = self.near(i, new) - self.near(i, old), None
        if self.model == "ewald":
            po, pn = self.k @ old, self.k @ new
            D = self.q[i] * torch.complex(torch.cos(pn) - torch.cos(po), torch.sin(pn) - torch.sin(po))
            du = du + (self.A * (2 * (self.Q.conj() * D).real + (D * D.conj()).real)).sum()
            m, dm = self.q @ self.x, self.q[i] * (new - old)
            du = du + self.surf * (2 * (m @ dm) + dm @ dm)
        return float(du), new, D

    def run(self, idx, disp, u, kT=1.0):
        du, acc = np.empty(len(idx)), np.zeros(len(idx), np.int32)
        disp = _t(disp)
        for t in range(len(idx)):
            i = int(idx[t])
            du[t], new, D = self.trial(i, disp[t])
            if not (u[t] > 0 and du[t] > -kT * math.log(u[t])):
                acc[t] = 1
                self.x[i] = new
                if D is not None:
                    self.Q += D
        return du, acc

    def energies(self):
        """(pairs, reciprocal, self, surface, total)"""
        n, pairs = len(self.x), 0.0
        for a in range(0, n, 512):
            d = self.x[a:a + 512, None, :] - self.x[None, :, :]
            d = d - self.L * torch.round(d / self.L)
            r2 = (d * d).sum(dim=2)
            i = torch.arange(a, min(a + 512, n), device=_dev())
            r2[torch.arange(n, device=_dev())[None, :] <= i[:, None]] = 1e12
            pairs += float(self.pair(r2, self.q[a:a + 512, None] * self.q[None, :]).sum())
        if self.model != "ewald":
            return np.array([pairs, 0.0, 0.0, 0.0, pairs])
        rec = float((self.A * (self.Q * self.Q.conj()).real).sum())
        own = -self.alpha / math.sqrt(math.pi) * n * self.lB
        m = self.q @ self.x
        srf = self.surf * float(m @ m)
        return np.array([pairs, rec, own, srf, srf + rec + own + pairs])


def _exact_ions(case, seed):
    p, xyz, _, _ = _ions(case, seed)
    return _Chain(case["model"], case["n"], xyz, case["kc"], p.box[0]), p.box[0]


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, int(seed))


def _exact_trial(case, seed):
    c, _ = _exact_ions(case, seed)
    du, acc = c.run(*_stream(_rng(seed, 9), case["n"], case["trials"]))
    return {"du": du, "acc": acc, "xyz": c.x.cpu().numpy()}


_exact_sweep = _exact_trial


def _exact_batch(case, seed):
    c, L = _exact_ions(case, seed)
    du, acc = c.run(*_device_stream(seed & 0x7FFFFFFF, 0, case["n"], L, case["trials"]))
    return {"accepted": None, "energy_change": None, "du0": du, "acc0": acc, "xyz0": c.x.cpu().numpy(), "du1": None, "acc1": None, "xyz1": None}


def _exact_tempering(case, seed):
    n = _sizes(case, case["replicas"])[0]
    p, xyz, _, _ = _ions(case, seed, n=n, model="salt")
    c = _Chain("salt", n, xyz, 0, p.box[0])
    c.run(*_device_stream(seed & 0x7FFFFFFF, 0, n, p.box[0], case["sweeps"] * n), kT=float(_temperatures(case)[0]))
    return {"accepted": None, "perm": None, "energies": None, "attempts": None, "accepts": None, "xyz0": c.x.cpu().numpy(), "xyz1": None}


def _exact_serve(case, seed):
    n = _sizes(case, case["jobs"])[0]
    p, xyz, _, _ = _ions(case, seed, n=n, model="salt")
    c = _Chain("salt", n, xyz, 0, p.box[0])
    c.run(*_device_stream(seed & 0x7FFFFFFF, 0, n, p.box[0], n), kT=float(workloads.pt_temperatures(case["jobs"])[0]))
    return {"accepted": None, "energy": None, "xyz": None, "xyz0": c.x.cpu().numpy()}


def _exact_mol(case, seed):
    p, cm, off, mu, types = _mol_box(case, seed, 0)
    st = _mol_stream(case, seed, 0)
    M, gs, L = case["molecules"], case["sites"], p.box[0]
    lB, rc, rfB = 7.1, p.rf_cutoff, -(2 * (p.rf_eps_rf - p.rf_eps_r) / (2 * p.rf_eps_rf + p.rf_eps_r)) / p.rf_eps_r
    a2 = -66.0 * 1494.0 / 56916.0
    X, q, dip = _t((cm[:, None, :] + off).reshape(-1, 3)), _t(types.reshape(-1) - 1.0), _t(1.5 * mu)
    mol = torch.arange(M * gs, device=_dev()) // gs

    def energy(g, x, m):
        """Molecule g with sites x and dipole m against all others."""
        d = x[:, None, :] - X[None, :, :]
        d = d - L * torch.round(d / L)
        r2 = (d * d).sum(dim=2)
        r2[:, mol == g] = 1e12
        r = torch.sqrt(r2)
        y = (3.5 ** 2 / r2) ** 3
        w = r / rc
        gal = (w - 1) ** 3 * (5 / 22 * w * w * a2 + 9 / 22 * w * a2 - 0.6 * w * w - 1.2 * w - 1)
        qi = q[g * gs:(g + 1) * gs]
        u = (0.8 * (y * y - y) + torch.where(r < rc, lB * qi[:, None] * q[None, :] / r * gal, 0.0)).sum()
        dk, rk = d[:, ::gs, :], r[:, ::gs]
        u = u + lB * (qi[:, None] * (dk * dip[None]).sum(dim=2) / rk ** 3).sum()   # its charges, the others' dipoles
        u = u - lB * (q * (d[0] @ m) / r[0] ** 3).sum()                             # its dipole, the others' charges
        v, s = dk[0], rk[0]
        t = 3 * (v @ m) * (v * dip).sum(dim=1) / s ** 2 - dip @ m + (dip @ m) * rfB * (s / rc) ** 3
        return u + torch.where(s < rc, -lB * t / s ** 3, 0.0).sum()

    du, acc = np.empty(case["trials"]), np.zeros(case["trials"], np.int32)
    cm, off, mu = cm.copy(), off.copy(), mu.copy()
    for t in range(case["trials"]):
        g = int(st["group"][t])
        o = _rotate(off[g], st["axis"][t], st["angle"][t])
        m = _rotate(mu[g][None], st["axis"][t], st["angle"][t])[0]
        c = _wrap(cm[g] + st["trans"][t], L)
        x = _t(c + o)
        du[t] = float(energy(g, x, _t(1.5 * m)) - energy(g, X[g * gs:(g + 1) * gs].clone(), dip[g].clone()))
        if not du[t] > -math.log(st["u"][t]):
            acc[t], cm[g], off[g], mu[g] = 1, c, o, m
            X[g * gs:(g + 1) * gs], dip[g] = x, _t(1.5 * m)
    mus = np.zeros((M * gs, 3))
    mus[::gs] = mu
    out = {"xyz": _wrap(X.cpu().numpy(), L), "mu": mus, "cm": cm}
    if case["systems"] == 1:
        return {"du": du, "acc": acc, **out}
    return {"accepted": None, "energy_change": None, **out}


def _exact_dip(case, seed):
    p, x, mu, mus, ids, q = _dipoles(case, seed, 0)
    st = _dip_stream(case, seed, 0)
    n, L, lB, al, rc = case["n"], p.box[0], p.bjerrum, p.ewald_alpha, p.ewald_cutoff
    k = 2 * math.pi * _kvectors(case["kc"]) / L
    k2 = (k * k).sum(axis=1)
    A = np.where(k[:, 0] > 0, 2.0, 1.0) * np.exp(-k2 / (4 * al * al)) / k2 * (2 * math.pi * lB / L ** 3)
    surf = 2 * math.pi * lB / ((2 * p.ewald_eps_surf + 1) * L ** 3)
    ion, dd = bool(case["ions"]), True
    ch = q if ion else np.zeros(n)
    x, mu = x.copy(), mu.copy()
    erfc = np.vectorize(math.erfc)

    def terms(r, m):
        e = np.exp(1j * (r @ k.T))
        return e * (0.0 + 1j * (m @ k.T)), e   # dipole factor, ion factor

    def near(i, r, m):
        d = r - np.delete(x, i, axis=0)
        d -= L * np.round(d / L)
        r2 = (d * d).sum(axis=1)
        s = np.sqrt(r2)
        w = np.delete(mu * mus[:, None], i, axis=0)
        qj = np.delete(ch, i)
        y = (p.type_sigma[0] ** 2 / r2) ** 3
        u = 4 * p.type_eps[0] * (y * y - y)
        ex, ec = np.exp(-al * al * r2), erfc(al * s)
        t1 = s * 2 * al / math.sqrt(math.pi) * ex + ec
        t2 = 3 * (t1 + 4 * al ** 3 / 3 / math.sqrt(math.pi) * s ** 3 * ex)
        e = ch[i] * qj * ec / s
        if ion:
            e = e + (ch[i] * (d * w).sum(axis=1) - qj * (d @ m)) * t1 / s ** 3
        e = e - ((d @ m) * (w * d).sum(axis=1) * t2 / s ** 5 - (w @ m) * t1 / s ** 3)
        return float((u + np.where(r2 <= rc * rc, lB * e, 0.0)).sum())

    fd, fi = terms(x, mu * mus[:, None])
    Q = fd.sum(axis=0) + (ch[:, None] * fi).sum(axis=0)
    S = (ch[:, None] * x + mu * mus[:, None]).sum(axis=0)
    du, acc = np.empty(case["trials"]), np.zeros(case["trials"], np.int32)
    for t in range(case["trials"]):
        i = int(st["idx"][t])
        rn, un = x[i], mu[i]
        if st["kind"][t] == 1:
            un = _rotate(mu[i][None], st["axis"][t], st["angle"][t])[0]
        else:
            rn = _wrap(x[i] + st["disp"][t], L)
        a, b = terms(rn, un * mus[i]), terms(x[i], mu[i] * mus[i])
        D = (a[0] + ch[i] * a[1]) - (b[0] + ch[i] * b[1])
        dS = ch[i] * (rn - x[i]) + mus[i] * (un - mu[i])
        du[t] = near(i, rn, un * mus[i]) - near(i, x[i], mu[i] * mus[i]) + float((A * (2 * (np.conj(Q) * D).real + np.abs(D) ** 2)).sum())
        du[t] += surf * float(2 * S @ dS + dS @ dS)
        if not du[t] > -math.log(st["u"][t]):
            acc[t], x[i], mu[i] = 1, rn, un
            Q, S = Q + D, S + dS
    if case["systems"] == 1:
        return {"du": du, "acc": acc, "xyz": x, "mu": mu}
    return {"accepted": None, "energy_change": None, "xyz": x, "mu": mu}


def _exact_npt(case, seed):
    c, L = _exact_ions(case, seed)
    e = c.energies()
    half, u = _npt_move(seed, 0)
    V = L ** 3
    Vn = math.exp(math.log(V) + half * 0.004)
    s = (Vn / V) ** (1.0 / 3.0)
    n = _Chain(case["model"], case["n"], c.x.cpu().numpy() * s, case["kc"], L * s)
    if case["model"] == "ewald":
        n.rc = c.rc
    du = n.energies()[4] - e[4] + _pressure(case) * (Vn - V) - (case["n"] + 1) * math.log(Vn / V)
    acc = not du > -math.log(u)
    return {"energy": np.append(e, du), "like": None, "unlike": None, "pairs": None, "accepted": None, "xyz": (n if acc else c).x.cpu().numpy()}
