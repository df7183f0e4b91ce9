"""Timed cases of the per-step MD path, through the package's public entry points.

Every case is bead-spring melt work at density 0.85 (rc 2.5, skin 0.3, dt 0.001, FENE + WCA bonds, harmonic
angles), the model of this repository's benchmark and tests: single systems as `fastmd <run.conf>` steps them,
batches of replicas as the throughput workloads run them, short runs between observations, the FP64 form, and
the reference-layout launchers on raw device pointers.

Starting states are made from the seed alone: chains laid along a snake through a slightly compressed lattice
(every bond near its rest length), displaced and given Maxwell velocities, so that no integrator run is needed
before the first pass; the lattice melts within the first passes.  A pass advances the state, so passes on one
state are a trajectory.

A pass ends as a production run's output does: the thermo row and the frame (positions) of every system; the
short passes of the driver and of the FP64 form return the velocities too.  (In a stiff bond an FP32 rounding of a
position turns into a velocity error that grows with every step, so velocities of long passes differ between any
two orders of summation.)  Mixed-form results are computed from FP32 forces and are returned as FP32 values;
positions are unwrapped, so that an atom at a box face does not jump by a box length.
"""
import ctypes as C
import math
import os
import tempfile

import numpy as np
import torch

import fastmd_b200 as fm

DENSITY, RC, SKIN, DT = 0.85, 2.5, 0.3, 0.001
FENE_K, FENE_R0, ANGLE_K = 30.0, 1.5, 5.0
LANGEVIN = "nvt_langevin 1.0 1.0 1.0 {seed}"
NVT = "nvt_nh 1.0 1.0 0.5 3"
NPT = "npt_nh 1.0 1.0 0.5 0.0 0.0 10.0 3"
# two-type pair parameters of the NPT workload: (i, j) -> (epsilon, sigma)
TWO_TYPES = {(0, 0): (1.0, 1.0), (0, 1): (0.8, 1.0), (1, 1): (1.0, 1.0)}
TABLE_POINTS, TABLE_LO, TABLE_HI = 2001, 0.05, 2.5
VERLET_ROWS = 128  # list rows a caller of the launchers allocates per atom


def listed():
    return [
        # a small melt run by the command-line program: a step's latency counts
        {"name": "single_3k_langevin", "kind": "single", "chains": 30, "length": 100, "ensemble": "langevin",
         "types": 1, "table": False, "steps": 100},
        # the benchmark's melt as one system
        {"name": "single_30k_langevin", "kind": "single", "chains": 300, "length": 100, "ensemble": "langevin",
         "types": 1, "table": False, "steps": 100},
        # two types with a tabulated cross interaction (run.conf `table`), Nose-Hoover
        {"name": "single_24k_table_nvt", "kind": "single", "chains": 240, "length": 100, "ensemble": "nvt",
         "types": 2, "table": True, "steps": 100},
        # a driver that reads the thermo row every few steps (odd size)
        {"name": "observed_9957_langevin", "kind": "observed", "chains": 3319, "length": 3, "ensemble": "langevin",
         "types": 1, "table": False, "steps": 5, "reads": 5},
        # the double-precision form of one system
        {"name": "plain_12k_langevin", "kind": "plain", "chains": 120, "length": 100, "ensemble": "langevin",
         "types": 1, "table": False, "steps": 50},
        # many small replicas, default settings, as a server holds them
        {"name": "batch_200x1k_langevin", "kind": "batch", "replicas": 200, "chains": 20, "length": 50,
         "spread": 1.0, "ensemble": "langevin", "types": 1, "tuned": False, "steps": 200},
        # replicas of uneven sizes (500 to 20,000 beads), autotuned
        {"name": "batch_uneven_64_langevin", "kind": "batch", "replicas": 64, "chains": 10, "length": 50,
         "spread": 40.0, "ensemble": "langevin", "types": 1, "tuned": True, "steps": 200},
        # deterministic thermostat on a medium batch
        {"name": "batch_16x30k_nvt", "kind": "batch", "replicas": 16, "chains": 300, "length": 100, "spread": 1.0,
         "ensemble": "nvt", "types": 1, "tuned": True, "steps": 200},
        # the benchmark's headline workload
        {"name": "batch_64x30k_langevin", "kind": "batch", "replicas": 64, "chains": 300, "length": 100,
         "spread": 1.0, "ensemble": "langevin", "types": 1, "tuned": True, "steps": 200},
        # one million beads, two types, constant pressure
        {"name": "batch_1x1m_npt", "kind": "batch", "replicas": 1, "chains": 10000, "length": 100, "spread": 1.0,
         "ensemble": "npt", "types": 2, "tuned": True, "steps": 100},
        # a program that owns its device buffers: Morton sort, Verlet list and LJ forces of one configuration
        {"name": "launch_100k", "kind": "launch", "chains": 1000, "length": 100, "types": 1},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["single", "single", "observed", "plain", "batch", "batch", "batch", "launch"])
    length = rng.choice([3, 20, 50, 77, 100])
    if kind in ("single", "observed", "plain"):
        top = {"single": 100_000, "observed": 40_000, "plain": 30_000}[kind]
        case = {"kind": kind, "chains": max(1, int(_log_uniform(rng, 2_500, top) / length)), "length": length,
                "ensemble": rng.choice(["langevin", "nvt", "npt"] if kind != "plain" else ["langevin"]),
                "types": 1, "table": False, "steps": 50}
        if kind == "single" and rng.random() < 0.4:
            case["types"] = 2
            case["table"] = case["ensemble"] != "npt" and rng.random() < 0.5
        if kind == "observed":
            case.update(steps=rng.choice([1, 3, 5]), reads=5)
        return case
    if kind == "batch":
        atoms = _log_uniform(rng, 50_000, 1_800_000)
        spread = rng.choice([1.0, 1.0, 20.0])
        each = _log_uniform(rng, max(600.0, atoms / 128), min(atoms, 200_000.0) / (4.0 if spread > 1 else 1.0))
        mean = 1.0 if spread == 1.0 else (spread - 1.0) / math.log(spread)
        return {"kind": "batch", "replicas": max(1, int(atoms / (each * mean))), "chains": max(1, int(each / length)),
                "length": length, "spread": spread, "ensemble": rng.choice(["langevin", "langevin", "nvt", "npt"]),
                "types": rng.choice([1, 2]), "tuned": rng.random() < 0.7, "steps": 100}
    return {"kind": "launch", "chains": max(1, int(_log_uniform(rng, 5_000, 400_000) / length)), "length": length,
            "types": rng.choice([1, 2])}


def _sizes(case):
    """Chains of each replica: `chains` times 1 to `spread`, evenly over the logarithm."""
    n = case.get("replicas", 1)
    spread = case.get("spread", 1.0)
    return [max(1, int(case["chains"] * spread ** (k / max(1, n - 1)))) for k in range(n)]


def _melt(chains, length, types, rng):
    """Chains along a snake through a lattice of the box, displaced, with Maxwell velocities."""
    n = chains * length
    L = (n / DENSITY) ** (1.0 / 3.0)
    m = math.ceil(n ** (1.0 / 3.0) - 1e-9)
    layers = -(-n // (m * m))
    k = np.arange(n)
    z, y, x = k // (m * m), (k // m) % m, k % m
    y = np.where(z % 2 == 0, y, m - 1 - y)
    x = np.where((k // m) % 2 == 0, x, m - 1 - x)
    xyz = (np.stack([x * (L / m), y * (L / m), z * (L / layers)], 1) + rng.uniform(-0.04, 0.04, (n, 3))) % L
    vel = rng.standard_normal((n, 3))
    vel -= vel.mean(0)
    inner = k.reshape(chains, length)
    bonds = np.stack([inner[:, :-1].ravel(), inner[:, 1:].ravel()], 1).astype(np.int32)
    angles = np.stack([inner[:, :-2].ravel(), inner[:, 1:-1].ravel(), inner[:, 2:].ravel()], 1).astype(np.int32)
    # types alternate in blocks of ten beads along each chain
    typ = ((k % length) // 10 % types).astype(np.int32)
    return fm.SystemDesc(xyz=xyz, box_L=L, type=typ, mol=(k // length + 1).astype(np.int32), vel=vel,
                         mass=np.ones(types), bonds=bonds, bond_type=np.zeros(len(bonds), np.int32), angles=angles,
                         angle_type=np.zeros(len(angles), np.int32), ntypes=types)


def _inputs(case, seed):
    """(melt, noise seed) of each replica."""
    rng = np.random.default_rng([int(seed), 11])
    return [(_melt(c, case["length"], case["types"], rng), int(rng.integers(1, 1 << 31))) for c in _sizes(case)]


def _pairs_of(case):
    pairs = {(0, 0): (1.0, 1.0)} if case["types"] == 1 else dict(TWO_TYPES)
    if case.get("table"):
        del pairs[(0, 1)]  # the table takes its place
    return pairs


def _table_columns():
    """A soft repulsion: r, F / r and energy at the table's points."""
    r = np.linspace(TABLE_LO, TABLE_HI, TABLE_POINTS)
    w = np.pi / TABLE_HI
    return r, 4.0 * w * np.sin(w * r) / r, 4.0 * (1.0 + np.cos(w * r))


def _run_conf(case, seed, table_file=None):
    ensemble = {"langevin": LANGEVIN.format(seed=seed), "nvt": NVT, "npt": NPT}[case["ensemble"]]
    lines = [f"ntypes {case['types']}", f"rc {RC}", f"skin {SKIN}", f"dt {DT}", "nsteps 100000000", ensemble,
             f"bond_type 0 {FENE_K} {FENE_R0} 1.0 1.0", f"angle_type 0 {ANGLE_K} 180.0", "thermo 1 100 thermo.dat"]
    lines += [f"lj {i} {j} {e} {s}" for (i, j), (e, s) in _pairs_of(case).items()]
    if table_file:
        lines.append(f"table 0 1 {table_file} SOFT")
    return "\n".join(lines) + "\n"


def _prepare_single(case, seed):
    (melt, noise), = _inputs(case, seed)
    form = fm.FMD_FORM_PLAIN_FP64 if case["kind"] == "plain" else fm.FMD_FORM_MIXED
    if not case["table"]:
        sim = fm.Simulation(_run_conf(case, noise), desc=melt, form=form)
    else:
        with tempfile.TemporaryDirectory() as tmp:
            path = os.path.join(tmp, "soft.table")
            r, f, e = _table_columns()
            with open(path, "w") as out:
                out.write(f"SOFT\nN {TABLE_POINTS} R {TABLE_LO} {TABLE_HI}\n\n")
                out.writelines(f"{k + 1} {a:.9g} {b:.9g} {c:.9g}\n" for k, (a, b, c) in enumerate(zip(r, e, f)))
            sim = fm.Simulation(_run_conf(case, noise, path), desc=melt, form=form)
    return {"kind": case["kind"], "sim": sim, "steps": case["steps"], "reads": case.get("reads", 1),
            "dtype": np.float64 if case["kind"] == "plain" else np.float32}


def _prepare_batch(case, seed):
    inputs = _inputs(case, seed)
    sizes = [len(m.type) for m, _ in inputs]
    # the NPT cells may grow; every replica's slots are padded to whole chunks
    batch = fm.Batch(max_replicas=len(inputs), max_atoms=sum(n + 256 for n in sizes) + 4096)
    slots = [batch.add(_run_conf(case, noise), desc=melt) for melt, noise in inputs]
    if case["tuned"]:
        batch.autotune(10)
    at = np.concatenate([[0], np.cumsum(sizes)])
    return {"kind": "batch", "batch": batch, "slots": slots, "steps": case["steps"], "at": at,
            "x": np.empty((at[-1], 3), np.float32), "thermo": np.empty((len(slots), 9), np.float32)}


def _prepare_launch(case, seed):
    (melt, _), = _inputs(case, seed)
    n, lib = len(melt.type), fm.lib()
    order = np.random.default_rng([int(seed), 12]).permutation(n)  # the caller's storage order
    place = np.empty(n, np.int64)
    place[order] = np.arange(n)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = melt.xyz[order]
    pos[:, 3] = melt.type[order].view(np.float32)
    vel = np.ones((n, 4), np.float32)
    vel[:, :3] = melt.vel[order]
    table = np.zeros((case["types"], case["types"], 2), np.float32)
    for (i, j), p in _pairs_of(case).items():
        table[i, j] = table[j, i] = p
    L = C.c_float(melt.box_L)
    verlet_bytes, morton_bytes = C.c_size_t(), C.c_size_t()
    assert lib.fmd_verlet_scratch_bytes(C.c_int32(n), C.c_float(RC + SKIN), L, C.byref(verlet_bytes)) == 0
    assert lib.fmd_morton_scratch_bytes(C.c_int32(n), C.byref(morton_bytes)) == 0
    scratch = torch.empty(max(verlet_bytes.value, morton_bytes.value), dtype=torch.uint8, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    return {"kind": "launch", "lib": lib, "n": n, "L": L, "types": case["types"], "scratch": scratch,
            "pos": torch.from_numpy(pos).cuda(), "vel": torch.from_numpy(vel).cuda(),
            "lj": torch.from_numpy(table).cuda(), "perm": torch.zeros(n, **i32),
            "nbr": torch.zeros((VERLET_ROWS, n), **i32), "count": torch.zeros(n, **i32),
            "flag": torch.zeros(1, **i32), "force": torch.zeros((n, 4), device="cuda"),
            "virial": torch.zeros(6, device="cuda")}


def prepare(case, seed):
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    if case["kind"] == "launch":
        return _prepare_launch(case, seed)
    return _prepare_single(case, seed)


def _run_single(s):
    sim = s["sim"]
    rows = []
    for _ in range(s["reads"]):
        sim.step(s["steps"])
        rows.append(sim.thermo().as_array())
    x, v, image = sim.state()
    out = {"x": (x + image * sim.box_L).astype(s["dtype"]), "thermo": np.array(rows, s["dtype"])}
    if s["kind"] != "single":
        out["v"] = v.astype(s["dtype"])
    return out


def _run_batch(s):
    batch, at = s["batch"], s["at"]
    batch.run(s["steps"])
    for k, slot in enumerate(s["slots"]):
        row = batch.thermo(slot)
        x, _, image = batch.state(slot)
        s["thermo"][k] = row.as_array()
        s["x"][at[k]:at[k + 1]] = x + image * row.box_L
    return {"x": s["x"], "thermo": s["thermo"]}


def _run_launch(s):
    lib, n, L = s["lib"], C.c_int32(s["n"]), s["L"]
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def ptr(name):
        return C.c_void_p(s[name].data_ptr())

    room = C.c_size_t(s["scratch"].numel())
    inv_L = C.c_float(1.0 / L.value)
    s["virial"].zero_()
    bad = lib.fmd_launch_morton_sort(ptr("pos"), ptr("vel"), n, inv_L, ptr("perm"), ptr("scratch"), room, stream)
    bad |= lib.fmd_launch_verlet_build(ptr("pos"), n, L, None, None, C.c_float(RC + SKIN), C.c_int32(VERLET_ROWS),
                                       ptr("nbr"), ptr("count"), ptr("scratch"), room, ptr("flag"), stream)
    bad |= lib.fmd_launch_lj(ptr("pos"), ptr("force"), ptr("virial"), ptr("lj"), ptr("nbr"), ptr("count"), n,
                             C.c_int32(s["types"]), C.c_float(RC * RC), L, inv_L, stream)
    if bad:
        raise RuntimeError("a launcher refused its arguments")
    return {k: s[k] for k in ("pos", "vel", "perm", "nbr", "count", "flag", "force", "virial")}


def run(state):
    return {"batch": _run_batch, "launch": _run_launch}.get(state["kind"], _run_single)(state)


def work(case):
    """Per atom and step: position, velocity and force read and written once, and the arithmetic of the pairs
    within rc (each counted once) and of the bonded terms."""
    atoms = sum(_sizes(case)) * case["length"]
    pairs = 0.5 * DENSITY * 4.0 / 3.0 * math.pi * RC ** 3
    if case["kind"] == "launch":
        listed_pairs = DENSITY * 4.0 / 3.0 * math.pi * (RC + SKIN) ** 3
        return {"bytes": atoms * (2 * 32 + 4 + 4 * listed_pairs + 4 + 16),
                "flops": atoms * (2 * pairs * 40.0 + 10.0 * listed_pairs)}
    steps = case["steps"] * case.get("reads", 1)
    real = 8 if case["kind"] == "plain" else 4
    return {"bytes": atoms * (steps * 2 * 9 * real + 2 * 6 * real), "flops": atoms * steps * (pairs * 40.0 + 200.0)}


# ---------------------------------------------------------------------------
# The same passes in 64 bits, in torch.

def _close_pairs(x, L, reach):
    """Index pairs (i, j), each once, within `reach` in the periodic box."""
    n, G = len(x), int(L / reach)
    if G < 3 or n < 4000:
        out, rows = [], max(1, 60_000_000 // n)
        for a in range(0, n, rows):
            d = x[a:a + rows, None, :] - x[None, :, :]
            d -= L * torch.round(d / L)
            i, j = torch.nonzero((d * d).sum(2) < reach * reach, as_tuple=True)
            out.append(torch.stack([i + a, j])[:, i + a < j])
        return torch.cat(out, 1)
    c = torch.clamp((x / (L / G)).long(), 0, G - 1)
    cell = (c[:, 2] * G + c[:, 1]) * G + c[:, 0]
    cell, order = torch.sort(cell)
    count = torch.bincount(cell, minlength=G ** 3)
    first = torch.cumsum(count, 0) - count
    room = int(count.max())
    table = torch.full((G ** 3, room), -1, dtype=torch.long, device=x.device)
    table[cell, torch.arange(n, device=x.device) - first[cell]] = order
    g = torch.arange(G, device=x.device)
    out, step = [], max(1, 30_000_000 // (room * room))
    half = [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1) if (dz, dy, dx) >= (0, 0, 0)]
    for dx, dy, dz in half:
        other = ((((g + dz) % G)[:, None, None] * G + ((g + dy) % G)[None, :, None]) * G
                 + ((g + dx) % G)[None, None, :]).reshape(-1)
        for a in range(0, G ** 3, step):
            i, j = table[a:a + step, :, None], table[other[a:a + step]][:, None, :]
            d = x[i] - x[j]
            d -= L * torch.round(d / L)
            ok = ((d * d).sum(3) < reach * reach) & (i >= 0) & (j >= 0)
            if (dx, dy, dz) == (0, 0, 0):
                ok &= i < j
            w = torch.nonzero(ok, as_tuple=True)
            out.append(torch.stack([i.expand(ok.shape)[w], j.expand(ok.shape)[w]]))
    return torch.cat(out, 1)


class _Exact:
    """One system: forces, energy and virial, and the integrators' steps."""

    def __init__(self, case, melt, noise):
        dev = "cuda" if torch.cuda.is_available() else "cpu"

        def t(a, dtype=torch.float64):
            return torch.as_tensor(np.ascontiguousarray(a)).to(dev, dtype)

        self.dev, self.n, self.L, self.seed = dev, len(melt.type), float(melt.box_L), noise
        self.x, self.v, self.img = t(melt.xyz), t(melt.vel), torch.zeros((self.n, 3), dtype=torch.float64, device=dev)
        self.type = t(melt.type, torch.long)
        self.bonds, self.angles = t(melt.bonds, torch.long).T, t(melt.angles, torch.long).T
        self.length, k = case["length"], case["types"]
        eps, sig = torch.zeros((k, k), dtype=torch.float64), torch.zeros((k, k), dtype=torch.float64)
        for (i, j), (e, s) in _pairs_of(case).items():
            eps[i, j] = eps[j, i] = e
            sig[i, j] = sig[j, i] = s
        self.eps, self.sig = eps.to(dev), sig.to(dev)
        self.table = None
        if case.get("table"):  # the points as the FP32 table holds them
            _, f, e = _table_columns()
            self.table = t(f.astype(np.float32)), t(e.astype(np.float32))
        self.listed_at = None
        self.ens, self.step_no = case["ensemble"], 0
        # Nose-Hoover chain of three and the barostat
        tdamp = {"langevin": 1.0, "nvt": 0.5, "npt": 0.5}[self.ens]
        self.M, self.Qr, self.Q1 = 3, tdamp * tdamp, 3.0 * self.n * tdamp * tdamp
        self.W, self.V0 = (3.0 * self.n + 3.0) * 100.0, self.L ** 3  # Pdamp 10
        self.c1 = math.exp(-DT / tdamp)
        self.xi, self.vxi, self.eps_V, self.veps, self.pending = [0.0] * 3, [0.0] * 3, 0.0, 0.0, 1.0
        self.Lpos = self.L
        self.forces()
        self.carry = self.kinetic()

    def kinetic(self):
        return 0.5 * float((self.v * self.v).sum())

    def image_of(self, d):
        return d - self.Lpos * torch.round(d / self.Lpos)

    def pairs(self):
        u = self.x + self.img * self.Lpos
        if self.listed_at is None or float((u - self.listed_at).square().sum(1).max()) > 0.2 ** 2:
            i, j = _close_pairs(self.x % self.Lpos, self.Lpos, RC + 0.5)
            bonded = ((i - j).abs() == 1) & (i // self.length == j // self.length)
            self.i, self.j, self.listed_at = i[~bonded], j[~bonded], u
        return self.i, self.j

    def forces(self):
        f = torch.zeros_like(self.x)
        pe, vir = 0.0, torch.zeros((3, 3), dtype=torch.float64, device=self.dev)

        def add(i, j, d, fr):
            nonlocal vir
            g = fr[:, None] * d
            f.index_add_(0, i, g)
            f.index_add_(0, j, -g)
            vir += g.T @ d

        i, j = self.pairs()
        d = self.image_of(self.x[i] - self.x[j])
        r2 = (d * d).sum(1)
        near = r2 < RC * RC
        i, j, d, r2 = i[near], j[near], d[near], r2[near]
        ti, tj = self.type[i], self.type[j]
        s6 = (self.sig[ti, tj] ** 2 / r2) ** 3
        e = self.eps[ti, tj]
        add(i, j, d, torch.clamp(24.0 * e / r2 * (2.0 * s6 * s6 - s6), -1000.0, 1000.0))
        pe += float((4.0 * e * (s6 * s6 - s6)).sum())
        if self.table is not None:
            cross = ti != tj
            rr = torch.clamp(r2[cross].sqrt(), TABLE_LO, TABLE_HI)
            at = (rr - TABLE_LO) * ((TABLE_POINTS - 1) / (TABLE_HI - TABLE_LO))
            k = torch.clamp(at.long(), 0, TABLE_POINTS - 2)
            w = at - k
            fr, et = ((1.0 - w) * c[k] + w * c[k + 1] for c in self.table)
            add(i[cross], j[cross], d[cross], fr)
            pe += float(et.sum())
        i, j = self.bonds
        d = self.image_of(self.x[i] - self.x[j])
        r2 = (d * d).sum(1)
        R2 = FENE_R0 ** 2
        s6 = r2 ** -3.0
        wca = r2 < 2.0 ** (1.0 / 3.0)
        add(i, j, d, -FENE_K * R2 / (R2 - r2) + torch.where(wca, 24.0 / r2 * (2.0 * s6 * s6 - s6), 0.0 * r2))
        pe += float((-0.5 * FENE_K * R2 * torch.log1p(-r2 / R2)).sum() + torch.where(wca, 4.0 * (s6 * s6 - s6) + 1.0, 0.0 * r2).sum())
        i, j, k = self.angles
        a, b = self.image_of(self.x[i] - self.x[j]), self.image_of(self.x[k] - self.x[j])
        ra, rb = a.norm(dim=1, keepdim=True), b.norm(dim=1, keepdim=True)
        cs = torch.clamp((a * b).sum(1, keepdim=True) / (ra * rb), -1.0, 1.0)
        sn = torch.linalg.cross(a, b).norm(dim=1, keepdim=True) / (ra * rb)
        off = torch.atan2(sn, cs) - math.pi
        pref = 2.0 * ANGLE_K * off / torch.clamp(sn, min=1e-6)
        fi = pref * (b / (ra * rb) - cs * a / ra ** 2)
        fk = pref * (a / (ra * rb) - cs * b / rb ** 2)
        f.index_add_(0, i, fi)
        f.index_add_(0, k, fk)
        f.index_add_(0, j, -(fi + fk))
        vir += fi.T @ a + fk.T @ b
        pe += float((ANGLE_K * off * off).sum())
        self.f, self.pe, self.vir = f, pe, vir

    def normals(self):
        """Philox4x32-10 (Salmon et al., SC'11) on (atom id, step, stream) and a Box-Muller transform."""
        lo = 0xFFFFFFFF
        ids = torch.arange(self.n, device=self.dev)
        c = [ids, torch.full_like(ids, self.step_no & lo), torch.full_like(ids, self.step_no >> 32),
             torch.full_like(ids, 0x4C414E47)]
        k0, k1 = self.seed & lo, self.seed >> 32

        def product(m, v):  # high and low words of a 32 x 32 bit product, in 16-bit limbs
            p0, p1 = m * (v & 0xFFFF), m * (v >> 16)
            mid = p1 + (p0 >> 16)
            return mid >> 16, ((mid & 0xFFFF) << 16) | (p0 & 0xFFFF)

        for r in range(10):
            h0, l0 = product(0xD2511F53, c[0])
            h1, l1 = product(0xCD9E8D57, c[2])
            c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
            k0, k1 = (k0 + 0x9E3779B9) & lo, (k1 + 0xBB67AE85) & lo

        def normal_pair(a, b):
            r = torch.sqrt(-2.0 * torch.log((a.double() + 1.0) * 2.0 ** -32))
            t = 0.5 * math.pi * ((b >> 30).double() + (b & 0x3FFFFFFF).double() * 2.0 ** -30)
            return r * torch.cos(t), r * torch.sin(t)

        n0, n1 = normal_pair(c[0], c[1])
        n2, _ = normal_pair(c[2], c[3])
        return torch.stack([n0, n1, n2], 1)

    def chain(self, ke, half):
        """Half a step of the thermostat chain; the velocity scale.  Its exponential is the truncated series,
        and the upper elements' accelerations start from zero, as the integrator defines them."""
        def ex(x):
            return 1.0 + x + x * x / 2 + x ** 3 / 6 + x ** 4 / 24 + x ** 5 / 120 + x ** 6 / 720

        M, v, Nf = self.M, self.vxi, 3.0 * self.n
        d4, d8 = 0.5 * half, 0.25 * half
        T = 2.0 * ke / Nf
        a0 = (Nf * T - Nf) / self.Q1
        for k in range(M - 1, 0, -1):
            e = ex(-d8 * v[k + 1]) if k + 1 < M else 1.0
            v[k] = v[k] * e * e
        e0 = ex(-d8 * v[1])
        v[0] = (v[0] * e0 + a0 * d4) * e0
        scale = ex(-half * v[0])
        a0 = (Nf * T * scale * scale - Nf) / self.Q1
        for k in range(M):
            self.xi[k] += half * v[k]
        v[0] = (v[0] * e0 + a0 * d4) * e0
        for k in range(1, M):
            e = ex(-d8 * v[k + 1]) if k + 1 < M else 1.0
            a = ((self.Q1 if k == 1 else self.Qr) * v[k - 1] ** 2 - 1.0) / self.Qr
            v[k] = (v[k] * e + a * d4) * e
        return scale

    def barostat(self, first):
        """Half a step of the coupled chain and barostat: (velocity scale, position scale, drift factor)."""
        ke = self.carry if first else self.kinetic()
        V = self.V0 * math.exp(3.0 * self.eps_V)
        if not first:
            P = (2.0 * ke + float(self.vir.trace())) / (3.0 * V)
            c = 2.0 ** (1.0 / 3.0)
            for w in (DT / (2.0 - c), -DT * c / (2.0 - c), DT / (2.0 - c)):
                half = self.veps + 0.5 * 3.0 * V * P * w
                self.eps_V += half * w / self.W
                self.veps += 3.0 * self.V0 * math.exp(3.0 * self.eps_V) * P * w
            V = self.V0 * math.exp(3.0 * self.eps_V)
        self.L = V ** (1.0 / 3.0)
        rate = self.veps / self.W
        shrink = math.exp(-(1.0 + 1.0 / self.n) * rate * 0.5 * DT)
        hx = 0.5 * rate * DT
        ratio = 1.0 + hx * hx / 6.0 if abs(hx) < 1e-6 else math.sinh(hx) / hx
        scale = self.chain(ke * shrink * shrink, 0.5 * DT)
        if not first:
            self.carry = ke * shrink * shrink * scale * scale
        return scale * shrink, math.exp(rate * DT), DT * math.exp(hx) * ratio

    def step(self):
        self.step_no += 1
        h = 0.5 * DT
        if self.ens == "langevin":
            self.v += h * self.f
            self.x = self.x + h * self.v
            self.v = self.c1 * self.v + math.sqrt(1.0 - self.c1 ** 2) * self.normals()
            self.x = self.x + h * self.v
        elif self.ens == "nvt":
            self.v = self.v * (self.pending * self.chain(self.carry, h)) + h * self.f
            self.x = self.x + DT * self.v
        else:
            scale, grow, drift = self.barostat(True)
            self.v = self.v * (self.pending * scale) + h * self.f
            self.x = self.x * grow + drift * self.v
        self.Lpos = self.L
        fl = torch.floor(self.x / self.Lpos)
        self.x, self.img = self.x - fl * self.Lpos, self.img + fl
        self.forces()
        self.v = self.v + h * self.f
        if self.ens == "nvt":
            ke = self.kinetic()
            self.pending = self.chain(ke, h)
            self.carry = ke * self.pending ** 2
        elif self.ens == "npt":
            self.pending = self.barostat(False)[0]

    def thermo(self):
        v = self.v * self.pending
        k = v.T @ v
        ke = 0.5 * float(k.trace()) / self.n
        p = ((k + self.vir) / self.L ** 3).cpu().numpy()
        return [ke, self.pe / self.n, 2.0 * ke / 3.0, p[0, 0], p[0, 1], p[0, 2], p[1, 1], p[1, 2], p[2, 2]]

    def state(self):
        return (self.x + self.img * self.L).cpu().numpy(), (self.v * self.pending).cpu().numpy()


def _exact_launch(case, seed):
    (melt, _), = _inputs(case, seed)
    n = len(melt.type)
    order = np.random.default_rng([int(seed), 12]).permutation(n)
    xyz, typ, L = melt.xyz[order].astype(np.float32), melt.type[order], np.float32(melt.box_L)
    cells = np.minimum((xyz * np.float32(1.0 / float(L)) * np.float32(1024.0)).astype(np.int64), 1023)
    key = np.zeros(n, np.int64)
    for bit in range(10):
        for axis in range(3):
            key |= ((cells[:, axis] >> bit) & 1) << (3 * bit + axis)
    perm = np.argsort(key, kind="stable")
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.as_tensor(xyz[perm].astype(np.float64)).to(dev)
    t = torch.as_tensor(typ[perm].astype(np.int64)).to(dev)
    L = float(L)
    i, j = _close_pairs(x % L, L, RC)
    d = x[i] - x[j]
    d -= L * torch.round(d / L)
    r2 = (d * d).sum(1)
    eps = torch.zeros((case["types"],) * 2, dtype=torch.float64, device=dev)
    for (a, b), (e, _) in _pairs_of(case).items():
        eps[a, b] = eps[b, a] = float(np.float32(e))
    e, s6 = eps[t[i], t[j]], r2 ** -3.0
    g = torch.clamp(24.0 * e / r2 * (2.0 * s6 * s6 - s6), -1000.0, 1000.0)[:, None] * d
    force = torch.zeros((n, 4), dtype=torch.float64, device=dev)
    half = 0.5 * (4.0 * e * (s6 * s6 - s6))[:, None]
    force.index_add_(0, i, torch.cat([g, half], 1))
    force.index_add_(0, j, torch.cat([-g, half], 1))
    vir = (g.T @ d)[torch.tensor([0, 0, 0, 1, 1, 2]), torch.tensor([0, 1, 2, 1, 2, 2])]
    return {"pos": None, "vel": None, "perm": None, "nbr": None, "count": None, "flag": None,
            "force": force.cpu().numpy(), "virial": vir.cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "launch":
        return _exact_launch(case, seed)
    # about 25 ms a step and system on a GPU for small systems, 60 ns an atom and step for large ones
    steps = case["steps"] * case.get("reads", 1)
    each = [0.012 + 60e-9 * c * case["length"] for c in _sizes(case)]
    if steps * sum(each) > 20.0:
        return None
    xs, vs, rows = [], [], []
    for melt, noise in _inputs(case, seed):
        sim = _Exact(case, melt, noise)
        for k in range(steps):
            sim.step()
            if (k + 1) % case["steps"] == 0:
                rows.append(sim.thermo())
        x, v = sim.state()
        xs.append(x)
        vs.append(v)
    out = {"x": np.concatenate(xs), "thermo": np.array(rows)}
    if case["kind"] in ("observed", "plain"):
        out["v"] = np.concatenate(vs)
    return out
