"""Performance cases of the force path: what a program that uses this library has it do, from the
smallest system to the largest, through the public entry points.

Every case is a dict of plain values; its ``kind`` names the call:

* ``step``   -- ``ForceField.step(n)``: n velocity-Verlet steps on device arrays (LJ, electrolyte with
                RBE, rigid water with SHAKE, EAM metal, flexible chains, batches of replicas);
* ``force``  -- ``ForceField.Execute()``: one force evaluation on device positions;
* ``host``   -- ``ForceField.compute_host()``: one force evaluation on host positions into host forces,
                the call of an MD driver that keeps its arrays on the host;
* ``rhok``   -- ``rbmd_rhok_noalloc``: structure factors of one box;
* ``train``  -- ``ForceField.train_proposal()``: fit of the learned k-proposal on a running system.

Systems come from ``copy_gpu_b200.systems`` in the shapes of the benchmark configurations.
"""
import math
import os
import tempfile

import numpy as np
import torch

from copy_gpu_b200 import Box, ForceField, library, rbmd_box, systems

# flexible chains: the periodic tile that larger boxes repeat (5^3 sites of 6 A)
TILE_CHAINS, TILE_LEN, TILE_IONS, TILE_CELL, TILE_SITES = 104, 12, 10, 6.0, 125
TILE_ATOMS = TILE_CHAINS * TILE_LEN + 2 * TILE_IONS


def listed():
    return [
        # the textbook LJ run in double precision, a few microseconds of arithmetic per step:
        # launches and host work dominate; library defaults
        dict(name="lj_4k_fp64_steps", kind="step", system="lj", ncell=10, precision="fp64", skin=0.3,
             tuned=False, steps=20),
        # a small odd-sized electrolyte as used for equilibration and screening; library defaults
        dict(name="electrolyte_16k_steps", kind="step", system="electrolyte", n=16381, P=200, ion_frac=0.1,
             proposal="gauss", precision="fp32", skin=0.3, tuned=False, steps=10),
        # the benchmark run: 1M atoms, learned proposal at the P of equal force error, autotuned
        dict(name="electrolyte_1m_learned_steps", kind="step", system="electrolyte", n=1000000, P=305,
             ion_frac=0.1, proposal="learned", precision="fp32", skin=0.3, tuned=True, steps=10),
        # a host-side MD engine calling for forces every step in its own float arrays; the list is
        # rebuilt on every call, as the reference does (no skin)
        dict(name="electrolyte_200k_host_f32", kind="host", system="electrolyte", n=200000, P=500, ion_frac=0.1,
             host="f32", precision="fp32", tuned=False),
        # double-precision forces of a strongly charged system (validation runs, energy minimisers)
        dict(name="electrolyte_50k_fp64_force", kind="force", system="electrolyte", n=50021, P=200, ion_frac=0.5,
             precision="fp64", tuned=False),
        # rigid water, the benchmark configuration: SHAKE / RATTLE, long lists, autotuned
        dict(name="water_30k_steps", kind="step", system="water", n_mol=10000, P=200, precision="fp32", skin=1.0,
             tuned=True, steps=5),
        # metal crystal, the benchmark configuration: two EAM passes per step, autotuned
        dict(name="eam_256k_steps", kind="step", system="eam", ncell=40, precision="fp32", skin=0.3, tuned=True,
             steps=10),
        # many uneven replicas advanced together, the batched benchmark configuration
        dict(name="replicas_512_steps", kind="step", system="replicas", n_rep=512, P=100, precision="fp32",
             skin=0.3, tuned=True, steps=4),
        # flexible chains in the reference's default RBL mode: list rebuilt every step, bonded terms
        dict(name="chains_101k_rbl_steps", kind="step", system="chains", kx=4, ky=4, kz=5, neighbor="RBL", P=100,
             precision="fp32", skin=0.0, tuned=False, steps=5),
        # a smaller box of the same chains with exact pair sums and list reuse; library defaults
        dict(name="chains_23k_verlet_steps", kind="step", system="chains", kx=2, ky=3, kz=3, neighbor="VERLETLIST",
             P=100, precision="fp32", skin=1.0, tuned=False, steps=5),
        # structure factors for a caller that cannot allocate (analysis of a trajectory frame)
        dict(name="rhok_20k", kind="rhok", n=20011, P=500),
        # fit of the learned proposal on a running system (forward and backward of the network)
        dict(name="train_20k", kind="train", system="electrolyte", n=20000, P=200, ion_frac=0.1, proposal="learned",
             precision="fp32", skin=0.3, tuned=False, snapshots=16, between=2, k=16384, iterations=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One case of the same ranges: sizes spread over their logarithm, odd sizes, both precisions."""
    kind = rng.choice(["lj", "electrolyte", "electrolyte", "host", "force", "water", "eam", "replicas", "rbl",
                       "verlet", "rhok", "train"])
    if kind == "lj":
        return dict(kind="step", system="lj", ncell=_log(rng, 5, 40), precision=rng.choice(["fp64", "fp32"]),
                    skin=rng.choice([0.0, 0.3]), tuned=rng.random() < 0.5, steps=rng.randint(2, 20))
    if kind == "electrolyte":
        n = _log(rng, 500, 400000)
        return dict(kind="step", system="electrolyte", n=n, P=rng.choice([100, 200, 305, 500]),
                    ion_frac=rng.choice([0.1, 0.1, 0.5, 1.0]),
                    proposal=rng.choice(["gauss", "gauss", "gauss_iid", "learned"]), precision="fp32",
                    skin=rng.choice([0.3, 0.3, 0.0]), tuned=rng.random() < 0.5, steps=rng.randint(2, 12))
    if kind == "host":
        return dict(kind="host", system="electrolyte", n=_log(rng, 1000, 400000), P=rng.choice([100, 200, 500]),
                    ion_frac=rng.choice([0.1, 0.5]), host=rng.choice(["f32", "f64"]),
                    precision=rng.choice(["fp32", "fp32", "fp64"]), tuned=False)
    if kind == "force":
        return dict(kind="force", system="electrolyte", n=_log(rng, 1000, 100000), P=rng.choice([100, 200, 500]),
                    ion_frac=rng.choice([0.1, 0.5, 1.0]), precision=rng.choice(["fp32", "fp64"]), tuned=False)
    if kind == "water":
        return dict(kind="step", system="water", n_mol=_log(rng, 1600, 20000), P=rng.choice([100, 200]),
                    precision="fp32", skin=rng.choice([1.0, 1.0, 0.0]), tuned=rng.random() < 0.5,
                    steps=rng.randint(2, 8))
    if kind == "eam":
        return dict(kind="step", system="eam", ncell=_log(rng, 6, 40), precision=rng.choice(["fp32", "fp32", "fp64"]),
                    skin=rng.choice([0.3, 0.3, 0.0]), tuned=rng.random() < 0.5, steps=rng.randint(2, 10))
    if kind == "replicas":
        return dict(kind="step", system="replicas", n_rep=_log(rng, 4, 256), P=100, precision="fp32", skin=0.3,
                    tuned=rng.random() < 0.5, steps=rng.randint(2, 8))
    if kind in ("rbl", "verlet"):
        k = [rng.randint(2, 4) for _ in range(3)]
        return dict(kind="step", system="chains", kx=k[0], ky=k[1], kz=k[2],
                    neighbor="RBL" if kind == "rbl" else "VERLETLIST", P=100, precision="fp32",
                    skin=0.0 if kind == "rbl" else rng.choice([0.0, 1.0]), tuned=rng.random() < 0.5,
                    steps=rng.randint(2, 6))
    if kind == "rhok":
        return dict(kind="rhok", n=_log(rng, 500, 262144), P=_log(rng, 16, 1024))
    return dict(kind="train", system="electrolyte", n=_log(rng, 2000, 50000), P=200, ion_frac=0.1,
                proposal="learned", precision="fp32", skin=0.3, tuned=False, snapshots=rng.randint(2, 24),
                between=2, k=rng.choice([4096, 8192, 16384]), iterations=rng.randint(20, 120))


# ---- systems --------------------------------------------------------------------------------------
def _chains(c, seed):
    """Flexible chains and ions: one seeded tile repeated kx x ky x kz times (every copy keeps its own
    molecules), thermal displacements of 0.02 A per copy, new velocities."""
    t = systems.molecular(n_chain=TILE_CHAINS, chain_len=TILE_LEN, n_ion_pairs=TILE_IONS, step=1.5,
                          cell=TILE_CELL, seed=1000 + seed)
    reps = c["kx"] * c["ky"] * c["kz"]
    n0, L0 = t["pos"].shape[0], t["hi"]
    rng = np.random.default_rng(seed)
    ijk = np.stack(np.unravel_index(np.arange(reps), (c["kx"], c["ky"], c["kz"])), 1)
    L = L0 * np.array([c["kx"], c["ky"], c["kz"]])
    pos = (t["pos"][None] + (ijk * L0)[:, None]).reshape(-1, 3) + rng.normal(scale=0.02, size=(reps * n0, 3))
    tile = lambda a: np.tile(a, (reps,) + (1,) * (a.ndim - 1))   # noqa: E731
    shift = lambda a, m: (a[None] + (np.arange(reps) * m).reshape((-1,) + (1,) * a.ndim)).reshape(   # noqa: E731
        (-1,) + a.shape[1:]).astype(np.int32)
    out = dict(t)
    for k in ("mass", "charge", "type", "bond_type", "angle_type", "dihedral_type"):
        out[k] = tile(t[k])
    nmol = int(t["molecule"].max()) + 1
    vel = rng.normal(size=pos.shape) * np.sqrt(1.9872067e-3 * 298.0 * 4.186e-4 / out["mass"][:, None])
    out.update(pos=np.mod(pos, L), vel=vel, molecule=shift(t["molecule"], nmol),
               bonds=shift(t["bonds"], n0), angles=shift(t["angles"], n0), dihedrals=shift(t["dihedrals"], n0),
               lo=np.zeros(3), hi=L)
    return out


def _replica_sizes(n_rep):
    """Atom counts of a batch, uniform in [500, 8000]: part of the case, whatever the seed."""
    return np.random.default_rng(n_rep).integers(500, 8001, size=n_rep)


def _replicas(n_rep, seed):
    parts = [systems.electrolyte(int(k), seed=seed * 1000 + r) for r, k in enumerate(_replica_sizes(n_rep))]
    s = {k: np.concatenate([p[k] for p in parts]) for k in ("pos", "vel", "mass", "charge", "type")}
    s.update(offsets=np.concatenate([[0], np.cumsum(_replica_sizes(n_rep))]).astype(np.int64),
             lo=np.stack([p["lo"] for p in parts]), hi=np.stack([p["hi"] for p in parts]),
             eps=parts[0]["eps"], sigma=parts[0]["sigma"])
    return s


def _system(c, seed):
    """(system, configuration, replica offsets or None) of a case."""
    name = c["system"]
    if name == "lj":
        cfg = systems.lj_config(cutoff=2.5, precision=c["precision"], ensemble="NVE")
        s = systems.lj_fcc(ncell=c["ncell"], seed=seed)
        # off the lattice sites, where every force would cancel
        s["pos"] = np.mod(s["pos"] + np.random.default_rng(seed).normal(scale=0.05, size=s["pos"].shape), s["hi"])
        return s, cfg, None
    if name == "electrolyte":
        cfg = systems.electrolyte_config(P=c["P"], precision=c["precision"], seed=7)
        cfg["hyper_parameters"]["coulomb"]["proposal"] = c.get("proposal", "gauss")
        return systems.electrolyte(c["n"], ion_frac=c["ion_frac"], seed=seed), cfg, None
    if name == "replicas":
        s = _replicas(c["n_rep"], seed)
        return s, systems.electrolyte_config(P=c["P"], precision=c["precision"], seed=7), s["offsets"]
    if name == "water":
        return systems.water(n_mol=c["n_mol"], seed=seed), systems.water_config(P=c["P"], precision=c["precision"]), None
    if name == "eam":
        return systems.eam_fcc(ncell=c["ncell"], seed=seed), systems.eam_config("", precision=c["precision"]), None
    s = _chains(c, seed)
    cfg = systems.molecular_config(P=c["P"], cutoff=12.0, alpha=0.074, neighbor=c["neighbor"], special=(0.0, 0.0, 0.0),
                                   dt=0.5, precision=c["precision"], r_core=6.0, sample_num=100)
    cfg["execution"].update(ensemble="NVT", temp_ctrl_type="BERENDSEN")
    return s, cfg, None


def _kset(c, L, seed, alpha):
    """P integer vectors of RBE's Gaussian (none of them zero), as a driver with its own sampler has."""
    rng = np.random.default_rng(seed + 77)
    sig = np.sqrt(alpha / 2.0) * np.asarray(L) / np.pi
    m = np.rint(rng.normal(size=(4 * c["P"] + 64, 3)) * sig).astype(np.int32)
    return np.ascontiguousarray(m[np.any(m != 0, 1)][:c["P"]])


def _rhok_inputs(c, seed):
    rng = np.random.default_rng(seed)
    n = c["n"]
    L = (n / 0.8) ** (1.0 / 3.0)
    pos = rng.uniform(0, L, size=(n, 3))
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    alpha = systems.electrolyte_alpha(2.5)
    return pos, q, L, _kset(c, [L] * 3, seed, alpha)


def prepare(case, seed):
    dev = torch.device("cuda")
    if case["kind"] == "rhok":
        pos, q, L, m = _rhok_inputs(case, seed)
        b = rbmd_box()
        for d in range(3):
            b.lo[d], b.hi[d] = 0.0, L
        return dict(kind="rhok", pos=torch.tensor(pos, device=dev), q=torch.tensor(q, device=dev),
                    m=torch.tensor(m, device=dev), box=b, n=case["n"], P=case["P"],
                    rho=torch.zeros((case["P"], 2), device=dev, dtype=torch.float64))
    s, cfg, offs = _system(case, seed)
    if case["system"] == "eam":
        with tempfile.TemporaryDirectory() as d:
            path = systems.write_johnson_setfl(os.path.join(d, "johnson.setfl"))
            cfg["hyper_parameters"]["force_field"].update(potential_file=path, potential_format="setfl")
            ff = _handle(case, s, cfg, offs)
    else:
        ff = _handle(case, s, cfg, offs)
    n = s["pos"].shape[0]
    t = {k: torch.tensor(s[k], device=dev, dtype=torch.float64).contiguous() for k in ("pos", "vel", "mass", "charge")}
    t["type"] = torch.tensor(s["type"], device=dev, dtype=torch.int32)
    t["force"] = torch.zeros((n, 3), device=dev, dtype=torch.float64)
    t["image"] = torch.zeros((n, 3), device=dev, dtype=torch.int32)
    if s.get("molecule") is not None:
        t["molecule"] = torch.tensor(s["molecule"], device=dev, dtype=torch.int32)
    if "hoh" in s:
        ff.set_water(s["hoh"], s["bond"][0], s["bond"][1], s["angle"][0], s["angle"][1])
    if "bonds" in s:
        ff.set_topology(s["molecule"], s["bonds"], s["bond_type"], s["bond_coeffs"], s["angles"], s["angle_type"],
                        s["angle_coeffs"], s["dihedrals"], s["dihedral_type"], s["dihedral_coeffs"])
    ff.Init(t["pos"], t["force"], vel=t["vel"], mass=t["mass"], charge=t["charge"], type=t["type"],
            molecule=t.get("molecule"), image=t["image"], replica_offsets=offs)
    st = dict(kind=case["kind"], ff=ff, t=t, case=case)
    if case["kind"] in ("force", "host"):
        alpha = cfg["hyper_parameters"]["coulomb"]["alpha"]
        ff.set_ksamples(_kset(case, s["hi"] - s["lo"], seed, alpha))
    if case["kind"] == "host":
        dt = torch.float32 if case["host"] == "f32" else torch.float64
        for k, v in (("ph", s["pos"]), ("fh", np.zeros((n, 3)))):
            h = torch.empty((n, 3), dtype=dt, pin_memory=True)
            h.copy_(torch.tensor(v))
            st[k] = h.numpy()
            st[k + "_pinned"] = h
        return st
    if case["kind"] == "step":
        if case.get("proposal") == "learned":
            ff.proposal_params(_network(seed))
        if case["tuned"]:
            ff.autotune()
        ff.Execute()   # the forces that the first kick uses
    if case["kind"] == "train":
        ff.Execute()
    return st


def _handle(case, s, cfg, offs):
    cfg["hyper_parameters"]["neighbor"]["skin"] = case.get("skin", 0.0)
    boxes = ([Box(tuple(s["lo"][r]), tuple(s["hi"][r])) for r in range(len(offs) - 1)] if offs is not None
             else Box(tuple(s["lo"]), tuple(s["hi"])))
    ff = ForceField(cfg, boxes)
    ff.set_pair_coeffs(s["eps"], s["sigma"])
    return ff


def _network(seed):
    """Parameters of a proposal network with output of order one, the size that training reaches."""
    rng = np.random.default_rng(seed + 5)
    p = np.zeros(5313, np.float32)
    p[:1024] = rng.normal(size=1024) / 4.0
    p[1088:5184] = rng.normal(size=4096) / 8.0
    p[5248:5312] = 0.1 * rng.normal(size=64)
    return p


def run(state):
    kind = state["kind"]
    if kind == "rhok":
        st = library().rbmd_rhok_noalloc(state["pos"].data_ptr(), state["q"].data_ptr(), state["n"], state["box"],
                                         state["m"].data_ptr(), state["P"], state["rho"].data_ptr(),
                                         torch.cuda.current_stream().cuda_stream)
        if st != 0:
            raise RuntimeError(library().rbmd_last_error().decode())
        return state["rho"]
    ff, t = state["ff"], state["t"]
    if kind == "force":
        ff.Execute()
        return t["force"]
    if kind == "host":
        ff.compute_host(state["ph"], state["fh"])
        return state["fh"]
    if kind == "step":
        ff.step(state["case"]["steps"])
        return dict(pos=t["pos"], vel=t["vel"], force=t["force"])
    c = state["case"]
    rep = ff.train_proposal(n_snapshots=c["snapshots"], steps_between=c["between"], k_per_snapshot=c["k"],
                            iterations=c["iterations"], seed=3)
    return dict(loss=[rep[k] for k in ("loss_gauss", "loss_first", "loss_final", "loss_optimum")],
                params=ff.proposal_params(), pos=t["pos"], vel=t["vel"], force=t["force"])


# ---- work -------------------------------------------------------------------------------------------
def _atoms(c):
    s = c.get("system")
    if s in ("lj", "eam"):
        return 4 * c["ncell"] ** 3
    if s == "water":
        return 3 * c["n_mol"]
    if s == "replicas":
        return int(_replica_sizes(c["n_rep"]).sum())
    if s == "chains":
        return TILE_ATOMS * c["kx"] * c["ky"] * c["kz"]
    return c["n"]


def work(case):
    """Bytes: per step positions and velocities read and written, forces written, masses and charges
    read; per force call positions and charges in, forces out.  Flops: 30 per pair inside the cutoff (both
    directions, as every atom's force is wanted), 20 per (charged atom, k) of the structure factors and
    the k-space force each (sine and cosine counted as one operation)."""
    c, k = case, case["kind"]
    if k == "rhok":
        return dict(bytes=32.0 * c["n"] + 28.0 * c["P"], flops=10.0 * c["n"] * c["P"])
    n = _atoms(c)
    charged = {"lj": 0.0, "eam": 0.0, "water": 1.0, "chains": 1.0, "replicas": 0.1}.get(c["system"], c.get("ion_frac", 0.1))
    dens, rc = {"lj": (0.8442, 2.5), "electrolyte": (0.8, 2.5), "replicas": (0.8, 2.5), "water": (0.1003, 10.0),
                "eam": (4 / 3.615 ** 3, 5.0), "chains": (TILE_ATOMS / (TILE_SITES * TILE_CELL ** 3), 12.0)}[c["system"]]
    pairs = n * dens * 4.0 / 3.0 * math.pi * rc ** 3
    if c.get("neighbor") == "RBL":   # core pairs, and about 100 kept shell pairs an atom
        pairs = n * min(pairs / n, dens * 4.0 / 3.0 * math.pi * 6.0 ** 3 + 100.0)
    kflops = 20.0 * charged * n * c.get("P", 0)
    flops = 30.0 * pairs + kflops
    if k == "step":
        return dict(bytes=136.0 * n * c["steps"], flops=flops * c["steps"])
    if k == "train":
        rows = 256.0 * c["snapshots"] * c["iterations"]
        net = rows * 6.0 * (16 * 64 + 64 * 64 + 64)
        data = 20.0 * charged * n * c["k"] * c["snapshots"]
        return dict(bytes=136.0 * n * c["snapshots"] * c["between"] + 8.0 * 5313 * c["iterations"],
                    flops=flops * c["snapshots"] * c["between"] + net + data)
    per = {"f32": 24.0, "f64": 48.0}[c.get("host", "f64")] + 8.0
    return dict(bytes=per * n, flops=flops)


# ---- tolerance --------------------------------------------------------------------------------------
def tolerance(case):
    """About four times the difference between the same call in 32 and in 64 bits, the size of a change
    of every rounding in 32 bits: positions rounded to floats carry 1e-5 into the pair forces, and the kept
    shell pairs of RBL change when a pair crosses r_core; in 64 bits only the order of sums is free.  The
    training rounds its activations to BF16, which moves single parameters."""
    c = case
    if c["kind"] == "train":
        return {"rel": 3e-3, "max": 0.2}
    if c["kind"] == "rhok":
        return {"rel": 4e-6, "max": 4e-5}
    if c["precision"] == "fp64" and c.get("host") != "f32":
        return {"rel": 1e-12, "max": 1e-10}
    if c["kind"] in ("host", "force"):
        return {"rel": 7e-5, "max": 4e-3}
    if c.get("neighbor") == "RBL":
        return {"rel": 7e-4, "max": 0.25}
    return {"rel": 2e-4, "max": 1.5e-2}


# ---- exact ------------------------------------------------------------------------------------------
def _pairs(pos, L, rc):
    """Chunks (i, j, r = p_j - p_i, d2, mask) of the pairs closer than rc in a periodic box of at least
    3 rc per edge, in 64 bits: cells of edge >= rc, every atom against the atoms of 27 cells."""
    dev = pos.device
    dims = torch.floor(L / rc).to(torch.int64)
    ncell = int(dims.prod())
    ci = torch.minimum((pos / (L / dims)).to(torch.int64).clamp_min(0), dims - 1)
    cid = (ci[:, 0] * dims[1] + ci[:, 1]) * dims[2] + ci[:, 2]
    order = torch.argsort(cid)
    cnt = torch.bincount(cid, minlength=ncell)
    M = int(cnt.max())
    start = torch.cumsum(cnt, 0) - cnt
    table = torch.full((ncell, M), -1, dtype=torch.int64, device=dev)
    table[cid[order], torch.arange(pos.shape[0], device=dev) - start[cid[order]]] = order
    o = torch.stack(torch.meshgrid(*[torch.arange(-1, 2, device=dev)] * 3, indexing="ij"), -1).reshape(-1, 3)
    step = max(1, int(1.5e7 // (27 * M * M)))
    for a in range(0, ncell, step):
        cells = torch.arange(a, min(ncell, a + step), device=dev)
        xyz = torch.stack([cells // (dims[1] * dims[2]), (cells // dims[2]) % dims[1], cells % dims[2]], -1)
        w = (xyz[:, None] + o) % dims
        j = table[(w[..., 0] * dims[1] + w[..., 1]) * dims[2] + w[..., 2]].reshape(len(cells), 1, -1)
        i = table[cells][:, :, None]
        r = pos[j] - pos[i]
        r = r - L * torch.round(r / L)
        d2 = (r * r).sum(-1)
        mask = (i >= 0) & (j >= 0) & (i != j) & (rc * rc - d2 > 1e-4) & (d2 > 1e-4)
        yield i, j, r, torch.where(mask, d2, torch.ones_like(d2)), mask


def _near(pos, L, rc, q=None, alpha=None):
    F = torch.zeros_like(pos)
    for i, j, r, d2, mask in _pairs(pos, L, rc):
        s6 = 1.0 / d2 ** 3
        f = -24.0 * (2.0 * s6 - 1.0) * s6 / d2
        if q is not None:
            d = torch.sqrt(d2)
            g = (torch.special.erfc(math.sqrt(alpha) * d) / d2
                 + 2.0 * math.sqrt(alpha / math.pi) * torch.exp(-alpha * d2) / d)
            f = f - q[i] * q[j] * g / d
        f = torch.where(mask, f, torch.zeros_like(f))
        keep = i[..., 0] >= 0
        F[i[..., 0][keep]] += (f[..., None] * r).sum(2)[keep]
    return F


def _eam(pos, L, rc):
    p = systems.JOHNSON_CU
    den = torch.zeros(pos.shape[0], dtype=torch.float64, device=pos.device)
    rho = lambda d: p["fe"] * torch.exp(-p["beta"] * (d / p["re"] - 1.0))        # noqa: E731
    phi = lambda d: p["phi_e"] * torch.exp(-p["gamma"] * (d / p["re"] - 1.0))    # noqa: E731
    for i, j, r, d2, mask in _pairs(pos, L, rc):
        keep = i[..., 0] >= 0
        den[i[..., 0][keep]] += torch.where(mask, rho(torch.sqrt(d2)), torch.zeros_like(d2)).sum(-1)[keep]
    fp = -0.5 * p["Ec"] / torch.sqrt(den * p["rho_e"])
    F = torch.zeros_like(pos)
    for i, j, r, d2, mask in _pairs(pos, L, rc):
        d = torch.sqrt(d2)
        dE = -p["gamma"] / p["re"] * phi(d) - (fp[i] + fp[j]) * p["beta"] / p["re"] * rho(d)
        f = torch.where(mask, dE / d, torch.zeros_like(d))
        keep = i[..., 0] >= 0
        F[i[..., 0][keep]] += (f[..., None] * r).sum(2)[keep]
    return F


def _kspace(pos, q, L, m, alpha):
    """RBE force of the given samples: (S / P) sum_l (-4 pi / (V k^2)) k (cos Im rho - sin Re rho) q_i."""
    S = 1.0
    for d in range(3):
        a = alpha * float(L[d]) ** 2
        S *= math.sqrt(a / math.pi) * sum(math.exp(-a * k * k) for k in range(-10, 11))
    S -= 1.0
    idx = torch.nonzero(q != 0)[:, 0]
    x, qq = pos[idx], q[idx]
    F = torch.zeros_like(pos)
    P = m.shape[0]
    for a in range(0, P, 50):
        k = 2.0 * math.pi * m[a:a + 50].to(torch.float64) / L
        ph = x @ k.T
        c, s = torch.cos(ph), torch.sin(ph)
        re, im = (qq[:, None] * c).sum(0), (qq[:, None] * s).sum(0)
        w = -4.0 * math.pi / (L.prod() * (k * k).sum(1)) * S / P
        F[idx] += qq[:, None] * ((c * im - s * re) * w) @ k
    return F


def exact(case, seed):
    dev = torch.device("cuda")
    f64 = lambda a: torch.tensor(np.asarray(a), device=dev, dtype=torch.float64)   # noqa: E731
    if case["kind"] == "rhok":
        pos, q, L, m = _rhok_inputs(case, seed)
        x, qq, out = f64(pos), f64(q), []
        for a in range(0, case["P"], 32):
            ph = x @ (2.0 * math.pi / L * f64(m[a:a + 32])).T
            out.append(torch.stack([(qq[:, None] * torch.cos(ph)).sum(0), (qq[:, None] * torch.sin(ph)).sum(0)], -1))
        return torch.cat(out)
    if case["kind"] in ("force", "host"):
        s, cfg, _ = _system(case, seed)
        pos = s["pos"].astype(np.float32) if case.get("host") == "f32" else s["pos"]
        alpha = cfg["hyper_parameters"]["coulomb"]["alpha"]
        L, q = f64(s["hi"]), f64(s["charge"])
        F = _near(f64(pos), L, 2.5, q, alpha)
        F += _kspace(f64(pos), q, L, torch.tensor(_kset(case, s["hi"], seed, alpha), device=dev), alpha)
        return F.to(torch.float32).cpu().numpy() if case.get("host") == "f32" else (
            F.cpu().numpy() if case["kind"] == "host" else F)
    if case["kind"] == "step" and case["system"] in ("lj", "eam") and _atoms(case) * case["steps"] <= 3000000:
        s, cfg, _ = _system(case, seed)
        L, x, v = f64(s["hi"]), f64(s["pos"]), f64(s["vel"])
        metal = case["system"] == "eam"
        acc = (1.0 / 1.0364269e-4) / s["mass"][0] if metal else 1.0   # force units to acceleration
        dt = cfg["execution"]["timestep"]
        force = (lambda p: _eam(p, L, 5.0)) if metal else (lambda p: _near(p, L, 2.5))
        F = force(x)
        for _ in range(case["steps"]):
            v = v + 0.5 * dt * acc * F
            x = x + dt * v
            x = torch.where(x < 0, x + L, torch.where(x > L, x - L, x))
            F = force(x)
            v = v + 0.5 * dt * acc * F
        return dict(pos=x, vel=v, force=F)
    # the other steps draw their own random k-vectors, and so does the training
    return None
