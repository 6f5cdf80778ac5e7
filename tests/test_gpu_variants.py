"""Kernel variants chosen by size, at the edges of their rules.

* EAM in FP32 with the spline rows in shared memory (the longest table that fits; one row more falls
  back to the global tables) against the FP64 passes on the same file and the same float positions, to
  what the float image positions allow (see the test); boxes of 2 cells per axis (per-pair minimum
  image) and of 3.
* RBL lists built by one warp per cell (the default) equal those of one thread per atom entry for
  entry, from a few atoms to cells of more than 32 atoms and several batches of candidates.
* Lanes per charged atom of the RBE force and short structure-factor chunks: one to a few thousand
  charged atoms against the FP64 oracle, no worse than 1e-5 of the largest force (FP32 bar).
* Lanes per atom with types, molecules, special bonds and boxes of two cells per axis (per-pair minimum
  image) against one thread per atom, forces and energies: the parity bars of each precision.
* A step call that starts with the graph of an earlier call: many short calls, with force calls, an
  injected k-set and velocities read back between them, bit for bit as without graphs.
* A step call replayed because its list overflowed draws the k-sets of the call's own steps and starts from
  its thermostat, noise counter and conditioning spectrum: bit for bit the trajectory of a run whose
  first capacity is large enough.
"""
import numpy as np
import pytest

from copy_gpu_b200 import systems
from tests.helpers import jitter, make_ff, rel_err, to_dev

pytestmark = pytest.mark.gpu


def _eam_force(s, path, prec, cuda):
    import torch
    cfg = systems.eam_config(path, precision=prec)
    cfg["hyper_parameters"]["force_field"]["potential_format"] = "setfl"
    dev = to_dev(s, cuda)
    ff = make_ff(cfg, s, dev)
    ff.Execute()
    torch.cuda.synchronize()
    assert ff.status() == 0
    e = ff.energy()
    return dev["force"].cpu().numpy(), e["eam_embed"] + e["eam_pair"]


@pytest.mark.parametrize("ncell,npts", [(4, 5000), (5, 5000), (5, 64), (9, 5000), (6, "longest"), (6, "one more"),
                                        (6, 9000)])
def test_eam_rows_in_shared_memory(cuda, tmp_path, ncell, npts):
    import torch
    if isinstance(npts, str):   # two tables of npts + 1 rows of 16 bytes in a block's shared memory
        limit = torch.cuda.get_device_properties(0).shared_memory_per_block_optin
        npts = limit // 32 - 1 + (npts == "one more")
    p = dict(systems.JOHNSON_CU, npts=npts)
    path = systems.write_johnson_setfl(str(tmp_path / "j.setfl"), p)
    s = systems.eam_fcc(ncell=ncell, seed=3)
    s["pos"] = s["pos"].astype(np.float32).astype(np.float64)
    s["pos"][s["pos"] >= s["hi"]] = 0.0
    f32, e32 = _eam_force(s, path, "fp32", cuda)
    f64, e64 = _eam_force(s, path, "fp64", cuda)
    # a neighbour's image lies within 2 L, where floats round to 2^-24 x 2 L; displacements of 0.131 A per axis
    # make the force, so that a shift of all neighbours by that much is 2^-23 L / 0.131 of its rms (8e-6 at 18 A
    # and 5e-6 at 33 A measured, the same with tables in global memory)
    bar = max(1e-5, 2.0 ** -23 * s["hi"][0] / 0.131)
    assert rel_err(f32, f64) <= bar, rel_err(f32, f64)
    assert abs(e32 - e64) <= 1e-6 * abs(e64)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("case", ["tiny", "chains", "dense", "wide", "outside"])
def test_rbl_cell_list_identical(cuda, prec, case):
    import torch
    if case == "chains":
        s = systems.molecular(n_chain=27, chain_len=12, n_ion_pairs=4, step=1.5, cell=8.0, seed=5)
        rc, rcore = 10.0, 5.0
    else:
        s = systems.lj_fcc(ncell={"tiny": 2, "dense": 8, "wide": 6, "outside": 7}[case], seed=4)
        s["pos"] = jitter(s["pos"], s["lo"], s["hi"], 0.08, seed=5)
        # tiny: fewer cells than the stencil; dense: about 75 atoms a cell; wide: num_cycles 3;
        # outside: atoms up to 1.2 beyond the faces, binned into the boundary cells
        rc, rcore = {"tiny": (1.6, 0.8), "dense": (8.0, 4.5), "wide": (3.4, 1.2), "outside": (3.0, 1.6)}[case]
        if case == "outside":
            rng = np.random.default_rng(8)
            s["pos"][:200] += rng.uniform(-1.2, 1.2, size=(200, 3))
    out = []
    for mode in ("auto", "thread"):
        cfg = systems.lj_config(cutoff=rc, precision=prec)
        cfg["hyper_parameters"]["neighbor"].update(type="RBL", r_core=rcore, neighbor_sample_num=20)
        cfg["tuning"] = {"rbl_list": mode}
        dev = to_dev(s, cuda)
        ff = make_ff(cfg, s, dev)
        ff.Execute()
        torch.cuda.synchronize()
        assert ff.status() == 0
        c, ids = ff.neighbors(1024)
        ncore, nshell, _ = ff.rbl_lists()
        out.append((c, ids, ncore, nshell, dev["force"].cpu().numpy()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("nq,P", [(2, 1), (2, 33), (66, 100), (258, 305), (3000, 64), (5000, 520)])
def test_kspace_small_counts(cuda, oracle_lib, nq, P):
    import torch
    s = systems.electrolyte(max(600, nq), ion_frac=min(1.0, nq / max(600, nq)), seed=5)
    cfg = systems.electrolyte_config(P=P, precision="fp32", seed=2)
    alpha = cfg["hyper_parameters"]["coulomb"]["alpha"]
    L = s["hi"] - s["lo"]
    m = oracle_lib.rbe_sample(alpha, L, seed=5, step=0, rep=0, P=P)
    dev = to_dev(s, cuda)
    ff = make_ff(cfg, s, dev)
    ff.set_ksamples(m)
    ff.Execute()
    torch.cuda.synchronize()
    rho = oracle_lib.rhok(s["pos"], s["charge"], L, m)
    far = oracle_lib.rbe_force(s["pos"], s["charge"], L, alpha, 1.0, m, rho)
    got = ff.far_force()
    assert np.abs(got - far).max() <= 1e-5 * np.abs(far).max()


@pytest.mark.parametrize("kind,skin", [("gauss", 0.3), ("gauss", 0.0), ("learned", 0.3), ("rescale", 0.3),
                                       ("nose_hoover", 0.3), ("langevin", 0.3)])
def test_step_calls_from_the_graph(cuda, kind, skin):
    import torch
    from oracle import mlp
    out = []
    for graph in (True, False):
        s = systems.electrolyte(1500, seed=21)
        cfg = systems.electrolyte_config(P=40, precision="fp32", seed=6)
        cfg["hyper_parameters"]["neighbor"]["skin"] = skin
        cfg["execution"]["cuda_graph"] = graph
        if kind == "learned":
            cfg["hyper_parameters"]["coulomb"]["proposal"] = "learned"
        elif kind != "gauss":
            cfg["execution"].update({"ensemble": "NVT", "temp_ctrl_type": {
                "rescale": "TEMP_RESCALE", "nose_hoover": "NOSE_HOOVER", "langevin": "LANGEVIN"}[kind],
                "temperature": [1.0, 1.0, 0.1]})
        dev = to_dev(s, cuda)
        ff = make_ff(cfg, s, dev)
        if kind == "learned":
            ff.proposal_params(mlp.init_params(2, scale=0.5))
        got = []
        for k, n in enumerate((1, 2, 1, 9, 1, 20, 3, 8, 1)):
            if k == 0 or k == 4:
                ff.Execute()
            if k == 6:
                ff.set_ksamples(np.array([[1, 0, 0], [0, 1, 0], [0, 0, 1], [1, 1, 0]] * 10, np.int32))
            ff.step(n)
            if k % 2:
                ff.sync_velocities()
                got.append(dev["vel"].cpu().numpy())
            got.append(dev["pos"].cpu().numpy())
        torch.cuda.synchronize()
        assert ff.status() == 0
        out.append((got, ff.list_builds()))
        ff.close()
    for a, b in zip(*[o[0] for o in out]):
        assert np.array_equal(a, b)
    assert out[0][1] == out[1][1]


@pytest.mark.parametrize("kind", ["gauss", "gauss_iid", "learned", "nose_hoover", "langevin"])
@pytest.mark.parametrize("n_steps,skin", [(1, 0.0), (1, 0.3), (5, 0.3), (12, 0.0)])
def test_step_replay_draws_its_own_k_sets(cuda, kind, n_steps, skin):
    import torch
    from oracle import mlp
    out = []
    for capacity in (0, 8):   # 0: by density; 8: every call's first attempt overflows on a fresh handle
        s = systems.electrolyte(1500, seed=23)
        cfg = systems.electrolyte_config(P=40, precision="fp32", seed=7)
        cfg["hyper_parameters"]["neighbor"]["skin"] = skin
        if kind in ("gauss", "gauss_iid", "learned"):
            cfg["hyper_parameters"]["coulomb"]["proposal"] = kind
        else:   # a thermostat with a state of its own
            cfg["execution"].update({"ensemble": "NVT", "temp_ctrl_type": kind.upper(), "temperature": [1.0, 1.0, 0.1]})
        if capacity:
            cfg["hyper_parameters"]["neighbor"]["capacity"] = capacity
        dev = to_dev(s, cuda)
        ff = make_ff(cfg, s, dev)
        if kind == "learned":
            ff.proposal_params(mlp.init_params(2, scale=0.5))
        ff.step(n_steps)
        torch.cuda.synchronize()
        assert ff.status() == 0
        got = [dev[k].cpu().numpy() for k in ("pos", "vel", "force")] + [ff.get_ksamples(40)]
        ff.step(2)
        torch.cuda.synchronize()
        out.append(got + [dev["pos"].cpu().numpy()])
        ff.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("case,skin", [("water", 0.0), ("water", 0.5), ("water_small", 0.0), ("chains", 0.0),
                                       ("chains", 0.5), ("chains_small", 0.0), ("chains_nospecial", 0.0),
                                       ("chains_nospecial", 0.5), ("types", 0.0), ("types", 0.3),
                                       ("types_small", 0.0), ("one_type", 0.0), ("one_type", 0.3)])
def test_lanes_match_one_thread(cuda, prec, case, skin):
    import torch
    if case.startswith("water"):
        s = systems.water(n_mol=300 if case == "water" else 90, seed=6)
        cfg = systems.water_config(P=16, precision=prec, cutoff=6.0)   # edges 20.8 and 13.9: 3 and 2 cells
    elif case.startswith("chains"):
        s = systems.molecular(n_chain=27 if case != "chains_small" else 8, chain_len=12, n_ion_pairs=4, step=1.5,
                              cell=8.0, seed=5)
        cfg = systems.molecular_config(P=16, cutoff=9.0, precision=prec,
                                       special=None if case == "chains_nospecial" else (0.0, 0.2, 0.5))
    else:   # two LJ coefficient pairs; one_type: the general pass forced by near_variant 0
        s = systems.electrolyte(200 if case == "types_small" else 1500, ion_frac=0.4, seed=8)   # 2 and 4 cells
        cfg = systems.electrolyte_config(P=16, precision=prec)
        if case != "one_type":
            s["eps"], s["sigma"] = np.array([1.0, 0.7, 0.7]), np.array([1.0, 0.9, 0.9])
    cfg["hyper_parameters"]["neighbor"]["skin"] = skin
    out = []
    for lanes in (1, 4, 8, 16, 32):
        cfg["tuning"] = {"force_lanes": lanes, "force_block": 128, "near_variant": 0 if case == "one_type" else 1}
        dev = to_dev(s, cuda)
        ff = make_ff(cfg, s, dev)
        if "bonds" in s:
            keys = ("molecule", "bonds", "bond_type", "bond_coeffs", "angles", "angle_type", "angle_coeffs",
                    "dihedrals", "dihedral_type", "dihedral_coeffs")
            ff.set_topology(*[s[k] for k in keys[:7 if case == "chains_nospecial" else 10]])
        ff.Execute()
        torch.cuda.synchronize()
        assert ff.status() == 0
        e = ff.energy()
        out.append((dev["force"].cpu().numpy(), e["lj"], e["coul_real"]))
        ff.close()
    # energies: the parity bar of FP64; in FP32 each lane adds up to 4 x 140 terms in a float, so that a row's
    # sum carries at most 560 x 2^-25 = 1.7e-5 of the terms it adds, of either sign from row to row
    bar, ebar = (1e-5, 1.7e-5) if prec == "fp32" else (1e-11, 1e-10)
    for f, lj, coul in out[1:]:
        assert rel_err(f, out[0][0]) <= bar
        scale = max(1.0, abs(out[0][1]), abs(out[0][2]))
        assert abs(lj - out[0][1]) <= ebar * scale
        assert abs(coul - out[0][2]) <= ebar * scale


@pytest.mark.parametrize("proposal", ["gauss", "gauss_iid"])
def test_steps_after_a_second_bind(cuda, proposal):
    """A handle bound to new arrays after steps draws their k-sets anew: bit for bit a fresh handle."""
    import torch
    cfg = systems.electrolyte_config(P=40, precision="fp32", seed=7)
    cfg["hyper_parameters"]["coulomb"]["proposal"] = proposal
    s = systems.electrolyte(1500, seed=23)
    out = []
    for first in (False, True):
        dev = to_dev(s, cuda)
        ff = make_ff(cfg, s, dev)
        if first:
            ff.step(3)
            dev = to_dev(s, cuda)
            ff.Init(dev["pos"], dev["force"], vel=dev["vel"], mass=dev["mass"], charge=dev["charge"],
                    type=dev["type"], image=dev["image"])
        ff.step(3)
        torch.cuda.synchronize()
        assert ff.status() == 0
        out.append([dev[k].cpu().numpy() for k in ("pos", "vel", "force")])
        ff.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
