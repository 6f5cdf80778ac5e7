"""Kernels chosen by size against the ones that a configuration can force: the same answers on both
sides of each line, and the choice no slower than what it replaced (event times of the phase, best of
15 calls, with a margin of 30 % for their spread)."""
import numpy as np
import pytest

from copy_gpu_b200 import systems
from tests.helpers import jitter, make_ff, rel_err, to_dev

pytestmark = pytest.mark.gpu


def _phase_us(s, cfg, phase, calls=15):
    """Shortest time of one phase of a force call, in microseconds."""
    dev = to_dev(s, "cuda", with_vel=False)
    ff = make_ff(cfg, s, dev)
    ff.Execute()
    ff.profile(True)
    best, last = 1e30, ff.phase_ms()[phase]
    for _ in range(calls):
        ff.Execute()
        now = ff.phase_ms()[phase]
        best, last = min(best, (now[0] - last[0]) / (now[1] - last[1])), now
    assert ff.status() == 0
    ff.close()
    return 1e3 * best


def _rbl_config(prec, rc, rcore, mode):
    cfg = systems.lj_config(cutoff=rc, precision=prec)
    cfg["hyper_parameters"]["neighbor"].update(type="RBL", r_core=rcore, neighbor_sample_num=50)
    cfg["tuning"] = {"rbl_list": mode}
    return cfg


# (atoms, density, cutoff, core radius): sparse cells (one thread per atom), few atoms (one warp per
# atom), and two sizes at which one warp per cell is the fastest
@pytest.mark.parametrize("n,rho,rc,rcore", [(150000, 0.1, 6.0, 2.0), (150000, 0.8, 2.5, 1.25), (2000, 0.8, 5.0, 2.5),
                                            (40000, 0.8, 5.0, 2.5), (150000, 0.8, 5.0, 2.5)])
def test_rbl_list_choice_is_not_slower(cuda, n, rho, rc, rcore):
    s = systems.electrolyte(n, rho=rho, ion_frac=0.0)
    us = {m: _phase_us(s, _rbl_config("fp32", rc, rcore, m), "neighbor_list") for m in ("auto", "warp", "thread")}
    assert us["auto"] <= 1.3 * min(us["warp"], us["thread"]), us


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("case", ["below", "above", "dense", "wide", "outside"])
def test_rbl_list_choice_same_lists(cuda, prec, case):
    import torch
    # below / above: the first size at which a warp takes a cell, and one atom less; dense: about 54 atoms
    # a cell and many batches of candidates; wide: 7 stencil cells per axis; outside: atoms beyond the faces
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if case in ("below", "above"):
        s = systems.electrolyte((100 if prec == "fp64" else 64) * sms - (case == "below"), ion_frac=0.0)
        rc, rcore = 5.0, 2.5
    else:
        s = systems.lj_fcc(ncell=16, seed=4)
        s["pos"] = jitter(s["pos"], s["lo"], s["hi"], 0.08, seed=5)
        rc, rcore = {"dense": (8.0, 4.2), "wide": (5.9, 2.0), "outside": (5.0, 2.6)}[case]
        if case == "outside":
            s["pos"][:500] += np.random.default_rng(8).uniform(-1.2, 1.2, size=(500, 3))
    out = []
    for mode in ("auto", "thread"):
        dev = to_dev(s, cuda)
        ff = make_ff(_rbl_config(prec, rc, rcore, mode), s, dev)
        ff.Execute()
        torch.cuda.synchronize()
        assert ff.status() == 0
        out.append(ff.neighbors(1024) + ff.rbl_lists()[:2] + (dev["force"].cpu().numpy(),))
        ff.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def _two_types(n, rho, prec, charged):
    """Atoms of two LJ types (the general near pass), one in ten charged."""
    s = systems.electrolyte(n, rho=rho, ion_frac=0.1)
    s["type"] = (np.arange(n) % 2).astype(np.int32)
    s["eps"], s["sigma"] = np.array([1.0, 0.8]), np.array([1.0, 0.95])
    if not charged:
        s["charge"][:] = 0
        return s, systems.lj_config(cutoff=2.5, precision=prec)
    return s, systems.electrolyte_config(P=32, precision=prec)


@pytest.mark.parametrize("n,rho,prec,charged", [(300000, 0.8, "fp64", True), (300000, 0.8, "fp64", False),
                                                (1000000, 0.1, "fp32", False), (60000, 0.1, "fp64", True),
                                                (30000, 0.8, "fp32", True), (4000, 0.8, "fp64", True)])
def test_near_lanes_choice_is_not_slower(cuda, n, rho, prec, charged):
    s, cfg = _two_types(n, rho, prec, charged)
    us = {}
    for lanes in (0, 1, 4, 8, 16):
        cfg["tuning"] = {"force_lanes": lanes} if lanes else {}
        us[lanes] = _phase_us(s, cfg, "force")
    assert us[0] <= 1.3 * min(us[k] for k in (1, 4, 8, 16)), us


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("charged", [False, True])
def test_every_forced_lane_count_runs(cuda, prec, charged):
    """Lanes 1 .. 32 of the pass for one LJ coefficient pair: the parity bars against one thread per atom,
    and in FP64 sums in another order for every count (rows of about 210 entries, 54 chunks; the butterfly
    adds rows of up to 32 chunks alike with 16 and 32 lanes), so that no count runs as another one (FP32
    adds the chunks in two-float sums, exact enough to agree)."""
    import torch
    s = systems.electrolyte(3000, ion_frac=0.2, seed=9)
    if not charged:
        s["charge"][:] = 0
    out = {}
    for lanes in (1, 4, 8, 16, 32):
        cfg = (systems.electrolyte_config(P=16, cutoff=4.0, precision=prec) if charged
               else systems.lj_config(cutoff=4.0, precision=prec))
        cfg["tuning"] = {"force_lanes": lanes}
        dev = to_dev(s, cuda)
        ff = make_ff(cfg, s, dev)
        if charged:
            ff.set_ksamples(np.array([[1, 0, 0], [0, 1, 0], [0, 0, 1], [1, 1, 0]] * 4, np.int32))
        ff.Execute()
        torch.cuda.synchronize()
        assert ff.status() == 0
        out[lanes] = dev["force"].cpu().numpy()
        ff.close()
    bar = 1e-5 if prec == "fp32" else 1e-11
    for a in out:
        assert rel_err(out[a], out[1]) <= bar
        for b in out:
            assert prec == "fp32" or a == b or not np.array_equal(out[a], out[b]), (a, b)


@pytest.mark.parametrize("skin", [0.0, 0.3])
@pytest.mark.parametrize("scale,sigma", [(2000.0, 2000.0), (1100.0, 1100.0), (2e5, 100.0), (1.0, 0.0)])
def test_lj_range_in_float(cuda, scale, sigma, skin):
    """LJ in units whose 48 eps sigma^12 (or d^-8) leaves the range of floats, and just inside it: the FP32
    pass against the FP64 pass at the same float positions, parity bar of FP32."""
    import torch
    s = systems.lj_fcc(ncell=7, seed=3)
    s["pos"] = (jitter(s["pos"], s["lo"], s["hi"], 0.05, seed=4) * scale).astype(np.float32).astype(np.float64)
    s["hi"] = s["hi"] * scale
    s["sigma"] = np.array([sigma])
    s["pos"] = np.minimum(s["pos"], np.nextafter(s["hi"].astype(np.float32), np.float32(0)).astype(np.float64))
    out = []
    for prec in ("fp32", "fp64"):
        cfg = systems.lj_config(cutoff=2.5 * scale, precision=prec)
        cfg["hyper_parameters"]["neighbor"]["skin"] = skin * scale
        dev = to_dev(s, cuda)
        ff = make_ff(cfg, s, dev)
        ff.Execute()
        torch.cuda.synchronize()
        assert ff.status() == 0
        out.append(dev["force"].cpu().numpy())
        ff.close()
    if sigma == 0.0:
        assert not out[0].any() and not out[1].any()
    else:
        assert rel_err(out[0], out[1]) <= 1e-5
