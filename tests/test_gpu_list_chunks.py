"""The cell-cooperative list build and the chunked list walk at the sizes where they can go wrong:
rows of 0, 1, 2, .. entries (the last chunk is filled with the slot itself), cells of more than 32
atoms and stencils of more than one batch of candidates, 3-cell boxes, an initial capacity that
overflows.  The lists are those of the per-atom build entry for entry and the oracle's pair sets;
forces to the parity bars (1e-5 of the force rms in FP32, 1e-11 in FP64)."""
import numpy as np
import pytest

from copy_gpu_b200 import systems
from tests.helpers import jitter, make_ff, pair_sets_equal, rel_err, to_dev

pytestmark = pytest.mark.gpu

TOL = {"fp32": 1e-5, "fp64": 1e-11}


def _gas(n, L, seed):
    """n atoms on a jittered lattice of edge L: at least 0.8 apart, few or no neighbours each."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    pos = np.stack(np.unravel_index(rng.permutation(m ** 3)[:n], (m, m, m)), 1) * (L / m) + 0.1
    s = dict(pos=np.mod(pos + rng.uniform(-0.1, 0.1, pos.shape), L), vel=np.zeros((n, 3)), mass=np.ones(n),
             charge=np.zeros(n), type=np.zeros(n, np.int32), molecule=None, lo=np.zeros(3), hi=np.full(3, L),
             eps=np.ones(1), sigma=np.ones(1))
    return s


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("case", ["one", "sparse", "dense", "small_cap"])
def test_cell_list_edges(cuda, oracle_lib, prec, case):
    import torch
    if case == "one":            # a single atom: an empty row
        s, rc = _gas(1, 9.0, 1), 2.5
    elif case == "sparse":       # rows of 0 .. about 8 entries
        s, rc = _gas(2000, 21.0, 2), 2.5
    elif case == "small_cap":    # overflow of the initial capacity (rounded up to whole chunks)
        s, rc = _gas(700, 10.5, 3), 2.5
    else:                        # about 66 atoms a cell, 1800 candidates: three batches
        s = systems.lj_fcc(ncell=8, seed=2)
        s["pos"] = jitter(s["pos"], s["lo"], s["hi"], 0.08, seed=5)
        rc = 4.2
    ref = None
    for block in (0, 128):
        cfg = systems.lj_config(cutoff=rc, precision=prec)
        cfg["tuning"] = {"list_block": block, "force_block": 64}
        if case == "small_cap":
            cfg["hyper_parameters"]["neighbor"]["capacity"] = 5
        dev = to_dev(s, cuda)
        ff = make_ff(cfg, s, dev)
        ff.Execute()
        torch.cuda.synchronize()
        assert ff.status() == 0
        c, ids = ff.neighbors(512)
        out = (c, ids, dev["force"].cpu().numpy())
        if ref is None:
            ref = out
        else:
            assert all(np.array_equal(a, b) for a, b in zip(ref, out))
    pr = s["pos"].astype(np.float32) if prec == "fp32" else s["pos"]
    nl = oracle_lib.neighbors(pr, s["lo"], s["hi"], rc, prec)
    assert pair_sets_equal(ref[0], ref[1], nl[0], nl[1]) == -1
    if case != "one":
        want = oracle_lib.near_force(pr, s["lo"], s["hi"], rc, nl, prec=prec, sum_mode=1)
        assert rel_err(ref[2], want) <= TOL[prec]
    else:
        assert ref[0][0] == 0 and not ref[2].any()


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("block", [0, 1, 128])
@pytest.mark.parametrize("far", [1e30, -1e30, np.inf, -np.inf])
def test_atom_far_outside(cuda, prec, block, far):
    """An atom whose cell index saturates has no neighbours and leaves the others' rows alone."""
    import torch
    s = systems.lj_fcc(ncell=6, seed=2)
    s["pos"] = jitter(s["pos"], s["lo"], s["hi"], 0.05, seed=5)
    out = []
    for k in (None, 0, 1, 2):   # nowhere, then along each axis
        p = dict(s, pos=s["pos"].copy())
        if k is not None:
            p["pos"][11, k] = far
        cfg = systems.lj_config(cutoff=2.5, precision=prec)
        cfg["tuning"] = {"list_block": block, "force_block": 64}
        dev = to_dev(p, cuda)
        ff = make_ff(cfg, p, dev)
        ff.Execute()
        torch.cuda.synchronize()
        c, ids = ff.neighbors(128)
        assert (ff.status() != 0) == (k is not None and not np.isfinite(far))
        out.append([set(ids[i, :c[i]].tolist()) for i in range(len(c))])
        ff.close()
    for rows in out[1:]:
        assert not rows[11] and all(r == ref - {11} for i, (r, ref) in enumerate(zip(rows, out[0])) if i != 11)
