"""The contact walks (a warp per eight agents for few rows, a thread per agent
for many) against the CPU oracle, bit for bit, where their lists can go wrong."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle
from oncolytica_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["even", "corner", "crowd", "scattered", "coincident"])
@pytest.mark.parametrize("n", [1, 7, 9, 65, 2500, 49152, 49153])
def test_contact_lists_bit_exact(cuda, olc, n, case):
    """Blocks with one agent and a last one that is not full; agents at the grid's
    faces; more candidates and near ones than a list holds (300 agents in one bin);
    a table whose bins do not follow one another in the order of their keys; and
    more than a list's worth of agents in one point."""
    import torch

    rng = np.random.default_rng(n)
    dims, vs = (24, 22, 20), 10.0
    top = np.array(dims) * vs
    pos = rng.uniform(0.0, 1.0, (n, 3)) * (top * (0.1 if n < 1000 else 1.0))
    if case == "corner":
        pos = np.where(rng.random((n, 3)) < 0.5, pos * 0.25, top - 0.25 * pos)
    if case == "crowd":
        pos[: min(n, 300)] = 100.0 + 9.9 * rng.random((min(n, 300), 3))
    if case == "coincident":
        pos[: min(n, 40)] = 55.0
    pos = np.minimum(pos, top - 0.01).astype(np.float32)
    ks, perm = oracle.sort_pairs(oracle.keys(pos, dims, vs))
    ranges = oracle.bin_ranges(ks, oracle.tissue_key(*dims)).reshape(-1, 2).copy()
    posr = np.concatenate([pos[perm], rng.uniform(4.0, 6.0, (n, 1))], axis=1).astype(np.float32)
    posr[rng.random(n) < 0.03, 3] = -1.0
    if case == "scattered":
        bins = rng.permutation(np.flatnonzero(ranges[:, 1] > ranges[:, 0]))
        order, at = [], 0
        for b in bins:
            lo, hi = ranges[b]
            order.append(np.arange(lo, hi))
            ranges[b] = at, at + hi - lo
            at += int(hi - lo)
        posr = posr[np.concatenate(order)]
    rows = len(posr)
    lo, hi = (0.1, 0.1, 0.1), tuple(float(t) - 0.1 for t in top)
    ref = oracle.contact(posr, ranges.reshape(-1), dims, vs, 1.0, 10.0, 1.0, 0.1, lo, hi)
    pr = torch.from_numpy(np.ascontiguousarray(posr)).to(cuda)
    rg = torch.from_numpy(ranges.astype(np.uint32).view(np.int32).copy()).to(cuda)
    xyz = [torch.from_numpy(np.ascontiguousarray(posr[:, a])).to(cuda) for a in range(3)]
    g = _lib.OlcGeom()
    g.tissue_dims[:] = dims
    g.tissue_voxel_size = vs
    g.chem_dims[:] = (0, 0, 0)
    g.chem_voxel_size = 1.0
    g.domain_lo[:] = (0, 0, 0)
    g.domain_hi[:] = tuple(float(t) for t in top)
    spec = _lib.OlcContact(enabled=1, radius_field=-1, radius_const=0.0, stiffness=1.0, mobility=10.0, max_disp=1.0,
                           margin=0.1)
    ptr = [C.c_void_p(t.data_ptr()) for t in (pr, rg, *xyz)]
    _lib.check(olc.olc_stage_contact(ptr[0], ptr[1], rows, C.byref(g), C.byref(spec), 0.1, *ptr[2:], None))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(np.stack([t.cpu().numpy() for t in xyz], axis=1), ref)



@pytest.mark.parametrize("per_bin", [17, 40, 127, 129])
@pytest.mark.parametrize("agents", [300, 3000])
def test_contact_lists_that_fill_in_mid_bin(cuda, olc, agents, per_bin):
    """Many bins so full that the warps' lists of near pairs fill up again and again,
    between and within the agents' shares: every pair listed just before must be seen
    by the lane that computes it."""
    import torch

    rng = np.random.default_rng(agents + per_bin)
    dims, vs = (12, 10, 8), 10.0
    top = np.array(dims) * vs
    bins = np.stack([rng.integers(0, d, -(-agents // per_bin)) for d in dims], axis=1)
    pos = (np.repeat(bins, per_bin, axis=0)[:agents] + 0.98 * rng.random((agents, 3))) * vs
    pos = np.minimum(pos, top - 0.01).astype(np.float32)
    ks, perm = oracle.sort_pairs(oracle.keys(pos, dims, vs))
    ranges = oracle.bin_ranges(ks, oracle.tissue_key(*dims)).reshape(-1, 2).copy()
    posr = np.concatenate([pos[perm], rng.uniform(4.0, 6.0, (agents, 1))], axis=1).astype(np.float32)
    lo, hi = (0.1, 0.1, 0.1), tuple(float(t) - 0.1 for t in top)
    ref = oracle.contact(posr, ranges.reshape(-1), dims, vs, 1.0, 10.0, 1.0, 0.1, lo, hi)
    pr = torch.from_numpy(posr).to(cuda)
    rg = torch.from_numpy(ranges.astype(np.uint32).view(np.int32).copy()).to(cuda)
    g = _lib.OlcGeom()
    g.tissue_dims[:] = dims
    g.tissue_voxel_size = vs
    g.chem_voxel_size = 1.0
    g.domain_hi[:] = tuple(float(t) for t in top)
    spec = _lib.OlcContact(enabled=1, radius_field=-1, stiffness=1.0, mobility=10.0, max_disp=1.0, margin=0.1)
    for _ in range(5):
        xyz = [torch.zeros(agents, device=cuda) for _ in range(3)]
        ptr = [C.c_void_p(t.data_ptr()) for t in (pr, rg, *xyz)]
        _lib.check(olc.olc_stage_contact(ptr[0], ptr[1], agents, C.byref(g), C.byref(spec), 0.1, *ptr[2:], None))
        torch.cuda.synchronize()
        np.testing.assert_array_equal(np.stack([t.cpu().numpy() for t in xyz], axis=1), ref)


@pytest.mark.parametrize("per_bin", [0.1, 0.4, 0.6, 2.4])
@pytest.mark.parametrize("agents", [19999, 20000, 24640, 30001, 49152])
def test_sparse_agents_get_a_thread_each(cuda, olc, agents, per_bin):
    """Sizes on either side of the least where sparse agents get a thread each, at grids
    of more and fewer bins than that takes: at faces, with dead agents, and with pairs
    that touch."""
    import torch

    rng = np.random.default_rng(agents + int(100 * per_bin))
    vs = 10.0
    d = max(4, 2 * int(round((agents / per_bin) ** (1 / 3) / 2)))
    dims = (min(d, 120),) * 3
    top = np.array(dims) * vs
    pos = rng.uniform(0.0, 1.0, (agents, 3)) * top
    pairs = rng.random(agents) < 0.3  # close to another one
    pos[pairs] = pos[rng.integers(0, agents, int(pairs.sum()))] + rng.uniform(-6, 6, (int(pairs.sum()), 3))
    pos = np.clip(pos, 0.0, top - 0.01).astype(np.float32)
    ks, perm = oracle.sort_pairs(oracle.keys(pos, dims, vs))
    ranges = oracle.bin_ranges(ks, oracle.tissue_key(*dims)).reshape(-1, 2).copy()
    posr = np.concatenate([pos[perm], rng.uniform(4.0, 6.0, (agents, 1))], axis=1).astype(np.float32)
    posr[rng.random(agents) < 0.1, 3] = -1.0
    lo, hi = (0.1, 0.1, 0.1), tuple(float(t) - 0.1 for t in top)
    ref = oracle.contact(posr, ranges.reshape(-1), dims, vs, 1.0, 10.0, 1.0, 0.1, lo, hi)
    pr = torch.from_numpy(posr).to(cuda)
    rg = torch.from_numpy(ranges.astype(np.uint32).view(np.int32).copy()).to(cuda)
    xyz = [torch.from_numpy(np.ascontiguousarray(posr[:, a])).to(cuda) for a in range(3)]
    g = _lib.OlcGeom()
    g.tissue_dims[:] = dims
    g.tissue_voxel_size = vs
    g.chem_voxel_size = 1.0
    g.domain_hi[:] = tuple(float(t) for t in top)
    spec = _lib.OlcContact(enabled=1, radius_field=-1, stiffness=1.0, mobility=10.0, max_disp=1.0, margin=0.1)
    ptr = [C.c_void_p(t.data_ptr()) for t in (pr, rg, *xyz)]
    _lib.check(olc.olc_stage_contact(ptr[0], ptr[1], agents, C.byref(g), C.byref(spec), 0.1, *ptr[2:], None))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(np.stack([t.cpu().numpy() for t in xyz], axis=1), ref)
