"""Per-member reductions of a batch against sums over the members' own rows:
runs of rows shorter and longer than a warp, than a warp's share and than a
block's, and members that begin in the middle of one."""
from __future__ import annotations

import numpy as np
import pytest

from oncolytica_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f32", "f16_sr"])
@pytest.mark.parametrize("counts", [(1, 31, 33, 2), (511, 1, 513, 64), (5000, 300, 1), (40,) * 24])
def test_member_reductions_match_their_rows(cuda, counts, storage):
    specs = [W.TumourSpec(name=f"m{k}", n_agents=n, domain=128.0, ball_radius=45.0, field_dims=(32, 32, 32),
                          r_lo=4.0, r_hi=6.0, has_drug=True, death_k=0.3, init_drug=0.4, v_lo=1.9, seed=k,
                          storage=storage, capacity=3 * n + 64) for k, n in enumerate(counts)]
    b = W.build_batch(specs)
    b.run_steps(2, collect_metrics=True)
    for k, (sp, red) in enumerate(zip(specs, b.get_reductions())):
        snap = b.snapshot(k)
        live = snap["life"] == 0
        cols = {c: v[live] for c, v in snap["cols"].items()}
        pos = np.stack([cols["pos.x"], cols["pos.y"], cols["pos.z"]], 1).astype(np.float64)
        r2 = ((pos - np.asarray(sp.center, np.float64)) ** 2).sum(1)
        assert red["n_live"] == int(live.sum())
        np.testing.assert_array_equal(red["state_counts"], np.bincount(cols["state"], minlength=8)[:8])
        hist = np.bincount(np.minimum((np.sqrt(r2) / sp.bin_size).astype(int), 63), minlength=64)
        np.testing.assert_array_equal(red["radial_hist"], hist)
        # sums of n FP64 terms in two orders: n rounding errors of the running sum at most
        tol = 4 * max(len(pos), 1) * 2.0 ** -53
        np.testing.assert_allclose(red["sum_pos"], pos.sum(0), rtol=tol)
        np.testing.assert_allclose(red["sum_r2"], r2.sum(), rtol=tol)
        np.testing.assert_allclose(red["max_r"], np.sqrt(r2).max() if len(r2) else 0.0, rtol=2.0 ** -50)
        if storage == "f32":
            for f in ("o2", "drug"):
                v = snap["fields"][f].astype(np.float64)
                np.testing.assert_allclose(red["field_mass"][f], v.sum(), rtol=4 * v.size * 2.0 ** -53)
                assert red["field_min"][f] == v.min() and red["field_max"][f] == v.max()


@pytest.mark.parametrize("counts", [(300,) * 40, (30,) * 80, (40_000, 20, 90_000, 33)])
def test_reductions_with_shares_of_every_size(cuda, counts):
    """Few rows, one 32-row run per warp; many, longer runs; members that change
    within and between them."""
    test_member_reductions_match_their_rows(cuda, counts, "f32")
