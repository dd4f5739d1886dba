"""The autotuner (oncolytica_b200.autotune) and the choices it makes.

Every kernel shape and variant it chooses between must give the same bits:
each stencil tile and contact walk of a solo engine, and each batched FP32
tile depth, are run from one initial state and compared with the defaults.
Tuning itself restores the engine's state (the run continues bit for bit as
if it had not been tuned), and a second tuning of the same shape comes from
the cache."""
from __future__ import annotations

import numpy as np
import pytest

from oncolytica_b200 import _lib, autotune
from oncolytica_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _spec(dense: bool = False):
    # dense: ~100 agents per 10 um bin
    return W.scaled(W.SCALE, n_agents=30_000, domain=320.0, ball_radius=40.0 if dense else 90.0,
                    field_dims=(64, 64, 64), capacity=150_000, seed=4, uptake=2.0, death_k=0.2, init_drug=0.1,
                    v_lo=1.85, v_hi=2.0)


def _same(a: dict, b: dict, what: str) -> None:
    assert a["rows"] == b["rows"], what
    np.testing.assert_array_equal(a["life"], b["life"], err_msg=what)
    for k in a["cols"]:
        np.testing.assert_array_equal(a["cols"][k], b["cols"][k], err_msg=f"{what} {k}")
    for k in a["fields"]:
        np.testing.assert_array_equal(a["fields"][k], b["fields"][k], err_msg=f"{what} {k}")


@pytest.mark.parametrize("tile", autotune.STENCIL_TILES)
@pytest.mark.parametrize("contact", autotune.CONTACT_VARIANTS)
def test_every_choice_gives_the_same_bits(cuda, tile, contact):
    spec = _spec()
    state = W.initial_state(spec)
    ref = W.build_engine(spec, state)
    ref.run_steps(3)
    eng = W.build_engine(spec, state)
    eng._backend_impl.set_tuning(stencil_tile=tile, contact_variant=contact)
    assert eng._backend_impl.get_tuning()["stencil_tile"] == tuple(tile)
    eng.run_steps(3)
    _same(eng._backend_impl.snapshot(), ref._backend_impl.snapshot(), f"tile {tile} contact {contact}")


@pytest.mark.parametrize("pair", [p for p in autotune.STENCIL_PAIRS if p[0]] + [(256, 7)])
def test_two_substeps_per_pass_give_the_same_bits(cuda, pair):
    spec = _spec()
    state = W.initial_state(spec)
    ref = W.build_engine(spec, state)
    ref.run_steps(3)
    eng = W.build_engine(spec, state)
    eng._backend_impl.set_tuning(stencil_pair=pair)
    assert eng._backend_impl.get_tuning()["stencil_pair"] == tuple(pair)
    eng.run_steps(3)
    _same(eng._backend_impl.snapshot(), ref._backend_impl.snapshot(), f"pair {pair}")


@pytest.mark.parametrize("keep", [k for k in autotune.L2_KEEP if k] + [100])
def test_l2_resident_slab_gives_the_same_bits(cuda, keep):
    spec = _spec()
    state = W.initial_state(spec)
    ref = W.build_engine(spec, state)
    ref.run_steps(3)
    eng = W.build_engine(spec, state)
    eng._backend_impl.set_tuning(l2_keep_pct=keep)
    assert eng._backend_impl.get_tuning()["l2_keep_pct"] == keep
    eng.run_steps(3)
    _same(eng._backend_impl.snapshot(), ref._backend_impl.snapshot(), f"l2 keep {keep}")


@pytest.mark.parametrize("contact", autotune.CONTACT_VARIANTS)
def test_contact_variants_agree_on_a_dense_population(cuda, contact):
    spec = _spec(dense=True)
    state = W.initial_state(spec)
    ref = W.build_engine(spec, state)
    ref.run_steps(2)
    eng = W.build_engine(spec, state)
    eng._backend_impl.set_tuning(contact_variant=contact)
    eng.run_steps(2)
    _same(eng._backend_impl.snapshot(), ref._backend_impl.snapshot(), f"dense, contact {contact}")


def test_tuning_restores_the_run_and_caches(cuda, tmp_path, monkeypatch):
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "tuning.json"))
    spec = _spec()
    state = W.initial_state(spec)
    ref = W.build_engine(spec, state)
    ref.run_steps(2)
    eng = W.build_engine(spec, state)
    eng.run_steps(1)
    rec = autotune.tune_engine(eng, steps=2)
    assert not rec["cached"]
    assert tuple(rec["tuning"]["stencil_tile"]) in autotune.STENCIL_TILES
    assert rec["tuning"]["contact_variant"] in autotune.CONTACT_VARIANTS
    assert {"substeps", "substep_pairs", "contact"} <= set(rec["measured_ms"])
    assert tuple(rec["tuning"]["stencil_pair"]) in autotune.STENCIL_PAIRS
    assert eng._backend_impl.get_tuning()["stencil_tile"] == tuple(rec["tuning"]["stencil_tile"])
    assert eng._step == 1 and eng._backend_impl.counters()["steps"] == 1
    eng.run_steps(1)
    _same(eng._backend_impl.snapshot(), ref._backend_impl.snapshot(), "after tuning")
    other = W.build_engine(spec, state)
    assert autotune.tune_engine(other, steps=2)["cached"]
    assert other._backend_impl.get_tuning() == eng._backend_impl.get_tuning()


def test_tuning_rejects_unknown_shapes(cuda):
    eng = W.build_engine(_spec())
    with pytest.raises(_lib.OlcError):
        eng._backend_impl.set_tuning(stencil_tile=(4, 4))
    with pytest.raises(_lib.OlcError):
        eng._backend_impl.set_tuning(batch_tile_depth=12)
    with pytest.raises(_lib.OlcError):
        eng._backend_impl.set_tuning(stencil_pair=(384, 0))
    with pytest.raises(_lib.OlcError):
        eng._backend_impl.set_tuning(l2_keep_pct=120)


def test_batch_tile_depths_give_the_same_bits(cuda, tmp_path, monkeypatch):
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "tuning.json"))
    specs = W.batched_specs(6, seed=3)
    states = [W.initial_state(sp) for sp in specs]
    ref = W.build_batch(specs, states)
    ref.run_steps(3)
    b = W.build_batch(specs, states)
    b.set_tile_depths([8, 32, 16, 32, 8, 0])
    b.run_steps(3)
    for k in range(len(specs)):
        _same(b.snapshot(k), ref.snapshot(k), f"member {k}")
    rec = autotune.tune_batch(lambda: W.build_batch(specs, states), steps=1)
    sizes = {"x".join(str(v) for v in sp.field_dims) for sp in specs}
    assert set(rec["depths"]) == sizes and all(d in autotune.BATCH_DEPTHS for d in rec["depths"].values())
    per = autotune.apply_batch(b, rec["depths"])
    assert len(per) == len(specs)
    assert autotune.tune_batch(lambda: W.build_batch(specs, states), steps=1)["cached"]


def _launches_per_step(eng, **tuning):
    be = eng._backend_impl
    be.set_tuning(**tuning)
    eng.run_steps(1)
    be.set_profiling(True)
    eng.run_steps(2)
    prof = be.profile()
    be.set_profiling(False)
    return prof["kernel_launches"] / 2, prof["substep_launches"] / 2


@pytest.mark.parametrize("dims", [(64, 64, 64), (50, 64, 64)])
def test_one_substep_per_pass_can_be_asked_for(cuda, dims):
    """(0, 1) takes a launch per substep, on rows that tensor maps describe and on
    others, where the library's own choice takes three per field; same bits."""
    spec = W.scaled(_spec(), field_dims=dims)
    state = W.initial_state(spec)
    ref = W.build_engine(spec, state)
    own, substeps = _launches_per_step(ref)
    eng = W.build_engine(spec, state)
    single, _ = _launches_per_step(eng, stencil_pair=(0, 1))
    fields = 2 if spec.S_drug else 1
    assert single - own == substeps - 3 * fields
    _same(eng._backend_impl.snapshot(), ref._backend_impl.snapshot(), "one substep per pass")


def test_pairs_that_a_field_does_not_allow_leave_the_choice_to_the_library(cuda):
    """Fewer than 16 rows: no two substeps per pass, and no single ones instead."""
    spec = W.scaled(_spec(), field_dims=(64, 12, 64))
    state = W.initial_state(spec)
    ref = W.build_engine(spec, state)
    eng = W.build_engine(spec, state)
    assert _launches_per_step(eng, stencil_pair=(256, 0)) == _launches_per_step(ref)
    _same(eng._backend_impl.snapshot(), ref._backend_impl.snapshot(), "pair on 12 rows")


@pytest.mark.parametrize("dims,tuning,route", [
    ((64, 64, 64), {}, "resident"), ((50, 64, 64), {}, "resident"), ((64, 64, 64), {"stencil_pair": (0, 1)}, "passes"),
    ((50, 64, 64), {"stencil_pair": (0, 1)}, "passes"), ((64, 64, 64), {"stencil_pair": (256, 0)}, "pairs"),
    ((64, 64, 64), {"stencil_tile": (16, 8)}, "passes"), ((128, 128, 128), {}, "resident"),
    ((160, 160, 160), {}, "pairs"), ((150, 160, 160), {}, "passes")])
def test_the_route_of_a_field_is_the_librarys_to_say(cuda, dims, tuning, route):
    """Small fields stay on chip, up to sizes beyond the least the pairs take; what
    olc_field_route says is what the launches show."""
    spec = W.scaled(_spec(), field_dims=dims)
    eng = W.build_engine(spec)
    got, substeps = _launches_per_step(eng, **tuning)
    assert [eng._backend_impl.field_route(n) for n in ("o2", "drug")] == [route] * 2
    ref = W.build_engine(W.scaled(spec, field_dims=(64, 64, 64)))
    own, _ = _launches_per_step(ref)  # three per field
    S = [spec.S_o2, spec.S_drug]
    per = {"resident": 6, "pairs": sum(s // 2 + s % 2 for s in S), "passes": sum(S)}[route]
    assert got - own == per - 6
    with pytest.raises(_lib.OlcError):
        _lib.check(eng._backend_impl.lib.olc_field_route(eng._backend_impl.handle, 7, None))
