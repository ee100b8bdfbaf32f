"""Failure paths made on the host, with no GPU fault: a device-memory budget
that the inputs exceed (FMMX_OVER_BUDGET, the reference GPU backend's
OverBudget, crates/visual/src/gpufmm.rs:1653-1672), walk buffers too small
for the walk (the overflow-and-retry path), and corrupted ensemble offsets.
After each failure the context stays usable and gives the same bits as a
context that never failed."""

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OVER_BUDGET, INVALID_ARG = 3, 1


def fx():
    import fmms_b200

    return fmms_b200


def test_over_budget_then_recovers():
    mass_big, pos_big = fx().gen_plummer(200_000, seed=3)
    mass, pos = fx().gen_plummer(2048, seed=4)
    kw = dict(mac="theta", theta=0.5, softening=1e-3)
    g = fx().Fmm(None, None, 6, 0.0, 16, device_budget_bytes=8 << 20, **kw)
    with pytest.raises(fx().FmmError) as e:
        g.refresh(mass_big, pos_big)
    assert e.value.status == OVER_BUDGET
    assert "budget 8.0 MiB" in str(e.value)
    assert g.stats()["device_bytes"] <= 8 << 20
    g.refresh(mass, pos)  # the same context, a system that fits
    r = g.run()
    ref = fx().Fmm(mass, pos, 6, 0.0, 16, **kw).run()
    assert np.array_equal(r.accel, ref.accel) and np.array_equal(r.pot, ref.pot)
    assert g.stats()["device_bytes"] <= 8 << 20


def test_over_budget_in_evaluate():
    """A budget that holds the tree but not the walk and expansions: the
    evaluation fails with OVER_BUDGET, a smaller system then runs."""
    mass, pos = fx().gen_plummer(100_000, seed=5)
    probe = fx().Fmm(mass, pos, 8, 1e-5, 16)
    after_build = probe.stats()["device_bytes"]
    probe.run()
    after_eval = probe.stats()["device_bytes"]
    probe.close()
    assert after_eval > after_build
    g = fx().Fmm(None, None, 8, 1e-5, 16, device_budget_bytes=(after_build + after_eval) // 2)
    g.refresh(mass, pos)
    with pytest.raises(fx().FmmError) as e:
        g.run()
    assert e.value.status == OVER_BUDGET
    m2, p2 = fx().gen_plummer(1000, seed=6)
    g.refresh(m2, p2)
    r = g.run()
    ref = fx().Fmm(m2, p2, 8, 1e-5, 16).run()
    assert np.array_equal(r.accel, ref.accel)


def test_walk_overflow_retry_gives_the_same_bits(monkeypatch):
    """A pool of 64 list entries, two chunks (FMMX_TEST_WALK_CAPACITY): the walk
    overflows and is redone with a larger one until it fits; the lists, and so every
    result bit, are those of a context sized for the tree."""
    mass, pos, _ = fx().gen_plummer_ic(30_000, 1.0, 1.0, 20.0, 8)
    kw = dict(mac="theta", theta=0.5, softening=1e-3)
    for precision in ("plain", "mixed"):
        ref = fx().Fmm(mass, pos, 8, 0.0, 32, precision=precision, **kw)
        r0 = ref.run()
        monkeypatch.setenv("FMMX_TEST_WALK_CAPACITY", "64")
        g = fx().Fmm(mass, pos, 8, 0.0, 32, precision=precision, **kw)
        monkeypatch.delenv("FMMX_TEST_WALK_CAPACITY")
        r1 = g.run()
        assert g.stats()["walk_retries"] > ref.stats()["walk_retries"]
        assert np.array_equal(r0.accel, r1.accel) and np.array_equal(r0.pot, r1.pot)
        assert g.stats()["n_m2l"] == ref.stats()["n_m2l"] and g.stats()["n_p2p"] == ref.stats()["n_p2p"]


@pytest.mark.parametrize("n,n_leaf,dense", [(1500, 8, False), (30_000, 4, True)])
def test_walk_capacity_between_used_and_reserved(monkeypatch, n, n_leaf, dense):
    """A block reserves several chunks at a time (6 or 16), so a pool may hold
    every chunk that is used while the tails of the last reservations lie beyond
    it: no overflow, and the lists are copied from inside the pool alone. Every
    capacity around the smallest one without a retry gives the same bits."""
    mass, pos, _ = fx().gen_plummer_ic(n, 1.0, 1.0, 20.0, 8)
    if dense:  # many cells per level: a warp each, thousands of reservations
        pos = np.concatenate([pos, pos[: n // 4] * 1e-3])
        mass = np.concatenate([mass, mass[: n // 4]])
    kw = dict(mac="theta", theta=0.5, softening=1e-3)
    ref = fx().Fmm(mass, pos, 2, 0.0, n_leaf, **kw)
    r0 = ref.run()
    lists0 = ref.export_lists()

    def with_chunks(chunks):
        monkeypatch.setenv("FMMX_TEST_WALK_CAPACITY", str(32 * chunks))
        g = fx().Fmm(mass, pos, 2, 0.0, n_leaf, **kw)
        monkeypatch.delenv("FMMX_TEST_WALK_CAPACITY")
        return g, g.run()

    lo, hi = 1, 1 << 20  # retries at lo, none at hi
    assert with_chunks(lo)[0].stats()["walk_retries"] > 0
    while hi - lo > 1:
        mid = (lo + hi) // 2
        if with_chunks(mid)[0].stats()["walk_retries"]:
            lo = mid
        else:
            hi = mid
    for chunks in list(range(max(hi - 6, 1), hi + 20)) + [hi + 100, 2 * hi]:
        g, r = with_chunks(chunks)
        assert np.array_equal(r.accel, r0.accel) and np.array_equal(r.pot, r0.pot), chunks
        for a, b in zip(g.export_lists(), lists0):
            assert np.array_equal(a, b), chunks


@pytest.mark.parametrize("precision", ["plain", "mixed"])
def test_near_field_partial_sums_bounded(monkeypatch, precision):
    """Leaves of 250 bodies with long lists have many partial sums. Where they
    are more than the 32-bit sums address (here: than a small bound,
    FMMX_TEST_P2P_PARTIALS) the shares are coarser, in the end one per leaf with
    no partial sums. Only the grouping of a body's sum changes: 100,000 terms in
    FP64 (plain, about 1e-16 each), or in FP32 groups of some 64 pairs (mixed)."""
    mass, pos = fx().gen_plummer(20_000, seed=8)
    kw = dict(mac="theta", theta=0.2, softening=1e-3, precision=precision)
    r0 = fx().Fmm(mass, pos, 2, 0.0, 256, **kw).run()
    rel = 1e-13 if precision == "plain" else 1e-6
    for bound in (5000, 0):
        monkeypatch.setenv("FMMX_TEST_P2P_PARTIALS", str(bound))
        g = fx().Fmm(mass, pos, 2, 0.0, 256, **kw)
        monkeypatch.delenv("FMMX_TEST_P2P_PARTIALS")
        r1 = g.run()
        r2 = g.run()  # the lists of the second evaluation, in the buffers of the first
        assert np.array_equal(r1.accel, r2.accel)
        for a, b in ((r1.accel, r0.accel), (r1.pot, r0.pot)):
            assert np.linalg.norm(a - b) <= rel * np.linalg.norm(b)
            assert not np.array_equal(a, b)


@pytest.mark.parametrize("precision,mib", [("plain", 77), ("mixed", 86)])
def test_budget_of_large_leaves(precision, mib):
    """100,000 bodies in leaves of up to 256 with lists of 10^3 leaves: 64 MB of
    partial sums that the budget does not hold; the shares are coarser instead."""
    mass, pos = fx().gen_plummer(100_000, seed=7)
    kw = dict(mac="theta", theta=0.2, precision=precision)
    r0 = fx().Fmm(mass, pos, 2, 0.0, 256, **kw).run()
    g = fx().Fmm(None, None, 2, 0.0, 256, device_budget_bytes=mib * 1_000_000, **kw)
    g.refresh(mass, pos)
    r1 = g.run()
    assert g.stats()["device_bytes"] <= mib * 1_000_000
    rel = 1e-13 if precision == "plain" else 1e-6
    assert np.linalg.norm(r1.accel - r0.accel) <= rel * np.linalg.norm(r0.accel)


@pytest.mark.parametrize("n,p,n_leaf,mb", [(1000, 8, 16, 1.65), (3000, 2, 4, 8.5), (20_000, 4, 8, 56.0)])
def test_budget_without_the_walk_expected_capacity(n, p, n_leaf, mb):
    """A budget that holds the lists but not the pool a walk starts with: the
    walk takes what there is, and the results are those without a budget. (The
    first budget is what the engine took with pair buffers in place of the pool.)"""
    mass, pos = fx().gen_plummer(n, seed=7)
    kw = dict(mac="theta", theta=0.5, softening=1e-3)
    r0 = fx().Fmm(mass, pos, p, 0.0, n_leaf, **kw).run()
    budget = int(mb * 1e6)
    g = fx().Fmm(None, None, p, 0.0, n_leaf, device_budget_bytes=budget, **kw)
    for _ in range(3):
        g.refresh(mass, pos)
        r = g.run()
        assert np.array_equal(r.accel, r0.accel) and np.array_equal(r.pot, r0.pot)
        assert g.stats()["device_bytes"] <= budget
    small = fx().gen_plummer(500, seed=9)  # a smaller system, then the first one again
    g.refresh(*small)
    g.run()
    g.refresh(mass, pos)
    assert np.array_equal(g.run().accel, r0.accel)


def test_corrupted_ensemble_offsets():
    m1, p1 = fx().gen_plummer(3000, seed=1)
    m2, p2 = fx().gen_plummer(2000, seed=2)
    mass, pos = np.concatenate([m1, m2]), np.concatenate([p1, p2])
    g = fx().Fmm(None, None, 6, 1e-4, 16)
    bad = [np.array([1, 3000, 5000], dtype=np.uint64),  # does not start at 0
           np.array([0, 3000, 3000, 5000], dtype=np.uint64),  # an empty system
           np.array([0, 4000, 3000, 5000], dtype=np.uint64)]  # decreasing
    for off in bad:
        with pytest.raises(fx().FmmError) as e:
            g.build_ensemble(off, mass, pos)
        assert e.value.status == INVALID_ARG
    g.build_ensemble(np.array([0, 3000, 5000], dtype=np.uint64), mass, pos)
    r = g.run()
    alone = fx().Fmm(m1, p1, 6, 1e-4, 16).run()
    assert np.array_equal(r.accel[:3000], alone.accel)
