"""The walk's forms -- 32, 8 and 1 warps per cell, the cells left to the heavy
form -- give the reference's pair sets: a dense clump with shallow leaves beside
it (lists of 10^4 and more), level sizes on both sides of the lines between the
forms, both criteria."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def clump(n_dense, n_wide, seed):
    rng = np.random.default_rng(seed)
    pos = np.concatenate([0.5 + 0.01 * rng.standard_normal((n_dense, 3)), rng.random((n_wide, 3))])
    return rng.random(len(pos)) + 0.5, pos


def pair_set(a):
    return np.sort(np.ascontiguousarray(a, dtype=np.uint32).view(np.uint64).ravel())


@pytest.mark.parametrize("mac", ["theta", "dehnen"])
@pytest.mark.parametrize("n_dense,n_wide,n_leaf", [(300, 100, 4), (5_000, 1_000, 4), (40_000, 2_000, 8),
                                                   (150_000, 300, 3)])
def test_pair_sets_equal_the_oracle(orc, mac, n_dense, n_wide, n_leaf):
    import fmms_b200 as fx

    if mac == "dehnen" and n_dense > 100_000:
        n_dense = 60_000
    mass, pos = clump(n_dense, n_wide, n_dense + n_leaf)
    kw = dict(mac="theta", theta=0.6) if mac == "theta" else {}
    okw = dict(mac=orc.MAC_THETA, theta=0.6) if mac == "theta" else {}
    g = fx.Fmm(mass, pos, 2, 1e-2, n_leaf, **kw)
    g.run()
    o = orc.Fmm(mass, pos, 2, 1e-2, n_leaf, **okw)
    o.run(nthreads=8)
    m2l, p2p = g.export_lists()
    m2l_o, p2p_o = o.lists()
    assert np.array_equal(pair_set(m2l), pair_set(m2l_o))
    assert np.array_equal(pair_set(p2p), pair_set(p2p_o))
    st = g.stats()
    assert st["n_m2l"] == len(m2l_o) and st["n_p2p"] == len(p2p_o)
    cnt = o.cells()["count"].astype(np.int64)
    a, b = cnt[p2p_o[:, 0]], cnt[p2p_o[:, 1]]
    assert st["p2p_interactions"] == int(np.where(p2p_o[:, 0] == p2p_o[:, 1], a * (a - 1), 2 * a * b).sum())
    assert st["walk_pops"] == o.pops


def test_results_do_not_depend_on_the_form():
    """A small system alone (many warps per cell) and in a forest large enough
    for a warp per cell: the same bits."""
    import fmms_b200 as fx

    parts = [clump(1500, 200, s) for s in range(40)] + [clump(30_000, 500, 99)]
    off = np.concatenate([[0], np.cumsum([len(m) for m, _ in parts])]).astype(np.uint64)
    for precision in ("plain", "mixed"):
        kw = dict(mac="theta", theta=0.5, softening=1e-4, precision=precision)
        g = fx.Fmm(None, None, 4, 0.0, 4, **kw)
        g.build_ensemble(off, np.concatenate([m for m, _ in parts]), np.concatenate([q for _, q in parts]))
        r = g.run()
        for s in (0, 17, 40):
            h = fx.Fmm(parts[s][0], parts[s][1], 4, 0.0, 4, **kw).run()
            a, b = int(off[s]), int(off[s + 1])
            assert np.array_equal(r.accel[a:b], h.accel) and np.array_equal(r.pot[a:b], h.pot)


def test_walk_time_does_not_grow_with_what_the_context_held():
    """A context that has evaluated a million bodies in small leaves (a pool of
    gigabytes) walks a small system in the time a new one does: nothing of the
    pool's size is cleared or read."""
    import fmms_b200 as fx

    mass, pos = fx.gen_plummer(1000, seed=2)
    kw = dict(mac="theta", theta=0.9, softening=1e-3)

    def walk_ms(g):
        g.refresh(mass, pos)
        t = []
        for _ in range(60):
            r = g.run()
            t.append(g.stats()["ms_walk"])
        return min(t), r.accel

    big_m, big_p = fx.gen_plummer(1 << 20, seed=3)
    used = fx.Fmm(big_m, big_p, 1, 0.0, 4, **kw)
    used.run()
    t1, a1 = walk_ms(used)
    t0, a0 = walk_ms(fx.Fmm(None, None, 1, 0.0, 4, **kw))
    assert np.array_equal(a0, a1)
    assert t1 < 1.12 * t0, (t0, t1)
