"""Tree construction from the sorted keys at its edges: leaf capacities from 0
to more than the bodies, body counts around the kernels' blocks, runs of equal
keys, and forests on both sides of the sort's system-length rule. Order, keys
and every cell field must equal the oracle's bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("first", "count", "level", "leaf", "children", "cen", "mass", "rho")


def bodies(kind, n, seed):
    rng = np.random.default_rng(seed)
    mass = rng.random(n) + 0.5
    if kind == "uniform":
        return mass, rng.random((n, 3))
    if kind == "clump":  # most bodies deep in one corner, some coincident
        pos = rng.random((n, 3)) * np.where(rng.random(n) < 0.8, 1e-5, 1.0)[:, None]
        pos[: n // 3] = pos[0]
        return mass, pos
    return mass, np.full((n, 3), 0.25)  # all coincident: one level-21 chain


@pytest.mark.parametrize("kind", ["uniform", "clump", "coincident"])
@pytest.mark.parametrize("n_leaf", [0, 1, 2, 33, 64, 5000])
@pytest.mark.parametrize("n", [1, 2, 33, 1023, 1024, 1025, 4500])
def test_tree_equals_oracle(orc, kind, n_leaf, n):
    import fmms_b200 as fx

    if n_leaf == 0 and n > 1100:
        pytest.skip("every body a level-21 chain")
    mass, pos = bodies(kind, n, 7 * n + n_leaf)
    g = fx.Fmm(mass, pos, 2, 1e-3, n_leaf)
    o = orc.Fmm(mass, pos, 2, 1e-3, n_leaf)
    order, keys, cells = g.export_tree()
    order_o, keys_o = o.order()
    assert np.array_equal(keys, keys_o) and np.array_equal(order, order_o)
    cells_o = o.cells()
    for k in FIELDS:
        assert np.array_equal(cells[k], cells_o[k]), k
    assert g.stats()["n_leaves"] == int(cells_o["leaf"].sum())


@pytest.mark.parametrize("sizes", [[4096, 4096, 1], [4097, 3, 4000], [2048, 1, 9000, 2047, 2], [1] * 70 + [5000]])
def test_forest_trees_equal_each_alone(sizes):
    import fmms_b200 as fx

    parts = [bodies("clump" if i % 2 else "uniform", n, i) for i, n in enumerate(sizes)]
    parts = [(m, q - 3.0 * i) for i, (m, q) in enumerate(parts)]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    g = fx.Fmm(None, None, 2, 1e-3, 16)
    g.build_ensemble(off, np.concatenate([m for m, _ in parts]), np.concatenate([q for _, q in parts]))
    order, keys, cells = g.export_tree()
    c0 = 0
    for s, (m, q) in enumerate(parts):
        a = int(off[s])
        h = fx.Fmm(m, q, 2, 1e-3, 16)
        order_a, keys_a, cells_a = h.export_tree()
        nc, n = len(cells_a["mass"]), len(m)
        assert np.array_equal(keys[a:a + n], keys_a)
        assert np.array_equal(order[a:a + n].astype(np.int64) - a, order_a.astype(np.int64))
        for k in FIELDS:
            v = cells[k][c0:c0 + nc]
            if k == "first":
                v = v - np.uint32(a)
            if k == "children":
                v = np.where(v >= 0, v - c0, v)
            assert np.array_equal(v, cells_a[k]), (s, k)
        c0 += nc
    assert c0 == len(cells["mass"])
