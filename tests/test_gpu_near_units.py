"""Near field at the edges of its work units: leaves of one body, of a unit's
32 targets and one more, of more bodies than a chunk's table holds, and lists
of more source leaves than one share. A large separation condition leaves no
M2L, so the result is the whole near field and must equal the direct sum."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["plain", "mixed"])
@pytest.mark.parametrize("n,n_leaf", [(1, 8), (2, 1), (3, 1), (700, 1), (1500, 2), (900, 31), (1100, 32), (1300, 33),
                                      (1900, 64), (2100, 65), (2049, 5000), (4500, 5000)])
def test_near_field_is_the_direct_sum(orc, precision, n, n_leaf):
    import fmms_b200 as fx

    rng = np.random.default_rng(n + n_leaf)
    mass, pos, soft = rng.random(n) + 0.1, rng.random((n, 3)), 1e-3
    # no M2L: no pair of cells is 1e6 softening lengths apart
    g = fx.Fmm(mass, pos, 4, 0.0, n_leaf, mac="theta", theta=0.5, softening=soft, soft_gap=1e6, precision=precision)
    res = g.run()
    st = g.stats()
    assert st["n_m2l"] == 0 and st["p2p_interactions"] == n * (n - 1)
    acc, pot = orc.direct(mass, pos, softening=soft)
    d = pos[None] - pos[:, None]
    r = np.sqrt((d ** 2).sum(2) + soft ** 2)
    np.fill_diagonal(r, np.inf)
    if precision == "plain":  # a term's roundings and those of n additions
        term = 16 * 2.0 ** -52 * (8 + np.log2(n))
    else:
        # FP32 terms (about 32 roundings of 2^-24), their differences taken of
        # coordinates up to a leaf's radius R (two bodies and an offset: the
        # error of a coordinate is a few R 2^-24, of the term three times that over r)
        cells = g.export_tree()[2]
        rmax = cells["rho"][cells["leaf"]].max()
        term = 2.0 ** -24 * (32 + 32 * rmax / r)
    assert np.all(np.linalg.norm(res.accel - acc, axis=1) <= (mass / r ** 2 * term).sum(1))
    assert np.all(np.abs(res.pot - pot) <= (mass / r * term).sum(1))
