"""Wide supports: rows of up to 441 entries, neighbour sets that leave tiles of 8
rows, blocks of 32 threads."""
import numpy as np
import pytest

from oracle import oracle as O
from taylor_b200 import _lib, cases, mega

pytestmark = pytest.mark.gpu


def _wide_bar():
    c = cases.taylor_bar(h=0.6e-3, R=4.2e-3, L=10e-3, seed=2, sy=40e6)
    c["win"] = 1.98 * c["win"]
    c["vinit"][:, 2] = -2.0e4 * c["coo"][:, 2]  # every node yields within a few steps
    nb = O.bin_search(c["coo"], c["win"], c["sm_len"], c["dist_max"])
    order = np.lexsort((nb["ijk"][:, 0], nb["ijk"][:, 1], nb["ijk"][:, 2]))
    rows = [nb["gstack"][s - 1:s - 1 + k] for s, k in zip(nb["gstart"], nb["gn"])]
    sets = {R: max(len(np.unique(np.concatenate([rows[i] for i in order[t:t + R]]))) for t in range(0, c["n"], R))
            for R in (8, 16)}
    assert sets[8] <= 1024 < sets[16] and c["n"] > 32 * 64  # more blocks than a block of 32 clears sums in one go
    return c


@pytest.mark.parametrize("variant", [0, 4])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_counts_of_the_last_step(mode, variant):
    c = _wide_bar()
    m = mega.Mega(c, _lib.params(**cases.param_kwargs(c)))
    m.search_and_shapes()
    m.set_variants(variant, variant, mode=mode)
    dt = cases.lattice_dt(c, 0.3)
    m.step(6, dt, mode=mode)
    before = m.scalars()
    m.step(1, dt, mode=mode)
    s = m.scalars()
    m.close()
    assert s["plastic_nodes"] > 0.9 * c["n"]
    assert s["plastic_nodes"] == s["plastic_nodes_total"] - before["plastic_nodes_total"]
    assert s["newton_iters"] == s["newton_iters_total"] - before["newton_iters_total"]


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("variant", [0, 3])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_bank_ordered_records_match_list_order(mode, variant, wide):
    """Records reordered by the tuner, in tiles of 64 rows (7,458 nodes) and in rows
    too long for the pass's shared memory (8 of up to 441 entries a warp), with the
    interpolation's and the body force's shape values following them.  20 steps of
    sums of up to 441 terms: 20 * 441 * 1.1e-16 = 1e-12 of the largest value, taken
    as 1e-10; mixed the same with 6e-8, 5.3e-4."""
    c = _wide_bar() if wide else cases.taylor_bar(h=0.5e-3, seed=6)
    c["bodyforce"] = np.random.default_rng(7).normal(scale=1.0e5, size=(c["n"], 3))
    p = _lib.params(**cases.param_kwargs(c, gravity=(0.0, 1.0e5, -2.0e5)))
    dt = cases.lattice_dt(c, 0.25)
    out = []
    for tuned in (False, True):
        m = mega.Mega(c, p)
        m.search_and_shapes()
        if tuned:
            m.autotune(dt, mode=mode, reps=1)
        m.set_variants(variant, variant, mode=mode)
        m.step(20, dt, mode=mode, interp_each_step=True)
        out.append([m.download(_lib.F_COO_CURRENT) - c["coo"]] +
                   [m.download(f) for f in (_lib.F_VEL, _lib.F_STRESS, _lib.F_FEXT)])
        m.close()
    tol = 1e-10 if mode == "fp64" else 5.3e-4
    assert any((a != b).any() for a, b in zip(*out))  # (the sums did run in another order)
    for want, got in zip(*out):
        assert np.abs(got - want).max() <= tol * np.abs(want).max()
