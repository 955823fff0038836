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
