"""The gathers' record slices (rows of a tile ordered by length, 8 at a time,
short rows padded) where they are ragged: fewer rows than a tile, one row in
the last tile, slices with absent rows, rows of very different lengths; with
the values that ride along in list order (interpolation, body force).  Against
the oracle.

Tolerances: FP64 sums of at most 125 terms, 20 steps, no amplification beyond
the stable step: 20 * 125 * 1.1e-16 = 3e-13 of the largest value, taken as
1e-10.  Mixed: the same with 6e-8, 1.5e-4."""
import numpy as np
import pytest

from oracle import oracle as O
from taylor_b200 import _lib, cases, mega

pytestmark = pytest.mark.gpu

H = 0.8e-3


@pytest.mark.parametrize("layers", [3, 5, 10, 40])  # 39, 65, 130 and 520 nodes of 13 a layer
@pytest.mark.parametrize("mode,variant", [("fp64", 0), ("fp64", 3), ("fp64", 6), ("fp64", 4), ("mixed", 0),
                                          ("mixed", 2), ("mixed", 5), ("mixed", 7)])
def test_ragged_slices_match_oracle(layers, mode, variant):
    c = cases.taylor_bar(h=H, R=2 * H, L=(layers - 1) * H, seed=layers)
    rng = np.random.default_rng(layers)
    c["bodyforce"] = rng.normal(scale=1.0e5, size=(c["n"], 3))
    assert c["n"] == 13 * layers
    kw = cases.param_kwargs(c, gravity=(0.0, 1.0e5, -2.0e5))
    m = mega.Mega(c, _lib.params(**kw))
    m.search_and_shapes()
    m.set_variants(variant, variant, mode=mode)
    r = O.Run(c, O.params(**kw), nthreads=2)
    dt = cases.lattice_dt(c, 0.3)
    m.step(20, dt, mode=mode, interp_each_step=True)
    r.step(20, dt)
    tol = 1e-10 if mode == "fp64" else 1.5e-4
    u = r.coo_cur.reshape(-1, 3) - c["coo"]
    for got, want in ((m.download(_lib.F_COO_CURRENT) - c["coo"], u), (m.download(_lib.F_VEL), r.vel.reshape(-1, 3)),
                      (m.download(_lib.F_STRESS), r.stress), (m.download(_lib.F_FEXT), r.fext.reshape(-1, 3))):
        assert np.abs(got - want).max() <= tol * np.abs(want).max()
    m.close()
