"""The row gather that goes on to the stress update of its tile, on either side
of the sizes that take it (all blocks resident at once; tiles of 32 rows up to
32 rows per SM): against the same steps with the two kernels apart, which a
run that interpolates each step takes.

The lanes and their sums are the same; the compiler may contract a product and
a sum in one and not in the other: 40 steps of four roundings, no amplification
beyond the stable step: 40 * 4 * 1.1e-16 = 2e-14 of the largest value, taken as
1e-12.  Mixed: the same with 6e-8, 1e-5."""
import numpy as np
import pytest

from taylor_b200 import _lib, cases, mega

pytestmark = pytest.mark.gpu

RATE = (90e6, 292e6, 0.31, 0.025, 1.0)


def _run(c, mode, variant, split):
    m = mega.Mega(c, _lib.params(**cases.param_kwargs(c, gravity=(0.0, 1.0e5, -2.0e5))))
    m.search_and_shapes()
    m.set_variants(variant, variant, mode=mode)
    dt = cases.lattice_dt(c, 0.3)
    k0 = m.kernel_launches()
    for k in (3, 36, 1):  # single steps, captured ones, a last step alone
        m.step(k, dt, mode=mode, interp_each_step=split)
    out = [m.download(_lib.F_COO_CURRENT) - c["coo"]]
    out += [m.download(f) for f in (_lib.F_VEL, _lib.F_STRESS, _lib.F_STRAIN, _lib.F_EPS)]
    s = m.scalars()
    launches = m.kernel_launches() - k0
    m.close()
    return out, s, launches


@pytest.mark.parametrize("h,variant,joined", [
    (0.8e-3, 0, True), (0.6e-3, 3, True), (0.6e-3, 7, True),  # 2,009 and 4,455 nodes: tiles of 32
    (0.5e-3, 0, True), (0.5e-3, 3, True), (0.5e-3, 7, False),  # 7,458: tiles of 64
    (0.4e-3, 0, True), (0.4e-3, 3, False), (0.35e-3, 0, False)])  # 16,154 and 23,782
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_joined_steps_match_split(h, variant, joined, mode):
    c = cases.taylor_bar(h=h, seed=2, rate_law=RATE if variant == 3 else None)
    got, s, launches = _run(c, mode, variant, False)
    want, t, split = _run(c, mode, variant, True)
    # of 40 steps three end a call and three form F afresh; the others join
    assert launches == split - (34 if joined else 0)
    assert s["plastic_nodes_total"] > 0
    tol = 1e-12 if mode == "fp64" else 1e-5
    for a, b in zip(got, want):
        assert np.abs(a - b).max() <= tol * np.abs(b).max()
    for k in ("int_energy", "kin_energy"):
        assert abs(s[k] - t[k]) <= max(tol, 1e-9) * abs(t[k])
    if mode == "fp64":
        for k in ("newton_iters", "plastic_nodes", "plastic_nodes_total", "newton_iters_total"):
            assert s[k] == t[k]
