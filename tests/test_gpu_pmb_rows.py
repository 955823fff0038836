"""The mixed PMB step's row layout (bonds in groups of 8 of distinct banks,
rows padded to 32, positions as sums of two floats) against the FP64 step, and
runs split into calls of any length."""
import numpy as np
import pytest

from taylor_b200 import cases, mega

pytestmark = pytest.mark.gpu

PLATES = [  # nx, ny, nz, horizon / h, jitter, offset: rows of 8 to 389 bonds, the last tile ragged
    (5, 4, 1, 2.2, 0.0, 0.0),
    (17, 9, 3, 3.015, 0.2, 1.0),
    (40, 33, 4, 3.015, 0.1, 0.0),
    (12, 13, 12, 4.6, 0.05, -3.0),
]


def _plate(nx, ny, nz, horizon, jitter, offset, seed=3):
    c = cases.pd_plate(h=0.5e-3, nx=nx, ny=ny, nz=nz, horizon=horizon, jitter=jitter, s_c=1e9)
    c["coo"] = c["coo"] + offset
    rng = np.random.default_rng(seed)
    c["vinit"] = rng.uniform(-1.0, 1.0, size=(c["n"], 3))
    return c


@pytest.mark.parametrize("plate", PLATES, ids=lambda p: "x".join(map(str, p[:3])))
def test_pmb_mixed_rows_match_fp64(plate):
    c = _plate(*plate)
    nb = mega.bin_search(c["coo"], c["win"], c["sm_len"], c["dist_max"], 0, 1)
    rng = np.random.default_rng(5)
    broken = (rng.uniform(size=nb["nnz"]) < 0.3).astype(np.uint8)
    rows = np.repeat(np.arange(c["n"]), nb["gn"])
    broken[rows == nb["gstack"] - 1] = 0  # the self entries stay
    dt = 1e-9  # u = dt v: strains of 1e-6 and up
    acl = {}
    for mode in ("fp64", "mixed"):
        p = mega.Pmb(c, broken, mode=mode)
        p.step(1, dt)
        np.testing.assert_array_equal(p.download(3)[0].astype(np.uint8), broken)
        dead = np.bincount(rows, weights=broken, minlength=c["n"])
        np.testing.assert_allclose(p.download(4)[0], dead / np.maximum(nb["gn"] - 1, 1), rtol=0, atol=1e-15)
        acl[mode] = p.download(2)[0].reshape(-1, 3)
        p.close()
    # a bond's stretch: offsets u - u_0 of up to 2 umax rounded to float (2 x 2^-25 x 2 umax, twice for the
    # difference) and a dozen float roundings of |s| <= 2 umax / L: at most 32 x 2^-24 umax / L in all
    umax, lmin = dt * np.sqrt(3.0), 0.5e-3 * (1.0 - 2.0 * plate[4] * np.sqrt(3.0))
    tol = 32 * 2.0 ** -24 * nb["gn"].max() * c["c"] * c["vol"][0] * umax / lmin / c["rho"]
    assert np.abs(acl["mixed"] - acl["fp64"]).max() <= tol
    assert np.abs(acl["fp64"]).max() > 100 * tol


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_pmb_steps_split_into_calls(mode):
    """Any split of a run into calls gives its bits: single steps, captured
    runs of steps, and an odd number before either."""
    c = _plate(17, 9, 3, 3.015, 0.2, 0.0)
    c["s_c"] = 1e-3
    got = []
    for split in ([53], [3, 2, 16, 1, 31], [1] * 5 + [48]):
        p = mega.Pmb(c, None, fixed=c["fixed"], mode=mode)
        for k in split:
            p.step(k, 2e-8)
        got.append([p.download(w)[0] for w in (0, 1, 2, 3)])
        p.close()
    assert got[0][3].sum() > 0  # bonds broke
    for g in got[1:]:
        for a, b in zip(got[0], g):
            np.testing.assert_array_equal(a, b)
