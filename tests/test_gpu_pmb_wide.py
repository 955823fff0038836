"""The mixed PMB step where bonds are short against the extent of the plate: pairs
that almost coincide, and a particle far from the rest, on both sides of the
line past which positions stay in double.  Against the FP64 step."""
import numpy as np
import pytest

from taylor_b200 import cases, mega

pytestmark = pytest.mark.gpu

H = 0.5e-3


@pytest.mark.parametrize("far", [None, 60.0, 140.0, 2.0 ** 16 * 3.015])  # in H; pairs are H / 2^13 apart
def test_short_bonds_match_fp64(far):
    c = cases.pd_plate(h=H, nx=17, ny=9, nz=3, horizon=3.015, jitter=0.2, s_c=1e9)
    rng = np.random.default_rng(4)
    way = rng.normal(size=(40, 3))
    way *= H / 2.0 ** 13 / np.linalg.norm(way, axis=1)[:, None]
    coo = np.concatenate([c["coo"], c["coo"][rng.permutation(c["n"])[:40]] + way])
    if far:
        coo = np.concatenate([coo, coo[:1] + [[far * H, 0.0, 0.0]]])
    n, grow = len(coo), len(coo) - c["n"]
    c = dict(c, n=n, coo=coo, vinit=rng.uniform(-1.0, 1.0, size=(n, 3)),
             vol=np.concatenate([c["vol"], np.repeat(c["vol"][:1], grow)]))
    win = np.full((n, 3), c["delta"])
    nb = mega.bin_search(coo, win, np.zeros((n, 6)), np.zeros(3), 0, 1)
    dt = 1e-9  # u = dt v
    acl = {}
    for mode in ("fp64", "mixed"):
        p = mega.Pmb(c, None, mode=mode)
        assert p.nnz == nb["nnz"]
        p.step(1, dt)
        acl[mode] = p.download(2)[0].reshape(-1, 3)
        p.close()
    # per bond: offsets u - u_0 of up to 2 umax rounded to float (2 x 2^-25 x 2 umax, twice for the difference) and
    # a dozen float roundings of |s| <= 2 umax / L: at most 32 x 2^-24 umax / L in all
    i = np.repeat(np.arange(n), nb["gn"])
    j = nb["gstack"][np.concatenate([s - 1 + np.arange(k) for s, k in zip(nb["gstart"], nb["gn"])])] - 1
    i, j = i[i != j], j[i != j]
    bond = 1.0 / np.linalg.norm(coo[i] - coo[j], axis=1)
    tol = 32 * 2.0 ** -24 * np.sqrt(3.0) * dt * c["c"] * c["vol"][0] / c["rho"] * np.bincount(i, bond, minlength=n)
    assert (np.abs(acl["mixed"] - acl["fp64"]).max(axis=1) <= tol).all()
    assert np.abs(acl["fp64"]).max() > 100 * tol.max()
