"""What the step's sums see in another order or from another place: FP64 records
in bank order (after the FP64 tuner), NSNI with a body force, a run restarted
from uploaded fields, and drop-in lists with gaps."""
import numpy as np
import pytest

from oracle import oracle as O
from taylor_b200 import _lib, cases, mega

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsni", [False, True])
@pytest.mark.parametrize("mode,variant", [("fp64", 0), ("fp64", 3), ("fp64", 4), ("mixed", 0), ("mixed", 3)])
def test_bank_ordered_records_match_oracle(nsni, mode, variant):
    """The body force's shape values follow their records.  FP64: 20 steps of
    sums of up to 125 terms, 20 * 125 * 1.1e-16 = 3e-13, taken as 1e-10; with NSNI
    second derivatives of 1/h^2 against gradients of 1/h, 1e-8.  Mixed 1.5e-4 (the
    same with 6e-8), with NSNI 1e-3."""
    c = cases.taylor_bar(h=0.8e-3, seed=6)
    rng = np.random.default_rng(7)
    c["bodyforce"] = rng.normal(scale=1.0e5, size=(c["n"], 3))
    kw = cases.param_kwargs(c, gravity=(0.0, 1.0e5, -2.0e5), itype_int=2 if nsni else 0)
    m = mega.Mega(c, _lib.params(**kw))
    m.search_and_shapes()
    dt = cases.lattice_dt(c, 0.25)
    m.autotune(dt, mode=mode, reps=1)
    m.set_variants(variant, variant, mode=mode)
    r = O.Run(c, O.params(**kw), nthreads=8)
    m.step(20, dt, mode=mode)
    r.step(20, dt)
    tol = {"fp64": (1e-10, 1e-8), "mixed": (1.5e-4, 1e-3)}[mode][nsni]
    u = r.coo_cur.reshape(-1, 3) - c["coo"]
    for got, want in ((m.download(_lib.F_COO_CURRENT) - c["coo"], u), (m.download(_lib.F_VEL), r.vel.reshape(-1, 3)),
                      (m.download(_lib.F_STRESS), r.stress), (m.download(_lib.F_FEXT), r.fext.reshape(-1, 3))):
        assert np.abs(got - want).max() <= tol * np.abs(want).max()
    m.close()


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("at", [32, 21])
def test_run_restarted_from_uploaded_fields(mode, at):
    """F is formed afresh from an uploaded displacement: bit for bit the unbroken
    run where that one forms it too (every 16 steps), else the rounding of the
    sum of at most 16 increments, 1e-12 (mixed: float increments, 1e-5)."""
    c = cases.taylor_bar(h=0.7e-3, seed=3)
    p = _lib.params(**cases.param_kwargs(c))
    dt = cases.lattice_dt(c, 0.3)
    fields = (_lib.F_DSP_TOT, _lib.F_VEL, _lib.F_ACL, _lib.F_STRESS, _lib.F_STRAIN, _lib.F_EPS)
    a, b = mega.Mega(c, p), mega.Mega(c, p)
    for m in (a, b):
        m.search_and_shapes()
    a.step(at, dt, mode=mode)
    for f in fields:
        b.upload(f, a.download(f))
    a.step(30, dt, mode=mode)
    b.step(30, dt, mode=mode)
    tol = 0.0 if at % 16 == 0 else (1e-12 if mode == "fp64" else 1e-5)
    for f in fields:
        x, y = a.download(f), b.download(f)
        assert np.abs(x - y).max() <= tol * np.abs(x).max()
    a.close()
    b.close()


def _call(c, lists, **change):
    rng = np.random.default_rng(9)
    n = c["n"]
    state = np.zeros((n, 20))
    state[:, 2] = np.abs(rng.normal(0.0, 0.02, n))
    k = dict(dinc=rng.normal(scale=1e-3 * c["h"], size=3 * n), dinc_tot=rng.normal(scale=1e-2 * c["h"], size=3 * n),
             stress=rng.normal(0.0, 60e6, (n, 6)), strain=rng.normal(0.0, 1e-3, (n, 6)), state=state)
    l = dict(lists, **change)
    return mega.construct_fint(_lib.params(**cases.param_kwargs(c)), c["coo"], c["win"], c["vol"], c["props"],
                               c["mat_type"], l["en"], k["state"], k["stress"], k["strain"], k["dinc"], k["dinc_tot"],
                               l["gn"], l["gstart"], l["gstack"], l["shp"], l["dshp"], False, 1e-8)


def test_dropin_lists_with_gaps_and_bad_ids():
    c = cases.taylor_bar(h=0.8e-3, seed=4)
    nb = mega.bin_search(c["coo"], c["win"], c["sm_len"], c["dist_max"])
    en = np.any(c["ebc"] == 1, axis=1).astype(np.int32)
    shp, dshp = mega.rk_shapes(_lib.params(**cases.param_kwargs(c)), c["coo"], c["win"], en, nb["gn"], nb["gstart"],
                               nb["gstack"])
    tight = dict(en=en, gn=nb["gn"], gstart=nb["gstart"], gstack=nb["gstack"], shp=shp, dshp=dshp)
    # rows last to first, three unused places (of no valid id or value) after each
    n, gn = c["n"], nb["gn"].astype(np.int64)
    start = np.zeros(n, np.int64)
    start[::-1] = np.concatenate([[0], np.cumsum(gn[::-1] + 3)[:-1]])
    total = int((gn + 3).sum())
    at = np.concatenate([start[i] + np.arange(gn[i]) for i in range(n)])
    was = np.concatenate([nb["gstart"][i] - 1 + np.arange(gn[i]) for i in range(n)])
    stack, s2, d2 = np.full(total, -7, np.int32), np.full(total, np.nan), np.full((total, 3), np.nan)
    stack[at], s2[at], d2[at] = nb["gstack"][was], np.ravel(shp)[was], np.reshape(dshp, (-1, 3))[was]
    gaps = dict(en=en, gn=nb["gn"], gstart=(start + 1).astype(np.int32), gstack=stack, shp=s2, dshp=d2)
    want, got = _call(c, tight), _call(c, gaps)
    for k in ("fint", "fext", "stress", "strain", "state", "gmax_wvel", "gstrain_eq"):
        np.testing.assert_array_equal(got[k], want[k])
    for bad in (0, -1, n + 1):
        ids = nb["gstack"].copy()
        ids[len(ids) // 2] = bad
        with pytest.raises(_lib.MegaError):
            _call(c, tight, gstack=ids)
    far = nb["gstart"].copy()
    far[-1] = len(nb["gstack"])  # its row runs past the list
    with pytest.raises(_lib.MegaError):
        _call(c, tight, gstart=far)
