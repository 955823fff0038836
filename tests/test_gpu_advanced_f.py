"""The deformation gradient that steps advance by their increments, where it may
not go on from the step before: against a context that starts from the same
fields, which forms it from the displacements.  Equal bits: both do."""
import numpy as np
import pytest

from taylor_b200 import _lib, cases, mega

pytestmark = pytest.mark.gpu

FIELDS = (_lib.F_DSP_TOT, _lib.F_VEL, _lib.F_ACL, _lib.F_STRESS, _lib.F_STRAIN, _lib.F_EPS)


def _pair(h=0.7e-3):
    c = cases.taylor_bar(h=h, seed=3)
    p = _lib.params(**cases.param_kwargs(c))
    a, b = mega.Mega(c, p), mega.Mega(c, p)
    for m in (a, b):
        m.search_and_shapes()
    return a, b, cases.lattice_dt(c, 0.3)


def _copy(a, b, fields=FIELDS):
    for f in fields:
        b.upload(f, a.download(f))


def _assert_equal(a, b):
    for f in FIELDS:
        np.testing.assert_array_equal(a.download(f), b.download(f))
    a.close()
    b.close()


@pytest.mark.parametrize("first,second", [("mixed", "fp64"), ("fp64", "mixed")])
@pytest.mark.parametrize("timed", [False, True])
def test_precision_changed_on_a_live_context(first, second, timed):
    a, b, dt = _pair()
    a.step(21, dt, mode=first)  # not a multiple of 16
    _copy(a, b)
    for m in (a, b):
        if timed:
            m.kernel_times(3, dt, mode=second)
        else:
            m.step(10, dt, mode=second)
    _assert_equal(a, b)


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_step_that_was_not_finite(mode):
    """After a call that ended with a status of lost sums F is formed afresh: the
    caller puts the fields right that were not finite, the displacements (which
    were) stay."""
    a, b, dt = _pair()
    a.step(21, dt, mode=mode)
    good = {f: a.download(f) for f in FIELDS}
    bad = good[_lib.F_STRESS].copy()
    bad[len(bad) // 2] = np.nan
    a.upload(_lib.F_STRESS, bad)
    assert a.step(1, dt, mode=mode, allow_status=True) & _lib.ST_NONFINITE
    assert np.isfinite(a.download(_lib.F_DSP_TOT)).all()
    for f in FIELDS[1:]:
        a.upload(f, good[f])
    _copy(a, b)
    for m in (a, b):
        m.step(10, dt, mode=mode)
    _assert_equal(a, b)
