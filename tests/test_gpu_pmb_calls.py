"""PMB runs in calls of 17 steps, which start from either displacement buffer in
turn: both buffers' captured steps, a change of dt between them, and calls of
two steps, against single steps."""
import numpy as np
import pytest

from taylor_b200 import cases, mega

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_calls_from_either_buffer(mode):
    c = cases.pd_plate(h=0.5e-3, nx=17, ny=9, nz=3, horizon=3.015, jitter=0.2, s_c=1e-3)
    c["vinit"] = np.random.default_rng(3).uniform(-1.0, 1.0, size=(c["n"], 3))
    calls = [(17, 2e-8), (17, 2e-8), (17, 2e-8), (2, 2e-8), (18, 1e-8), (3, 1e-8), (2, 1e-8), (17, 1e-8), (34, 2e-8)]
    got = []
    for single in (False, True):
        p = mega.Pmb(c, None, fixed=c["fixed"], mode=mode)
        for k, dt in calls:
            for n in [1] * k if single else [k]:
                p.step(n, dt)
        got.append([p.download(w)[0] for w in (0, 1, 2, 3)])
        p.close()
    assert got[0][3].sum() > 0  # bonds broke
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


def test_calls_of_odd_length_do_not_capture_again():
    """Steps of a small plate in calls of 17 cost what they cost in calls of 18
    (a capture in each call would cost three times as much)."""
    c = cases.pd_plate(h=0.5e-3, nx=40, ny=40, nz=1, horizon=3.015, s_c=1e9)
    p = mega.Pmb(c, None, mode="fp64")

    def per_step(k):
        p.step(k, 1e-9), p.step(k, 1e-9)
        return min(p.step(k, 1e-9, timed=True) for _ in range(20)) / k

    t18, t17 = per_step(18), per_step(17)
    p.close()
    assert t17 < 1.6 * t18
