"""The pinned stage of the process: downloads longer than it may grow go in
rounds, and it is given back with the cached device memory."""
import numpy as np
import pytest

from taylor_b200 import _lib, cases, mega

pytestmark = pytest.mark.gpu


def _resident():
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) for line in f if line.startswith("VmRSS")) << 10


def test_downloads_in_rounds_and_the_stage_given_back():
    c = cases.taylor_bar(h=0.3e-3)  # 41,093 nodes
    m = mega.Mega(c, _lib.params(**cases.param_kwargs(c)))
    m.search_and_shapes()
    m.step(5, cases.lattice_dt(c, 0.3))
    want = m.download(_lib.F_STRESS).ravel()
    _lib.lib().mega_release_cached_memory()
    codes = np.full(80, _lib.F_STRESS, np.int32)  # 158 MB
    out = np.ones((len(codes), want.size))
    before = _resident()
    assert _lib.lib().mega_snapshot(m.h, len(codes), _lib.ptr(codes), _lib.ptr(out)) == 0
    grown = _resident() - before
    for row in out:
        np.testing.assert_array_equal(row, want)
    held = _resident()
    _lib.lib().mega_release_cached_memory()
    freed = held - _resident()
    print("grown", grown, "freed", freed)
    np.testing.assert_array_equal(m.download(_lib.F_STRESS).ravel(), want)
    m.close()
    assert grown <= 136 << 20 and freed >= 120 << 20
