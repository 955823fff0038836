"""The drop-in's lists as a caller may hold them: rows a fixed number of places
apart, in any order and sharing places, from several threads at once.  The
sums see the same entries in the same order: equal bits."""
import threading

import numpy as np
import pytest

from taylor_b200 import _lib, cases, mega

pytestmark = pytest.mark.gpu

OUT = ("fint", "fext", "stress", "strain", "state", "gmax_wvel", "gstrain_eq")


def _lists(c):
    nb = mega.bin_search(c["coo"], c["win"], c["sm_len"], c["dist_max"])
    en = np.any(c["ebc"] == 1, axis=1).astype(np.int32)
    shp, dshp = mega.rk_shapes(_lib.params(**cases.param_kwargs(c)), c["coo"], c["win"], en, nb["gn"], nb["gstart"],
                               nb["gstack"])
    return dict(en=en, gn=nb["gn"], gstart=nb["gstart"], gstack=nb["gstack"], shp=np.ravel(shp),
                dshp=np.reshape(dshp, (-1, 3)))


def _moved(l, start):
    """The same rows from 0-based places `start` on (no valid id or value between)."""
    gn, n = l["gn"].astype(np.int64), len(l["gn"])
    total = int((start + gn).max())
    at = np.concatenate([start[i] + np.arange(gn[i]) for i in range(n)])
    was = np.concatenate([l["gstart"][i] - 1 + np.arange(gn[i]) for i in range(n)])
    stack, shp, dshp = np.full(total, -7, np.int32), np.full(total, np.nan), np.full((total, 3), np.nan)
    stack[at], shp[at], dshp[at] = l["gstack"][was], l["shp"][was], l["dshp"][was]
    return dict(l, gstart=(start + 1).astype(np.int32), gstack=stack, shp=shp, dshp=dshp)


def _call(c, l, seed=9):
    rng = np.random.default_rng(seed)
    n = c["n"]
    state = np.zeros((n, 20))
    state[:, 2] = np.abs(rng.normal(0.0, 0.02, n))
    return mega.construct_fint(_lib.params(**cases.param_kwargs(c)), c["coo"], c["win"], c["vol"], c["props"],
                               c["mat_type"], l["en"], state, rng.normal(0.0, 60e6, (n, 6)),
                               rng.normal(0.0, 1e-3, (n, 6)), rng.normal(scale=1e-3 * c["h"], size=3 * n),
                               rng.normal(scale=1e-2 * c["h"], size=3 * n), l["gn"], l["gstart"], l["gstack"],
                               l["shp"], l["dshp"], False, 1e-8)


def _assert_equal(got, want):
    for k in OUT:
        np.testing.assert_array_equal(got[k], want[k])


def test_rows_far_apart_take_no_device_memory():
    import torch

    c = cases.taylor_bar(h=0.8e-3, seed=4)
    tight = _lists(c)
    wide = _moved(tight, np.arange(c["n"], dtype=np.int64) * 4096)
    want = _call(c, tight)

    def held(l):
        _lib.lib().mega_release_cached_memory()
        free = torch.cuda.mem_get_info()[0]
        _assert_equal(_call(c, l), want)
        return free - torch.cuda.mem_get_info()[0]

    base = held(tight)
    assert held(wide) <= base + (32 << 20)  # 36 bytes for each of 8.2 M places would be 296 MB


def test_rows_in_any_order_and_shared():
    """57 MB of gradients, many pieces of the upload; then the last nodes' rows are
    the first one's, in its places."""
    c = cases.taylor_bar(h=0.3e-3, seed=4)
    tight = _lists(c)
    gn = tight["gn"].astype(np.int64)
    order = np.random.default_rng(1).permutation(c["n"])
    start = np.zeros(c["n"], np.int64)
    start[order] = np.concatenate([[0], np.cumsum(gn[order])[:-1]])
    _assert_equal(_call(c, _moved(tight, start)), _call(c, tight))
    # rows that share places, against the same rows each with its own
    shared = dict(tight, gn=tight["gn"].copy(), gstart=tight["gstart"].copy())
    shared["gn"][-9:], shared["gstart"][-9:] = shared["gn"][0], shared["gstart"][0]
    g = shared["gn"].astype(np.int64)
    own = _moved(shared, np.concatenate([[0], np.cumsum(g)[:-1]]))
    _assert_equal(_call(c, shared), _call(c, own))


def test_calls_from_two_threads():
    work = [cases.taylor_bar(h=0.5e-3, seed=4), cases.taylor_bar(h=0.6e-3, seed=5)]
    lists = [_lists(c) for c in work]
    lists[1] = _moved(lists[1], np.arange(work[1]["n"], dtype=np.int64) * 160)
    want = [_call(c, l) for c, l in zip(work, lists)]
    errors = []

    def run(k):
        try:
            for _ in range(8):
                _assert_equal(_call(work[k], lists[k]), want[k])
        except BaseException as e:  # noqa: BLE001 - handed to the main thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k % 2,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
