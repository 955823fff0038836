"""The tuner where device memory has no room for its second set of records: it
tunes on the records as they are, and the steps keep their bits."""
import numpy as np
import pytest

from taylor_b200 import _lib, cases, mega

pytestmark = pytest.mark.gpu

FIELDS = (_lib.F_DSP_TOT, _lib.F_VEL, _lib.F_STRESS, _lib.F_EPS)


def test_autotune_without_room_for_reordered_records():
    import torch

    c = cases.taylor_bar(h=0.2e-3)  # 129,911 nodes: records of 200 MB a gather, state of 72 MB
    dt = cases.lattice_dt(c, 0.3)
    out = []
    for tune in (False, True):
        m = mega.Mega(c, _lib.params(**cases.param_kwargs(c)))
        m.set_precisions(fp64=True, mixed=False)
        m.search_and_shapes()
        if tune:
            _lib.lib().mega_release_cached_memory()
            hold = torch.empty(torch.cuda.mem_get_info()[0] - (250 << 20), dtype=torch.uint8, device="cuda")
            m.autotune(dt, mode="fp64", reps=1)
            del hold
            torch.cuda.empty_cache()
        m.set_variants(0, 0, mode="fp64")
        m.step(20, dt)
        out.append([m.download(f) for f in FIELDS])
        m.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_device_bytes_after_the_tuner(mode):
    """The reordered records take the place of the ones before: the context holds
    one array more, the interpolation's shape values in the records' order."""
    c = cases.taylor_bar(h=0.5e-3)
    m = mega.Mega(c, _lib.params(**cases.param_kwargs(c)))
    nnz = m.search_and_shapes()["nnz"]
    held = m.device_bytes()
    m.autotune(cases.lattice_dt(c, 0.3), mode=mode, reps=1)
    assert m.device_bytes() == held + 8 * nnz
    m.close()
