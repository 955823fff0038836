"""A run in calls of any length has the bits of the run in one: the last step of a
call takes other kernels than the steady ones (row gather and stress update
apart, the outputs only a caller reads), captured steps and single ones, with
the row gather that goes on to the stress update (4,455 nodes) and without
(23,782).  Energies are summed by atomics: 53 steps of 64 slots, 1e-12."""
import numpy as np
import pytest

from taylor_b200 import _lib, cases, mega

pytestmark = pytest.mark.gpu

FIELDS = (_lib.F_DSP_TOT, _lib.F_COO_CURRENT, _lib.F_VEL, _lib.F_ACL, _lib.F_STRESS, _lib.F_STRAIN, _lib.F_EPS)
KINDS = {
    "j2": {},
    "rate": {},
    "nsni": dict(itype_int=2),
    "body": dict(gravity=(0.0, 1.0e5, -2.0e5)),
    "small": dict(finite_strain=0),
    "interp": {},
}


@pytest.mark.parametrize("h", [0.6e-3, 0.35e-3])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_any_split_has_the_bits_of_one_call(mode, kind, h):
    c = cases.taylor_bar(h=h, seed=2, rate_law=(90e6, 292e6, 0.31, 0.025, 1.0) if kind == "rate" else None)
    dt = cases.lattice_dt(c, 0.3)
    out = []
    for split in ([53], [3, 2, 16, 1, 31], [20, 20, 13]):
        m = mega.Mega(c, _lib.params(**cases.param_kwargs(c, **KINDS[kind])))
        m.search_and_shapes()
        for k in split:
            m.step(k, dt, mode=mode, interp_each_step=kind == "interp")
        out.append(([m.download(f) for f in FIELDS], m.scalars()))
        m.close()
    (want, t), rest = out[0], out[1:]
    assert t["plastic_nodes_total"] > 0
    for got, s in rest:
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
        for k in ("int_energy", "kin_energy"):
            assert abs(s[k] - t[k]) <= 1e-12 * abs(t[k])
        for k in ("newton_iters", "plastic_nodes", "newton_iters_total", "plastic_nodes_total"):
            assert s[k] == t[k]
