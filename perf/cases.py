"""The work this framework is asked to do, as cases that can be run and timed.

Each case is one call sequence a program makes through taylor_b200.mega, over
the sizes of the repository's own configurations (the copper Taylor bar of
D = 6.4 mm, L = 32.4 mm on lattices of 0.6 to 0.1 mm, the notched PMB plate):

  sweep  a resident model is started again from rest with new initial
         velocities (a study over impact speeds, or a restart), stepped, and
         its fields are read back.  Direct or stabilised nodal integration,
         J2 or the rate-dependent law, FP64 or mixed precision.
  batch  the same for many bars of uneven size stepped as one context, each
         with its own stable step.
  job    a whole short run with nothing kept: upload, neighbour search,
         shape functions, steps, download.
  pmb    a whole bond-based peridynamics run of a notched plate.
  fint   one call of the stateless drop-in CONSTRUCT_FINT on host arrays, as
         the Fortran program calls it once per step.

Mixed-precision runs carry single precision (their forces and stresses are
sums of floats), so their fields are returned, as such a program would store
them, as float32; FP64 runs return float64.
"""
import math

import numpy as np
import torch

from taylor_b200 import _lib, cases, mega

RATE_LAW = (90e6, 292e6, 0.31, 0.025, 1.0)  # A, B, n, C, epsdot0 of annealed copper
FIELDS = (_lib.F_COO_CURRENT, _lib.F_VEL, _lib.F_STRESS, _lib.F_EPS)
BAR_R, BAR_L = 3.2e-3, 32.4e-3


def listed():
    sw = dict(kind="sweep", law="j2", nsni=False)
    return [
        # the coarsest bar anyone steps: every launch is short, latency counts
        dict(sw, name="sweep_fp64_4k", h=0.6e-3, prec="fp64", steps=200, tune=False),
        # the survey's 16 k-node bar in the precision of long runs
        dict(sw, name="sweep_mixed_16k", h=0.4e-3, prec="mixed", steps=200, tune=False),
        # a medium bar (0.2 mm), plain FP64 as the Fortran drop-in steps it
        dict(sw, name="sweep_fp64_130k", h=0.2e-3, prec="fp64", steps=200, tune=False),
        # the rate-dependent law, whose return mapping iterates on transcendentals
        dict(sw, name="sweep_rate_mixed_255k", h=0.16e-3, prec="mixed", steps=200, tune=True, law="rate"),
        # the benchmark's 1.04 M-node bar, both precisions
        dict(sw, name="sweep_mixed_1m", h=0.1e-3, prec="mixed", steps=300, tune=True),
        dict(sw, name="sweep_fp64_1m", h=0.1e-3, prec="fp64", steps=150, tune=True),
        # stabilised nodal integration, the reference's default ITYPE_INT (its
        # probed tangent amplifies float rounding, so mixed runs are read often)
        dict(sw, name="nsni_fp64_38k", h=0.3e-3, prec="fp64", steps=100, tune=False, nsni=True),
        dict(sw, name="nsni_mixed_130k", h=0.2e-3, prec="mixed", steps=30, tune=False, nsni=True),
        # a parameter study: 24 bars of uneven size in one context
        dict(kind="batch", name="batch_mixed_24", bars=24, h=0.25e-3, prec="mixed", steps=200, tune=False),
        # a short run end to end: set-up counts as much as the steps
        dict(kind="job", name="job_mixed_1m", h=0.1e-3, prec="mixed", steps=20, law="j2", nsni=False),
        # a notched glass plate, bonds breaking
        dict(kind="pmb", name="pmb_mixed_320k", nx=200, ny=200, nz=8, prec="mixed", steps=150),
        # the drop-in force subroutine on host arrays
        dict(kind="fint", name="fint_fp64_38k", h=0.3e-3, prec="fp64"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "nsni", "batch", "job", "pmb", "fint"])
    prec = rng.choice(["fp64", "mixed"])
    if kind in ("sweep", "nsni"):
        nsni = kind == "nsni"
        h = _log(rng, 0.16e-3 if nsni else 0.105e-3, 0.62e-3)
        steps = rng.randint(80, 150) if not nsni else rng.randint(40, 90) if prec == "fp64" else rng.randint(15, 35)
        return dict(kind="sweep", h=h, prec=prec, steps=steps, tune=rng.random() < 0.4, nsni=nsni,
                    law="j2" if nsni else rng.choice(["j2", "j2", "rate"]))
    if kind == "batch":
        return dict(kind="batch", bars=rng.randint(5, 29), h=rng.uniform(0.25e-3, 0.35e-3), prec=prec,
                    steps=rng.randint(60, 150), tune=False)
    if kind == "job":
        return dict(kind="job", h=_log(rng, 0.105e-3, 0.5e-3), prec=prec, steps=rng.randint(7, 40),
                    law=rng.choice(["j2", "rate"]), nsni=False)
    if kind == "pmb":
        return dict(kind="pmb", nx=rng.randint(61, 230), ny=rng.randint(60, 230), nz=rng.randint(4, 9), prec=prec,
                    steps=rng.randint(50, 120))
    return dict(kind="fint", h=_log(rng, 0.25e-3, 0.62e-3), prec="fp64")


# ---- inputs

def _bar(case, seed):
    rng = np.random.default_rng(seed)
    return cases.taylor_bar(h=case["h"], seed=1 + seed, v0=float(rng.uniform(150.0, 240.0)),
                            rate_law=RATE_LAW if case.get("law") == "rate" else None)


def _bars(case, seed):
    """Bars of the study: spacings set by the case, speeds and yield stresses by the seed."""
    hs = np.random.default_rng(case["bars"]).uniform(case["h"], 0.6e-3, case["bars"])
    rng = np.random.default_rng(seed)
    bars = [cases.taylor_bar(h=float(h), v0=float(rng.uniform(100.0, 300.0)), sy=float(rng.uniform(200e6, 600e6)),
                             seed=1000 * (1 + seed) + k) for k, h in enumerate(hs)]
    keys = ("coo", "win", "vol", "mass", "ebc", "vinit", "props", "mat_type", "body_id", "sm_len")
    c = {k: np.concatenate([b[k] for b in bars]) for k in keys}
    c.update(n=len(c["coo"]), counts=np.array([b["n"] for b in bars], np.int32), bodyforce=None,
             dist_max=np.stack([b["dist_max"] for b in bars]), ql_len=float(min(b["ql_len"] for b in bars)),
             dt=np.array([cases.lattice_dt(b) for b in bars]))
    return c


def _plate(case, seed):
    rng = np.random.default_rng(seed)
    return cases.pd_plate(nx=case["nx"], ny=case["ny"], nz=case["nz"], jitter=0.02, seed=1 + seed,
                          notch=0.2 * case["nx"] * 0.25e-3, v_edge=float(rng.uniform(4.0, 6.0)))


def _pmb_dt(pl):
    return 0.4 * pl["h"] / math.sqrt(72e9 / pl["rho"])


def _params(c, nsni=False):
    return _lib.params(**cases.param_kwargs(c, itype_int=2 if nsni else 0))


def _model(case, c):
    m = mega.Mega(c, _params(c, case.get("nsni", False)))
    m.set_precisions(fp64=case["prec"] == "fp64", mixed=case["prec"] == "mixed")
    if case["kind"] == "batch":
        m.set_instances(c["counts"], c["dist_max"])
    m.search_and_shapes()
    if case["kind"] == "batch":
        m.set_instance_dt(c["dt"])
    return m


def _deformed(c, seed):
    """A bar some way into its impact, for one force call: a smooth finite
    displacement, a small increment, and stresses and plastic strains to match."""
    rng = np.random.default_rng(seed + 1000)
    x = c["coo"] / np.array([BAR_R, BAR_R, BAR_L])
    a, b, k = rng.uniform(0.5, 1.5, (3, 3)), rng.uniform(0.0, 6.0, (3, 3)), rng.uniform(0.5, 2.0, (3, 3))
    f = lambda s: np.stack([sum(a[i, j] * np.sin(k[i, j] * x[:, j] + b[i, j]) for j in range(3)) for i in range(3)], 1) * s
    strs = rng.normal(0.0, 60e6, (c["n"], 6))
    state = np.zeros((c["n"], 20))
    state[:, 2] = np.abs(rng.normal(0.0, 0.02, c["n"]))
    return dict(dinc=(0.002 * f(c["h"])).reshape(-1), dinc_tot=f(0.3 * c["h"]).reshape(-1), stress=strs,
                strain=rng.normal(0.0, 1e-3, (c["n"], 6)), state=state)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pmb":
        pl = _plate(case, seed)
        return dict(case=case, plate=pl, rect=cases.notch_rect(pl), dt=_pmb_dt(pl))
    c = _bars(case, seed) if kind == "batch" else _bar(case, seed)
    dt = float(c["dt"].min()) if kind == "batch" else cases.lattice_dt(c, 0.3)
    if kind == "job":
        return dict(case=case, bar=c, dt=dt)
    if kind == "fint":
        p = _params(c)
        nb = mega.bin_search(c["coo"], c["win"], c["sm_len"], c["dist_max"])
        en = np.any(c["ebc"] == 1, axis=1).astype(np.int32)
        shp, dshp = mega.rk_shapes(p, c["coo"], c["win"], en, nb["gn"], nb["gstart"], nb["gstack"])
        return dict(case=case, bar=c, p=p, nb=nb, en=en, shp=shp, dshp=dshp, dt=dt, **_deformed(c, seed))
    m = _model(case, c)
    if case["tune"]:
        m.autotune(dt, case["prec"])
    n = c["n"]
    zero = {_lib.F_DSP_TOT: np.zeros((n, 3)), _lib.F_ACL: np.zeros((n, 3)), _lib.F_STRESS: np.zeros((n, 6)),
            _lib.F_STRAIN: np.zeros((n, 6)), _lib.F_EPS: np.zeros(n)}
    if case.get("nsni"):
        zero[_lib.F_NSNI_SGRAD] = np.zeros((n, 18))
    start = dict(zero)
    start[_lib.F_VEL] = np.where(c["ebc"] == 1, 0.0, c["vinit"])
    return dict(case=case, m=m, dt=dt, start=start)


def _out(case, a):
    t = torch.from_numpy(a)
    return t.to(torch.float32) if case["prec"] == "mixed" else t


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pmb":
        pl = state["plate"]
        p = mega.Pmb(pl, fixed=pl["fixed"], mode=case["prec"])
        p.cut(*state["rect"])
        p.step(case["steps"], state["dt"])
        out = [_out(case, p.download(k)[0]) for k in (0, 1, 4)]
        p.close()
        return out
    if kind == "fint":
        c, nb = state["bar"], state["nb"]
        r = mega.construct_fint(state["p"], c["coo"], c["win"], c["vol"], c["props"], c["mat_type"], state["en"],
                                state["state"], state["stress"], state["strain"], state["dinc"], state["dinc_tot"],
                                nb["gn"], nb["gstart"], nb["gstack"], state["shp"], state["dshp"], False, state["dt"])
        return [r["fint"], r["stress"], r["strain"], r["state"]]
    if kind == "job":
        m = _model(case, state["bar"])
        m.step(case["steps"], state["dt"], case["prec"])
        out = [_out(case, m.download(f)) for f in FIELDS]
        m.close()
        return out
    m = state["m"]
    for f, a in state["start"].items():
        m.upload(f, a)
    m.step(case["steps"], state["dt"], case["prec"])
    return [_out(case, m.download(f)) for f in FIELDS]


# ---- what a pass cannot do without

def _bar_nodes(h):
    return math.pi * (BAR_R / h) ** 2 * (BAR_L / h + 1.0)


def work(case):
    w = 8 if case["prec"] == "fp64" else 4
    if case["kind"] == "pmb":
        n = case["nx"] * case["ny"] * case["nz"]
        bonds = 104.0 * n
        # per step: a neighbour id and a broken bit a bond; position, volume,
        # displacement, velocity and acceleration of each particle
        return {"bytes": case["steps"] * (bonds * 2.125 + n * (32 + 6 * 24)) + n * 18 * 8, "flops": case["steps"] * bonds * 40.0}
    if case["kind"] == "batch":
        hs = np.linspace(case["h"], 0.6e-3, 64)
        n = case["bars"] * float(np.mean([_bar_nodes(h) for h in hs]))
    else:
        n = _bar_nodes(case["h"])
    nsni = case.get("nsni", False)
    nnz = n * (107.0 if nsni else 61.0)
    entry = 3 * w + 2 + (6 * w if nsni else 0)  # gradients (and second derivatives) and a neighbour id
    node = 30 * 8 + 24 * 8                      # state read and written: u, du, v, a, f, stress, strain, eps, mass, volume
    if case["kind"] == "fint":
        return {"bytes": nnz * (32 + 4) + n * 8 * (9 + 30 + 2 * 32 + 6 + 3), "flops": nnz * 54.0 + n * 600.0}
    if nsni:
        node += 36 * 8
    flops = case["steps"] * (nnz * (54.0 + (72.0 if nsni else 0.0)) + n * 600.0)
    io = n * 8 * (13 + (22 if case["kind"] in ("sweep", "batch") else 60))
    if case["kind"] == "job":
        flops += nnz * 400.0
        io += nnz * entry
    return {"bytes": case["steps"] * (nnz * entry + n * node) + io, "flops": flops}


# ---- the same in 64 bits with plain torch

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_dev(), torch.float64)


def _pairs(x, reach, ball=None):
    """All (i, j) with |x_i - x_j| < reach per axis (and inside the ball), i ascending."""
    n = len(x)
    lo = x.min(0).values
    cell = torch.floor((x - lo) / reach).long()
    dim = cell.max(0).values + 3
    key = ((cell[:, 0] + 1) * dim[1] + cell[:, 1] + 1) * dim[2] + cell[:, 2] + 1
    order = torch.argsort(key)
    count = torch.bincount(key, minlength=int(dim.prod()))
    start = torch.cumsum(count, 0) - count
    most = int(count.max())
    me = torch.arange(n, device=x.device)
    ri, ci = [], []
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            for c in (-1, 0, 1):
                k = key + (a * dim[1] + b) * dim[2] + c
                s, m = start[k], count[k]
                for q in range(most):
                    ok = me[q < m]
                    j = order[s[ok] + q]
                    d = x[ok] - x[j]
                    keep = (d.abs() < reach).all(1)
                    if ball is not None:
                        keep &= (d / ball).square().sum(1).sqrt() < 1.0
                    ri.append(ok[keep])
                    ci.append(j[keep])
    r, c = torch.cat(ri), torch.cat(ci)
    o = torch.argsort(r * n + c)
    return r[o], c[o]


def _rk(x, pt, win, sing, rows, cols, ql_len, ql_coef=0.001):
    """Shape gradients (and values) of every pair at the rows' points pt."""
    n = len(x)
    d = pt[rows] - x[cols]
    w = win[cols]
    r = d / w
    a = r.abs()
    phi1 = torch.where(a <= 0.5, 2 / 3 - 4 * a ** 2 + 4 * a ** 3, torch.where(a <= 1, 4 / 3 - 4 * a + 4 * a ** 2 - 4 / 3 * a ** 3, 0.0))
    dph1 = torch.where(a <= 0.5, -8 * a + 12 * a ** 2, torch.where(a <= 1, -4 + 8 * a - 4 * a ** 2, 0.0)) * torch.sign(r)
    phi = phi1.prod(1)
    w1 = w[:, :1]
    dphi = torch.stack([dph1[:, 0] * phi1[:, 1] * phi1[:, 2], phi1[:, 0] * dph1[:, 1] * phi1[:, 2],
                        phi1[:, 0] * phi1[:, 1] * dph1[:, 2]], 1) / w1
    s = sing[cols]
    wm = 1.0 / (r.square().sum(1).sqrt() + float(np.float32(1e-15)))
    dphi = torch.where(s[:, None], dphi * wm[:, None] - (phi * wm ** 3)[:, None] * r / w, dphi)
    phi = torch.where(s, phi * wm, phi)
    H = torch.cat([torch.ones_like(d[:, :1]), d], 1)

    def rowsum(v):
        return torch.zeros(n, dtype=v.dtype, device=v.device).index_add_(0, rows, v)

    M = torch.zeros(n, 4, 4, dtype=x.dtype, device=x.device)
    Md = torch.zeros(3, n, 4, 4, dtype=x.dtype, device=x.device)
    for j in range(4):
        for k in range(j, 4):
            M[:, j, k] = M[:, k, j] = rowsum(H[:, j] * H[:, k] * phi)
            for q in range(3):
                v = H[:, j] * H[:, k] * dphi[:, q]
                if j == q + 1:
                    v = v + H[:, k] * phi
                if k == q + 1:
                    v = v + H[:, j] * phi
                Md[q, :, j, k] = Md[q, :, k, j] = rowsum(v)
    star = torch.zeros(4, 4, dtype=x.dtype, device=x.device)
    hq = torch.zeros(4, dtype=x.dtype, device=x.device)
    for ax in range(3):
        for sg in (1.0, -1.0):
            hv = torch.zeros(4, dtype=x.dtype, device=x.device)
            hv[0], hv[1 + ax] = 1.0, -sg * ql_len
            star += torch.outer(hv, hv)
            hq += hv
    M = M + star * rowsum(phi)[:, None, None] * ql_coef
    sc = torch.tensor([1.0] + 3 * [float(1.0 / w.max())], dtype=x.dtype, device=x.device)  # balanced, then inverted
    Mi = torch.linalg.inv(M * sc[:, None] * sc) * sc[:, None] * sc
    b = Mi[:, 0, :]
    Hs = H + hq * ql_coef
    c = (b[rows] * Hs).sum(1)
    g = torch.empty_like(d)
    for q in range(3):
        bq = -torch.einsum("ni,nij,njk->nk", b, Md[q], Mi)
        g[:, q] = ((bq[rows] * Hs).sum(1) + b[rows, q + 1]) * phi + c * dphi[:, q]
    return c * phi, g


def _inv3(A):  # the adjugate times the determinant, as the reference writes it
    det = torch.linalg.det(A)
    adj = torch.stack([torch.linalg.cross(A[:, :, 1], A[:, :, 2]), torch.linalg.cross(A[:, :, 2], A[:, :, 0]),
                       torch.linalg.cross(A[:, :, 0], A[:, :, 1])], 1)
    return adj * det[:, None, None]


def _v2t(v):
    return torch.stack([v[:, 0], v[:, 5], v[:, 4], v[:, 5], v[:, 1], v[:, 3], v[:, 4], v[:, 3], v[:, 2]], 1).view(-1, 3, 3)


def _t2v(t):
    return torch.stack([t[:, 0, 0], t[:, 1, 1], t[:, 2, 2], t[:, 1, 2], t[:, 0, 2], t[:, 0, 1]], 1)


def _rot(R, v):
    return _t2v(R @ _v2t(v) @ R.transpose(1, 2))


def _eng(e):
    return torch.cat([e[:, :3], 2 * e[:, 3:]], 1)


def _cmul(lam, mu, e):
    tr = (e[:, :3].sum(1) * lam)[:, None]
    return torch.cat([tr + 2 * mu[:, None] * e[:, :3], mu[:, None] * e[:, 3:]], 1)


def _dev6(s):
    kk = s[:, :3].sum(1) / 3
    return torch.cat([s[:, :3] - kk[:, None], s[:, 3:]], 1), kk


def _norm6(s):
    return (s[:, :3].square().sum(1) + 2 * s[:, 3:].square().sum(1)).sqrt()


def _norm6e(e):
    return e.square().sum(1).sqrt()  # engineering shears, weighted as the reference does


class _Exact:
    """The explicit step of a case's bar(s) in double, sums by sparse products."""

    def __init__(self, c, nsni=False, rate=None):
        self.n = n = c["n"]
        self.nsni, self.rate = nsni, rate
        x, win = _t(c["coo"]), _t(c["win"])
        sml = _t(c["sm_len"])
        sing = torch.from_numpy(np.any(c["ebc"] == 1, axis=1)).to(x.device)
        rows, cols, o = [], [], 0
        for k in (c["counts"] if "counts" in c else [n]):
            e = o + int(k)
            reach = float(win[o:e].max()) + (float(sml[o:e].max()) if nsni else 0.0)
            r, q = _pairs(x[o:e], reach)
            rows.append(r + o)
            cols.append(q + o)
            o = e
        rows, cols = torch.cat(rows), torch.cat(cols)
        self.shp, g = _rk(x, x, win, sing, rows, cols, c["ql_len"])
        crow = torch.zeros(n + 1, dtype=torch.int64, device=x.device)
        crow[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
        order = torch.argsort(cols * n + rows)
        ccol = torch.zeros_like(crow)
        ccol[1:] = torch.cumsum(torch.bincount(cols, minlength=n), 0)
        trow = rows[order]
        mat = lambda v: torch.sparse_csr_tensor(crow, cols, v, (n, n))
        tmat = lambda v: torch.sparse_csr_tensor(ccol, trow, v[order], (n, n))
        self.G = [mat(g[:, k].contiguous()) for k in range(3)]
        self.Gt = [tmat(g[:, k].contiguous()) for k in range(3)]
        self.P = mat(self.shp)
        if nsni:
            D = [[None] * 3 for _ in range(3)]
            for a in range(3):
                f = []
                for sg, q in ((1.0, 2 * a), (-1.0, 2 * a + 1)):
                    pt = x.clone()
                    pt[:, a] += sg * sml[:, q]
                    f.append(_rk(x, pt, win, sing, rows, cols, c["ql_len"])[1])
                wd = (sml[:, 2 * a] + sml[:, 2 * a + 1])[rows]
                for b in range(3):
                    D[a][b] = (f[0][:, b] - f[1][:, b]) / wd
            S = [D[0][0], D[1][1], D[2][2], 0.5 * (D[0][1] + D[1][0]), 0.5 * (D[1][2] + D[2][1]), 0.5 * (D[0][2] + D[2][0])]
            self.S = [mat(v.contiguous()) for v in S]
            self.St = [tmat(v.contiguous()) for v in S]
            self.fac = torch.stack([(sml[:, 2 * a] + sml[:, 2 * a + 1]).square() / 12 for a in range(3)])
        self.x, self.vol = x, _t(c["vol"])
        p = _t(c["props"])
        self.E, self.nu, self.s0, self.B, self.C = p[:, 1], p[:, 0], p[:, 3], p[:, 4], p[:, 5]
        self.p7, self.p8, self.lam, self.mu = p[:, 6], p[:, 7], p[:, 27], p[:, 28]
        self.mass = _t(c["mass"])
        self.fixed = torch.from_numpy(c["ebc"] == 1).to(x.device)
        self.vel = torch.where(self.fixed, 0.0, _t(c["vinit"]))
        z3, z6 = torch.zeros_like(x), torch.zeros(n, 6, dtype=x.dtype, device=x.device)
        self.u, self.acl, self.stress, self.strain = z3.clone(), z3.clone(), z6.clone(), z6.clone()
        self.eps = torch.zeros_like(self.vol)
        self.sg = [z6.clone() for _ in range(3)]

    def returned(self, sp, dt):
        """Radial return of the trial stress to J2 with linear or rate-dependent hardening."""
        d, kk = _dev6(sp)
        q = _norm6(d)
        r = math.sqrt(2.0 / 3.0)
        mu = self.E / (2 * (1 + self.nu))
        if self.rate is None:  # sigma_y = s0 (1 + B eps), C = 1: linear in the multiplier
            f = q - r * self.s0 * (1 + self.B * self.eps)  # an overstress below 1e-5 of the yield stress is left
            dg = torch.where(f > r * self.s0 * float(np.float32(1e-5)), f, 0.0) / (2 * mu + r * r * self.s0 * self.B)
        else:
            dte = dt if torch.is_tensor(dt) else torch.full_like(q, dt)

            def over(g):
                ep = self.eps + r * g
                sy = self.s0 + self.B * ep.clamp(min=0) ** self.C * (1 + self.p7 * torch.log(torch.clamp(r * g / dte / self.p8, min=1.0)))
                return q - 2 * mu * g - r * sy
            on = q - r * (self.s0 + self.B * self.eps ** self.C) > 0
            lo, hi = torch.zeros_like(q), q / (2 * mu)
            idx = on.nonzero()[:, 0]
            dg = torch.zeros_like(q)
            if len(idx):
                keep = (self.eps, self.s0, self.B, self.C, self.p7, self.p8)
                full_q, full_mu = q, mu
                self.eps, self.s0, self.B, self.C, self.p7, self.p8 = (t[idx] for t in keep)
                q, mu, dte = full_q[idx], full_mu[idx], dte[idx]
                y0, y1 = torch.log(hi[idx]) - 60.0, torch.log(hi[idx])
                for _ in range(70):  # bisection in ln(dg), over() falls with dg
                    ym = 0.5 * (y0 + y1)
                    up = over(torch.exp(ym)) > 0
                    y0, y1 = torch.where(up, ym, y0), torch.where(up, y1, ym)
                dg[idx] = torch.exp(0.5 * (y0 + y1))
                self.eps, self.s0, self.B, self.C, self.p7, self.p8 = keep
                q, mu = full_q, full_mu
        new = d * (1 - 2 * mu * dg / torch.where(q > 0, q, 1.0))[:, None]
        new[:, :3] += kk[:, None]
        return new, self.eps + r * dg

    def force(self, u, du, dt):
        """Updates stress, strain and plastic strain; returns the internal force."""
        eye = torch.eye(3, dtype=u.dtype, device=u.device)
        both = torch.cat([u, du], 1)
        FG = torch.stack([g @ both for g in self.G], 2)  # (n, 6, 3)
        F, G0 = eye + FG[:, :3], FG[:, 3:]
        det = torch.linalg.det(F).abs()
        IF = _inv3(F)
        L = G0 @ IF
        A1 = _inv3(eye + 0.5 * L)
        Gm = L @ A1
        W = 0.5 * (Gm - Gm.transpose(1, 2))
        R = eye + _inv3(eye - 0.5 * W) @ W
        de = _eng(_t2v(0.5 * (Gm + Gm.transpose(1, 2))))
        s0 = _rot(R, self.stress)
        self.strain = _rot(R, self.strain) + de
        self.stress, self.eps = self.returned(s0 + _cmul(self.lam, self.mu, de), dt)
        vj = (self.vol * det)[:, None, None]
        T = vj * _v2t(self.stress) @ IF.transpose(1, 2)
        f = sum(self.Gt[m] @ T[:, :, m].contiguous() for m in range(3))
        if self.nsni:
            gs, ks = self.E / (2 * (1 + self.nu)), self.E / (3 * (1 - 2 * self.nu))
            sd, sk = _dev6(self.stress - s0)
            ed, ek = _dev6(de)
            a, b = _norm6(sd), _norm6e(ed)
            gs = torch.where((a > 1e-8) & (b > 1e-8), torch.minimum(a / b / 2, gs), gs)
            a, b = math.sqrt(3.0) * sk.abs(), math.sqrt(3.0) * ek.abs()
            ks = torch.where((a > 1e-8) & (b > 1e-8), torch.minimum(a / b / 3, ks), ks)
            H = torch.stack([s @ du for s in self.S], 2)  # (n, k, q)
            at = ((0, 3, 5), (3, 1, 4), (5, 4, 2))
            Wq = torch.zeros_like(H)
            for ax in range(3):
                La = H[:, :, list(at[ax])] @ IF
                E = La @ A1 - L @ (A1 @ (0.5 * La) @ A1)
                dea = _eng(_t2v(0.5 * (E + E.transpose(1, 2))))
                self.sg[ax] = _rot(R, self.sg[ax]) + _cmul(ks - 2 * gs / 3, gs, dea)
                Wa = self.fac[ax][:, None, None] * vj * _v2t(self.sg[ax]) @ IF.transpose(1, 2)
                for m in range(3):
                    Wq[:, :, at[ax][m]] += Wa[:, :, m]
            f = f + sum(self.St[q] @ Wq[:, :, q].contiguous() for q in range(6))
        return f

    def steps(self, k, dt):
        dn = dt if not torch.is_tensor(dt) else dt[:, None]
        for _ in range(k):
            du = dn * self.vel + 0.5 * dn * dn * self.acl
            self.u = self.u + du
            v = self.vel + 0.5 * dn * self.acl
            f = self.force(self.u, du, dt)
            self.acl = torch.where(self.fixed, 0.0, -f / self.mass)
            self.vel = torch.where(self.fixed, 0.0, v + 0.5 * dn * self.acl)
        return [self.x + self.P @ self.u, self.vel, self.stress, self.eps]


def _exact_pmb(case, seed):
    pl = _plate(case, seed)
    dt = _pmb_dt(pl)
    x, vol = _t(pl["coo"]), _t(pl["vol"])
    rows, cols = _pairs(x, pl["delta"], pl["delta"])
    off = rows != cols
    rows, cols = rows[off], cols[off]
    xi = x[cols] - x[rows]
    L0 = xi.square().sum(1).sqrt()
    y = pl["ymid"]
    a, b = x[rows], x[cols]
    cross = (a[:, 1] - y) * (b[:, 1] - y) < 0
    t = (y - a[:, 1]) / torch.where(cross, b[:, 1] - a[:, 1], 1.0)
    broken = cross & (a[:, 0] + t * (b[:, 0] - a[:, 0]) < pl["notch"])
    fixed = torch.from_numpy(pl["fixed"] != 0).to(x.device)[:, None]
    v, acl = _t(pl["vinit"]), torch.zeros_like(x)
    u = dt * v
    for _ in range(case["steps"]):
        last = u
        eta = xi + (u[cols] - u[rows])
        ln = eta.square().sum(1).sqrt()
        s = (ln - L0) / L0
        broken = broken | (s > pl["s_c"])
        w = torch.where(broken, 0.0, pl["c"] * s * vol[cols] / ln)
        f = torch.zeros_like(x).index_add_(0, rows, w[:, None] * eta)
        new = f / pl["rho"]
        v = torch.where(fixed, v, v + 0.5 * dt * (acl + new))
        acl = torch.where(fixed, acl, new)
        u = u + dt * v + torch.where(fixed, 0.0, 0.5 * dt * dt * new)
    bonds = torch.bincount(rows, minlength=len(x))
    dam = torch.bincount(rows[broken], minlength=len(x)).double() / bonds.clamp(min=1)
    return [last.reshape(-1).cpu(), v.reshape(-1).cpu(), dam.cpu()]


def exact(case, seed):
    kind = case["kind"]
    if not torch.cuda.is_available():
        return None  # over 20 seconds without one
    if kind == "pmb":
        return _exact_pmb(case, seed)
    c = _bars(case, seed) if kind == "batch" else _bar(case, seed)
    e = _Exact(c, case.get("nsni", False), RATE_LAW if case.get("law") == "rate" else None)
    if kind == "fint":
        d = _deformed(c, seed)
        e.stress, e.strain, e.eps = _t(d["stress"]), _t(d["strain"]), _t(d["state"][:, 2])
        f = e.force(_t(d["dinc_tot"]).view(-1, 3), _t(d["dinc"]).view(-1, 3), cases.lattice_dt(c, 0.3))
        state = _t(d["state"])
        state[:, 2] = e.eps
        return [f.reshape(-1).cpu(), e.stress.cpu(), e.strain.cpu(), state.cpu()]
    dt = _t(np.repeat(c["dt"], c["counts"])) if kind == "batch" else cases.lattice_dt(c, 0.3)
    return [o.cpu() for o in e.steps(case["steps"], dt)]
