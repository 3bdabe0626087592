"""The work that a user of this engine has it do, as cases that can be timed
and compared: single evaluations, the fits of one trial period, the
convexity pre-pass, scans in every form, the learned cascade, a packed
multi-object launch and the training of the stop predictor, each through the
package's public entry points.

Photometry is synthetic, of the shapes that this repository's benchmark and
tests use: sparse calibrated points over 8 years and dense relative
lightcurves of 3 h, a convex body with random Laplace coefficients, Gaussian
magnitude noise."""
from __future__ import annotations

import math

import numpy as np

from periodsearch_gb300 import Engine, InputData, Pack, PS_FORM_FP64, PS_FORM_MIXED, learned

N_POLES = 10
YEAR = 365.25
TINY_MU = 1e-8
ROW_FIELDS = ("period_h", "rms", "chi2", "dark_or_conw", "lambda_deg", "beta_deg")
FIT_FIELDS = ("dev", "dark", "totarea", "period_h", "lambda_deg", "beta_deg", "chisq", "niter", "err_code")
BETA_POLE = (0, 0, 0, 0, 60, 60, 60, -60, -60, -60)
LAMBDA_POLE = (0, 90, 180, 270, 60, 180, 300, 60, 180, 300)

# A case's object: n_dense relative lightcurves of dense_points each, n_sparse
# calibrated points, a Laplace series of degree and order lmax on 8 nrows^2
# facets, the LM stop rule (> 1: iterations; < 1: smallest improvement of rms)
# and whether the Lambert weight is free.
OBJECT = dict(n_dense=8, dense_points=60, n_sparse=500, lmax=6, nrows=6, stop=50.0, free_cl=False)


def listed():
    return [
        # one evaluation of the model (chi^2, normal matrix, facet areas): the
        # smallest call, all latency; the benchmark's object
        dict(name="eval_fp64", do="eval", form="fp64", **OBJECT),
        dict(name="eval_mixed", do="eval", form="mixed", **OBJECT),
        # a look at one trial period: ten fits, far fewer than the device holds
        dict(name="period_fp64", do="fits", form="fp64", periods=1, **OBJECT),
        dict(name="period_mixed", do="fits", form="mixed", periods=1, **OBJECT),
        # the convexity pre-pass that every job starts with: launches of 100
        # FP64 fits; a work unit of sparse survey photometry
        dict(name="prepass_fp64", do="prepass", form="fp64", **{**OBJECT, "n_dense": 0, "n_sparse": 200}),
        # the drop-in's scan, 400 fits: a few waves with a ragged last one
        dict(name="scan_fp64", do="scan", form="fp64", periods=40, **OBJECT),
        # the mixed form's scan: a window of the benchmark's
        dict(name="scan_mixed", do="scan", form="mixed", periods=301, **OBJECT),
        # the same with a Laplace series of degree 8 on 512 facets
        dict(name="scan_mixed_wide", do="scan", form="mixed", periods=101, **{**OBJECT, "lmax": 8, "nrows": 8}),
        # a work unit of relative lightcurves only, odd sizes
        dict(name="scan_mixed_relative", do="scan", form="mixed", periods=151,
             **{**OBJECT, "n_dense": 19, "dense_points": 43, "n_sparse": 0}),
        # the whole job in its fastest form: screening, completion, FP64 refit
        dict(name="scan_learned", do="learned", form="mixed", periods=1001, **OBJECT),
        # many work units of 100 to 5000 points in one launch
        dict(name="pack_mixed", do="pack", form="mixed", objects=40, periods=4, points_lo=100, points_hi=5000,
             **OBJECT),
        # training of the stop predictor on recorded trajectories
        dict(name="train", do="train", samples=20000, batch=512, epochs=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["eval", "fits", "prepass", "scan", "scan", "learned", "pack", "train"])
    if do == "train":
        return dict(do=do, samples=_log_int(rng, 2000, 20000), batch=rng.choice([128, 256, 500, 512]),
                    epochs=rng.randint(1, 6))
    form = "fp64" if do == "prepass" else "mixed" if do in ("learned", "pack") else rng.choice(["fp64", "mixed"])
    n_dense = rng.choice([0, rng.randint(1, 8), rng.randint(1, 19)])
    case = dict(do=do, form=form, n_dense=n_dense, dense_points=rng.randint(15, 90),
                n_sparse=_log_int(rng, 60, 1000) if n_dense == 0 or rng.random() < 0.6 else 0,
                lmax=rng.choice([3, 4, 6, 6, 7, 8]), nrows=rng.randint(5, 8), stop=rng.choice([50.0, 50.0, 30.0, 0.001]),
                free_cl=rng.random() < 0.25)
    if form == "fp64" and _eval_flops(case) > 2 * _eval_flops(OBJECT):
        case.update(lmax=6, nrows=6, n_dense=min(n_dense, 8))
    if do == "pack":
        case.update(objects=rng.randint(4, 40), points_lo=100, points_hi=_log_int(rng, 400, 5000))
    if do != "eval" and do != "prepass":
        # as many periods as half of the largest listed case's work holds
        one = _fit_flops({**case, "periods": 1}) * (8.0 if form == "fp64" else 1.0)
        most = 0.5 * _fit_flops(listed()[5]) * 8.0 / one
        top = dict(fits=12, scan=300, learned=1000, pack=6)[do]
        case["periods"] = max(1, min(_log_int(rng, 1, top), int(most)))
    elif do == "prepass":   # up to seven launches
        case.update(lmax=min(case["lmax"], 6), nrows=min(case["nrows"], 6))
        if case["n_sparse"] + n_dense * case["dense_points"] > 350:
            case.update(n_dense=rng.randint(0, 3), n_sparse=_log_int(rng, 60, 250))
    return case


# ---------------------------------------------------------------------------
# Objects: the facet grid, a body, its photometry (plain numpy)
# ---------------------------------------------------------------------------
def _grid(nrows, lmax):
    """Normals [F,3], areas [F] and the Laplace basis [F,C] of the octant
    triangulation (unnormalised Legendre functions, m outer, l inner, cos
    before sin)."""
    theta, phi, rows = [0.0], [0.0], [[0]]
    ring = list(range(1, nrows + 1)) + list(range(nrows - 1, 0, -1))
    for k, r in enumerate(ring):
        first = len(theta)
        theta += [(k + 1) * math.pi / (2 * nrows)] * (4 * r)
        phi += [j * math.pi / (2 * r) for j in range(4 * r)]
        rows.append(list(range(first, first + 4 * r)) + [first])
    theta.append(math.pi)
    phi.append(0.0)
    rows.append([len(theta) - 1])
    tri = []
    for r in range(1, nrows + 1):
        up, low = rows[r - 1], rows[r]
        for o in range(4):
            j0 = o * r
            tri.append((up[j0 - o], low[j0], low[j0 + 1]))
            for j in range(j0 + 1, j0 + r):
                tri.append((low[j], up[j - o], up[j - 1 - o]))
                tri.append((up[j - o], low[j], low[j + 1]))
    for r in range(nrows + 1, 2 * nrows + 1):
        up, low = rows[r - 1], rows[r]
        w = 2 * nrows - r
        for o in range(4):
            j0 = o * w
            tri.append((low[j0], up[j0 + 1 + o], up[j0 + o]))
            for j in range(j0 + 1, j0 + w + 1):
                tri.append((low[j], up[j + o], low[j - 1]))
                tri.append((low[j], up[j + 1 + o], up[j + o]))
    th, ph, tri = np.array(theta), np.array(phi), np.array(tri)
    v = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], 1)
    n = np.cross(v[tri[:, 1]] - v[tri[:, 0]], v[tri[:, 2]] - v[tri[:, 0]])
    size = np.linalg.norm(n, axis=1)
    nor = n / size[:, None]
    t, f = np.arccos(nor[:, 2]), np.arctan2(nor[:, 1], nor[:, 0])
    ct, st = np.cos(t), np.sin(t)
    cols = []
    for m in range(lmax + 1):
        p0, p1 = np.zeros_like(t), np.full_like(t, float(np.prod(np.arange(1, 2 * m, 2)))) * st ** m
        for l in range(m, lmax + 1):
            if l > m:
                p0, p1 = p1, ((2 * l - 1) * ct * p1 - (l + m - 1) * p0) / (l - m)
            cols.append(p1 * np.cos(m * f))
            if m:
                cols.append(p1 * np.sin(m * f))
    return nor, 0.5 * size, np.stack(cols, 1)


def _body(rng, lmax):
    """Laplace coefficients of a slightly irregular convex body."""
    cg = []
    for m in range(lmax + 1):
        for l in range(m, lmax + 1):
            norm = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            sd = 0.15 / (l + 1) * norm * (math.sqrt(2.0) if m else 1.0)
            cg.append(0.0 if l == 0 else rng.normal(0.0, sd))
            if m:
                cg.append(rng.normal(0.0, sd))
    return np.array(cg)


def _pole_matrix(beta, lam):
    """The pole rotation and its derivatives by beta and lambda."""
    cb, sb, cl, sl = math.cos(beta), math.sin(beta), math.cos(lam), math.sin(lam)
    return (np.array([[cb * cl, cb * sl, -sb], [-sl, cl, 0], [sb * cl, sb * sl, cb]]),
            np.array([[-sb * cl, -sb * sl, -cb], [0, 0, 0], [cb * cl, cb * sl, -sb]]),
            np.array([[-cb * sl, cb * cl, 0], [-cl, -sl, 0], [-sb * sl, sb * cl, 0]]))


def _spin(w, t, x):
    """x (points in the pole's frame) turned by the rotation phase."""
    c, s = np.cos(w * t), np.sin(w * t)
    return np.stack([c * x[:, 0] + s * x[:, 1], c * x[:, 1] - s * x[:, 0], x[:, 2]], 1)


def _object(case, seed, salt=0, sizes=None):
    """(InputData, the parameters that the brightness was made from)."""
    rng = np.random.default_rng([int(seed), salt])
    n_dense, n_sparse = sizes or (case["n_dense"], case["n_sparse"])
    lam, sin_b, period = rng.uniform(0, 2 * math.pi), rng.uniform(-1, 1), rng.uniform(4, 12)
    body = _body(rng, case["lmax"])
    incl, node, a0, e0 = math.radians(rng.uniform(-5, 5)), *rng.uniform(0, 2 * math.pi, 3)

    def positions(t):
        ta, te = 2 * math.pi * t / (YEAR * 2.6 ** 1.5) + a0, 2 * math.pi * t / YEAR + e0
        x, y = 2.6 * np.cos(ta), 2.6 * np.sin(ta)
        cn, sn, ci, si = math.cos(node), math.sin(node), math.cos(incl), math.sin(incl)
        return (np.stack([cn * x - sn * ci * y, sn * x + cn * ci * y, si * y], 1),
                np.stack([np.cos(te), np.sin(te), np.zeros_like(te)], 1))

    def epochs(n):
        got = np.zeros(0)
        while len(got) < n:
            t = rng.uniform(0, 8 * YEAR, 4 * n + 16)
            ra, re = positions(t)
            d = ra - re
            far = np.sum(d * -re, 1) < math.cos(math.radians(100)) * np.linalg.norm(d, axis=1) * np.linalg.norm(re, axis=1)
            got = np.concatenate([got, t[far]])
        return np.sort(got[:n])

    blocks = [(s + np.linspace(0, 0.125, case["dense_points"]), 0, 0.02) for s in (epochs(n_dense) if n_dense else ())]
    if n_sparse:
        ts = epochs(n_sparse)
        blocks += [(ts[i:i + 1000], 1, 0.1) for i in range(0, n_sparse, 1000)]
    t = np.concatenate([b[0] for b in blocks])
    jd = 2455000.5 + t
    zero = math.floor(jd.min())
    ra, re = positions(t)
    sun, earth = -ra, re - ra
    nor, darea, basis = _grid(9, case["lmax"])
    area = darea * np.exp(basis @ body)
    omega = 2 * math.pi * 24 / period
    B = _pole_matrix(math.pi / 2 - math.asin(sin_b), lam)[0]
    ee, ee0 = (v / np.linalg.norm(v, axis=1)[:, None] for v in (earth, sun))
    mu, mu0 = (_spin(omega, jd - zero, v @ B.T) @ nor.T for v in (ee, ee0))
    lit = (mu > TINY_MU) & (mu0 > TINY_MU)
    law = np.where(lit, mu * mu0 * (0.1 + 1 / np.where(lit, mu + mu0, 1.0)), 0.0)
    al = np.arccos(np.clip(np.sum(ee * ee0, 1), -1, 1))
    bright = (law @ area) * (1 + 0.5 * np.exp(-al / 0.1) - 0.5 * al)
    noise = np.concatenate([rng.normal(0, b[2], len(b[0])) for b in blocks])
    n_periods = 40000
    header = dict(per_start=2.0, per_end=50.0, per_step_coef=(1 / 2.0 - 1 / 50.0) * (jd.max() - jd.min()) * 48 / (n_periods - 0.5),
                  ia_prd=1, jd00=float(zero), phi0_deg=0.0, conw=0.1, lmax=case["lmax"], mmax=case["lmax"],
                  nrows=case["nrows"], par=[0.5, 0.1, -0.5], ia_par=[1, 1, 1], cl=0.1, ia_cl=int(case["free_cl"]),
                  stop_condition=case["stop"], n_iter_min=10, alamda_incr=5.0, alamda_start=0.1)
    data = InputData(header=header, lc_points=np.array([len(b[0]) for b in blocks], np.int32),
                     lc_calibrated=np.array([b[1] for b in blocks], np.int32), lc_weight=np.full(len(blocks), -1.0),
                     jd=jd, brightness=bright * 10 ** (-0.4 * noise), sun=sun, earth=earth)
    truth = np.concatenate([body, [math.pi / 2 - math.asin(sin_b), lam, omega, 0.5, 0.1, -0.5, math.log(0.1), 1.0]])
    return data, truth, rng


def _near(truth, rng):
    """Parameters as they are half-way through a fit."""
    cg = truth * (1 + rng.normal(0, 0.05, len(truth)))
    cg[-1] = 1.0
    cg[-6] = truth[-6] * (1 + rng.normal(0, 1e-7))
    return cg


def _window(rng, periods):
    return int(rng.integers(2, 39000 - periods))


def _pack_objects(case, seed):
    rng = np.random.default_rng([int(seed), 99])
    got = []
    for k in range(case["objects"]):
        n = int(round(math.exp(rng.uniform(math.log(case["points_lo"]), math.log(case["points_hi"])))))
        dense = int(min(8, max(0, (n - 100) // case["dense_points"]), rng.integers(0, 9)))
        got.append((dense, n - dense * case["dense_points"]))
    return got


# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["do"] == "train":
        rng = np.random.default_rng([int(seed), 7])
        n = case["samples"]
        chi = np.cumsum(-np.abs(rng.normal(0.4, 0.5, (n, 4))), axis=1)
        lam = np.cumsum(rng.choice([-1.4, 0.7], (n, 4), p=[0.8, 0.2]), axis=1) - 1
        x = np.concatenate([chi, lam, rng.uniform(5.3, 8, (n, 1)), rng.uniform(0.7, 4.6, (n, 1))], 1).astype(np.float32)
        y = (0.12 * chi[:, 3] - 0.2 * (chi[:, 3] - chi[:, 1]) * np.tanh(lam[:, 3]) + rng.normal(0, 0.03, n)).astype(np.float32)
        return dict(case=case, x=x, y=y, w=learned.init_weights(x, y, seed=int(seed) % 1000))
    form = PS_FORM_FP64 if case["form"] == "fp64" else PS_FORM_MIXED
    if case["do"] == "pack":
        objects = [_object(case, seed, 1 + k, s) for k, s in enumerate(_pack_objects(case, seed))]
        engines = [Engine(o[0], form=form) for o in objects]
        rng = objects[0][2]
        at = np.array([_window(rng, case["periods"]) for _ in engines])
        ob, per, pole = (a.ravel() for a in np.meshgrid(np.arange(len(engines)), np.arange(case["periods"]),
                                                        np.arange(1, N_POLES + 1), indexing="ij"))
        return dict(case=case, engines=engines, pack=Pack(engines, form), conw=[e.info.conw_r0 for e in engines],
                    object=ob, period=at[ob] + per, pole=pole)
    data, truth, rng = _object(case, seed)
    s = dict(case=case, engine=Engine(data, form=form), cg=_near(truth, rng))
    s["conw"] = s["engine"].info.conw_r0
    if "periods" in case:
        s["lo"] = _window(rng, case["periods"])
    return s


def run(state):
    case, do = state["case"], state["case"]["do"]
    if do == "train":
        w, loss = learned.train(state["x"], state["y"], epochs=case["epochs"], batch=case["batch"], weights=state["w"])
        return dict(weights=w, loss=loss)
    if do == "pack":
        f = state["pack"].fit(state["conw"], state["object"], state["period"], state["pole"])
        return {k: f[k] for k in FIT_FIELDS}
    eng, lo = state["engine"], state.get("lo", 0)
    if do == "eval":
        alpha, beta, chisq, area = eng.eval(0.1, state["cg"])
        return dict(alpha=alpha, beta=beta, chisq=chisq, area=area)
    if do == "prepass":
        conw, new = eng.precalc_conw()
        return dict(conw=conw, new=new)
    if do == "fits":
        per = np.arange(lo, lo + case["periods"])
        f = eng.fit_batch(state["conw"], np.repeat(per, N_POLES), np.tile(np.arange(1, N_POLES + 1), len(per)))
        return {k: f[k] for k in FIT_FIELDS}
    hi = lo + case["periods"] - 1
    rows = eng.scan(state["conw"], lo, hi) if do == "scan" else eng.scan_learned(state["conw"], lo, hi)[0]
    return {k: rows[k] for k in ROW_FIELDS}


# ---------------------------------------------------------------------------
def _sizes(case):
    c = (case["lmax"] + 1) ** 2
    return case["n_dense"] * case["dense_points"] + case["n_sparse"], 8 * case["nrows"] ** 2, c, c + 6


def _eval_flops(case, n=None):
    """Of one evaluation: the facet law and the contraction over the lit
    facets (about 0.47 of them), the normal matrix, the curvature."""
    n0, f, c, m = _sizes(case)
    n = n0 if n is None else n
    return (70 + 2 * c) * 0.47 * n * f + 10.0 * n * f + n * m * (m + 1.0) + 9.0 * f * c


def _fit_flops(case):
    """Of the case's fits: 51 evaluations and 50 solves each (a fit that
    stops by the rms rule: about 20)."""
    m = _sizes(case)[3]
    it = case["stop"] if case["stop"] > 1 else 20
    if case["do"] == "learned":
        it = 0.25 * it   # most fits stop after the screening
    fits, n = case["periods"] * N_POLES, None
    if case["do"] == "pack":
        fits *= case["objects"]
        n = (case["points_hi"] - case["points_lo"]) / math.log(case["points_hi"] / case["points_lo"])
    return fits * ((it + 1) * _eval_flops(case, n) + it * 2.0 * m ** 3)


def work(case):
    if case["do"] == "train":
        steps = case["epochs"] * (case["samples"] // case["batch"])
        return dict(bytes=case["samples"] * 44.0 * case["epochs"] + 4951 * 8.0,
                    flops=steps * case["batch"] * 6.0 * (64 * 10 + 64 * 64 + 64) + steps * 4800 * 12.0)
    n, f, c, m = _sizes(case)
    data = n * 12 * 8.0 + f * (c + 4) * 8.0
    if case["do"] == "eval":
        return dict(bytes=data + 8.0 * (m * m + m + 1 + f), flops=_eval_flops(case))
    if case["do"] == "prepass":   # two launches of ten periods
        return dict(bytes=data + 8.0, flops=_fit_flops({**case, "periods": 20}))
    if case["do"] == "pack":
        data *= case["objects"]
    return dict(bytes=data + case["periods"] * N_POLES * 80.0, flops=_fit_flops(case))


# ---------------------------------------------------------------------------
# The same in 64-bit numpy: the model evaluation (chi^2, its derivatives by
# the parameters, the normal matrix) and the Levenberg-Marquardt loop on it
# ---------------------------------------------------------------------------
class _Model:
    def __init__(self, case, data, conw_r=None):
        h = data.header
        self.nor, self.darea, self.basis = _grid(case["nrows"], case["lmax"])
        self.t = data.jd - h["jd00"]
        self.ee, self.ee0 = (v / np.linalg.norm(v, axis=1)[:, None] for v in (data.earth, data.sun))
        self.al = np.arccos(np.sum(self.ee * self.ee0, 1))
        self.y = data.brightness
        ends = np.cumsum(data.lc_points)
        self.curves = [(int(e - n), int(e), bool(c)) for e, n, c in zip(ends, data.lc_points, data.lc_calibrated)]
        self.sig = np.concatenate([np.full(e - b, self.y[b:e].mean()) for b, e, _ in self.curves])
        self.rel_only = not any(c for _, _, c in self.curves)
        c = self.basis.shape[1]
        free = np.ones(c + 8, bool)
        free[0] = not self.rel_only
        free[-2], free[-1] = bool(h["ia_cl"]), False
        self.free, self.h = np.flatnonzero(free), h
        # size of the starting ellipsoid, from the point of smallest phase angle
        first = [b for b, _, cal in self.curves if cal or self.rel_only]
        q = min(first, key=lambda b: self.al[b])
        r = math.sqrt(2 * self.sig[q] / (0.5 * math.pi * (1 + math.cos(self.al[q]))))
        self.size = r / math.sqrt((1.05 * 1 + 1 * 0.95 + 1.05 * 0.95) / 3) * (1.0 if self.rel_only else 0.8)
        self.conw = h["conw"] / self.size / self.size if conw_r is None else conw_r

    def start(self):
        a, b, c = 1.05 * self.size, self.size, 0.95 * self.size
        s = np.sum((self.nor * np.array([a, b, c])) ** 2, 1)
        return np.linalg.solve(self.basis.T @ self.basis, self.basis.T @ (2 * (np.log(a * b * c) - np.log(s))))

    def evaluate(self, cg):
        nor, basis, C = self.nor, self.basis, self.basis.shape[1]
        area = self.darea * np.exp(basis @ cg[:C])
        B = _pole_matrix(cg[C], cg[C + 1])
        w, (p0, p1, p2), cl, cls = cg[C + 2], cg[C + 3:C + 6], math.exp(cg[C + 6]), cg[C + 7]
        ph = np.fmod(w * self.t + self.h["phi0_deg"] * math.pi / 180, 2 * math.pi)
        turn = lambda v, m: _spin(1.0, ph, v @ m.T)  # noqa: E731
        e, e0 = turn(self.ee, B[0]), turn(self.ee0, B[0])
        mu, mu0 = e @ nor.T, e0 @ nor.T
        lit = (mu > TINY_MU) & (mu0 > TINY_MU)
        mu, mu0, ar = np.where(lit, mu, 1.0), np.where(lit, mu0, 1.0), lit * area
        den = mu + mu0
        law = mu * mu0 * (cl + cls / den) * ar
        u, v = (cls * (mu0 / den) ** 2 + cl * mu0) * ar, (cls * (mu / den) ** 2 + cl * mu) * ar
        ex = np.exp(-self.al / p1)
        scale = 1 + p0 * ex + p2 * self.al
        br = law.sum(1)
        J = np.zeros((len(br), C + 8))
        J[:, :C] = scale[:, None] * (law @ basis)
        U, V = u @ nor, v @ nor
        by_w = lambda x: self.t[:, None] * np.stack([x[:, 1], -x[:, 0], np.zeros(len(x))], 1)  # noqa: E731
        for k, (d, d0) in enumerate(((turn(self.ee, B[1]), turn(self.ee0, B[1])),
                                     (turn(self.ee, B[2]), turn(self.ee0, B[2])), (by_w(e), by_w(e0)))):
            J[:, C + k] = scale * (np.sum(d * U, 1) + np.sum(d0 * V, 1))
        J[:, C + 3], J[:, C + 4], J[:, C + 5] = br * ex, br * p0 * ex * self.al / p1 ** 2, br * self.al
        J[:, C + 6], J[:, C + 7] = scale * (mu * mu0 * ar).sum(1) * cl, scale * (mu * mu0 / den * ar).sum(1)
        ym = br * scale
        for b, e_, cal in self.curves:
            if not cal:
                total = ym[b:e_].sum()
                coef = self.sig[b:e_] * (e_ - b) / total
                J[b:e_] = coef[:, None] * (J[b:e_] - ym[b:e_, None] * J[b:e_].sum(0) / total)
                J[b:e_, 0] = 0
                ym[b:e_] *= coef
        chk = area @ nor   # the convexity rows
        K = np.zeros((3, C + 8))
        K[:, :C] = (area[:, None] * nor).T @ basis
        J, dy = np.concatenate([J, K])[:, self.free], np.concatenate([self.y - ym, -chk])
        wt = np.concatenate([1 / self.sig ** 2, np.full(3, self.conw ** 2)])
        return (J * wt[:, None]).T @ J, J.T @ (wt * dy), float(np.sum(wt * dy * dy)), area, chk

    def fit(self, n, pole):
        h, C = self.h, self.basis.shape[1]
        step = 0.5 / (self.t.max() - self.t.min()) / 24 * h["per_step_coef"]
        prd = 1 / (1 / h["per_start"] - (n - 1) * step)
        cg = np.concatenate([self.start(), [math.radians(90 - BETA_POLE[pole - 1]), math.radians(LAMBDA_POLE[pole - 1]),
                                            48 * math.pi / prd], h["par"], [math.log(h["cl"]), 1.0]])
        stop = h["stop_condition"]
        n_max, least, n_min = (int(stop), 0.0, 0) if stop > 1 else (100, stop, h["n_iter_min"])
        alpha, beta, best, area, chk = self.evaluate(cg)
        lam, it, gain, dev_old, total, acc, reg = h["alamda_start"], 0, 1e40, 1e30, 0.0, chk, 0.0
        while (it < n_max and gain > least) or it < n_min:
            A = alpha.copy()
            A[np.diag_indices(len(A))] *= 1 + lam
            trial = cg.copy()
            trial[self.free] += np.linalg.solve(A, beta)
            a1, b1, c1, area1, chk1 = self.evaluate(trial)
            it, total, better = it + 1, area1.sum(), c1 < best
            lam = lam / h["alamda_incr"] if better else lam * h["alamda_incr"]
            if better:
                alpha, beta, best, cg, acc = a1, b1, c1, trial, chk1
            if better or it == 1:
                total = area1.sum() if better else area.sum()
                reg = best - float(acc @ acc) * self.conw ** 2
            dev = math.sqrt(reg / len(self.y))
            if dev_old - dev > 1e-10:
                gain, dev_old = dev_old - dev, dev
        return dict(dev=dev, dark=math.sqrt(float(acc @ acc)), totarea=total, period_h=48 * math.pi / cg[C + 2],
                    lambda_deg=math.degrees(cg[C + 1]), beta_deg=90 - math.degrees(cg[C]), chisq=best)


def exact(case, seed):
    """An evaluation, and the ten FP64 fits of one period.  The end points of
    more fits take too long here, and those of the mixed form's fits have no
    64-bit value: 50 unconverged steps carry its rounding far."""
    if case["do"] == "eval":
        data, truth, rng = _object(case, seed)
        alpha, beta, chisq, area, _ = _Model(case, data, 0.1).evaluate(_near(truth, rng))
        return dict(alpha=alpha, beta=beta, chisq=chisq, area=area)
    if case["do"] == "fits" and case["form"] == "fp64" and _fit_flops(case) < 1.5 * _fit_flops({**listed()[2]}):
        data, _, rng = _object(case, seed)
        _near(np.zeros(_sizes(case)[2] + 8), rng)
        model, lo = _Model(case, data), _window(rng, case["periods"])
        got = [model.fit(lo + k, pole) for k in range(case["periods"]) for pole in range(1, N_POLES + 1)]
        return {**{k: np.array([g[k] for g in got]) for k in got[0]}, "niter": None, "err_code": None}
    return None
