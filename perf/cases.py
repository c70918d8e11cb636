"""Performance cases: what a user of this framework has it do, through its public entry
points, over the sizes, precisions and options of its own workloads.

A step case is a simulation: a problem (the granular column, the slope, the biaxial sample,
one of the reference's example inputs, or a batch of columns) in one of the two precision
forms.  One pass is the work between two outputs: `steps` steps, then the output fields;
with `restart` the pass begins by uploading the problem's initial state and ends with it
advanced (one run of a parameter study), otherwise it continues the run.  The surrogate cases
train the constitutive network on captured-like tuples and evaluate it.

`exact` restates the step and the training in 64-bit numpy for the sizes where that is quick.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(os.getcwd(), "stress-particle-sph_gb300"))

import sps_gb300  # noqa: E402
from sps_gb300 import surrogate  # noqa: E402

FIELDS = ("x", "vel", "stress", "rho", "intvars1", "displ", "bc_or_not", "f_drucker")
EXAMPLES = {"soil_failure": "soil_failure_bui_et_al_2008/inside_approach/SP1",
            "soil_failure_outside": "soil_failure_bui_et_al_2008/outside_approach",
            "localisation": "strain_localisation_in_soil_sample/SP1",
            "localisation_sp3": "strain_localisation_in_soil_sample/SP3"}
EXACT_PARTICLE_STEPS = 660_000  # about 15 s of numpy


def listed():
    return [
        # the smallest call: one step and its output, as an output-every-step loop does it
        dict(name="column_600_fp64", kind="column", form="fp64", dx=0.008, steps=1, restart=False),
        # the reference's soil failure example as its input file says: a whole 10-step run with
        # output after every step (XSPH, artificial viscosity, walls)
        dict(name="soil_failure_fp64", kind="soil_failure", form="fp64", dx=0.0, steps=10,
             restart=True),
        # the strain-localisation example between two outputs (every 100 steps): von Mises with
        # Perzyna flow, CSPM, segment boundary conditions
        dict(name="localisation_fp32", kind="localisation", form="fp32", dx=0.0, steps=100,
             restart=True),
        # the column collapse at its stated size, one run of a parameter study
        dict(name="column_10k_fp32", kind="column", form="fp32", dx=0.002, steps=50, restart=True),
        # a biaxial test between platens in the bit-exact form
        dict(name="biaxial_40k_fp64", kind="biaxial", form="fp64", dx=0.0005, steps=10,
             restart=True),
        # a slope with the stabilisation options on
        dict(name="slope_320k_stabilised_fp32", kind="slope", form="fp32", dx=0.03, steps=5,
             restart=False, xsph=True, alpha=0.1),
        # a coupled loop: every step's state comes from the host and goes back to it
        dict(name="slope_320k_coupled_fp32", kind="slope", form="fp32", dx=0.03, steps=1,
             restart=True),
        # a mid-sized slope in the bit-exact form
        dict(name="slope_115k_fp64", kind="slope", form="fp64", dx=0.05, steps=5, restart=False),
        # the benchmark's slope, both forms: the largest runs of one problem
        dict(name="slope_2m_fp32", kind="slope", form="fp32", dx=0.012, steps=10, restart=False),
        dict(name="slope_2m_fp64", kind="slope", form="fp64", dx=0.012, steps=2, restart=False),
        # an ensemble: 64 columns with drawn friction angles in one batch context
        dict(name="batch_64_columns_fp32", kind="batch", form="fp32", dx=0.004, count=64, steps=10,
             restart=False),
        # one epoch of surrogate training
        dict(name="training_64k", kind="training", batch=4096, rows=65536),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("column", "column", "slope", "slope", "slope", "biaxial", "batch",
                       "example", "training"))
    form = rng.choice(("fp64", "fp32"))
    restart = rng.random() < 0.5
    if kind == "training":
        batch = 64 * int(round(_log(rng, 8, 128)))
        return dict(kind=kind, batch=batch, rows=int(batch * rng.uniform(4, 12)) + rng.randrange(64))
    if kind == "example":
        return dict(kind=rng.choice(sorted(EXAMPLES)), form=form, dx=0.0,
                    steps=rng.randint(1, 10), restart=True)
    if kind == "batch":
        return dict(kind=kind, form=form, dx=round(_log(rng, 0.004, 0.009), 5),
                    count=int(_log(rng, 2, 60)), steps=rng.randint(1, 10), restart=False)
    c = dict(kind=kind, form=form, restart=restart)
    if kind == "column":
        c.update(dx=round(_log(rng, 0.0009, 0.009), 6), steps=rng.randint(1, 10))
    elif kind == "biaxial":
        c.update(dx=round(_log(rng, 0.0002, 0.004), 7), steps=rng.randint(1, 10))
    else:
        c.update(dx=round(_log(rng, 0.018, 0.2), 4), steps=rng.randint(1, 4))
    if kind != "biaxial" and rng.random() < 0.3:
        c.update(xsph=rng.random() < 0.5, alpha=0.1)
    return c


# ------------------------------------------------------------------------ the problems
def _problem(case, rng, k=0):
    """The case's problem with a seeded initial state: the set-up's own state with every node
    and stress-point moved by up to 2% of the spacing, a smooth velocity field and a smooth
    few-percent variation of the stress, as a run in progress has them."""
    kind = case["kind"]
    opt = dict(xsph=case.get("xsph", False), alpha=case.get("alpha", 0.0),
               beta=case.get("alpha", 0.0))
    if kind in EXAMPLES:
        prob = sps_gb300.Problem.from_dir(os.path.join(
            os.getcwd(), "tests", "golden", "example_problems", EXAMPLES[kind]))
    elif kind == "column":
        prob = sps_gb300.Problem.column(dx=case["dx"], **opt)
    elif kind == "batch":
        prob = sps_gb300.Problem.column(dx=case["dx"], phi_deg=float(rng.uniform(19.0, 35.0)))
    elif kind == "slope":
        prob = sps_gb300.Problem.slope(dx=case["dx"], **opt)
    else:
        prob = sps_gb300.Problem.biaxial(dx=case["dx"])
    nt, dx = prob.ntotal, float(prob.params.dx)
    x, v, s = prob.x[:2 * nt].reshape(nt, 2), prob.vel[:2 * nt].reshape(nt, 2), \
        prob.stress[:4 * nt].reshape(nt, 4)
    x += 0.02 * dx * (2.0 * rng.random((nt, 2)) - 1.0)
    prob.x00[:2 * nt] = prob.x[:2 * nt]
    span = float(np.ptp(x[:, 1]))
    wave = np.sin((2.0 * math.pi / span) * x @ rng.uniform(-1.0, 1.0, 2) + rng.uniform(0.0, 6.0))
    v += (1e-3 * span * rng.uniform(0.5, 1.0, 2)) * wave[:, None]
    s *= 1.0 + 0.03 * wave[:, None]
    return prob


def _pinned(shape, dtype):
    kind = {np.dtype(np.float64): torch.float64, np.dtype(np.int32): torch.int32}[np.dtype(dtype)]
    return torch.empty(shape, dtype=kind, pin_memory=True).numpy()


def _output(prob, make):
    """The arrays a program keeps for the output fields."""
    n2, nt, nn = prob.ntotal2, prob.ntotal, prob.nnode
    size = dict(x=2 * n2, vel=2 * n2, stress=4 * n2, rho=n2, intvars1=nt, displ=2 * nn,
                bc_or_not=nt, f_drucker=nt)
    return {k: make(n, np.int32 if k == "bc_or_not" else np.float64) for k, n in size.items()}


def _tuples(rng, n):
    """Training tuples as sps_capture collects them: scale-free inputs of loading
    stress-points and the Drucker-Prager plastic source."""
    tanfi, coh = np.tan(np.radians(rng.uniform(19.0, 35.0, n))), rng.uniform(0.0, 2e4, n)
    nu, young, rho = rng.uniform(0.22, 0.34, n), 10.0 ** rng.uniform(6.5, 7.7, n), \
        rng.uniform(1800.0, 2700.0, n)
    den = np.sqrt(9.0 + 12.0 * tanfi ** 2)
    alpha, kc = tanfi / den, 3.0 * coh / den
    p = -(10.0 ** rng.uniform(3.0, 5.3, n))
    d = rng.normal(size=(n, 4))
    d[:, 3] = -(d[:, 0] + d[:, 1])
    sj = np.sqrt(d[:, 2] ** 2 + 0.5 * (d[:, 0] ** 2 + d[:, 1] ** 2 + d[:, 3] ** 2))
    d *= ((kc - 3.0 * alpha * p) / sj)[:, None]  # on the cone
    sj = kc - 3.0 * alpha * p
    s = d.copy()
    s[:, [0, 1, 3]] += p[:, None]
    g = rng.normal(size=(n, 4))  # grad_u(a, b) at a + 2 b
    e11, e22, e12, w = g[:, 0], g[:, 3], 0.5 * (g[:, 2] + g[:, 1]), 0.5 * (g[:, 2] - g[:, 1])
    en = np.sqrt(e11 ** 2 + e22 ** 2 + 2.0 * e12 ** 2)
    size = np.sqrt((s ** 2).sum(axis=1))
    gm, km = young / (2.0 * (1.0 + nu)), young / (3.0 * (1.0 - 2.0 * nu))
    s_eps = d[:, 0] * e11 + 2.0 * d[:, 2] * e12 + d[:, 1] * e22
    rate = (3.0 * alpha * km * (e11 + e22) + gm / sj * s_eps) / gm
    t = np.empty((n, surrogate.TUPLE))
    t[:, 0:4] = s / size[:, None]
    t[:, 4], t[:, 5], t[:, 6], t[:, 7], t[:, 8] = e11 / en, e22 / en, e12 / en, 0.0, w / en
    t[:, 9], t[:, 10], t[:, 11] = tanfi, coh / size, nu
    t[:, 12], t[:, 13] = np.log10(young) - 7.0, rho / 2000.0 - 1.0
    t[:, 14:18] = -d * (rate / (sj * en))[:, None]
    return t.astype(np.float32)


def _training_inputs(case, seed):
    rng = np.random.default_rng(seed)
    return _tuples(rng, case["rows"]), _init_params(rng)


def prepare(case, seed):
    if case["kind"] == "training":
        tuples, params = _training_inputs(case, seed)
        net = surrogate.Mlp(batch=case["batch"], seed=seed, lr=2e-3)
        net.set_params(params)
        net.set_data(tuples)
        return dict(case=case, net=net)
    rng = np.random.default_rng(seed)
    prec = sps_gb300.SPS_PREC_FP32_FAST if case["form"] == "fp32" else \
        sps_gb300.SPS_PREC_FP64_PLAIN
    if case["kind"] == "batch":
        probs = [_problem(case, rng, k) for k in range(case["count"])]
        ctx = sps_gb300.Batch(probs, precision=prec)
        ctx.upload_all()
        return dict(case=case, ctx=ctx, out=[_output(p, np.empty) for p in probs])
    prob = _problem(case, rng)
    ctx = sps_gb300.Solver(prob, precision=prec)
    st = dict(case=case, ctx=ctx, out=_output(prob, _pinned))
    if case["restart"]:
        st["start"] = {}
        for k, v in prob.state().items():
            st["start"][k] = _pinned(v.shape, v.dtype)
            st["start"][k][:] = v
        st["bcs"] = (np.array(prob.bc_or_not), np.array(prob.bc_info))
    return st


def run(state):
    case = state["case"]
    if case["kind"] == "training":
        loss = state["net"].train(1)
        return dict(loss=loss, params=state["net"].params())
    ctx = state["ctx"]
    if case["kind"] == "batch":
        ctx.step(case["steps"])
        ctx.snapshot()
        for r, out in enumerate(state["out"]):
            ctx.snapshot_wait(r, out)
        return {k: np.concatenate([f[k] for f in state["out"]]) for k in FIELDS}
    if case["restart"]:
        ctx.upload(**state["start"])
        ctx.upload_bcs(*state["bcs"])
        ctx.time_sph = 0.0
    if case["kind"] in EXAMPLES and case["kind"].startswith("soil"):
        for _ in range(case["steps"]):  # print, save, plot 1,1,1
            ctx.time_integration()
            ctx.download(state["out"])
        return state["out"]
    ctx.time_integration(case["steps"])
    return ctx.download(state["out"])


def _count(case):
    """Nodes plus stress-points."""
    kind = case["kind"]
    if kind in EXAMPLES:
        return {"soil_failure": 1661, "soil_failure_outside": 2583, "localisation": 6521,
                "localisation_sp3": 12921}[kind]
    area = {"column": 0.02, "batch": 0.02 * case.get("count", 1), "biaxial": 0.005,
            "slope": 144.0}[kind]
    return 2.0 * area / case["dx"] ** 2


def work(case):
    if case["kind"] == "training":
        rows = case["rows"] // case["batch"] * case["batch"]
        macs = 14 * 128 + 2 * 128 * 128 + 128 * 4
        return dict(bytes=rows * surrogate.TUPLE * 4.0 + 4 * 4.0 * surrogate.NPARAM,
                    flops=6.0 * macs * rows)
    n, steps = _count(case), case["steps"]
    # per particle and step: x, v, stress, mass, rho, h, intvars1, f_drucker read, all but the
    # masses written; the pass's output (and the upload of a restart)
    state, out = 13 * 8 + 10 * 8, 100
    # per stress-point and step about 18 nodes in the support (h = 1.2 dx): kernel values, five
    # interpolations and four derivative sums of both sides of every pair
    pair = 40 + 5 * 16 + 4 * 46
    return dict(bytes=n * (state * steps + out + (124 if case["restart"] else 0)),
                flops=n / 2 * 18 * pair * steps)


# ------------------------------------------------------------------------ 64-bit statement
def exact(case, seed):
    if case["kind"] == "training":
        return _exact_training(case, seed)
    if case["kind"] == "soil_failure_outside" or _count(case) * case["steps"] > EXACT_PARTICLE_STEPS:
        return None
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        per = [_Exact(_problem(case, rng, k)).steps(case["steps"]) for k in range(case["count"])]
        return {k: None if per[0][k] is None else np.concatenate([f[k] for f in per])
                for k in FIELDS}
    return _Exact(_problem(case, rng)).steps(case["steps"])


class _Exact:
    """The step of the inside approach (cubic kernel; Drucker-Prager, von Mises or elastic)
    in 64 bits."""

    def __init__(self, prob):
        self.prob, self.p = prob, prob.params  # (the params live as long as their problem)
        p = self.p
        self.nn, self.nt, self.n2 = prob.nnode, prob.ntotal, prob.ntotal2
        self.x = np.array(prob.x).reshape(-1, 2)
        self.v = np.array(prob.vel).reshape(-1, 2)
        self.s = np.array(prob.stress).reshape(-1, 4)
        self.x00 = np.array(prob.x00).reshape(-1, 2)
        self.m, self.rho, self.h = np.array(prob.mass), np.array(prob.rho), np.array(prob.hsml)
        self.iv, self.f = np.array(prob.intvars1), np.array(prob.f_drucker)
        self.wall = np.array(prob.wall_position, np.float64)
        self.horiz = np.array(prob.horizontal_or_not) == 1.0
        self.disp = np.zeros((self.nn, 2))
        self.gu = np.zeros((self.nt, 4))
        self.kind = np.zeros(self.n2, np.int64)
        self.kind[self.nn:self.nt], self.kind[self.nt:] = 1, 2
        self.props = np.array(p.props)
        tanfi, coh = self.props[12], self.props[13]
        den = math.sqrt(9.0 + 12.0 * tanfi ** 2)
        self.alpha, self.kc = tanfi / den, 3.0 * coh / den
        self.plastic, self.ncrit = int(self.props[0]) > 1, int(self.props[1])
        info = np.array(prob.bc_info).reshape(-1, 8)
        fixed = (np.array(prob.bc_or_not) == 1) & (info[:, 1] != 0) & (p.no_bcs > 0)
        if p.bc_nodes_only:
            fixed[self.nn:] = False
        bc = np.ctypeslib.as_array(p.bc_list, shape=(p.no_bcs, 8)) if p.no_bcs else None
        self.bcs = []  # in the reference's order: the particles, the variable, its curve, factor
        for r in range(2, 7):
            for b in range(p.no_bcs):
                who = np.nonzero(fixed & (info[:, r] == b + 1))[0]
                if len(who):
                    self.bcs.append((who, int(bc[b, 1]), int(bc[b, 2]), float(bc[b, 3])))
        self.t = 0.0

    def curve(self, k):
        p, n = self.p, self.p.nptstcurves[k - 1]
        tt = [p.ttcurves[k - 1 + i * p.ntcurves] for i in range(n)]
        ff = [p.ftcurves[k - 1 + i * p.ntcurves] for i in range(n)]
        for i in range(n - 1):
            if tt[i] <= self.t <= tt[i + 1]:
                xi = (self.t - tt[i]) / (tt[i + 1] - tt[i])
                return (1.0 - xi) * ff[i] + xi * ff[i + 1]
        return 0.0

    def pairs(self):
        """Every pair within the support: i, j, W and its gradient with respect to i."""
        x, cell = self.x, 2.0 * self.h.max()
        ij = ((x - x.min(axis=0)) / cell).astype(np.int64)
        nx = ij[:, 0].max() + 3
        key = (ij[:, 1] + 1) * nx + ij[:, 0] + 1
        order = np.argsort(key, kind="stable")
        skey, found = key[order], []
        for off in (0, 1, nx - 1, nx, nx + 1):
            lo = np.searchsorted(skey, skey + off, "left")
            hi = np.searchsorted(skey, skey + off, "right")
            if off == 0:
                lo = np.arange(len(skey)) + 1
            n = np.maximum(hi - lo, 0)
            a = np.repeat(np.arange(len(skey)), n)
            b = np.arange(n.sum()) - np.repeat(np.cumsum(n) - n, n) + lo[a]
            a, b = order[a], order[b]
            d = x[a] - x[b]
            keep = (d ** 2).sum(axis=1) < (self.h[a] + self.h[b]) ** 2
            found.append((a[keep], b[keep]))
        i, j = (np.concatenate(q) for q in zip(*found))
        d = x[i] - x[j]
        r, h = np.sqrt((d ** 2).sum(axis=1)), 0.5 * (self.h[i] + self.h[j])
        q, fac = r / h, 15.0 / (7.0 * math.pi * h * h)
        t = np.maximum(2.0 - q, 0.0)
        w = np.where(q <= 1.0, fac * (2.0 / 3.0 - q ** 2 + 0.5 * q ** 3), fac / 6.0 * t ** 3)
        a = np.where(q <= 1.0, fac * (-2.0 + 1.5 * q) / h ** 2,
                     -0.5 * fac * t ** 2 / (h * np.maximum(r, 1e-300)))
        return i, j, w, a[:, None] * d

    def build(self):
        i, j, w, g = self.pairs()
        ki, kj = self.kind[i], self.kind[j]

        def pick(a, b):  # the pairs of kinds a and b, the particle of kind a first
            fwd, rev = (ki == a) & (kj == b), (ki == b) & (kj == a) & (a != b)
            return (np.concatenate([i[fwd], j[rev]]), np.concatenate([j[fwd], i[rev]]),
                    np.concatenate([w[fwd], w[rev]]), np.concatenate([g[fwd], -g[rev]]))

        self.sp_n, self.sp_d, self.n_d = pick(1, 0), pick(1, 2), pick(0, 2)
        self.nn_, self.ss_ = pick(0, 0), pick(1, 1)

    def sums(self, idx, *cols):
        return np.stack([np.bincount(idx, c, self.nt) for c in cols], axis=1)

    def adapt(self):
        if self.ncrit != 12:
            return
        s = self.s[:self.nt]
        n = (0, 1, 3)
        mean = (s[:, 0] + s[:, 1] + s[:, 3]) / 3.0
        cut = self.kc - 3.0 * self.alpha * mean < 0
        apex = self.kc / (3.0 * self.alpha) if self.alpha else 0.0
        for k in n:
            s[cut, k] += apex - mean[cut]
        mean = np.where(cut, apex, mean)
        d = s.copy()
        for k in n:
            d[:, k] -= mean
        sj = np.sqrt(d[:, 2] ** 2 + 0.5 * (d[:, 0] ** 2 + d[:, 1] ** 2 + d[:, 3] ** 2))
        y = np.maximum(self.kc - 3.0 * self.alpha * mean, 0.0)
        back = y < sj
        rn = np.where(sj <= 1e-5, 0.0, y / np.maximum(sj, 1e-300))
        d *= rn[:, None]
        for k in n:
            d[:, k] += mean
        s[back] = d[back]

    def fix(self):
        for who, var, curve, factor in self.bcs:
            val = self.curve(curve) * factor
            if var in (5, 6):
                self.v[who, var - 5] = val
            else:
                self.s[who, {1: 0, 2: 1, 3: 2}[var]] = val

    def interpolate(self):
        sp, n, w, _ = self.sp_n
        vol = self.m / self.rho
        hn, hs = vol[n] * w, vol[sp] * w
        a = self.sums(sp, self.v[n, 0] * hn, self.v[n, 1] * hn, hn)
        b = self.sums(n, *(self.s[sp, k] * hs for k in range(4)), self.iv[sp] * hs, hs)
        ok = a[:, 2] != 0
        self.v[:self.nt][ok] = a[ok, :2] / a[ok, 2:]
        ok = b[:, 5] != 0
        self.s[:self.nt][ok] = b[ok, :4] / b[ok, 5:]
        self.iv[:self.nt][ok] = b[ok, 4] / b[ok, 5]
        self.v[:self.nn][~ok[:self.nn]] = 0.0

    def cspm(self, g, idx, other, gx, gy):
        d = self.x[other] - self.x[idx]
        e = self.sums(idx, d[:, 0] * gx, d[:, 1] * gx, d[:, 0] * gy, d[:, 1] * gy)
        det = e[:, 0] * e[:, 3] - e[:, 1] * e[:, 2]
        off = np.abs(det) < self.p.cspm_det_min
        e[off] = (1.0, 0.0, 0.0, 1.0)
        q = 1.0 / np.where(off, 1.0, det)
        half = g.shape[1] // 2
        for k in range(2):
            g[:, k] = q * (e[:, 0] * g[:, k] + e[:, 1] * g[:, k + half])
            g[:, k + half] = q * (e[:, 2] * g[:, k] + e[:, 3] * g[:, k + half])

    def rates(self):
        """(stress-point rates, node accelerations, plastic strain rate)."""
        p, nn, nt = self.p, self.nn, self.nt
        vol = self.m / self.rho
        sp, n, w, dw = self.sp_n
        hx, hy = dw[:, 0] * vol[n], dw[:, 1] * vol[n]
        dv = self.v[n] - self.v[sp]
        g = self.sums(sp, dv[:, 0] * hx, dv[:, 1] * hx, dv[:, 0] * hy, dv[:, 1] * hy)
        ws, wd, _, wg = self.sp_d
        if len(ws):
            axis = np.where(self.horiz[wd], 1, 0)
            da = np.abs(self.x[ws, axis] - self.wall[wd])
            db = np.abs(self.x[wd, axis] - self.wall[wd])
            beta = np.minimum(1.5, 1.0 + db / da)
            vb, kx, ky = self.v[ws] * beta[:, None], -wg[:, 0] * vol[wd], -wg[:, 1] * vol[wd]
            g += self.sums(ws, vb[:, 0] * kx, vb[:, 1] * kx, vb[:, 0] * ky, vb[:, 1] * ky)
        a = self.s[:, :3] / (self.rho ** 2)[:, None]
        term = self.m[sp][:, None] * (a[sp] + a[n])
        g2 = -self.sums(n, *(dw[:, 0] * term[:, k] for k in range(3)),
                        *(dw[:, 1] * term[:, k] for k in range(3)))
        dn, dd, _, dg = self.n_d
        if len(dn):
            term = self.m[dd][:, None] * (a[dn] + self.s[dn, :3] / (self.rho[dd] ** 2)[:, None])
            g2 += self.sums(dn, *(dg[:, 0] * term[:, k] for k in range(3)),
                            *(dg[:, 1] * term[:, k] for k in range(3)))
        if p.cspm:
            self.cspm(g, sp, n, hx, hy)
            self.cspm(g2, n, sp, -dw[:, 0] * vol[sp], -dw[:, 1] * vol[sp])
        g[:nn] = 0.0
        self.gu = g
        g11, g21, g12, g22 = g.T
        r = np.stack([p.D11 * g11 + p.D12 * g22, p.D12 * g11 + p.D22 * g22, p.D33 * (g21 + g12),
                      p.D41 * g11 + p.D42 * g22], axis=1)
        s = self.s[:nt]
        if p.update_x:
            om = 0.5 * (g12 - g21)
            r[:, 0] += 2.0 * om * s[:, 2]
            r[:, 1] -= 2.0 * om * s[:, 2]
            r[:, 2] += om * (s[:, 1] - s[:, 0])
        flow = self.flow(s, g)
        r -= flow[0]
        acc = np.stack([g2[:nn, 0] + g2[:nn, 5], g2[:nn, 2] + g2[:nn, 4]], axis=1)
        if p.ic_grav == 1:
            acc += self.curve(p.tcurve_grav) * p.ft_grav * np.array(p.cgrav)
        acc -= p.damping * self.v[:nn]
        acc += self.wall_force()
        if p.alpha > 0 or p.beta > 0:
            i, j, _, q = self.nn_
            d, dv = self.x[i] - self.x[j], self.v[i] - self.v[j]
            h, rho = 0.5 * (self.h[i] + self.h[j]), 0.5 * (self.rho[i] + self.rho[j])
            div = (d * dv).sum(axis=1)
            th = h * div / ((d ** 2).sum(axis=1) + 0.01 * h * h)
            vis = np.where(div < 0, (-600.0 * p.alpha * th + p.beta * th * th) / rho, 0.0)
            av = self.sums(i, *(vis[:, None] * q * self.m[j][:, None]).T) - \
                self.sums(j, *(vis[:, None] * q * self.m[i][:, None]).T)
            acc -= av[:nn]
        return r, acc, flow[1]

    def flow(self, s, g):
        """The plastic source and the plastic strain rate of every stress-point."""
        props, gs, viv = self.props, np.zeros_like(s), np.zeros_like(s)
        young, nu = props[2], props[3]
        mean = (s[:, 0] + s[:, 1] + s[:, 3]) / 3.0
        d = s - mean[:, None] * np.array([1.0, 1.0, 0.0, 1.0])
        sj = np.sqrt(d[:, 2] ** 2 + 0.5 * (d[:, 0] ** 2 + d[:, 1] ** 2 + d[:, 3] ** 2))
        gm = young / (2.0 * (1.0 + nu))
        safe = np.maximum(sj, 1e-300)[:, None]
        if self.plastic and self.ncrit == 12:
            km = young / (3.0 * (1.0 - 2.0 * nu))
            f = sj - (self.kc - 3.0 * self.alpha * mean)
            e11, e22, e12 = g[:, 0], g[:, 3], 0.5 * (g[:, 1] + g[:, 2])
            rate = (3.0 * self.alpha * km * (e11 + e22) + gm / safe[:, 0] * (
                d[:, 0] * e11 + 2.0 * d[:, 2] * e12 + d[:, 1] * e22)) / gm
            on = (f >= 0) & (f >= self.f[:self.nt]) & (sj >= 1e-5) & (self.t > 0)
            rate = np.where(on, rate, 0.0)[:, None]
            gs, viv = gm / safe * d * rate, d / safe * rate
            viv = viv * np.array([0.5, 0.5, 1.0, 0.5])
            self.f[self.nn:self.nt] = f[self.nn:]
        elif self.plastic and self.ncrit == 2:
            f0 = props[6]
            size = f0 * np.maximum(np.abs(f0 + props[7] * self.iv) / abs(f0), 0.1)
            over = (math.sqrt(3.0) * sj - size) / size
            rate = np.where(over >= 0.01, props[9] * over ** props[10], 0.0)[:, None]
            viv = rate * math.sqrt(3.0) * d / safe * np.array([0.5, 0.5, 1.0, 0.5])
            gs = 2.0 * gm * viv * np.array([1.0, 1.0, 0.5, 1.0])
        der = np.sqrt((2.0 * (viv[:, 0] ** 2 + viv[:, 1] ** 2 + viv[:, 3] ** 2) +
                       viv[:, 2] ** 2) / 3.0)
        return gs, der

    def wall_force(self):
        p, out = self.p, np.zeros((self.nn, 2))
        i, j = self.n_d[:2]
        keep = j < self.nt + p.ndummy2
        i, j = i[keep], j[keep]
        if not (p.inside_approach and len(i)):
            return out
        d = self.x[i] - self.x[j]
        r, h = np.sqrt((d ** 2).sum(axis=1)), 0.5 * (self.h[i] + self.h[j])
        reach = 0.75 * p.dx
        near = np.where(r < reach, 1.0 - r / reach, 0.0)
        b = r / (0.75 * h)
        shape = np.where(b <= 2.0 / 3.0, 2.0 / 3.0,
                         np.where(b <= 1.0, 2.0 * b - 1.5 * b * b,
                                  np.where(b < 2.0, 0.5 * (2.0 - b) ** 2, 0.0)))
        k = (4.0 * near * shape / r ** 2)[:, None] * d
        return self.sums(i, k[:, 0], k[:, 1])[:self.nn]

    def steps(self, count):
        p, nn, nt, dt = self.p, self.nn, self.nt, self.p.dt_sph
        for _ in range(count):
            self.build()
            x0, v0, s0 = self.x.copy(), self.v.copy(), self.s.copy()
            self.v[:] = 0.0
            self.s[:] = 0.0
            r, a = np.zeros((nt, 4)), np.zeros((nn, 2))
            rs, ra, rd = np.zeros((nt, 4)), np.zeros((nn, 2)), np.zeros(nt)
            for f1, f2 in ((0.0, 1.0), (0.5, 2.0), (0.5, 2.0), (1.0, 1.0)):
                self.v[:nn] = v0[:nn] + f1 * dt * a
                self.s[nn:nt] = s0[nn:nt] + f1 * dt * r[nn:]
                self.adapt()
                self.fix()
                self.interpolate()
                self.adapt()
                self.fix()
                r, a, der = self.rates()
                rs += f2 * r
                ra += f2 * a
                rd += f2 * der
            self.v[:nn] = v0[:nn] + dt / 6.0 * ra
            self.s[nn:nt] = s0[nn:nt] + dt / 6.0 * rs[nn:]
            self.adapt()
            self.fix()
            self.iv[nn:nt] += dt * rd[nn:] / 6.0
            self.interpolate()
            self.adapt()
            self.fix()
            if p.xsph:
                vs, vol = np.zeros((nt, 2)), self.m / self.rho
                for i, j, w, _ in (self.nn_, self.ss_):
                    dv = (self.v[j] - self.v[i]) * w[:, None]
                    vs += self.sums(i, *(dv * vol[j][:, None]).T)
                    vs -= self.sums(j, *(dv * vol[i][:, None]).T)
                self.x[:nt] = x0[:nt] + dt * (self.v[:nt] + 0.5 * vs)
            else:
                self.x[:nt] = x0[:nt] + dt * 0.5 * (v0[:nt] + self.v[:nt])
            self.disp = self.x[:nn] - self.x00[:nn]
            self.t += dt
        self.s[nt:] = 0.0
        # the loading flag and the strain that it gates switch on the last bit of f, the
        # surface flags on a region's edge: no 64-bit value stands for these
        return dict(x=self.x.ravel(), vel=self.v.ravel(), stress=self.s.ravel(), rho=self.rho,
                    intvars1=None, displ=self.disp.ravel(), bc_or_not=None, f_drucker=None)


def _init_params(rng):
    """Glorot-uniform weights (row-major W[k][n], then the bias, layer by layer)."""
    parts = []
    for kin, nout, rows, cols in ((14, 128, 16, 128), (128, 128, 128, 128), (128, 128, 128, 128),
                                  (128, 4, 128, 8)):
        w = np.zeros((rows, cols), np.float32)
        lim = math.sqrt(6.0 / (kin + nout))
        w[:kin, :nout] = rng.uniform(-lim, lim, (kin, nout))
        parts += [w.ravel(), np.zeros(cols, np.float32)]
    return np.concatenate(parts)


def _bf16(a):
    """To the nearest bfloat16 (ties to even) of each value."""
    b = np.asarray(a, np.float32).view(np.uint32).astype(np.uint64)
    b = (b + 0x7FFF + ((b >> 16) & 1)) & 0xFFFF0000
    return b.astype(np.uint32).view(np.float32).astype(np.float64)


def _shuffled(n, seed):
    """The epoch's order: Fisher-Yates on a splitmix64 stream."""
    order, s, mask = list(range(n)), seed & (2 ** 64 - 1), 2 ** 64 - 1
    for i in range(n - 1, 0, -1):
        s = (s + 0x9E3779B97F4A7C15) & mask
        z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (i + 1)
        order[i], order[j] = order[j], order[i]
    return np.array(order)


def _exact_training(case, seed):
    """One epoch in 64 bits: BF16-rounded weights and activations, straight-through gradients,
    mean squared error, Adam."""
    tuples, params = _training_inputs(case, seed)
    n, batch = case["rows"], case["batch"]
    p = params.astype(np.float64)
    m, v, loss, count = np.zeros_like(p), np.zeros_like(p), 0.0, n // batch
    shape = ((16, 128), (128, 128), (128, 128), (128, 8))
    order = _shuffled(n, seed)
    for it in range(count):
        rows = tuples[order[it * batch:(it + 1) * batch]]
        ws, at = [], 0
        for k, c in shape:
            ws.append((_bf16(p[at:at + k * c]).reshape(k, c), p[at + k * c:at + k * c + c]))
            at += k * c + c
        act, zs = [np.zeros((batch, 16))], []
        act[0][:, :14] = _bf16(rows[:, :14])
        for w, b in ws[:3]:
            z = act[-1] @ w + b
            zs.append(z)
            act.append(_bf16(z / (1.0 + np.exp(-z))))
        y = act[-1] @ ws[3][0] + ws[3][1]
        d = np.zeros_like(y)
        d[:, :4] = y[:, :4] - rows[:, 14:]
        loss += (d ** 2).sum()
        d *= 2.0 / (4.0 * batch)
        grads = []
        for layer in range(3, -1, -1):
            grads.append(np.concatenate([(act[layer].T @ d).ravel(), d.sum(axis=0)]))
            if layer:
                sg = 1.0 / (1.0 + np.exp(-zs[layer - 1]))
                d = (d @ ws[layer][0].T) * sg * (1.0 + zs[layer - 1] * (1.0 - sg))
        g = np.concatenate(grads[::-1])
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - 2e-3 * (m / (1.0 - 0.9 ** (it + 1))) / (
            np.sqrt(v / (1.0 - 0.999 ** (it + 1))) + 1e-8)
    return dict(loss=np.array([loss / (count * batch * 4.0)]), params=p)
