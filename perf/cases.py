"""Performance cases of the batched reactor path, through its public entry points.

Mechanisms: the seeded synthetic ones of zerork_b200/mechgen.py (the sizes of
the benchmark configurations), and for integrations also the dimethyl ether
mechanism of the tests (tests/golden/mech).  Kinds of case:

  jac       Mechanism.rates_jac with the Jacobian: net rates and the sparse
            reactor Jacobian of n independent device states
  rates     Mechanism.rates_jac without the Jacobian: net rates and the
            reactor right-hand side (explicit or operator-split solvers)
  tc        Mechanism.rates_tc: net, creation and destruction rates and rates
            of progress from temperature and concentrations, device arrays
  tc_host   Mechanism.rates_tc_host: the same from and to host arrays (a code
            that asks for single states or small blocks)
  solve     Plugin.solve: n reactors through one time step on host arrays, as
            a CFD code calls it between its transport steps
  mlp       the learned predictor: a few training minibatches (gradients and
            Adam) and a validation forward pass

States: "mixed" draws every mass fraction (Dirichlet(0.5)); "fresh" is fuel in
air, most mass fractions exactly zero, where the Jacobian's clamp is active.
"""
import functools
import gzip
import os
import tempfile

import numpy as np
import torch

from zerork_b200 import Mechanism, mechgen

P_ATM = 101325.0
RU = 8.314462618e3
TROE3, TROE4 = 1, 2  # falloff types in the mechanism tables (0: Lindemann)
# largest n of each kind and mechanism: (smallest, largest)
RANGES = {
    ("jac", "c1_h2"): (16, 262144), ("jac", "c2_53"): (64, 131072),
    ("jac", "c3_160"): (32, 16384), ("jac", "c4_650"): (16, 1024),
    ("rates", "c1_h2"): (16, 262144), ("rates", "c2_53"): (64, 200000),
    ("rates", "c3_160"): (32, 32768), ("rates", "c4_650"): (16, 2048),
    ("tc", "c1_h2"): (16, 262144), ("tc", "c2_53"): (64, 262144),
    ("tc", "c3_160"): (32, 32768), ("tc", "c4_650"): (16, 2048),
    ("tc_host", "c1_h2"): (1, 256), ("tc_host", "c2_53"): (1, 256),
    ("solve", "c1_h2"): (8, 2048), ("solve", "dme_24"): (8, 2048), ("solve", "c3_160"): (8, 296),
}
SPAN = {"c1_h2": 1e-3, "dme_24": 1e-5, "c3_160": 1e-6}  # longest time step of a solve


def listed():
    return [
        # one block of cells of a small hydrogen mechanism: launches and latency
        dict(name="jac_h2_64", kind="jac", mech="c1_h2", n=64, pad=0, states="mixed", ydot=False),
        # the headline workload: a large batch of 53-species states
        dict(name="jac_53sp_131072", kind="jac", mech="c2_53", n=131072, pad=0, states="mixed", ydot=False),
        # a detailed fuel before ignition, ragged and padded, with the right-hand side
        dict(name="jac_160sp_fresh_9001", kind="jac", mech="c3_160", n=9001, pad=7, states="fresh", ydot=True),
        # the largest mechanism, whose workspace does not fit in shared memory
        dict(name="jac_650sp_500", kind="jac", mech="c4_650", n=500, pad=0, states="mixed", ydot=False),
        # right-hand sides alone, for explicit integrators
        dict(name="rates_53sp_100003", kind="rates", mech="c2_53", n=100003, pad=0, states="mixed", ydot=True),
        # the reference GPU class's entry point at its largest batch
        dict(name="tc_53sp_262144", kind="tc", mech="c2_53", n=262144, limiter=False),
        # one state at a time from a host program
        dict(name="tc_host_53sp_1", kind="tc_host", mech="c2_53", n=1, limiter=True),
        # hydrogen ignition, a small batch over a millisecond
        dict(name="solve_h2_64", kind="solve", mech="c1_h2", n=64, dt=1e-3, fp32=False, cp=False),
        # a CFD time step of a thousand cells with the dimethyl ether mechanism
        dict(name="solve_dme_1000", kind="solve", mech="dme_24", n=1000, dt=1e-5, fp32=False, cp=False),
        # a detailed mechanism, two reactors per SM
        dict(name="solve_160sp_296", kind="solve", mech="c3_160", n=296, dt=1e-6, fp32=False, cp=True),
        # the same with the single-precision preconditioner
        dict(name="solve_160sp_fp32_148", kind="solve", mech="c3_160", n=148, dt=1e-7, fp32=True, cp=False),
        # training the predictor of a 160-species mechanism
        dict(name="mlp_163x256x3_4096", kind="mlp", n_in=163, n_out=161, hidden=256, layers=3, batch=4096,
             steps=8, rows=5001),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["jac", "jac", "rates", "tc", "tc_host", "solve", "solve", "solve", "mlp"])
    if kind == "mlp":
        nsp = rng.choice([10, 53, 160])
        return dict(kind=kind, n_in=nsp + 3, n_out=nsp + 1, hidden=rng.choice([64, 100, 128, 256]),
                    layers=rng.randint(1, 4), batch=16 * _log_int(rng, 1, 256), steps=rng.randint(1, 8),
                    rows=_log_int(rng, 1, 5001))
    mech = rng.choice([m for k, m in RANGES if k == kind])
    n = _log_int(rng, *RANGES[kind, mech])
    if kind in ("jac", "rates"):
        return dict(kind=kind, mech=mech, n=n, pad=rng.choice([0, 0, 1, 7, 32]),
                    states=rng.choice(["mixed", "fresh"]) if mech != "c1_h2" else "mixed",
                    ydot=rng.random() < 0.5)
    if kind in ("tc", "tc_host"):
        return dict(kind=kind, mech=mech, n=n, limiter=rng.random() < 0.3)
    dt = SPAN[mech] * 0.1 ** (2.0 * rng.random())
    fp32 = rng.random() < 0.25
    if fp32:  # no dearer than the listed ones
        n, dt = min(n, RANGES[kind, mech][1] // 2), 0.1 * dt
    if mech == "dme_24":
        dt = min(dt, 1e-5 * min(1.0, 1000.0 / n))
    elif mech == "c1_h2":
        dt = min(dt, 1e-3 * min(1.0, 64.0 / n))
    return dict(kind=kind, mech=mech, n=n, dt=float(f"{dt:.3g}"), fp32=fp32, cp=rng.random() < 0.3)


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _mech(name):
    """(generated mechanism, its files, parse-only handle for sizes and tables)."""
    to, g = tempfile.mkdtemp(prefix="zrk_cases_"), None
    if name == "dme_24":
        files = []
        for f in ("dme_24_mech.txt", "dme_24_therm.txt"):
            files.append(os.path.join(to, f))
            with gzip.open(os.path.join("tests", "golden", "mech", f + ".gz")) as a, open(files[-1], "wb") as b:
                b.write(a.read())
    else:
        g = mechgen.generate(mechgen.SPECS[name])
        files = g.write(to)
    return g, files, Mechanism(*files, device=False)


def _fuels(g):
    return [i for i, (_, c) in enumerate(g.species)
            if c.get("C", 0) >= 1 and c.get("H", 0) >= 2 and c.get("O", 0) == 0 and c.get("N", 0) == 0]


def _weights(g):
    w = {"C": 12.0107, "H": 1.00794, "O": 15.9994, "N": 14.0067, "AR": 39.948}
    return np.array([sum(w[e] * k for e, k in c.items()) for _, c in g.species])


def _host_states(g, n, seed, states):
    """T U[300, 3000] K, log10 P U[0, 2] atm, Y [n, nsp] (made on the device
    when there is one: the values are the same for a seed on one kind of
    device, and these arrays can be large)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    r = torch.Generator(device=dev).manual_seed(1000003 * seed + 17)
    kw = dict(generator=r, dtype=torch.float64, device=dev)
    T = 300.0 + 2700.0 * torch.rand(n, **kw)
    P = P_ATM * 10.0 ** (2.0 * torch.rand(n, **kw))
    S = len(g.species)
    if states == "mixed":  # squares of normals, normalised: Dirichlet(0.5)
        Y = torch.randn((S, n), **kw).square_()
    else:
        X = torch.zeros((S, n), dtype=torch.float64, device=dev)
        fuels = torch.tensor(_fuels(g), device=dev)
        for _ in range(3):
            at = fuels[torch.randint(0, len(fuels), (n,), generator=r, device=dev)]
            X[at, torch.arange(n, device=dev)] += 0.02 * torch.rand(n, **kw)
        rest = 1.0 - X.sum(0)
        X[g.index("O2")] += 0.21 * rest
        X[g.index("N2")] += 0.79 * rest
        Y = X * torch.from_numpy(_weights(g)).to(dev)[:, None]
    Y /= Y.sum(0)
    return T, P, Y  # Y species-major [nsp, n]


def _reactors(g, mech, n, seed):
    """Reactor-major host arrays of a solve: the workloads of the benchmark,
    and dimethyl ether in air at equivalence ratios U[0.3, 2], T U[700, 1500]
    K, P U[1, 50] atm."""
    if mech == "dme_24":
        pm, r = _mech(mech)[2], np.random.default_rng(seed)
        T, P, phi = r.uniform(700.0, 1500.0, n), P_ATM * r.uniform(1.0, 50.0, n), r.uniform(0.3, 2.0, n)
        sp = [s.lower() for s in pm.species]
        Y = np.zeros((n, pm.nsp))
        Y[:, sp.index("ch3och3")] = phi
        Y[:, sp.index("o2")], Y[:, sp.index("n2")] = 3.0, 3.0 * 3.76
        Y *= pm.table("mw")
        return T, P, Y / Y.sum(1, keepdims=True)
    return mechgen.reactor_states(g, n, "c1" if mech == "c1_h2" else "c3", seed=seed)


def _mlp_inputs(c, seed):
    r = np.random.default_rng(seed + 5)
    dims = [c["n_in"]] + [c["hidden"]] * c["layers"] + [c["n_out"]]
    pad = [(d + 15) // 16 * 16 for d in dims]
    w, b = [], []
    for l in range(len(dims) - 1):
        m = np.zeros((pad[l], pad[l + 1]), np.float32)
        bound = np.sqrt(6.0 / dims[l])
        m[:dims[l], :dims[l + 1]] = r.uniform(-bound, bound, (dims[l], dims[l + 1]))
        w.append(m)
        v = np.zeros(pad[l + 1], np.float32)
        v[:dims[l + 1]] = r.uniform(-0.1, 0.1, dims[l + 1])
        b.append(v)
    n = c["batch"] * c["steps"]
    mix = r.standard_normal((c["n_in"], c["n_out"])) / np.sqrt(c["n_in"])

    def pairs(k):  # standardised features and smooth targets
        x = r.standard_normal((k, c["n_in"]))
        return x.astype(np.float32), np.tanh(x @ mix).astype(np.float32)

    x, t = pairs(n)
    xv, _ = pairs(c["rows"])
    return dims, w, b, x, t, xv


def prepare(case, seed):
    c = dict(case)
    s = {"c": c}
    if c["kind"] == "mlp":
        from zerork_b200.predictor import Mlp
        dims, w, b, x, t, xv = _mlp_inputs(c, seed)
        net = Mlp(c["n_in"], c["n_out"], c["hidden"], c["layers"], seed)
        net.set_params(np.concatenate([m.ravel() for m in w]), np.concatenate(b))
        k = c["batch"]
        s.update(net=net, x=torch.from_numpy(x).cuda().split(k), t=torch.from_numpy(t).cuda().split(k),
                 xv=torch.from_numpy(xv).cuda(), loss=torch.zeros(c["steps"], device="cuda"))
        return s
    g, files, sizes = _mech(c["mech"])
    n = c["n"]
    if c["kind"] == "solve":
        from zerork_b200.plugin import Plugin
        # a CFD code gives its cells enough steps for a whole ignition
        p = Plugin(*files, max_steps=20000, lu_fp32=int(c["fp32"]), constant_volume=int(not c["cp"]))
        T, P, Y = _reactors(g, c["mech"], n, seed)
        s.update(p=p, T=T, P=P, Y=np.ascontiguousarray(Y))
        p.load_mechanism()
        return s
    pm = Mechanism(*files)
    T, P, Y = _host_states(g, n, seed, c.get("states", "mixed"))
    if c["kind"] in ("tc", "tc_host"):
        iw = 1.0 / torch.from_numpy(sizes.table("mw")).to(Y.device)[:, None]
        C = (P / (RU * T) / (Y * iw).sum(0)) * (Y * iw)
        lim = torch.full((pm.nstep,), 1e22, dtype=torch.float64, device=Y.device) if c["limiter"] else None
        if c["kind"] == "tc":
            s.update(pm=pm, T=T, C=C.contiguous(), lim=lim)
        else:
            s.update(pm=pm, T=T.cpu().numpy(), C=C.cpu().numpy(), lim=None if lim is None else lim.cpu().numpy())
        return s
    ld = n + c["pad"]
    new = lambda k: torch.zeros((k, ld), dtype=torch.float64, device="cuda")  # noqa: E731
    Yp = new(pm.nsp)
    Yp[:, :n] = Y
    s.update(pm=pm, T=T, P=P, Y=Yp, W=new(pm.nsp), J=new(pm.nnz) if c["kind"] == "jac" else None,
             D=new(pm.nsp + 1) if c["ydot"] else None)
    return s


def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind in ("jac", "rates"):
        s["pm"].rates_jac(s["T"], s["P"], s["Y"], s["W"], s["J"], s["D"], n=c["n"],
                          stream=torch.cuda.current_stream().cuda_stream)
        return [a for a in (s["W"], s["J"], s["D"]) if a is not None]
    if kind == "tc":
        return s["pm"].rates_tc(s["T"], s["C"], s["lim"], stream=torch.cuda.current_stream().cuda_stream)
    if kind == "tc_host":
        return s["pm"].rates_tc_host(s["T"], s["C"], s["lim"])
    if kind == "solve":
        T, P, Y = s["T"].copy(), s["P"].copy(), s["Y"].copy()
        s["p"].solve(c["dt"], T, P, Y, raise_on_fail=False)
        return T, P, Y
    net, loss = s["net"], s["loss"]
    for i in range(c["steps"]):
        net.gradients(s["x"][i], s["t"][i], loss[i:i + 1])
        net.adam(1e-3)
    y = net.forward(s["xv"])
    w, b = net.params()
    return loss, y, w, b


# ------------------------------------------------------- work and tolerance

def _rhs_flops(pm):
    """Floating-point operations of one right-hand side: two transcendentals
    (about 25 operations each) and the products of every step, its creation
    and destruction sums, and the thermodynamic fits."""
    return 60.0 * pm.nstep + 60.0 * pm.nsp


# mean accepted steps of a reactor over one call, counted once per mechanism
# for the listed time steps
STEPS = {"c1_h2": 2000.0, "dme_24": 450.0, "c3_160": 1000.0}


def work(case):
    c = case
    if c["kind"] == "mlp":
        d = [c["n_in"]] + [c["hidden"]] * c["layers"] + [c["n_out"]]
        mac = sum(a * b for a, b in zip(d, d[1:]))
        par = mac + sum(d[1:])
        rows = c["batch"] * c["steps"]
        # forward, weight gradient and input gradient (not for the first layer)
        fl = 2.0 * (rows * (3 * mac - d[0] * d[1]) + c["rows"] * mac)
        by = 4.0 * (rows * (d[0] + d[-1]) + c["rows"] * (d[0] + d[-1]) + 6 * par * c["steps"])
        return {"bytes": by, "flops": fl}
    _, _, pm = _mech(c["mech"])
    n, S, N = c["n"], pm.nsp, pm.nstep
    if c["kind"] == "solve":
        m = S + 1.0
        steps = STEPS[c["mech"]]
        # per step one and a half right-hand sides and solves with a kept
        # factor, and a tenth of a Jacobian and a factorization
        fl = steps * (1.5 * (_rhs_flops(pm) + 2 * m * m) + 0.1 * (2 * m ** 3 / 3 + 4.0 * pm.nnz))
        return {"bytes": 16.0 * n * (S + 2), "flops": n * fl}
    if c["kind"] in ("tc", "tc_host"):
        return {"bytes": 8.0 * n * (1 + 4 * S + N), "flops": n * _rhs_flops(pm)}
    by = 8.0 * n * (2 + 2 * S + (pm.nnz if c["kind"] == "jac" else 0) + (S + 1 if c["ydot"] else 0))
    fl = n * _rhs_flops(pm)
    if c["kind"] == "jac":  # the perturbed right-hand side, and about six operations a nonzero
        fl = 2 * fl + 6.0 * n * pm.nnz
    return {"bytes": by, "flops": fl}


def tolerance(case):
    if case["kind"] == "mlp":  # BF16 products, and Adam's sign-like first steps
        return {"rel": 2e-2}
    if case["kind"] == "solve":
        # rtol 1e-8 per step, carried through an ignition: sums in another
        # order (other thread counts) move end temperatures by up to 6e-7
        return {"rel": 5e-6}
    # Jacobians: up to 2e-10 (a few dozen hydrogen states) from the noise of
    # the difference quotient of the temperature column; rates are at 1e-14
    return {"rel": 1e-9 if case["kind"] == "jac" else 1e-13 if case.get("states") != "fresh" else 1e-12}


# -------------------------------------------------------------------- exact

def _steps_of(t, N):
    """Reactant and product species of every step."""
    rp, rs, pp, ps = (t[k].tolist() for k in ("reac_ptr", "reac_spc", "prod_ptr", "prod_spc"))
    return [rs[rp[i]:rp[i + 1]] for i in range(N)], [ps[pp[i]:pp[i + 1]] for i in range(N)]


class _Kinetics:
    """Rates of a mechanism in extended precision, states along the last
    axis: NASA-7 fits, Arrhenius, equilibrium reverse rates, third bodies,
    Lindemann and Troe falloff and the step limiter."""

    def __init__(self, pm):
        self.t, self.S, self.N = pm.tables(), pm.nsp, pm.nstep
        self.reac, self.prod = _steps_of(self.t, self.N)
        self.X = np.longdouble

    def thermo(self, T):
        """cp/R, h/RT, g/RT [S, n]."""
        th = self.t["thermo"].reshape(self.S, 16)
        lo, hi = th[:, 1:8, None].astype(self.X), th[:, 8:15, None].astype(self.X)
        a = np.where(T[None, None, :] < th[:, 0, None, None], lo, hi)
        cp = a[:, 0] + T * (a[:, 1] + T * (a[:, 2] + T * (a[:, 3] + T * a[:, 4])))
        h = a[:, 0] + T * (a[:, 1] / 2 + T * (a[:, 2] / 3 + T * (a[:, 3] / 4 + T * a[:, 4] / 5))) + a[:, 5] / T
        s = a[:, 0] * np.log(T) + T * (a[:, 1] + T * (a[:, 2] / 2 + T * (a[:, 3] / 3 + T * a[:, 4] / 4))) + a[:, 6]
        return cp, h, h - s

    def rop(self, T, C, gRT, lim):
        """Rates of progress [N, n]; lim: one limit per step, or None."""
        t, X, n = self.t, self.X, T.shape[0]
        lnT, inv = np.log(T), 1 / T
        k = np.zeros((self.N, n), X)
        for i, st in enumerate(t["arr_step"]):
            k[st] = np.exp(X(t["arr_lnA"][i]) + X(t["arr_n"][i]) * lnT - X(t["arr_Ta"][i]) * inv)
        lnp = np.log(X(P_ATM) / (X(RU) * T))
        for i, st in enumerate(t["keq_step"]):
            f = t["keq_fwd"][i]
            dg = sum(gRT[p] for p in self.prod[f]) - sum(gRT[r] for r in self.reac[f])
            k[st] = np.exp(dg - X(t["keq_dn"][i]) * lnp) * k[f]
        Cs = C.sum(0)
        for i, f in enumerate(t["tb_fwd"]):
            M = Cs.copy()
            for e in range(t["tb_ptr"][i], t["tb_ptr"][i + 1]):
                M = M + C[t["tb_spc"][e]] * X(t["tb_alpha"][e])
            k[f] = k[f] * M
            if t["tb_rev"][i] >= 0:
                k[t["tb_rev"][i]] = k[t["tb_rev"][i]] * M
        for i, f in enumerate(t["fo_fwd"]):
            p = t["fo_par"].reshape(-1, 8)[i].astype(X)
            if t["fo_spc"][i] >= 0:
                M = C[t["fo_spc"][i]]
            else:
                M = Cs.copy()
                for e in range(t["fo_ptr"][i], t["fo_ptr"][i + 1]):
                    M = M + C[t["fo_eff_spc"][e]] * X(t["fo_alpha"][e])
            Pr = np.maximum(np.exp(p[0] + p[1] * lnT - p[2] * inv) * M / k[f], X(1e-300))
            F = X(1)
            if t["fo_type"][i] in (TROE3, TROE4):
                Fc = np.zeros_like(T)
                if p[4] != 0:
                    Fc = Fc + (1 - p[3]) * np.exp(-T / p[4])
                if p[5] != 0:
                    Fc = Fc + p[3] * np.exp(-T / p[5])
                if t["fo_type"][i] == TROE4:
                    Fc = Fc + np.exp(-p[6] * inv)
                lF = np.log10(np.maximum(Fc, X(1e-300)))
                x = np.log10(Pr) - (X("0.4") + X("0.67") * lF)
                x = x / ((X("0.75") - X("1.27") * lF) - X("0.14") * x)
                F = 10 ** (lF / (1 + x * x))
            m = F * Pr / (1 + Pr)
            k[f] = k[f] * m
            if t["fo_rev"][i] >= 0:
                k[t["fo_rev"][i]] = k[t["fo_rev"][i]] * m
        for st in range(self.N):
            if lim is not None and 0 < lim[st] < 1e300:
                k[st] = k[st] * (X(lim[st]) / (X(lim[st]) + k[st]))
            for r in self.reac[st]:
                k[st] = k[st] * C[r]
        return k

    def sums(self, k):
        """Creation and destruction rates [S, n]."""
        cre, des = np.zeros((self.S, k.shape[1]), self.X), np.zeros((self.S, k.shape[1]), self.X)
        for st in range(self.N):
            for s in self.prod[st]:
                cre[s] += k[st]
            for s in self.reac[st]:
                des[s] += k[st]
        return cre, des


def _exact_states(c, K, T, P, Y, mw, cp_, ri):
    """(wdot, jac, ydot) of rates_jac in extended precision, species-major."""
    X, S = K.X, K.S
    T, P, Y, mw = (a.astype(X) for a in (T, P, Y, mw))
    ru, lim, mmf = X(RU), np.full(K.N, 1e22), X("1e-30")
    v = ru * T * (Y / mw[:, None]).sum(0) / P

    def rhs(T, Y, yS):
        C = Y / mw[:, None] / v
        cp, h, g = K.thermo(T)
        k = K.rop(T, C, g, lim)
        cre, des = K.sums(k)
        net = cre - des
        cv = ((cp - 1) * (ru / mw)[:, None] * Y).sum(0)
        Td = -((h - 1) * net).sum(0) * v * ru * yS / cv
        return net, net * mw[:, None] * v, Td, k, cv, h - 1, cp

    net, yd, Td, k, cv, u, cp = rhs(T, Y, T)
    ydot = np.concatenate([yd, Td[None]])
    if c["kind"] == "rates":
        return net, None, ydot
    Yc = np.where(np.abs(Y) < mmf, np.where(Y < 0, -mmf, mmf), Y)
    _, _, Tdc, kc, cvc, _, _ = rhs(T, Yc, T)
    # the temperature of the difference quotient is the double nearest T + T sqrt(eps)
    T64 = T.astype(np.float64)
    Tp = (T64 + T64 * np.sqrt(np.finfo(np.float64).eps)).astype(X)
    _, ydp, Tdp, _, _, _, _ = rhs(Tp, Y, Tp)
    at = {}
    for j in range(S):
        for p in range(cp_[j], cp_[j + 1]):
            at[int(ri[p]), j] = p
    jac = np.zeros((ri.shape[0], T.shape[0]), X)
    for st in range(K.N):
        for r in K.reac[st]:
            d = kc[st] * (mw[r] * v / Yc[r])
            for s in K.reac[st]:
                jac[at[s, r]] -= d
            for s in K.prod[st]:
                jac[at[s, r]] += d
    for j in range(S):
        a, b = cp_[j], cp_[j + 1] - 1
        tr = (jac[a:b] * u[ri[a:b]]).sum(0) * ru * T + Tdc * ((cp[j] - 1) * ru / mw[j]) * mw[j]
        jac[b] = -tr / mw[j] / cvc
        jac[a:b] *= (mw[ri[a:b]] / mw[j])[:, None]
    for p in range(cp_[S], cp_[S + 1]):
        f1, f0 = (ydp[ri[p]], yd[ri[p]]) if ri[p] < S else (Tdp, Td)
        jac[p] = (f1 - f0) / (Tp - T)
    return net, jac, ydot


def _exact_mlp(c, seed):
    """The training loop and the forward pass in 64 bits, nothing rounded."""
    dims, w, b, x, t, xv = _mlp_inputs(c, seed)
    L = len(w)
    w = [torch.from_numpy(a).double() for a in w]
    b = [torch.from_numpy(a).double() for a in b]
    pad = lambda a, k: torch.nn.functional.pad(torch.from_numpy(a).double(), (0, k - a.shape[1]))  # noqa: E731
    x, xv, t = pad(x, w[0].shape[0]), pad(xv, w[0].shape[0]), torch.from_numpy(t).double()

    def forward(a):
        for l in range(L):
            a = a @ w[l] + b[l]
            if l + 1 < L:
                a = a * torch.sigmoid(a)
        return a[:, :dims[-1]]

    par = w + b
    m, v = [torch.zeros_like(a) for a in par], [torch.zeros_like(a) for a in par]
    loss = []
    for i in range(c["steps"]):
        for a in par:
            a.requires_grad_(True)
        k = c["batch"]
        sq = (forward(x[i * k:(i + 1) * k]) - t[i * k:(i + 1) * k]).square().sum()
        loss.append(sq.item())
        gr = torch.autograd.grad(sq / (k * dims[-1]), par)
        with torch.no_grad():
            for a, d, p, q in zip(par, gr, m, v):
                a.requires_grad_(False)
                p.mul_(0.9).add_(d, alpha=0.1)
                q.mul_(0.999).addcmul_(d, d, value=0.001)
                a -= 1e-3 * (p / (1 - 0.9 ** (i + 1))) / ((q / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8)
    y = forward(xv)
    return (torch.tensor(loss), y, torch.cat([a.reshape(-1) for a in w]), torch.cat(b))


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "solve":  # a stiff integration at tight tolerances takes minutes
        return None
    if c["kind"] == "mlp":
        return _exact_mlp(c, seed)
    g, _, pm = _mech(c["mech"])
    if c["n"] * pm.nstep > 1.2e7:  # over about 20 s on one core
        return None
    K = _Kinetics(pm)
    T, P, Y = (a.cpu().numpy() for a in _host_states(g, c["n"], seed, c.get("states", "mixed")))
    mw = pm.table("mw")
    f8 = lambda a: np.asarray(a, np.float64)  # noqa: E731
    if c["kind"] in ("tc", "tc_host"):
        Tt, Pt, Yt = _host_states(g, c["n"], seed, "mixed")
        iw = 1.0 / torch.from_numpy(mw).to(Yt.device)[:, None]
        C = ((Pt / (RU * Tt) / (Yt * iw).sum(0)) * (Yt * iw)).cpu().numpy().astype(K.X)
        Tx = T.astype(K.X)
        k = K.rop(Tx, C, K.thermo(Tx)[2], np.full(K.N, 1e22) if c["limiter"] else None)
        cre, des = K.sums(k)
        return f8(cre - des), f8(cre), f8(des), f8(k)
    net, jac, ydot = _exact_states(c, K, T, P, Y, mw, *pm.jac_pattern())
    out = [a for a in (net, jac, ydot if c["ydot"] else None) if a is not None]
    return [f8(np.pad(np.asarray(a, np.float64), ((0, 0), (0, c["pad"])))) for a in out]
