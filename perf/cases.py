"""The work a user of this framework has it do, as cases that can be timed.

Eight kinds of call, each through a public entry point of the package:

  dslash     one operator application on device fields (apply_dev): D, D^dag or
             a normal operator, domain wall (Ls > 1) or Wilson (Ls = 1), FP64 or FP32
  prop       the analyzers' propagator solves of a set of boundary sources on
             one configuration (propagators_dev, even-odd mixed solver)
  measure    a whole analyzer call on host data: all sources of several
             configurations and their contractions (measure)
  corr       the Wilson analyzer's pseudoscalar correlator over several
             configurations (pseudoscalar_correlator, FP64 CG)
  hmc        one domain-wall HMC trajectory (hmc_trajectory, mixed CG)
  whmc       one Wilson HMC step with its Metropolis decision (hmc_step, FP64 CG)
  net        the learned preconditioner applied to a batch of fields (lp_apply_dev)
  netgrad    its training direction: loss and weight gradients (lp_loss_grad_dev)

Solves run to 1e-12, the tolerance of the repository's golden runs: there the
solution no longer depends on the path taken to it, so outputs can be compared.
Gauge fields are pure-gauge configurations at the study's couplings
(independent von Mises plaquettes, then a random gauge rotation), built here.
"""
import math

import numpy as np
import torch

import three_part_dwf_study_b200 as T

RTOL = 1e-12
MAXITER = 20000
M5 = 1.0

# ---------------------------------------------------------------- cases


def listed():
    return [
        # the smallest call: D on one field of a test-sized lattice, launch bound
        dict(name="dslash_16x16x8_f64", kind="dslash", Nt=16, Nx=16, Ls=8, n=1, prec=64, op="D"),
        # the standalone domain-wall operator on the bench's large lattice
        dict(name="dslash_512x512x16_f64", kind="dslash", Nt=512, Nx=512, Ls=16, n=1, prec=64,
             op="D"),
        # a ragged lattice (no whole warps in x, odd Ls), single precision, the normal operator
        dict(name="normal_100x90x13_f32", kind="dslash", Nt=100, Nx=90, Ls=13, n=16, prec=32,
             op="DdagD"),
        # the Wilson operator, large, single precision
        dict(name="wilson_2048x2048_f32", kind="dslash", Nt=2048, Nx=2048, Ls=1, n=1, prec=32,
             op="Ddag"),
        # the headline: one configuration's 28 sources (8 point, 16 noise, 4 wall)
        dict(name="prop_64x64x16_28", kind="prop", Nt=64, Nx=64, Ls=16, mf=0.05, nsrc=28),
        # the finite-volume study's largest extent, two configurations' worth of sources
        dict(name="prop_64x96x16_56", kind="prop", Nt=64, Nx=96, Ls=16, mf=0.05, nsrc=56),
        # the finite-volume study's smallest extent, host data in, correlators out
        dict(name="measure_64x32x16_4conf", kind="measure", Nt=64, Nx=32, Ls=16, mf=0.05, nconf=4),
        # the Wilson analyzer on a few configurations, extents not multiples of 32
        dict(name="corr_48x40_8conf", kind="corr", Nt=48, Nx=40, m0=0.05, beta=3.0, nconf=8),
        # a generator's trajectory at the study's domain-wall lattice (a quarter of its steps)
        dict(name="hmc_64x64x16", kind="hmc", Nt=64, Nx=64, Ls=16, mf=0.05, steps=10),
        # the Wilson generator's trajectory: tau = 1 in 20 steps at 32x32
        dict(name="whmc_32x32", kind="whmc", Nt=32, Nx=32, m0=0.1, beta=2.0, steps=20),
        # the network at the bench's width on one configuration's sources
        dict(name="net_64x64x16_h32", kind="net", Nt=64, Nx=64, Ls=16, hidden=32, n=28),
        # one training step's gradient at the bench's batch
        dict(name="netgrad_64x64x16_h32", kind="netgrad", Nt=64, Nx=64, Ls=16, hidden=32, n=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dslash", "dslash", "prop", "prop", "measure", "corr", "hmc", "whmc", "net",
                       "netgrad"])
    if kind == "dslash":
        wilson = rng.random() < 0.4
        Ls = 1 if wilson else rng.randint(2, 24)
        while True:
            Nt, Nx, n = (_log(rng, 8, 2048 if wilson else 512), _log(rng, 8, 2048 if wilson else 512),
                         _log(rng, 1, 32))
            if rng.random() < 0.5:
                Nx = max(8, 8 * (Nx // 8))  # half the extents are round, as lattices mostly are
            if Nt * Nx * Ls * n <= 4 * 1024 * 1024:
                break
        return dict(kind=kind, Nt=Nt, Nx=Nx, Ls=Ls, n=n, prec=rng.choice([64, 32]),
                    op=rng.choice(["D", "Ddag", "DDdag", "DdagD"]))
    if kind in ("prop", "measure"):
        while True:
            Nt, Nx = 2 * rng.randint(6, 32), 2 * rng.randint(4, 48)
            if rng.random() < 0.5:  # the scans' own extents
                Nt, Nx = rng.choice([16, 32, 48, 64]), 8 * rng.randint(2, 12)
            elif rng.random() < 0.2:  # an odd extent: no even-odd split
                Nx += 1
            Ls = rng.choice([4, 6, 8, 8, 12, 12, 16, 16, 16, 24])
            most = 64 * 96 * 16 * (56 if Nx % 2 == 0 else 14)
            k = rng.randint(2, 56) if kind == "prop" else rng.randint(1, 6)
            if Nt * Nx * Ls * k * (1 if kind == "prop" else 28) <= most:
                break
        c = dict(kind=kind, Nt=Nt, Nx=Nx, Ls=Ls, mf=round(rng.uniform(0.04, 0.1), 3))
        c["nsrc" if kind == "prop" else "nconf"] = k
        return c
    if kind == "corr":
        return dict(kind=kind, Nt=_log(rng, 8, 64), Nx=_log(rng, 8, 64),
                    m0=round(rng.uniform(0.02, 0.2), 3), beta=rng.choice([2.0, 3.0, 4.0, 6.0]),
                    nconf=rng.randint(1, 16))
    if kind == "hmc":
        return dict(kind=kind, Nt=_log(rng, 8, 64), Nx=_log(rng, 8, 64), Ls=rng.randint(4, 16),
                    mf=round(rng.uniform(0.04, 0.1), 3), steps=rng.randint(4, 10))
    if kind == "whmc":
        return dict(kind=kind, Nt=_log(rng, 8, 64), Nx=_log(rng, 8, 64),
                    m0=round(rng.uniform(0.08, 0.2), 3), beta=rng.choice([2.0, 3.0, 4.0]),
                    steps=rng.randint(8, 20))
    wilson = rng.random() < 0.3
    return dict(kind=kind, Nt=rng.randint(8, 64), Nx=rng.choice([16, 20, 32, 40, 48, 64]),
                Ls=1 if wilson else rng.choice([4, 8, 12, 16]),
                hidden=8 if wilson else rng.choice([8, 16, 24, 32]), n=rng.randint(2, 28))


# ---------------------------------------------------------------- inputs


def _np(case, seed):
    return np.random.default_rng([int(seed) & 0xFFFFFFFF, case["Nt"], case["Nx"], case.get("Ls", 1)])


def _gauge(rng, Nt, Nx, beta):
    """A pure-gauge configuration's link angles [2 Nt Nx] in [-pi, pi)."""
    P = rng.vonmises(0.0, beta, size=(Nt, Nx))
    th = np.zeros((2, Nt, Nx))
    th[1, 0] = rng.uniform(-np.pi, np.pi, Nx)
    th[1, 1:] = th[1, 0] + np.cumsum(P[:-1], axis=0)
    step = th[1, 0, :-1] - th[1, Nt - 1, :-1] - P[Nt - 1, :-1]
    th[0, Nt - 1, 1:] = np.cumsum(step)
    phi = rng.uniform(-np.pi, np.pi, (Nt, Nx))
    th[0] += phi - np.roll(phi, -1, 0)
    th[1] += phi - np.roll(phi, -1, 1)
    return (np.mod(th + np.pi, 2 * np.pi) - np.pi).reshape(-1)


def _beta(case):
    return case.get("beta", 3.0)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _gauss(case, seed, n, dtype):
    """n Gaussian fields on the GPU, complex [n, Ls, Nt, Nx, 2]."""
    return torch.randn(n, case["Ls"], case["Nt"], case["Nx"], 2, generator=_gen(seed), device="cuda",
                       dtype=dtype)


def _sources(case, seed):
    """Boundary sources [nsrc, Ls, Nt, Nx, 2]: spin 1 on s = 0, spin 0 on s = Ls - 1;
    2 of 7 are points, 1 of 7 walls, the rest Z4 noise (the analyzer's 8 : 4 : 16)."""
    Nt, Nx, Ls, n = case["Nt"], case["Nx"], case["Ls"], case["nsrc"]
    v = torch.zeros(n, Ls, Nt, Nx, 2, dtype=torch.complex128, device="cuda")
    digits = torch.randint(0, 4, (n, Nt, Nx, 2), generator=_gen(seed + 17), device="cuda")
    z4 = torch.tensor([1, 1j, -1, -1j], dtype=torch.complex128, device="cuda")[digits]
    npoint, nwall = max(1, 2 * n // 7), n // 7
    for k in range(n):
        t, b = ((k // 2) * (Nt // 4)) % Nt, k % 2
        s = 0 if b else Ls - 1
        if k < npoint:
            v[k, s, t, 0, b] = 1.0
        elif k < npoint + nwall:
            v[k, s, t, :, b] = 1.0
        else:
            v[k, 0, :, :, 1] = z4[k, :, :, 1]
            v[k, Ls - 1, :, :, 0] = z4[k, :, :, 0]
    return v


def _measure_inputs(case, seed):
    rng = _np(case, seed)
    th = np.stack([_gauge(rng, case["Nt"], case["Nx"], _beta(case)) for _ in range(case["nconf"])])
    z4 = rng.integers(0, 4, size=case["nconf"] * 16 * case["Nt"] * case["Nx"] * 2).astype(np.int8)
    return th, z4


def _max_momentum(case):
    return min(5, case["Nx"] // 2)


def _hmc_inputs(case, seed):
    """Start angles, heat-bath draw, momenta and the Metropolis uniform (host)."""
    rng = _np(case, seed)
    th = _gauge(rng, case["Nt"], case["Nx"], _beta(case))
    nd = case.get("Ls", 1) * case["Nt"] * case["Nx"] * 2
    chi = (rng.normal(size=nd) + 1j * rng.normal(size=nd)) / math.sqrt(2.0)
    mom = rng.normal(size=2 * case["Nt"] * case["Nx"])
    return th, chi, mom, float(rng.uniform())


def _epsilon(case):
    return 0.01 if case["kind"] == "hmc" else 0.05


def _net_inputs(case, seed):
    """Four layers of weights [9, cout, cin]: a damped identity in the first
    offset plus noise, as a network on its way to D^-1 has them."""
    rng = _np(case, seed)
    th = _gauge(rng, case["Nt"], case["Nx"], _beta(case))
    C0, H = 2 * case["Ls"], case["hidden"]
    ch = [C0, H, H, H, C0]
    ws = []
    for co, ci in zip(ch[1:], ch[:-1]):
        w = (rng.normal(size=(9, co, ci)) + 1j * rng.normal(size=(9, co, ci))) / math.sqrt(18.0 * ci)
        w[0] += 0.7 * np.eye(co, ci)
        ws.append(w.astype(np.complex64))
    return th, ws


def _pairs(case, seed):
    e = _gauss(case, seed + 3, case["n"], torch.complex64)
    return _gauss(case, seed + 5, case["n"], torch.complex64) + 2.0 * e, e


def _context(case):
    if case.get("Ls", 1) == 1:
        return T.Wilson(case["Nt"], case["Nx"], case.get("m0", 0.1), _beta(case))
    return T.DomainWall(case["Nt"], case["Nx"], case["Ls"], M5, case.get("mf", 0.05), _beta(case))


_OPS = {"D": "OP_D", "Ddag": "OP_DDAG", "DDdag": "OP_DDDAG", "DdagD": "OP_DDAGD"}


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, d=_context(case))
    d = s["d"]
    if kind == "dslash":
        d.set_gauge(_gauge(_np(case, seed), case["Nt"], case["Nx"], _beta(case)))
        s["in"] = _gauss(case, seed, case["n"], torch.complex128 if case["prec"] == 64 else torch.complex64)
        s["out"] = torch.empty_like(s["in"])
    elif kind == "prop":
        d.set_gauge(_gauge(_np(case, seed), case["Nt"], case["Nx"], _beta(case)))
        s["src"] = _sources(case, seed)
        s["x"] = torch.empty_like(s["src"])
    elif kind == "measure":
        s["theta"], s["z4"] = _measure_inputs(case, seed)
    elif kind == "corr":
        rng = _np(case, seed)
        s["theta"] = np.stack([_gauge(rng, case["Nt"], case["Nx"], _beta(case))
                               for _ in range(case["nconf"])])
    elif kind in ("hmc", "whmc"):
        s["theta"], s["chi"], s["mom"], s["u"] = _hmc_inputs(case, seed)
    else:
        th, ws = _net_inputs(case, seed)
        d.set_gauge(th)
        d.lp_init(hidden=case["hidden"], seed=1)
        d.lp_set_weights(ws)
        if kind == "net":
            s["in"] = _gauss(case, seed, case["n"], torch.complex64)
            s["out"] = torch.empty_like(s["in"])
        else:
            s["rho"], s["e"] = _pairs(case, seed)
    return s


# ---------------------------------------------------------------- one pass


def run(s):
    case, d = s["case"], s["d"]
    kind = case["kind"]
    if kind == "dslash":
        d.apply_dev(getattr(T, _OPS[case["op"]]), s["in"], s["out"])
        return s["out"]
    if kind == "prop":
        d.propagators_dev(s["src"], s["x"], rtol=RTOL, maxiter=MAXITER, solver=T.SOLVER_EO_MIXED)
        return s["x"]
    if kind == "measure":
        m = d.measure(s["theta"], z4=s["z4"], n_point_times=4, n_wall_times=2, n_noise=16,
                      max_momentum=_max_momentum(case), rtol=RTOL, maxiter=MAXITER,
                      solver=T.SOLVER_EO_MIXED)
        return {k: m[k] for k in ("cpp", "cj5", "loop", "mom_cpp")}
    if kind == "corr":
        return d.pseudoscalar_correlator(s["theta"], 0, 0, RTOL, MAXITER)
    if kind == "hmc":
        th, i = d.hmc_trajectory(s["theta"], s["chi"], s["mom"], _epsilon(case), case["steps"],
                                 rtol=RTOL, maxiter=MAXITER, solver=T.SOLVER_MIXED)
        return {"theta": th, "H0": i["H0"], "H": i["H"], "plaquette": i["plaquette"]}
    if kind == "whmc":
        th, i = d.hmc_step(s["theta"], s["mom"], s["chi"], s["u"], _epsilon(case), case["steps"],
                           RTOL, MAXITER)
        return {"theta": th, "H0": i["H0"], "H": i["H"], "accepted": int(i["accepted"])}
    if kind == "net":
        d.lp_apply_dev(s["in"], s["out"])
        return s["out"]
    loss, grads = d.lp_loss_grad_dev(s["rho"], s["e"])
    return {"loss": loss, "grads": grads}


# ---------------------------------------------------------------- what a pass cannot do without


def work(case):
    """Inputs read once, outputs written once; arithmetic of the operator
    applications, with a nominal count of Krylov iterations for the solves
    (per even-odd iteration, the four half-lattice hops cost two D)."""
    kind, V, Ls = case["kind"], case["Nt"] * case["Nx"], case.get("Ls", 1)
    site = 2 * V * Ls  # complex numbers of one field
    dflops = 100.0 * V * Ls  # one D: four projected hops of a two-spinor, diagonal and fifth dimension
    if kind == "dslash":
        w = case["prec"] // 4
        reps = 2 if case["op"] in ("DDdag", "DdagD") else 1
        return dict(bytes=case["n"] * site * w * 2 + 2 * V * w, flops=reps * case["n"] * dflops)
    if kind == "prop":
        return dict(bytes=case["nsrc"] * site * 32 + 16 * V, flops=case["nsrc"] * 350 * 2.5 * dflops)
    if kind == "measure":
        n = 28 * case["nconf"]
        return dict(bytes=case["nconf"] * (16 * V + 32 * V + 16 * V), flops=n * 350 * 2.5 * dflops)
    if kind == "corr":
        return dict(bytes=case["nconf"] * 16 * V, flops=2 * case["nconf"] * 250 * 2.5 * dflops)
    if kind in ("hmc", "whmc"):
        return dict(bytes=site * 16 + 48 * V, flops=(case["steps"] + 1) * 500 * 2.5 * dflops)
    C0, H = 2 * Ls, case["hidden"]
    mac = 8.0 * 9 * V * case["n"] * (2 * C0 * H + 2 * H * H)
    wts = 9 * (2 * C0 * H + 2 * H * H)
    if kind == "net":
        return dict(bytes=case["n"] * site * 16 + wts * 8, flops=mac)
    return dict(bytes=case["n"] * site * 16 + wts * 16, flops=3 * mac)


# ---------------------------------------------------------------- 64-bit values, plain torch


class _Op:
    """D and D^dag on complex128 fields [n, Ls, Nt, Nx, 2] (n fields on one
    configuration, or one configuration per field). theta: [c, 2, Nt, Nx]."""

    def __init__(self, case, theta):
        Nt, Nx = case["Nt"], case["Nx"]
        self.fifth = case.get("Ls", 1) > 1
        self.diag = 3.0 - M5 if self.fifth else 2.0 + case.get("m0", 0.1)
        self.mf = case.get("mf", 0.05)
        th = theta.reshape(-1, 2, 1, Nt, Nx)
        U = torch.polar(torch.ones_like(th), th)
        sign = torch.ones(Nt, 1, dtype=torch.float64, device=th.device)
        sign[-1] = -1.0  # fermions antiperiodic in t
        self.Ut, self.Ux = U[:, 0] * sign, U[:, 1]

    def D(self, v, dag=False):
        k = 1.0 if dag else -1.0
        a, b = v[..., 0], v[..., 1]
        up = self.diag * a
        lo = self.diag * b
        w = self.Ut * (a + k * b).roll(-1, 2)
        up = up - 0.5 * w
        lo = lo - 0.5 * k * w
        w = (self.Ut.conj() * (a - k * b)).roll(1, 2)
        up = up - 0.5 * w
        lo = lo + 0.5 * k * w
        w = self.Ux * (a - (1j * k) * b).roll(-1, 3)
        up = up - 0.5 * w
        lo = lo - (0.5j * k) * w
        w = (self.Ux.conj() * (a + (1j * k) * b)).roll(1, 3)
        up = up - 0.5 * w
        lo = lo + (0.5j * k) * w
        if self.fifth:
            f, g = (a, b) if not dag else (b, a)
            dn, un = f.roll(1, 1), g.roll(-1, 1)  # s - 1 and s + 1, m_f across the walls
            dn = torch.cat([-self.mf * dn[:, :1], dn[:, 1:]], 1)
            un = torch.cat([un[:, :-1], -self.mf * un[:, -1:]], 1)
            up, lo = (up - dn, lo - un) if not dag else (up - un, lo - dn)
        return torch.stack([up, lo], -1)

    def cg(self, b, dag_first, x=None):
        """(D^dag D)^-1 b, or (D D^dag)^-1 b when dag_first, to 1e-14."""
        def dot(u, v):
            return torch.view_as_real(u * v.conj())[..., 0].flatten(1).sum(1)

        def A(v):
            return self.D(self.D(v, dag_first), not dag_first)

        def ex(c):
            return c.reshape(-1, 1, 1, 1, 1)

        x = torch.zeros_like(b) if x is None else x.clone()
        r = b - A(x)
        p = r.clone()
        rr, stop = dot(r, r), 1e-28 * dot(b, b)
        for it in range(MAXITER):
            t = self.D(p, dag_first)
            al = rr / dot(t, t).clamp_min(1e-300)
            x += ex(al) * p
            r -= ex(al) * self.D(t, not dag_first)
            rn = dot(r, r)
            p = r + ex(rn / rr.clamp_min(1e-300)) * p
            rr = rn
            if it % 25 == 24 and bool((rr <= stop).all()):
                break
        return x


def _theta(th):
    return torch.as_tensor(th, dtype=torch.float64, device="cuda")


def _plaq(th):
    return th[0] + th[1].roll(-1, 0) - th[0].roll(-1, 1) - th[1]


def _trajectory(case, seed):
    th0, chi, mom, u = _hmc_inputs(case, seed)
    Nt, Nx, eps, wil = case["Nt"], case["Nx"], _epsilon(case), case["kind"] == "whmc"
    case = dict(case, Ls=case.get("Ls", 1))
    th = _theta(th0).reshape(2, Nt, Nx)
    p = _theta(mom).reshape(2, Nt, Nx)
    chi = torch.as_tensor(chi, device="cuda").reshape(1, case["Ls"], Nt, Nx, 2)
    phi = _Op(case, th).D(chi)
    eta = None

    def force(th):
        nonlocal eta
        op = _Op(case, th)
        eta = op.cg(phi, True, eta)
        xi = op.D(eta, True)
        q = th.clone().requires_grad_()
        Sg = _beta(case) * (1.0 - torch.cos(_plaq(q))).sum()
        lin = -2.0 * torch.view_as_real(eta.conj() * _Op(case, q).D(xi))[..., 0].sum()
        f, = torch.autograd.grad(Sg + lin, q)
        return f, float(Sg) + float(torch.view_as_real(phi.conj() * eta)[..., 0].sum())

    f, S = force(th)
    H0 = S + 0.5 * float((p * p).sum())
    p = p - 0.5 * eps * f
    for k in range(case["steps"]):
        th = th + eps * p
        if wil:
            th = torch.remainder(th + math.pi, 2 * math.pi) - math.pi
        f, S = force(th)
        p = p - (eps if k + 1 < case["steps"] else 0.5 * eps) * f
    H = S + 0.5 * float((p * p).sum())
    if not wil:
        return {"theta": th.reshape(-1), "H0": H0, "H": H,
                "plaquette": float(torch.cos(_plaq(th)).mean())}
    acc = u < min(1.0, math.exp(-(H - H0)))
    return {"theta": th.reshape(-1) if acc else _theta(th0), "H0": H0, "H": H, "accepted": int(acc)}


def _measure_exact(case, seed):
    Nt, Nx, Ls, nc = case["Nt"], case["Nx"], case["Ls"], case["nconf"]
    ths, z4 = _measure_inputs(case, seed)
    z4 = torch.as_tensor(z4.reshape(nc, 16, Nt, Nx, 2).astype(np.int64), device="cuda")
    ph = torch.tensor([1, 1j, -1, -1j], dtype=torch.complex128, device="cuda")[z4]
    nm = _max_momentum(case) + 1
    x = torch.arange(Nx, device="cuda", dtype=torch.float64)
    cosw = torch.cos(2 * math.pi / Nx * torch.arange(nm, device="cuda", dtype=torch.float64)[:, None] * x)
    res = {k: [] for k in ("cpp", "cj5", "loop", "mom_cpp")}
    for c in range(nc):
        v = torch.zeros(28, Ls, Nt, Nx, 2, dtype=torch.complex128, device="cuda")
        for k in range(12):
            t = (k // 2) * Nt // 4 if k < 8 else ((k - 8) // 2) * Nt // 2
            b = k % 2
            v[k, 0 if b else Ls - 1, t, slice(0, 1) if k < 8 else slice(None), b] = 1.0
        v[12:, 0, :, :, 1] = ph[c, :, :, :, 1]
        v[12:, Ls - 1, :, :, 0] = ph[c, :, :, :, 0]
        op = _Op(case, _theta(ths[c]))
        s = op.cg(op.D(v, True), False)
        q = torch.stack([s[:, Ls - 1, ..., 0], s[:, 0, ..., 1]], -1)  # [28, Nt, Nx, 2]
        qq = (q.abs() ** 2).sum(-1)
        j5 = torch.view_as_real(s[:, Ls // 2].conj() * q)[..., 0].sum(-1)
        cpp, cj5 = torch.zeros(2, Nt, dtype=torch.float64, device="cuda")
        for k in range(8, 12):
            ts = ((k - 8) // 2) * Nt // 2
            cpp = cpp + qq[k].sum(1).roll(-ts) / 2
            cj5 = cj5 + j5[k].sum(1).roll(-ts) / 2
        mom = torch.zeros(nm, Nt, dtype=torch.float64, device="cuda")
        for k in range(8):
            mom = mom + (cosw @ qq[k].T).roll(-((k // 2) * Nt // 4), 1) / 4
        g5 = torch.tensor([1.0, -1.0], dtype=torch.float64, device="cuda")
        loop = (ph[c].conj() * g5 * q[12:]).sum(-1).mean(0).reshape(-1)
        for k, val in (("cpp", cpp), ("cj5", cj5), ("loop", loop), ("mom_cpp", mom)):
            res[k].append(val)
    return {k: torch.stack(val) for k, val in res.items()}


_OFFSETS = ((0, 0), (1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (1, -1), (-1, 1), (-1, -1))


class _Net:
    """The four-layer network in 64 bits, fields [n, C, Nt, Nx]."""

    def __init__(self, case, th):
        U = _Op(case, th)
        self.U = (U.Ut[0, 0], U.Ux[0, 0])

    def hop(self, v, mu, sg):
        """Transport of v one step along mu: from y + mu to y, or from y - mu."""
        ax = v.dim() - 2 + mu
        if sg > 0:
            return self.U[mu] * v.roll(-1, ax)
        return (self.U[mu].conj() * v).roll(1, ax)

    def moved(self, v, dt, dx):
        if dt and dx:
            return 0.5 * (self.hop(self.hop(v, 1, dx), 0, dt) + self.hop(self.hop(v, 0, dt), 1, dx))
        if dt:
            return self.hop(v, 0, dt)
        return self.hop(v, 1, dx) if dx else v

    def __call__(self, ws, v):
        for w in ws:
            out = 0
            for k, (dt, dx) in enumerate(_OFFSETS):
                out = out + torch.einsum("oi,nitx->notx", w[k], self.moved(v, dt, dx))
            v = out
        return v


def _to_net(f):
    n, Ls, Nt, Nx, _ = f.shape
    return f.to(torch.complex128).permute(0, 1, 4, 2, 3).reshape(n, 2 * Ls, Nt, Nx)


def exact(case, seed):
    kind = case["kind"]
    if kind == "dslash":
        op = _Op(case, _theta(_gauge(_np(case, seed), case["Nt"], case["Nx"], _beta(case))))
        v = _gauss(case, seed, case["n"], torch.complex128 if case["prec"] == 64 else torch.complex64)
        v = v.to(torch.complex128)
        for dag in {"D": (False,), "Ddag": (True,), "DDdag": (True, False), "DdagD": (False, True)}[case["op"]]:
            v = op.D(v, dag)
        return v
    if kind == "prop":
        op = _Op(case, _theta(_gauge(_np(case, seed), case["Nt"], case["Nx"], _beta(case))))
        return op.cg(op.D(_sources(case, seed), True), False)
    if kind == "measure":
        return _measure_exact(case, seed)
    if kind == "corr":
        rng = _np(case, seed)
        out = []
        for _ in range(case["nconf"]):
            op = _Op(case, _theta(_gauge(rng, case["Nt"], case["Nx"], _beta(case))))
            v = torch.zeros(2, 1, case["Nt"], case["Nx"], 2, dtype=torch.complex128, device="cuda")
            v[0, 0, 0, 0, 0] = v[1, 0, 0, 0, 1] = 1.0
            out.append((op.cg(op.D(v, True), False).abs() ** 2).sum((0, 1, 3, 4)))
        return torch.stack(out)
    if kind in ("hmc", "whmc"):
        return _trajectory(case, seed)
    th, ws = _net_inputs(case, seed)
    net = _Net(case, _theta(th))
    ws = [torch.as_tensor(w, device="cuda").to(torch.complex128) for w in ws]
    n, C0 = case["n"], 2 * case["Ls"]
    if kind == "net":
        with torch.no_grad():
            out = net(ws, _to_net(_gauss(case, seed, n, torch.complex64)))
        return out.reshape(n, case["Ls"], 2, case["Nt"], case["Nx"]).permute(0, 1, 3, 4, 2).contiguous()
    rho, e = (_to_net(v) for v in _pairs(case, seed))
    ws = [w.requires_grad_() for w in ws]
    diff = torch.view_as_real(net(ws, rho) - e).square().flatten(1).sum(1)
    loss = (diff / torch.view_as_real(e).square().flatten(1).sum(1)).mean()
    grads = torch.autograd.grad(loss, ws)
    return {"loss": float(loss), "grads": list(grads)}
