"""The work a user of hipft_b200 has it do, as cases that can be timed.

Every case drives the public Python binding (hipft_b200.HipftGPU, .MisfitAdjoint,
.FluxTransport) the way HipFT's main loop, or a program that calibrates its
parameters, drives it: a handle is built once with the run's mesh, realizations
and switches, and then steps, assimilates, analyses or differentiates.

Step cases put the handle's field back to the initial map first (one device
copy), so that every pass does the same work: the number of diffusion subcycles
and RKG2 stages follows from the field (HipFT's practical time step limit).

Grids: HipFT's test suite (180 x 360 and the 150 x 300 class of remeshed HMI
maps), its production sizes (512 x 1024, 1024 x 2048, 2048 x 4096), and sizes of
no particular factor in between.  Flows: HipFT's analytic differential rotation
and meridional flow; attenuated flows, which are rebuilt from the field before
every step; flows from files.  Diffusion: 25 to 1000 km^2/s.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import hipft_b200 as H
from hipft_b200.adjoint import FluxTransport, MisfitAdjoint

M_S = 5.172413793103448e-06        # m/s in solar radii per hour
DEG_DAY = (math.pi / 180.0) / 86400.0 * 6.96e8
D_FACTOR = 7.43162901307967e-09    # km^2/s in solar radii^2 per hour
BASE = dict(kind="step", nt=180, np=360, nr=1, refined=False, ragged=False, graph=False, cfl=0.9, hours=0.0,
            flow="analytic", adv=4, strang=True, dif=3, subcycles=0, grid_d=False, d_lo=300.0, d_hi=300.0, steps=1,
            checkpoint=64, balance=False)


def _case(name=None, **kw):
    c = dict(BASE)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the test suite's grid, one realization, a short step: latency of one call
        _case("step_180x360", hours=0.25, d_lo=300.0, d_hi=300.0),
        # the test suite's attenuated run: flows rebuilt from the field, CFL limit, step and history row every 15 minutes
        _case("atten_cycle_151x300_x5", kind="cycle", nt=151, np=300, nr=5, flow="attenuated", hours=0.25, d_lo=25.0,
              d_hi=25.0, strang=False),
        # plain diffusion in daily steps, no flows
        _case("diffuse_day_256x512", nt=256, np=512, flow="none", hours=24.0, d_lo=500.0, d_hi=500.0),
        # the other methods HipFT offers: upwind SSPRK(3,3), grid-dependent D, RKL2 with fixed subcycles, Lie splitting
        _case("upwind_gridD_rkl2_181x361_x4", nt=181, np=361, nr=4, adv=2, dif=2, grid_d=True, subcycles=2, strang=False,
              d_lo=20.0, d_hi=200.0),
        # one forward step of the calibration grid
        _case("step_512x1024", nt=512, np=1024),
        # a small ensemble on the reference's one shared schedule, sizes of no particular factor
        _case("shared_359x722_x9", nt=359, np=722, nr=9, d_lo=100.0, d_hi=700.0),
        # the production grid, one realization
        _case("step_1024x2048", nt=1024, np=2048, refined=True),
        # the production ensemble: 64 parameter sets, each on its own schedule, one CUDA graph per step
        _case("ensemble_1024x2048_x64", nt=1024, np=2048, nr=64, refined=True, ragged=True, graph=True, d_lo=100.0,
              d_hi=1000.0),
        # high resolution with convective flows from files: many short steps
        _case("fileflow_2048x4096_x4", kind="cycle", nt=2048, np=4096, nr=4, refined=True, ragged=True, flow="file",
              hours=0.004, d_lo=100.0, d_hi=1000.0),
        # a daily observation blended into an ensemble, flux-balanced, with its history rows
        _case("assimilate_1024x2048_x16", kind="assimilate", nt=1024, np=2048, nr=16, refined=True, balance=True,
              d_lo=100.0, d_hi=1000.0),
        # gradient of a map misfit over several steps
        _case("gradient_512x1024", kind="gradient", nt=512, np=1024, steps=6, checkpoint=3),
        # the autograd function inside a small torch program
        _case("autograd_90x181_x2", kind="autograd", nt=90, np=181, nr=2, steps=4, checkpoint=2, hours=2.0, d_lo=200.0,
              d_hi=400.0),
    ]


def draw(rng):
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return n if rng.random() < 0.5 else n - n % 8

    kind = rng.choice(["single", "diffuse", "shared", "ragged", "atten", "file", "other", "assimilate", "gradient",
                       "autograd"])
    if kind in ("single", "diffuse"):
        nt = size(64, 1200)
        return _case(nt=nt, np=2 * nt + rng.randrange(0, 9), refined=rng.random() < 0.4,
                     flow="none" if kind == "diffuse" else "analytic",
                     hours=float(rng.choice([6.0, 24.0])) if kind == "diffuse" else 0.0,
                     cfl=round(rng.uniform(0.3, 0.95), 3), strang=rng.random() < 0.8, d_lo=300.0,
                     d_hi=round(rng.uniform(100.0, 700.0), 1), dif=3 if rng.random() < 0.8 else 2)
    if kind in ("shared", "ragged"):
        nt = size(90, 800)
        nr = max(2, min(48, int(3.0e7 / (2.0 * nt * nt) * rng.uniform(0.3, 1.0))))
        return _case(nt=nt, np=2 * nt + rng.randrange(0, 9), nr=nr, refined=rng.random() < 0.5, ragged=kind == "ragged",
                     graph=rng.random() < 0.5, cfl=round(rng.uniform(0.5, 0.95), 3), d_lo=100.0,
                     d_hi=round(rng.uniform(300.0, 1000.0), 1))
    if kind == "atten":
        nt = size(90, 500)
        return _case(kind="cycle", nt=nt, np=2 * nt + rng.randrange(0, 5), nr=rng.randrange(1, 7), flow="attenuated",
                     hours=0.25, d_lo=25.0, d_hi=round(rng.uniform(25.0, 300.0), 1), strang=rng.random() < 0.5)
    if kind == "file":
        nt = size(256, 1200)
        return _case(kind="cycle", nt=nt, np=2 * nt + rng.randrange(0, 9), nr=rng.randrange(1, 6), refined=True,
                     ragged=rng.random() < 0.5, flow="file", hours=round(rng.uniform(0.004, 0.05), 4), d_lo=100.0,
                     d_hi=round(rng.uniform(200.0, 1000.0), 1))
    if kind == "other":
        nt = size(64, 400)
        return _case(nt=nt, np=2 * nt + rng.randrange(0, 5), nr=rng.randrange(1, 7), adv=rng.choice([1, 2, 3]),
                     dif=rng.choice([2, 3]), grid_d=rng.random() < 0.6, subcycles=rng.choice([0, 2]),
                     strang=rng.random() < 0.5, d_lo=20.0, d_hi=200.0, cfl=0.5)
    if kind == "assimilate":
        nt = size(150, 1024)
        return _case(kind="assimilate", nt=nt, np=2 * nt + rng.randrange(0, 5), nr=rng.randrange(1, 17),
                     refined=rng.random() < 0.5, balance=rng.random() < 0.5)
    nt = size(64, 400) if kind == "gradient" else size(48, 128)
    return _case(kind=kind, nt=nt, np=2 * nt + rng.randrange(0, 5), nr=1 if kind == "gradient" else rng.randrange(1, 4),
                 steps=rng.randrange(2, 7), checkpoint=rng.randrange(1, 5), hours=0.0 if kind == "gradient" else 2.0,
                 d_lo=200.0, d_hi=round(rng.uniform(200.0, 500.0), 1))


# ------------------------------------------------------------------ inputs
def _theta(c):
    n = c["nt"]
    if not c["refined"]:
        return np.linspace(0.0, np.pi, n)
    x = np.linspace(0.0, np.pi, 20001)  # spacing halved within 15 degrees of each pole
    pole = np.minimum(x, np.pi - x)
    dens = 1.0 + 0.5 * (1.0 - np.tanh((pole - np.deg2rad(15.0)) / np.deg2rad(2.0)))
    cdf = np.concatenate([[0.0], np.cumsum(0.5 * (dens[1:] + dens[:-1]) * np.diff(x))])
    t = np.interp(np.linspace(0.0, 1.0, n), cdf / cdf[-1], x)
    t[0], t[-1] = 0.0, np.pi
    return t


def _grid(c):
    return _theta(c), np.linspace(0.0, 2.0 * np.pi, c["np"] + 1)


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _map(c, seed, pairs=60):
    """An active Sun: a polar dipole of 5 G and bipolar Gaussian pairs of up to
    some hundred Gauss at +-15 degrees; (ntm, npm1), periodic."""
    t, p = _grid(c)
    rng = np.random.default_rng([seed, 11])
    dev = _dev()
    T, P = torch.as_tensor(t, device=dev)[:, None], torch.as_tensor(p, device=dev)[None, :]
    st, ct = torch.sin(T), torch.cos(T)
    f = 5.0 * ct + 0.0 * P
    for _ in range(pairs):
        hemi = rng.choice([-1.0, 1.0])
        lat = hemi * abs(rng.normal(15.0, 7.0))
        lon, peak, sep = rng.uniform(0.0, 360.0), rng.lognormal(math.log(100.0), 0.6), rng.uniform(3.0, 10.0)
        tilt = math.radians(0.5 * abs(lat))
        for sign in (1.0, -1.0):
            la = math.radians(lat - hemi * sign * 0.5 * sep * math.sin(tilt))
            lo = math.radians(lon + sign * 0.5 * sep * math.cos(tilt))
            dot = ct * math.sin(la) + st * math.cos(la) * torch.cos(P - lo)
            f = f + hemi * sign * peak * torch.exp((dot - 1.0) * (2.0 / math.radians(2.0) ** 2))
    f[:, -1] = f[:, 0]
    return f.cpu().numpy()


def _params(c):
    """Per-realization parameters; they belong to the case."""
    nr = c["nr"]
    rng = np.random.default_rng(5)
    D = np.exp(np.linspace(math.log(c["d_lo"]), math.log(c["d_hi"]), nr)) if nr > 1 else np.array([float(c["d_hi"])])
    D = D[rng.permutation(nr)]
    v0 = rng.uniform(10.0, 20.0, nr)
    return dict(D=D, p0=np.zeros(nr), p2=-2.40 * DEG_DAY * rng.uniform(0.9, 1.1, nr),
                p4=-1.80 * DEG_DAY * rng.uniform(0.9, 1.1, nr), p1=2.0 * v0, p3=-2.0 * v0, p5=np.zeros(nr))


def _file_flow(c):
    """A smooth random divergent flow of some 100 m/s as HipFT's flow files hold
    it: vt (nt, npm1), vp (ntm, np), m/s; it fades out at the poles."""
    t, p = _grid(c)
    rng = np.random.default_rng(7)
    th = 0.5 * (t[1:] + t[:-1])
    ph = 0.5 * (p[1:] + p[:-1])
    vt, vp = np.zeros((len(t) + 1, len(p))), np.zeros((len(t), len(p) + 1))
    for _ in range(24):
        m, n = int(rng.integers(2, 60)), int(rng.integers(2, 60))
        a, b, s = rng.uniform(0.0, 2 * np.pi), rng.uniform(0.0, 2 * np.pi), 40.0 * rng.normal()
        vt[1:-1] += s * (np.sin(th) ** 2 * np.cos(n * th + b))[:, None] * np.cos(m * p + a)[None, :]
        vp[:, 1:-1] += s * (np.sin(t) ** 2 * np.sin(n * t + b))[:, None] * np.sin(m * ph + a)[None, :]
    vp[:, 0], vp[:, -1] = vp[:, -2], vp[:, 1]
    return vt, vp


# ------------------------------------------------- what the library is given
def _handle(c, prm, t, p):
    flow = c["flow"] != "none"
    g = H.HipftGPU(t, p, c["nr"], advance_flow=flow, flow_num_method=c["adv"], strang_splitting=c["strang"],
                   advance_diffusion=True, diffusion_num_method=c["dif"], diffusion_subcycles=c["subcycles"],
                   diffusion_coef_grid=c["grid_d"], diffusion_coef_constants=prm["D"])
    g.set_stream(torch.cuda.current_stream().cuda_stream)
    if c["flow"] == "file":
        g.set_flow_from_files(*_file_flow(c))
    if flow:
        g.set_flow(dr_model=1, mf_model=1, dr_p0=prm["p0"], dr_p2=prm["p2"], dr_p4=prm["p4"], mf_p1=prm["p1"],
                   mf_p3=prm["p3"], mf_p5=prm["p5"], attenuate=c["flow"] == "attenuated", attenuate_values=500.0)
    return g


def _dt(c, prm):
    return c["hours"] if c["hours"] > 0.0 else c["cfl"] * Scheme(c, prm).cfl()


def _observation(c, seed):
    t, p = _grid(c)
    rng = np.random.default_rng([seed, 13])
    mu = np.sin(t)[:, None] * np.cos(p - rng.uniform(0.0, 2 * np.pi))[None, :]
    d = 10.0 * np.cos(t)[:, None] + rng.normal(0.0, 2.0, (len(t), len(p)))
    return np.stack([d, np.where(mu > 0.1, mu, 0.0) ** 4, mu])


def _target(c, f0):
    """The map a calibration compares with: the initial one a little weaker and turned by some degrees."""
    n2 = f0.shape[1] - 2
    core = np.roll(0.9 * f0[:, 1:-1], n2 // 90 + 1, axis=1)
    return np.concatenate([core[:, -1:], core, core[:, :1]], axis=1)


def prepare(case, seed):
    c = _case(**case)
    prm = _params(c)
    t, p = _grid(c)
    br = _map(c, seed)
    s = dict(case=c, prm=prm, dt=_dt(c, prm))
    if c["kind"] == "autograd":
        f0 = Scheme(c, prm).load(br)
        s["fn"] = FluxTransport(t, p, [s["dt"]] * c["steps"], checkpoint_every=c["checkpoint"])
        s["leaf"] = {k: torch.as_tensor(v).requires_grad_(k not in ("p0", "p5")) for k, v in prm.items()}
        s["f0"] = torch.as_tensor(f0).requires_grad_(True)
        s["target"] = torch.as_tensor(_target(c, f0))
        return s
    g = s["g"] = _handle(c, prm, t, p)
    g.load_initial_map(br[None])
    if c["flow"] != "none":
        g.update_flow()
    if c["ragged"]:
        g.set_ragged(True)
    if c["graph"]:
        g.set_graph(True)
    if c["kind"] == "gradient":
        s["f0"] = g.get_field()
        s["target"] = _target(c, s["f0"])
        s["adj"] = MisfitAdjoint(g, prm["D"], {k: prm[k] for k in ("p0", "p2", "p4", "p1", "p3", "p5")},
                                 checkpoint_every=c["checkpoint"])
        return s
    s["start"] = g.field_tensor().clone()
    if c["kind"] == "assimilate":
        s["obs"] = _observation(c, seed)
    return s


def _field(s):
    """The handle's own field: a view, which keeps the handle alive."""
    f = s["g"].field_tensor()[:, :, :s["case"]["nt"]]
    f.handle = s["g"]
    return f


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "autograd":
        for x in [s["f0"], *s["leaf"].values()]:
            x.grad = None
        f = s["fn"](s["f0"], s["leaf"]["D"], {k: s["leaf"][k] for k in ("p0", "p2", "p4", "p1", "p3", "p5")})
        ((f - s["target"]) ** 2).mean().backward()
        return dict(field=f.detach(), f0=s["f0"].grad, **{k: s["leaf"][k].grad for k in ("D", "p1", "p2", "p3", "p4")})
    if kind == "gradient":
        loss, gr = s["adj"].run(s["f0"], s["target"], [s["dt"]] * c["steps"])
        return dict(loss=loss, **{k: gr[k] for k in ("f0", "D", "p1", "p2", "p3", "p4")})
    g = s["g"]
    g._ck(g.L.hipft_gpu_set_field_device(g.h, ctypes.c_void_p(s["start"].data_ptr())), "set_field_device")
    if kind == "assimilate":
        g.assimilate(s["obs"], custom_from_mu=True, mu_power=4.0, mu_limit=0.1, balance_flux=c["balance"])
        return dict(field=_field(s), history=g.analysis(0.0))
    if kind == "cycle":
        g.update_flow()
        limit = g.flow_dtmax()
        g.flux_transport_step(s["dt"])
        return dict(field=_field(s), history=g.analysis(s["dt"]), limit=limit)
    g.flux_transport_step(s["dt"])
    return dict(field=_field(s))


def work(case):
    """The field read and written once (with its map, flows, or gradients), and
    the arithmetic of the least number of stages: one RKG2 super-step over the
    whole step (HipFT's subcycles, which follow from the field, need more), at
    20 operations per cell and stage, and 130 per cell for a WENO3 stage."""
    c = _case(**case)
    prm = _params(c)
    S = Scheme(c, prm, light=True)
    cells = float(c["nt"]) * c["np"]
    dt = _dt(c, prm)
    if c["kind"] == "assimilate":
        return {"bytes": 8.0 * cells * (2 * c["nr"] + 3), "flops": 40.0 * cells * c["nr"]}
    subs = max(1, c["subcycles"])
    euler = [S.euler_dt(i) for i in range(c["nr"])]
    if not c["ragged"]:
        euler = [min(euler)] * c["nr"]
    stages = sum(subs * _stages(c["dif"], dt / subs, e) for e in euler)
    adv = 0 if c["flow"] == "none" else (2 if c["strang"] else 1) * {1: 1, 2: 3, 3: 3, 4: 4}[c["adv"]] * c["nr"]
    one = 20.0 * stages + (130.0 if c["adv"] >= 3 else 20.0) * adv
    nbytes = 16.0 * c["nr"] + (16.0 if c["flow"] == "file" else 0.0)
    if c["kind"] in ("gradient", "autograd"):
        return {"bytes": cells * 40.0 * c["nr"], "flops": cells * 3.0 * c["steps"] * one}
    return {"bytes": cells * nbytes, "flops": cells * one}


# ----------------------------------------------- the same in plain torch
def _stages(method, dt, euler):
    r = dt / euler
    s = math.ceil(0.5 * (math.sqrt(9.0 + 16.0 * r) - 1.0) if method == 2 else 0.5 * (math.sqrt(25.0 + 24.0 * r) - 3.0))
    s = max(s, 3)
    return s + 1 if s % 2 == 0 else s


class Scheme:
    """HipFT's discrete step in plain 64-bit torch, on the core columns
    (nr, npm - 2, ntm), periodic in phi: src/hipft.f90 set_mesh 6495-6653,
    load_weno 6846-6938, set_lf_alpha 6940-7048, the operators 7615-7990, the
    integrators 7409-7582 and 5163-5475, the subcycles 4551-4695 with the
    practical time step limit 5042-5161.  Differences are taken before they are
    multiplied and increments are summed up apart from the field."""

    def __init__(self, c, prm, light=False):
        self.c, self.prm = c, prm
        t, p = _grid(c)
        ntm, n2 = c["nt"], c["np"]
        self.ntm, self.n2, self.nr = ntm, n2, c["nr"]
        th = np.zeros(ntm + 1)   # faces 1..nt at th[0..ntm]
        dth = np.zeros(ntm + 1)
        th[1:ntm], dth[1:ntm] = 0.5 * (t[1:] + t[:-1]), t[1:] - t[:-1]
        dth[0], dth[ntm] = dth[1], dth[ntm - 1]
        th[0], th[ntm] = th[1] - dth[1], th[ntm - 1] + dth[ntm - 1]
        st = np.sin(t)
        st[0] = st[-1] = 0.0
        sth, cth, ct = np.sin(np.abs(th)), np.cos(th), np.cos(t)
        ct[0] = ct[-1] = 1.0
        # core column q (0-based) is phi column q + 2: the node p[q + 1], its lower face between p[q] and p[q + 1]
        dph = p[1:] - p[:-1]
        dp = 0.5 * (dph + np.roll(dph, -1))
        self.np_mesh = dict(t=t, p=p, th=th, dth=dth, dt=th[1:] - th[:-1], st=st, sth=sth, cth=cth, ct=ct, dp=dp, dph=dph)
        if light:
            return
        dev = self.dev = _dev()
        T = self.T = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)
        self.dth, self.dt, self.sth, self.dp, self.dph = (T(self.np_mesh[k]) for k in ("dth", "dt", "sth", "dp", "dph"))
        sti = np.zeros(ntm)
        sti[1:-1] = 1.0 / st[1:-1]
        self.sti = T(sti)

        def weno(d, lo, hi):
            w = (d / (d + hi), d / (lo + d), lo / (lo + d + hi), (d + hi) / (lo + d + hi), hi / (lo + d + hi),
                 (lo + d) / (lo + d + hi))
            return [T(x) for x in w]

        d = self.np_mesh["dt"]
        self.wt = weno(d, np.concatenate([d[:1], d[:-1]]), np.concatenate([d[1:], d[-1:]]))
        self.wp = weno(dp, np.roll(dp, 1), np.roll(dp, -1))

    # -- input
    def load(self, br):
        """load_initial_map: transpose, seam, pole means; (nr, npm, ntm) numpy."""
        core = br[:, 1:].T.copy()
        w = self.np_mesh["dp"] / (2.0 * np.pi)
        core[:, 0], core[:, -1] = (core[:, 0] * w).sum(), (core[:, -1] * w).sum()
        f = np.concatenate([core[-1:], core, core[:1]])
        return np.ascontiguousarray(np.broadcast_to(f, (self.nr,) + f.shape))

    # -- flows: vt (nr, n2 or 1, nt), vp (nr, n2 or 1, ntm) at the lower phi face of each core column
    def flows_np(self, field=None):
        m, q = self.np_mesh, self.prm
        col = lambda k: q[k][:, None]
        vt = -M_S * m["sth"] * (col("p1") * m["cth"] + col("p3") * m["cth"] ** 3 + col("p5") * m["cth"] ** 5)
        vp = M_S * m["st"] * (col("p0") + col("p2") * m["ct"] ** 2 + col("p4") * m["ct"] ** 4)
        vt, vp = vt[:, None], vp[:, None]
        if self.c["flow"] == "file":
            a, b = _file_flow(self.c)
            vt, vp = vt + M_S * a[:, 1:].T[None], vp + M_S * b[:, 1:-1].T[None]
        return vt, vp

    def flows(self, f=None, coef=None):
        if coef is not None:
            m = {k: self.T(v) for k, v in self.np_mesh.items()}
            col = lambda k: coef[k][:, None, None]
            vt = -M_S * m["sth"] * (col("p1") * m["cth"] + col("p3") * m["cth"] ** 3 + col("p5") * m["cth"] ** 5)
            vp = M_S * m["st"] * (col("p0") + col("p2") * m["ct"] ** 2 + col("p4") * m["ct"] ** 4)
        else:
            vt, vp = (self.T(x) for x in self.flows_np())
        if self.c["flow"] == "attenuated":
            a = f.abs()
            vt = vt.expand(-1, self.n2, -1).clone()
            vt[..., 1:-1] *= 1.0 - torch.tanh(torch.maximum(a[..., :-1], a[..., 1:]) / 500.0)
            vp = vp * (1.0 - torch.tanh(torch.maximum(a.roll(1, 1), a) / 500.0))
        av = vt.abs()
        pad = torch.cat([torch.zeros_like(av[..., :2]), av, torch.zeros_like(av[..., :2])], -1)
        at = torch.stack([pad[..., o:o + self.ntm] for o in range(6)]).amax(0)
        bv = vp.abs()
        ap = bv if bv.shape[1] == 1 else torch.stack([bv.roll(o, 1) for o in (2, 1, 0, -1, -2, -3)]).amax(0)
        return vt, at, vp, ap

    def cfl(self):
        m = self.np_mesh
        vt, vp = (np.abs(x) for x in self.flows_np())
        kt = np.maximum(vt[..., 1:-2], vt[..., 2:-1]) / m["dt"][1:-1]
        kp = np.maximum(vp, np.roll(vp, -1, axis=1))[..., 1:-1] / m["st"][1:-1]
        kp = (kp / m["dp"][None, :, None]).max(1, keepdims=True) if vp.shape[1] == 1 else kp / m["dp"][None, :, None]
        return 0.95 * float(0.5 / (kt + kp).max()) * (2.0 if self.c["strang"] else 1.0) * (2.0 if self.c["adv"] == 4 else 1.0)

    # -- diffusion
    def dcoef(self, D):
        """D on the half mesh: (nr, n2, nt), at the lower phi face of each core column."""
        if not self.c["grid_d"]:
            return (D_FACTOR * D)[:, None, None]
        b = self.dph[:, None] * self.sth[None, :]
        return D_FACTOR * (D[:, None, None] + (self.dth ** 2 + b ** 2)[None])

    def coefs(self, D):
        d = self.dcoef(D)
        up = d.roll(-1, 1)  # upper phi face
        lo, hi = (d[..., 1:-2], d[..., 2:-1]) if d.shape[2] > 1 else (d, d)
        ulo, uhi = (up[..., 1:-2], up[..., 2:-1]) if d.shape[2] > 1 else (d, d)
        s, dti, dpi = self.sti[1:-1], 1.0 / self.dt[1:-1], (1.0 / self.dp)[:, None]
        dphi = (1.0 / self.dph)[:, None]
        c1 = 0.5 * (lo + hi) * dphi * dpi * s * s
        c5 = 0.5 * (ulo + uhi) * dphi.roll(-1, 0) * dpi * s * s
        c2 = 0.5 * (lo + ulo) * dti * s * (self.sth[1:-2] / self.dth[1:-2])
        c4 = 0.5 * (hi + uhi) * dti * s * (self.sth[2:-1] / self.dth[2:-1])
        if d.shape[2] > 1:
            n, so = d[..., 0] + d[..., 1], d[..., -2] + d[..., -1]
        else:
            n = so = (2.0 * d[..., 0]).expand(-1, self.n2)
        return c1, c2, c4, c5, n * self.dp, so * self.dp

    def lap(self, x, C):
        c1, c2, c4, c5, n, so = C
        xc = x[..., 1:-1]
        y = (c1 * (x.roll(1, 1)[..., 1:-1] - xc) + c5 * (x.roll(-1, 1)[..., 1:-1] - xc) + c2 * (x[..., :-2] - xc) +
             c4 * (x[..., 2:] - xc))
        north = (n * (x[..., 1] - x[..., 0])).sum(1) / (math.pi * self.dth[1] ** 2)
        south = -(so * (x[..., -1] - x[..., -2])).sum(1) / (math.pi * self.dth[-2] ** 2)
        return torch.cat([north[:, None, None].expand(-1, self.n2, 1), y, south[:, None, None].expand(-1, self.n2, 1)], 2)

    def euler_dt(self, i=None):
        """The explicit limit of realization i (of all: None), get_dtime_diffusion_euler."""
        m, D = self.np_mesh, self.prm["D"]
        j = slice(1, -1)
        s, a = 1.0 / m["st"][j], 1.0 / (m["dph"] * m["dp"])
        cp = (a + np.roll(1.0 / m["dph"], -1) / m["dp"])
        ct = (m["sth"][1:-2] / m["dth"][1:-2] + m["sth"][2:-1] / m["dth"][2:-1]) * s / m["dt"][j]
        Dm = D.max() if i is None else D[i]
        if not self.c["grid_d"]:
            return 0.95 / (D_FACTOR * Dm * (cp.max() * s * s + ct).max())
        g = Dm + m["dth"][None, :] ** 2 + (m["dph"][:, None] * m["sth"][None, :]) ** 2
        u = np.roll(g, -1, 0)
        e = (0.5 * (g[:, 1:-2] + g[:, 2:-1]) * (1.0 / (m["dph"] * m["dp"]))[:, None] * s * s +
             0.5 * (u[:, 1:-2] + u[:, 2:-1]) * (np.roll(1.0 / m["dph"], -1) / m["dp"])[:, None] * s * s +
             0.5 * (g + u)[:, 1:-2] * (m["sth"][1:-2] / m["dth"][1:-2] * s / m["dt"][j]) +
             0.5 * (g + u)[:, 2:-1] * (m["sth"][2:-1] / m["dth"][2:-1] * s / m["dt"][j]))
        return 0.95 / (D_FACTOR * e.max())

    def sts(self, f, dt, euler, C):
        """One RKL2 / RKG2 super-step; the stages advance the increment z = y - f."""
        meth = self.c["dif"]
        s = _stages(meth, dt, euler)
        if meth == 2:
            w = 4.0 / (s * s + s - 2)
            b = lambda j: 1.0 / 3.0 if j <= 2 else (j * j + j - 2.0) / (2.0 * j * (j + 1))
        else:
            w = 6.0 / ((s + 4) * (s - 1))
            b = lambda j: 1.0 / 3.0 if j <= 1 else 1.0 / 15.0 if j == 2 else 4.0 * (j - 1) * (j + 4) / (3.0 * j * (j + 1) * (j + 2) * (j + 3))
        d0 = dt * self.lap(f, C)
        z2, z1 = torch.zeros_like(f), (w / 3.0 if meth == 2 else w) * d0
        for j in range(2, s + 1):
            if j == 2:
                mu, nu = (1.5, -0.5) if meth == 2 else (0.5, -0.1)
                g = -w if meth == 2 else 0.0
            elif meth == 2:
                mu, nu = b(j) / b(j - 1) * (2.0 - 1.0 / j), b(j) / b(j - 2) * (1.0 / j - 1.0)
                g = (b(j - 1) - 1.0) * mu * w
            else:
                mu, nu = b(j) / b(j - 1) * (2.0 + 1.0 / j), -b(j) / b(j - 2) * (1.0 / j + 1.0)
                g = (0.5 * j * (j + 1.0) * b(j - 1) - 1.0) * mu * w
            z1, z2 = mu * z1 + nu * z2 + (mu * w * dt) * self.lap(z1, C) + (g + mu * w) * d0, z1
        return f + z1

    def ptl(self, f, dt, C):
        """get_dtime_diffusion_ptl of the realizations in f together."""
        with torch.no_grad():
            a = self.lap(f, C)
            big = float(torch.where(f.abs() > 1e-14, a.abs(), torch.zeros_like(a)).max())
            if not big > 0.0:
                return 1.7976931348623157e308
            at = ((a[..., 1:-1].abs() == big) & (f[..., 1:-1].abs() > 1e-14)).nonzero()
            best = 1.7976931348623157e308
            for i, k, j in at[:64].tolist():
                j += 1
                for kk, jj in ((k, j - 1), (k, j + 1), ((k - 1) % self.n2, j), ((k + 1) % self.n2, j)):
                    du, df = float(f[i, k, j] - f[i, kk, jj]), float(a[i, k, j] - a[i, kk, jj])
                    if du * df < -1e-14:
                        best = min(best, -du / df)
        return max(0.95 * best, dt)

    def diffuse(self, f, dt, D, euler):
        C = self.coefs(D)
        if self.c["subcycles"]:
            for _ in range(self.c["subcycles"]):
                f = self.sts(f, dt / self.c["subcycles"], euler, C)
            return f
        done, d, i = 0.0, 0.0, 1
        while True:
            d = self.ptl(f, d, C)
            last = done + d >= dt or i == 59
            if last:
                d = dt - done
            f = self.sts(f, d, euler, C)
            done, i = done + d, i + 1
            if last:
                return f

    # -- advection
    def upwind(self, v, hi, lo):
        return v * torch.where(v >= 0, lo, hi)

    def face(self, LN, LP, W, eps):
        """Face values from LN at cells -2, -1, 0, LP at cells -1, 0, 1; W, eps at cells -1 and 0."""
        (cp1, mc1, _, _, p1, mct1), (cp0, mc0, m0, cpt0, _, _) = W
        t = (mc1 * (LN[1] - LN[0]), cp1 * (LN[2] - LN[1]), cp0 * (LP[2] - LP[1]), mc0 * (LP[1] - LP[0]))
        e = [(x + 4.0 * y * y) ** 2 for x, y in zip((eps[0], eps[0], eps[1], eps[1]), t)]
        wa, wb, wc, wd = p1 / e[0], mct1 / e[1], m0 / e[2], cpt0 / e[3]
        um = (wa * (LN[1] + t[0]) + wb * (mc0 * LN[1] + cp1 * LN[2])) / (wa + wb)
        up = (wc * (LP[1] - t[2]) + wd * (cp1 * LP[1] + mc0 * LP[0])) / (wc + wd)
        return um + up

    def adv(self, x, fl):
        vt, at, vp, ap = fl
        n = self.ntm
        if self.c["adv"] <= 2:
            ft = self.upwind(vt[..., 1:n], x[..., 1:], x[..., :-1])
            fp = self.upwind(vp, x, x.roll(1, 1))[..., 1:-1]
        else:
            LN, LP = 0.5 * x * (vt[..., :n] + at), 0.5 * x * (vt[..., 1:] - at)
            cut = lambda w, o: [q[o:o + n - 3] for q in w]
            mid = self.face([LN[..., o:o + n - 3] for o in (0, 1, 2)], [LP[..., o:o + n - 3] for o in (1, 2, 3)],
                            (cut(self.wt, 1), cut(self.wt, 2)), (self.dt[1:n - 2], self.dt[2:n - 1]))
            ft = torch.cat([self.upwind(vt[..., 1:2], x[..., 1:2], x[..., :1]), mid,
                            self.upwind(vt[..., n - 1:n], x[..., n - 1:], x[..., n - 2:n - 1])], 2)
            LN, LP = (0.5 * x * (vp + ap))[..., 1:-1], (0.5 * x * (vp.roll(-1, 1) - ap))[..., 1:-1]
            col = lambda w: [q[:, None] for q in w]
            fp = self.face([LN.roll(2, 1), LN.roll(1, 1), LN], [LP.roll(1, 1), LP, LP.roll(-1, 1)],
                           (col([q.roll(1, 0) for q in self.wp]), col(self.wp)),
                           (self.dp.roll(1, 0)[:, None], self.dp[:, None]))
        s = self.sti[1:-1]
        flux = self.sth[1:-1] * ft
        y = (flux[..., 1:] - flux[..., :-1]) * s / self.dt[1:-1] + (fp.roll(-1, 1) - fp) * s / self.dp[:, None]
        north = (ft[..., 0] * self.dp).sum(1) * (2.0 / (math.pi * self.dth[1]))
        south = -(ft[..., -1] * self.dp).sum(1) * (2.0 / (math.pi * self.dth[-2]))
        return torch.cat([north[:, None, None].expand(-1, self.n2, 1), y, south[:, None, None].expand(-1, self.n2, 1)], 2)

    def advect(self, f, dt, fl):
        L = lambda x: self.adv(x, fl)
        if self.c["adv"] == 1:
            return f - dt * L(f)
        if self.c["adv"] in (2, 3):
            a = f - dt * L(f)
            a = 0.75 * f + 0.25 * a - 0.25 * dt * L(a)
            return f / 3.0 + 2.0 / 3.0 * a - 2.0 / 3.0 * dt * L(a)
        a = f - 0.5 * dt * L(f)
        a = a - 0.5 * dt * L(a)
        a = 2.0 / 3.0 * f + a / 3.0 - dt / 6.0 * L(a)
        return a - 0.5 * dt * L(a)

    def step(self, f, dt, D, fl):
        h = 0.5 * dt if self.c["strang"] else dt
        if fl is not None:
            f = self.advect(f, h, fl)
        if self.c["ragged"]:
            f = torch.cat([self.diffuse(f[i:i + 1], dt, D[i:i + 1], self.euler_dt(i)) for i in range(self.nr)])
        else:
            f = self.diffuse(f, dt, D, self.euler_dt())
        return self.advect(f, h, fl) if fl is not None and self.c["strang"] else f

    def areas(self):
        """get_flux's cell areas of the columns 1..npm-1, (npm - 1, ntm)."""
        m = self.np_mesh
        a = m["st"] * m["dt"]
        a[0] = 0.25 * math.sin(0.5 * (m["t"][0] + m["t"][1])) * m["dth"][1]
        a[-1] = 0.25 * math.sin(0.5 * (m["t"][-1] + m["t"][-2])) * m["dth"][-2]
        b = np.concatenate([[0.5 * m["dph"][-1]], m["dp"][:-1], [0.5 * m["dph"][-1]]])
        return self.T(b[:, None] * a[None, :])


def _full(core):
    return torch.cat([core[:, -1:], core, core[:, :1]], 1)


def exact(case, seed):
    c = _case(**case)
    cells = c["nt"] * c["np"] * c["nr"]
    if cells > (3.0e5 if c["kind"] in ("gradient", "autograd") else 4.0e7):
        return None  # too long, or too much memory, in plain torch
    prm = _params(c)
    S = Scheme(c, prm)
    f0 = S.T(S.load(_map(c, seed)))[:, 1:-1].contiguous()
    dt = _dt(c, prm)
    D = S.T(prm["D"])
    if c["kind"] == "assimilate":
        d, w, mu = (S.T(x) for x in _observation(c, seed))
        f = _full(f0)
        w = torch.where(mu > 0.1, mu, torch.zeros_like(mu)) ** 4
        delta = (w * (d - f[:, :-1].transpose(1, 2))).transpose(1, 2)
        delta = _full(delta[:, 1:])
        if c["balance"]:
            fl = delta[:, :-1] * S.areas()
            r = torch.sqrt((fl.clamp(min=0.0).sum((1, 2)) / fl.clamp(max=0.0).sum((1, 2))).abs())[:, None, None]
            delta = torch.where(delta > 0, delta / r, delta * r)
        return dict(field=f + delta, history=None)
    if c["kind"] in ("step", "cycle"):
        with torch.no_grad():
            f = S.step(f0, dt, D, None if c["flow"] == "none" else S.flows(f0))
        out = dict(field=_full(f))
        return dict(out, history=None, limit=None) if c["kind"] == "cycle" else out
    lead = {k: S.T(v).requires_grad_(True) for k, v in prm.items()}
    x = f = f0.clone().requires_grad_(True)
    fl = S.flows(None, lead)
    for _ in range(c["steps"]):
        f = torch.utils.checkpoint.checkpoint(S.step, f, dt, lead["D"], fl, use_reentrant=False)
    r = _full(f) - S.T(_target(c, _full(f0).cpu().numpy()))
    loss = (r ** 2).mean() if c["kind"] == "autograd" else 0.5 * (S.areas() * r[:, :-1] ** 2).sum()
    loss.backward()
    z = torch.zeros_like(x.grad[:, :1])
    out = dict(f0=torch.cat([z, x.grad, z], 1), **{k: lead[k].grad for k in ("D", "p1", "p2", "p3", "p4")})
    return dict(out, field=_full(f.detach())) if c["kind"] == "autograd" else dict(out, loss=float(loss.detach()))
