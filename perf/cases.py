"""What a user of this framework has it do, as cases that can be timed.

Kinds of case:

  start     host arrays to a first step and back: init_profile with
            Navier-Stokes shear, step, max_temperature, get_state
  step      device-resident state: set the state, take `steps` steps (one
            call, or one call and a max-temperature read per step as the
            reference's main loop makes them), read the state
  batch     an ensemble of boost-invariant events: init every event, run,
            read every event and its observables
  adjoint   eps_p after `steps` steps and its gradients
  freezeout the surface swept by `steps` steps and the spectrum it emits

Inputs are made here from the seed: a lumpy fireball on a floor (or the
Cartesian shock tube), already flowing and sheared, as in the middle of a
run.  exact() is the same step in plain torch, 64 bits.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from viral_b200 import _abi as A
from viral_b200.batch import Batch
from viral_b200.configs import eos_table
from viral_b200.hydro import A_QGP, HBARC, Config, Hydro, cooper_frye_2d_device, cooper_frye_3d_device

NG = 3
F64 = torch.float64
SIDES = (64, 96, 128, 160, 200)  # the ensemble's grid sides

# Arithmetic of one cell, counted on the scheme itself: per direction 23 WENO5
# stencils (both faces, about 50 operations each) and the fluxes; per stage
# the shear and geometric sources and about 2.5 Newton steps of the 4x4
# root-find.  A generalized-minmod stencil costs about 12 operations.
WENO_FLOPS, MINMOD_FLOPS, UPDATE_FLOPS = 23 * 50 + 80, 19 * 12 + 4 * 50 + 80, 1300


def _case(name, kind, nx, ny, nz, steps, **more):
    c = dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, steps=steps, mixed=False, minmod=False, cart=False,
             table=True, mirror=False, read=False, events=0, every=0)
    c.update(more)
    return c


def listed():
    return [
        # the smallest call there is: a 33x33 Gubser grid from host arrays, one step, the result back
        _case("start_33", "start", 33, 33, 0, 1, table=False, mirror=True),
        # the reference's Gubser test at its size, main-loop style: a step, then the maximum temperature
        _case("gubser_129", "step", 129, 129, 0, 10, table=False, mirror=True, read=True),
        # one boost-invariant event at the ensemble's largest side, single precision state
        _case("event_200_mixed", "step", 200, 200, 0, 20, mixed=True),
        # the headline event, in double precision and in the mixed mode
        _case("glauber_161x161x41", "step", 161, 161, 41, 4),
        _case("glauber_161x161x41_mixed", "step", 161, 161, 41, 4, mixed=True),
        # the reference's Cartesian shock tube: thin and long
        _case("shocktube_10x10x101", "step", 10, 10, 101, 5, cart=True, table=False),
        # the generalized-minmod option on a ragged grid
        _case("minmod_97x61x23", "step", 97, 61, 23, 4, minmod=True),
        # a large event on sizes that divide by nothing
        _case("large_257x251x63", "step", 257, 251, 63, 2),
        # an ensemble: 20 events of the five sides, mixed precision
        _case("ensemble_20", "batch", 0, 0, 0, 48, mixed=True, events=20),
        # sensitivities of eps_p, boost-invariant and 3+1D
        _case("adjoint_128", "adjoint", 128, 128, 0, 50, every=25),
        _case("adjoint_97x97x33", "adjoint", 97, 97, 33, 6, every=3),
        # analysis after the evolution: the surface of a few steps and its spectrum
        _case("freezeout_121x121x31", "freezeout", 121, 121, 31, 3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step2", "step2", "step3", "step3", "step3", "cart", "minmod", "start", "batch", "adjoint",
                       "adjoint3", "freezeout"])
    mixed = rng.random() < 0.5
    if kind == "start":
        return _drawn("start", _log(rng, 10, 200), _log(rng, 10, 200), 0, rng.randint(1, 5), table=False,
                      mirror=rng.random() < 0.5)
    if kind == "step2":
        return _drawn("step", _log(rng, 16, 600), _log(rng, 16, 600), 0, rng.randint(2, 20), mixed=mixed,
                      table=rng.random() < 0.7, read=rng.random() < 0.4)
    if kind == "step3":
        return _drawn("step", _log(rng, 20, 250), _log(rng, 20, 250), _log(rng, 7, 60), rng.randint(1, 3), mixed=mixed,
                      table=rng.random() < 0.7, read=rng.random() < 0.3)
    if kind == "cart":
        return _drawn("step", _log(rng, 8, 100), _log(rng, 8, 100), _log(rng, 20, 200), rng.randint(1, 4), mixed=mixed,
                      cart=True, table=False)
    if kind == "minmod":
        three = rng.random() < 0.7
        return _drawn("step", _log(rng, 16, 200), _log(rng, 16, 200), _log(rng, 7, 50) if three else 0,
                      rng.randint(1, 4), mixed=mixed, minmod=True)
    if kind == "batch":
        return _drawn("batch", 0, 0, 0, rng.randint(16, 48), mixed=mixed, events=rng.randint(3, 20))
    if kind == "adjoint":
        return _drawn("adjoint", _log(rng, 24, 160), _log(rng, 24, 160), 0, rng.randint(8, 50),
                      every=rng.randint(5, 25))
    if kind == "adjoint3":
        return _drawn("adjoint", _log(rng, 16, 97), _log(rng, 16, 97), _log(rng, 7, 33), rng.randint(2, 6),
                      every=rng.randint(2, 6))
    three = rng.random() < 0.6
    return _drawn("freezeout", _log(rng, 100, 161), _log(rng, 100, 161), _log(rng, 9, 41) if three else 0,
                  rng.randint(1, 5))


def _drawn(*a, **k):
    c = _case("", *a, **k)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs

def _config(c, nx=None, ny=None):
    bi = c["nz"] == 0
    return Config(nx=nx or c["nx"], ny=ny or c["ny"], nz=1 if bi else c["nz"], boost_invariant=bi,
                  coords=A.COORD_CARTESIAN if c["cart"] else A.COORD_MILNE,
                  precision=A.PREC_MIXED if c["mixed"] else A.PREC_FP64,
                  recon=A.RECON_MINMOD if c["minmod"] else A.RECON_WENO5, dx=0.1, dy=0.1,
                  dz=0.1 if c["cart"] else 0.25, tau0=1.0, dtau=0.01 if c["mirror"] or c["cart"] else 0.02,
                  eos_kind=A.EOS_TABLE if c["table"] else A.EOS_CONFORMAL,
                  eos_table=eos_table() if c["table"] else None, etas0=0.2 if c["mirror"] else 0.08,
                  etas1=1.0 if c["kind"] == "adjoint" else 0.0,
                  taupi_kind=A.TAUPI_5_ETA_OVER_EPP if c["mirror"] else A.TAUPI_15_ETA_OVER_P,
                  gubser_mirror=c["mirror"])


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _inputs(cfg, seed):
    """The 18 canonical fields (18, gz, gy, gx) of a lumpy, flowing, sheared event at cfg.tau0."""
    r = np.random.RandomState(seed % (1 << 31))
    dev = _dev()
    gx, gy, gz = cfg.gdims()
    cart = cfg.coords == A.COORD_CARTESIAN
    tau, dt = cfg.tau0, cfg.dtau
    ax = lambda n, h: (torch.arange(n, dtype=F64, device=dev) - n // 2) * h  # noqa: E731
    x, y, z = ax(gx, cfg.dx), ax(gy, cfg.dy), ax(gz, cfg.dz)
    X, Y, Z = x[None, None, :], y[None, :, None], z[:, None, None]
    one = torch.ones(gz, gy, gx, dtype=F64, device=dev)
    ph = r.uniform(0, 2 * math.pi, 8)
    amp = r.uniform(0.5, 1.0, 8)
    wig = (amp[0] * torch.sin(1.1 * X + 0.7 * Y + ph[0]) + amp[1] * torch.cos(0.8 * X - 1.3 * Y + 0.4 * Z + ph[1])) / 2
    if cart:
        # 16 : 1 across z = 0, with smooth structure on both sides
        e = torch.where(Z + 0 * one < 0, 16.0, 1.0) * (1 + 0.1 * wig)
        flow, p_scale = 0.02, 0.0
    else:
        npart = 180
        cx = torch.tensor(r.normal(0, 1.9, npart), dtype=F64, device=dev)
        cy = torch.tensor(r.normal(0, 2.6, npart), dtype=F64, device=dev)
        g = lambda s, c: torch.exp(-((s[None, :] - c[:, None]) ** 2) / (2 * 0.5 ** 2))  # noqa: E731
        e2 = g(y, cy).T @ g(x, cx)
        env = torch.exp(-torch.clamp(Z.abs() - 1.5, min=0) ** 2 / (2 * 1.3 ** 2))
        e = (0.5 + 25.0 * (e2 / e2.max())[None] * env * (1 + 0.05 * wig)) / cfg.hbarc
        flow, p_scale = 0.15, 0.5
    t2 = 1.0 if cart else tau * tau
    u1 = flow * (X / (1 + X.abs() / 6) + 0.2 * wig) + 0 * one
    u2 = flow * (Y / (1 + Y.abs() / 6) + 0.2 * amp[2] * torch.sin(0.9 * X + 0.5 * Y + ph[2])) + 0 * one
    if gz > 1:
        u3 = 0.05 / math.sqrt(t2) * (torch.tanh(Z + 0.1 * amp[3]) + 0.3 * wig) + 0 * one
    else:
        u3 = 0 * one
    u = torch.stack([torch.sqrt(1 + u1 * u1 + u2 * u2 + t2 * u3 * u3), u1, u2, u3])
    back = 1 - dt / (tau + 1)
    tp2 = 1.0 if cart else (tau - dt) ** 2
    v = u[1:] * back
    pu = torch.cat([torch.sqrt(1 + v[0] ** 2 + v[1] ** 2 + tp2 * v[2] ** 2)[None], v])
    P, _, T = _eos(cfg, e)
    eta = _etas(cfg, T, None) * (e + P) / T
    p = p_scale * 2 * eta / (3 * tau)
    cross = 0.0 if gz == 1 else 0.05
    pi = torch.stack([p * (1 + 0.1 * wig), p * (1 - 0.1 * wig), 0.05 * p * wig, cross * p * wig, -cross * p * wig])
    return torch.cat([e[None], u, pi, _tmunu(cfg, e, u, pi, t2), pu])


def _profile(cfg, seed):
    S = _inputs(cfg, seed).reshape(18, -1).cpu().numpy()
    return dict(e=S[0].copy(), ux=S[2].copy(), uy=S[3].copy(), pi5=S[5:10].copy(), prevu=S[14:18].copy())


def _sides(c):
    return [SIDES[k % len(SIDES)] for k in range(c["events"])]


# ------------------------------------------------------------------- cases

def prepare(case, seed):
    c = dict(case)
    s = {"case": c, "seed": seed}
    if c["kind"] == "batch":
        sides = _sides(c)
        cfg = _config(c, 64, 64)
        s["batch"] = Batch(cfg, sides, tau0=cfg.tau0, dtau=cfg.dtau, tau_max=15.0, t_freeze_gev=0.01)
        s["events"] = [_profile(_config(c, n, n), seed + 31 * k) for k, n in enumerate(sides)]
        return s
    cfg = _config(c)
    s["cfg"], s["tau"] = cfg, cfg.tau0
    s["h"] = Hydro(cfg)
    if c["kind"] == "start":
        s["profile"] = _profile(cfg, seed)
        return s
    s["state"] = _inputs(cfg, seed).reshape(18, -1).contiguous()
    s["out"] = torch.empty_like(s["state"])
    if c["kind"] == "freezeout":
        # an isotherm inside the fireball's range of temperatures, and the bins of a pion spectrum
        s["t_fo"] = 0.2 / cfg.hbarc
        s["rows"] = (cfg.nx - 1) * (cfg.ny - 1) * (1 if c["nz"] == 0 else 4 * (cfg.nz - 1))
        s["pt"] = np.linspace(0.2, 3.0, 8) / cfg.hbarc
        s["phi"] = np.arange(16) * (2 * math.pi / 16)
    return s


def _fields(S, mixed):
    """The state by tensor group; a mixed handle's values are single precision numbers."""
    S = S.float() if mixed else S
    return {"e": S[0], "u": S[1:5], "pi": S[5:10], "T": S[10:14], "prevu": S[14:18]}


def _set(s):
    A.check(A.lib().vh_set_state_device(s["h"].h, ctypes.c_void_p(s["state"].data_ptr()), s["tau"]), s["h"].h)


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "batch":
        return _run_batch(s)
    h = s["h"]
    if kind == "start":
        p = s["profile"]
        h.init_profile(s["tau"], p["e"], p["ux"], p["uy"], None, p["prevu"], A.PI_NS)
        h.step(c["steps"])
        return {"tmax": h.max_temperature(), **_fields(h.get_state(), False)}
    _set(s)
    if kind == "step":
        out = {}
        if c["read"]:
            for _ in range(c["steps"]):
                h.step(1)
                out["tmax"] = h.max_temperature()
        else:
            h.step(c["steps"])
        A.check(A.lib().vh_get_state_device(h.h, ctypes.c_void_p(s["out"].data_ptr())), h.h)
        return {**out, **_fields(s["out"], c["mixed"])}
    if kind == "adjoint":
        eps, gs, ge, gc = h.adjoint_eps_p(c["steps"], c["every"])
        return {"eps_p": np.float64(eps), "grad_e0": ge, "grad_etas": gc,
                **{"grad_" + k: v for k, v in _fields(gs, False).items()}}
    h.freezeout_step(s["t_fo"])
    h.step(c["steps"])
    el = h.freezeout_step(s["t_fo"])
    spectrum = cooper_frye_2d_device if c["nz"] == 0 else cooper_frye_3d_device
    rap = () if c["nz"] == 0 else (0.0,)
    # as many rows for every event of this size, the surface's first
    rows = torch.zeros(s["rows"], el.shape[1], dtype=F64, device=el.device)
    rows[:el.shape[0]] = el[:s["rows"]]
    return {"count": el.shape[0], "elements": rows, "spectrum": spectrum(el, s["t_fo"], 0.14 / HBARC, 1.0, *rap, s["pt"], s["phi"])}


def _run_batch(s):
    b, c = s["batch"], s["case"]
    for k, p in enumerate(s["events"]):
        b.init_event(k, p["e"], p["ux"], p["uy"], p["prevu"], A.PI_GIVEN, p["pi5"])
    A.check(A.lib().vh_batch_reset(b.h))
    b.run(c["steps"])
    tau, steps, state = b.events()
    eps_p, eps_2 = b.observables()
    kind = np.float32 if c["mixed"] else np.float64
    out = {"tau": tau, "steps": steps, "state": state, "eps_p": eps_p.astype(kind), "eps_2": eps_2.astype(kind)}
    for k in range(b.n):
        out["event_%02d" % k] = b.event_state(k).astype(kind)
    return out


def _cells(c):
    if c["kind"] == "batch":
        return sum(SIDES[i % len(SIDES)] ** 2 for i in range(c["events"]))
    return c["nx"] * c["ny"] * max(1, c["nz"])


def work(case):
    c = dict(case)
    cells, dirs = _cells(c), 3 if c["nz"] else 2
    word = 4 if c["mixed"] else 8
    per_stage = dirs * (MINMOD_FLOPS if c["minmod"] else WENO_FLOPS) + UPDATE_FLOPS
    flops = 2.0 * cells * c["steps"] * per_stage
    # the state in and out of the call in double precision, and once in and
    # out of every step
    nbytes = cells * 36 * 8.0 + c["steps"] * cells * 36.0 * word
    if c["kind"] == "adjoint":
        # forward, recomputation and a reverse of about twice the forward
        flops *= 4
        nbytes *= 4
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------- the scheme in plain torch, 64 bits

def _table(cfg, dev):
    return torch.tensor(np.asarray(cfg.eos_table), dtype=F64, device=dev)


def _eos(cfg, e, slope=False):
    """P, c_s^2 and T of e; with slope, the derivative of P as interpolated in c_s^2's place."""
    if cfg.eos_kind == A.EOS_CONFORMAL:
        return e / 3, torch.full_like(e, 1 / 3), (e / cfg.eos_a) ** 0.25
    te, tp, tc, tt = _table(cfg, e.device)
    n = te.numel()
    i = torch.clamp(torch.searchsorted(te, e.detach().contiguous(), right=True) - 1, 0, n - 2)
    w = (e - te[i]) / (te[i + 1] - te[i])
    lin = lambda q: q[i] + w * (q[i + 1] - q[i])  # noqa: E731
    lo, hi = e <= te[0], e >= te[-1]
    quart = lambda a, b: b * torch.sqrt(torch.sqrt(torch.clamp(e, min=1e-300) / a))  # noqa: E731
    P = torch.where(lo, tc[0] * e, torch.where(hi, tp[-1] + tc[-1] * (e - te[-1]), lin(tp)))
    cs = (tp[i + 1] - tp[i]) / (te[i + 1] - te[i]) if slope else lin(tc)
    cs = torch.where(lo, tc[0], torch.where(hi, tc[-1], cs))
    T = torch.where(lo, quart(te[0], tt[0]), torch.where(hi, quart(te[-1], tt[-1]), lin(tt)))
    return P, cs, T


def _etas(cfg, T, par):
    c0, c1 = (cfg.etas0, cfg.etas1) if par is None else par
    return c0 + c1 * torch.clamp(T * cfg.hbarc - cfg.etas_tc, min=0)


def _pi4(u, p, t2):
    """The symmetric 4x4 shear tensor from its five evolved components."""
    u0, u1, u2, u3 = u
    D = u0 * u0 - t2 * u3 * u3
    Q = u1 * u1 * p[0] + 2 * u1 * u2 * p[2] + u2 * u2 * p[1] + 2 * t2 * u3 * (u1 * p[3] + u2 * p[4])
    tt = (Q - t2 * u3 * u3 * (p[0] + p[1])) / D
    ee = (Q - u0 * u0 * (p[0] + p[1])) / (t2 * D)
    tx = (p[0] * u1 + p[2] * u2 + p[3] * u3 * t2) / u0
    ty = (p[2] * u1 + p[1] * u2 + p[4] * u3 * t2) / u0
    te = (u1 * p[3] + u2 * p[4] + t2 * u3 * ee) / u0
    return [[tt, tx, ty, te], [tx, p[0], p[2], p[3]], [ty, p[2], p[1], p[4]], [te, p[3], p[4], ee]]


def _tmunu(cfg, e, u, pi, t2):
    P, _, _ = _eos(cfg, e)
    q = _pi4(u, pi, t2)
    ep = e + P
    return torch.stack([ep * u[0] * u[0] - P + q[0][0]] + [ep * u[0] * u[l] + q[0][l] for l in (1, 2, 3)])


def _weno(q):
    """Both face values of every 5-point stencil along the last axis: right face, left face."""
    a, b, c, d, f = (q[..., k:q.shape[-1] - 4 + k] for k in range(5))
    b0 = 13 / 12 * (c - 2 * d + f) ** 2 + 0.25 * (3 * c - 4 * d + f) ** 2
    b1 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b2 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    w0, w1, w2 = ((1e-6 + k) ** -2 for k in (b0, b1, b2))
    l0, l1, l2 = 0.3 * w0, 0.6 * w1, 0.1 * w2
    L = (l0 * (2 * c + 5 * d - f) + l1 * (-b + 5 * c + 2 * d) + l2 * (2 * a - 7 * b + 11 * c)) / (6 * (l0 + l1 + l2))
    r0, r1, r2 = 0.1 * w0, 0.6 * w1, 0.3 * w2
    R = (r0 * (11 * c - 7 * d + 2 * f) + r1 * (2 * b + 5 * c - d) + r2 * (-a + 5 * b + 2 * c)) / (6 * (r0 + r1 + r2))
    return L, R


def _minmod(q, th):
    b, c, d = (q[..., k:q.shape[-1] - 4 + k] for k in (1, 2, 3))
    s = [th * (c - b), 0.5 * (d - b), th * (d - c)]
    m = torch.minimum(torch.minimum(s[0].abs(), s[1].abs()), s[2].abs())
    ok = (s[0] * s[1] > 0) & (s[1] * s[2] > 0)
    m = torch.where(ok, torch.sign(s[0]) * m, torch.zeros_like(m))
    return c + 0.5 * m, c - 0.5 * m


class _Grid:
    def __init__(self, cfg):
        self.cfg = cfg
        self.gx, self.gy, self.gz = cfg.gdims()
        self.bi = cfg.boost_invariant
        self.cart = cfg.coords == A.COORD_CARTESIAN

    def inner(self, q):
        q = q[..., NG:-NG, NG:-NG]
        return q if self.bi else q[..., NG:-NG, :, :]

    def lines(self, q, d):
        """q with the lines along direction d last, interior across."""
        s = [slice(None) if self.bi else slice(NG, -NG), slice(NG, -NG), slice(NG, -NG)]
        s[2 - d] = slice(None)
        return q[(Ellipsis, *s)].transpose(-1, -1 - d)


def _sweep(G, d, e, u, pi, T, tau):
    """Flux divergence (9) and d_d u^mu (4) on the interior."""
    cfg, cart = G.cfg, G.cart
    h = (cfg.dx, cfg.dy, cfg.dz)[d]
    e, u, pi, T = G.lines(e, d), G.lines(u, d), G.lines(pi, d), G.lines(T, d)
    t2, tf = (1.0, 1.0) if cart else (tau * tau, tau)
    P, _, _ = _eos(cfg, e)
    q = _pi4(u, pi, t2)
    ep, un = e + P, u[1 + d]
    gi = (1.0, 1.0, 1.0 / t2)[d]
    F = [tf * (q[1 + d][l] + un * u[l] * ep + (P * gi if l == 1 + d else 0)) for l in range(4)]
    vf = un / u[0] * (tf if d == 2 else 1.0)
    F = torch.stack(F + [pi[l] * vf for l in range(5)])
    V = torch.cat([tf * T, pi])
    inside = torch.zeros(e.shape[-1], dtype=F64, device=e.device)
    inside[NG:-NG] = 1
    spd = vf * inside
    rec = (lambda x: _minmod(x, cfg.minmod_theta)) if cfg.recon == A.RECON_MINMOD else _weno
    (FL, FR), (VL, VR), (sL, sR) = rec(F), rec(V), rec(spd)
    amax = torch.maximum(sL[..., :-1].abs(), sR[..., 1:].abs())
    first = torch.ones(amax.shape[-1], dtype=F64, device=e.device)
    first[0] = 0  # the face left of the first interior cell has no dissipation
    amax = amax * first
    H = 0.5 * (FL[..., :-1] + FR[..., 1:]) - 0.5 * amax * (VR[..., 1:] - VL[..., :-1])
    uL, uR = _weno(u)
    du = ((uL - uR) / h)[..., 1:-1]
    return (-(H[..., 1:] - H[..., :-1]) / h).transpose(-1, -1 - d), du.transpose(-1, -1 - d)


def _shear(cart, tau, u, du):
    """sigma^{mu nu}, theta and a_mu of du[l][a] = d_a u^l."""
    t2 = 1.0 if cart else tau * tau
    g, gi = (1.0, -1.0, -1.0, -t2), (1.0, -1.0, -1.0, -1.0 / t2)
    Dm = [list(r) for r in du]
    if not cart:
        Dm[0][3] = Dm[0][3] + tau * u[3]
        Dm[3][0] = Dm[3][0] + u[3] / tau
        Dm[3][3] = Dm[3][3] + u[0] / tau
    R = range(4)
    Dl = [[g[b] * Dm[b][a] for b in R] for a in R]
    theta = sum(Dm[a][a] for a in R)
    Dt = [[(gi[a] if a == b else 0.0) - u[a] * u[b] for b in R] for a in R]
    tr = sum(Dt[a][b] * Dl[a][b] for a in R for b in R)
    S = [[0.5 * (Dl[a][b] + Dl[b][a]) for b in R] for a in R]
    M = [[sum(Dt[m][a] * S[a][b] for a in R) for b in R] for m in R]
    sig = [[sum(M[m][b] * Dt[v][b] for b in R) - Dt[m][v] * tr / 3 for v in R] for m in R]
    acc = [g[v] * sum(u[a] * Dm[v][a] for a in R) for v in R]
    return sig, theta, acc


def _source(G, e, u, p, du, tau, par):
    cfg, cart = G.cfg, G.cart
    t2 = 1.0 if cart else tau * tau
    P, _, T = _eos(cfg, e)
    eta = _etas(cfg, T, par) * (e + P) / T
    tp = 5 * eta / (e + P) if cfg.taupi_kind == A.TAUPI_5_ETA_OVER_EPP else 1.5 * eta / P
    q = _pi4(u, p, t2)
    sig, th, acc = _shear(cart, tau, u, du)
    pa = [sum(q[v][a] * acc[a] for a in range(4)) for v in range(4)]
    divv = sum(du[i][i] / u[0] - u[i] * du[0][i] / (u[0] * u[0]) for i in (1, 2, 3))
    out = []
    for m, v in ((1, 1), (2, 2), (1, 2), (1, 3), (2, 3)):
        rhs = -(q[m][v] - 2 * eta * sig[m][v]) / tp - 4 / 3 * q[m][v] * th - (u[m] * pa[v] + u[v] * pa[m])
        if not cart and v == 3:
            rhs = rhs - (u[0] * q[3][m] + u[3] * q[0][m]) / tau
        out.append(rhs / u[0] + q[m][v] * divv)
    s5 = torch.stack(out)
    if cart:
        if not G.bi:  # the last three interior z layers carry no shear source
            keep = torch.ones(s5.shape[-3], 1, 1, dtype=F64, device=e.device)
            keep[-NG:] = 0
            s5 = s5 * keep
        return torch.cat([torch.zeros_like(s5[:4]), s5])
    ep, zero = e + P, torch.zeros_like(e)
    geo = [-P - t2 * (q[3][3] + ep * u[3] * u[3]), zero, zero, -2 * (q[0][3] + ep * u[0] * u[3])]
    return torch.cat([torch.stack(geo), s5])


def _residual(cfg, T, p, t2, x, jac=False, slope=False):
    e, u1, u2, u3 = x
    P, a, _ = _eos(cfg, e, slope)
    W, X, Y, Z = T
    S = 1 + u1 * u1 + u2 * u2 + t2 * u3 * u3
    u0, ep = torch.sqrt(S), e + P
    y = [(W - e) * u0 - X * u1 - Y * u2 - t2 * Z * u3,
         X * u0 - e * u1 - u1 * (P + p[0] + ep * u1 * u1) - u2 * (p[2] + ep * u1 * u2) - t2 * u3 * (p[3] + ep * u1 * u3),
         Y * u0 - e * u2 - u1 * (p[2] + ep * u1 * u2) - u2 * (P + p[1] + ep * u2 * u2) - t2 * u3 * (p[4] + ep * u2 * u3),
         Z * u0 - p[3] * u1 - p[4] * u2 - u3 * (P + W - p[0] - p[1])]
    if not jac:
        return y
    k = 1 / u0
    J = [[-u0, (W - e) * u1 * k - X, (W - e) * u2 * k - Y, t2 * ((W - e) * u3 * k - Z)],
         [-(1 + a) * u1 * S, X * u1 * k - p[0] - ep * (S + 2 * u1 * u1), X * u2 * k - p[2] - 2 * ep * u1 * u2,
          t2 * (X * u3 * k - p[3] - 2 * ep * u1 * u3)],
         [-(1 + a) * u2 * S, Y * u1 * k - p[2] - 2 * ep * u1 * u2, Y * u2 * k - p[1] - ep * (S + 2 * u2 * u2),
          t2 * (Y * u3 * k - p[4] - 2 * ep * u2 * u3)],
         [-a * u3, Z * u1 * k - p[3], Z * u2 * k - p[4], t2 * Z * u3 * k - (P + W - p[0] - p[1])]]
    return y, J


def _solve(J, y):
    """J s = y by elimination, cell by cell (the Jacobian is dominated by its diagonal)."""
    M, b = [list(r) for r in J], list(y)
    for c in range(4):
        for r in range(c + 1, 4):
            m = M[r][c] / M[c][c]
            for k in range(c + 1, 4):
                M[r][k] = M[r][k] - m * M[c][k]
            b[r] = b[r] - m * b[c]
    for c in (3, 2, 1, 0):
        for k in range(c + 1, 4):
            b[c] = b[c] - M[c][k] * b[k]
        b[c] = b[c] / M[c][c]
    return b


def _root(G, T, p, e, u, tau):
    """e and u^mu of the conserved set; differentiable through one Newton step at the root."""
    t2 = 1.0 if G.cart else tau * tau
    with torch.no_grad():
        x = [e.detach(), u[1].detach(), u[2].detach(), u[3].detach()]
        Td, pd = T.detach(), p.detach()
        for _ in range(7):
            y, J = _residual(G.cfg, Td, pd, t2, x, True)
            s = _solve(J, y)
            x = [a - b for a, b in zip(x, s)]
        _, J = _residual(G.cfg, Td, pd, t2, x, True, True)
    y = _residual(G.cfg, T, p, t2, x)
    x = [a - b for a, b in zip(x, _solve(J, y))]
    u0 = torch.sqrt(1 + x[1] ** 2 + x[2] ** 2 + t2 * x[3] ** 2)
    return x[0], torch.stack([u0, x[1], x[2], x[3]])


def _ghosts(G, S, new):
    """S with the interior replaced by new and the face ghosts copied from it (corners keep their values)."""
    S = S.clone()
    z = slice(None) if G.bi else slice(NG, -NG)
    i = slice(NG, -NG)
    S[:, z, i, i] = new
    n = new.shape
    mir = G.cfg.gubser_mirror
    for m in range(NG):
        for at, frm, mfrm in ((m, 0, NG - 1 - m), (NG + n[3] + m, n[3] - 1, n[3] - 1 - m)):
            S[:, z, i, at] = new[..., frm]
            if mir:
                S[2:4, z, i, at] = new[2:4, ..., mfrm]
        for at, frm, mfrm in ((m, 0, NG - 1 - m), (NG + n[2] + m, n[2] - 1, n[2] - 1 - m)):
            S[:, z, at, i] = new[..., frm, :]
            if mir:
                S[2:4, z, at, i] = new[2:4, ..., mfrm, :]
        if not G.bi:
            S[:, m, i, i] = new[:, 0]
            S[:, NG + n[1] + m, i, i] = new[:, -1]
    return S


def _rhs(G, S, tau, par):
    e, u, pi, T, pu = S[0], S[1:5], S[5:10], S[10:14], S[14:18]
    ui = G.inner(u)
    zero = torch.zeros_like(ui[0])
    du = [[(ui[l] - G.inner(pu)[l]) / G.cfg.dtau, zero, zero, zero] for l in range(4)]
    div = 0
    for d in range(2 if G.bi else 3):
        r, g = _sweep(G, d, e, u, pi, T, tau)
        div = div + r
        for l in range(4):
            du[l][1 + d] = g[l]
    return div + _source(G, G.inner(e), ui, G.inner(pi), du, tau, par)


def _step(G, S, tau, par=None):
    ts, cart = G.cfg.dtau, G.cart
    t1 = tau + ts
    i = G.inner(S)
    tf, tn = (1.0, 1.0) if cart else (tau, t1)
    var0 = torch.cat([tf * i[10:14], i[5:10]])
    var1 = var0 + ts * _rhs(G, S, tau, par)
    T, p = var1[:4] / tn, var1[4:]
    e, u = _root(G, T, p, i[0], i[1:5], t1)
    S1 = _ghosts(G, S, torch.cat([e[None], u, p, T, i[1:5]]))
    var2 = 0.5 * var0 + 0.5 * var1 + 0.5 * ts * _rhs(G, S1, t1, par)
    T, p = var2[:4] / tn, var2[4:]
    e2, u2 = _root(G, T, p, e, u, t1)
    return _ghosts(G, S1, torch.cat([e2[None], u2, p, T, i[1:5]]))


def _evolve(G, S, tau, steps):
    with torch.no_grad():
        for _ in range(steps):
            S = _step(G, S, tau)
            tau += G.cfg.dtau
    return S


def _tmax(G, S):
    return float(_eos(G.cfg, G.inner(S[0]))[2].max() * G.cfg.hbarc)


def _ns_state(cfg, seed):
    """The boost-invariant state init_profile makes with Navier-Stokes shear: gradients where their stencils
    fit on interior rows and columns, zero elsewhere."""
    S = _inputs(cfg, seed)
    e, pu = S[0], S[14:18]
    u = torch.stack([torch.sqrt(1 + S[2] ** 2 + S[3] ** 2), S[2], S[3], torch.zeros_like(e)])
    zero = torch.zeros_like(u)
    dt, dx, dy = zero.clone(), zero.clone(), zero.clone()
    i, m = slice(NG, -NG), slice(2, -2)
    dt[:, :, i, i] = ((u - pu) / cfg.dtau)[:, :, i, i]
    L, R = _weno(u)
    dx[:, :, i, m] = ((L - R) / cfg.dx)[:, :, i, :]
    L, R = _weno(u.transpose(-1, -2))
    dy[:, :, m, i] = ((L - R) / cfg.dy).transpose(-1, -2)[:, :, :, i]
    du = [[dt[l], dx[l], dy[l], zero[l]] for l in range(4)]
    sig, _, _ = _shear(False, cfg.tau0, u, du)
    P, _, T = _eos(cfg, e)
    eta = _etas(cfg, T, None) * (e + P) / T
    pi = torch.stack([2 * eta * sig[a][b] for a, b in ((1, 1), (2, 2), (1, 2), (1, 3), (2, 3))])
    return torch.cat([e[None], u, pi, _tmunu(cfg, e, u, pi, cfg.tau0 ** 2), pu])


def _exact_adjoint(c, cfg, seed):
    G = _Grid(cfg)
    S0 = _inputs(cfg, seed).requires_grad_()
    de = torch.zeros_like(S0[0]).requires_grad_()
    par = [torch.tensor(v, dtype=F64, device=S0.device, requires_grad=True) for v in (cfg.etas0, cfg.etas1)]
    t2 = cfg.tau0 ** 2
    e, u, pi = S0[0].detach(), S0[1:5].detach(), S0[5:10].detach()
    dT = _tmunu(cfg, e + de, u, pi, t2) - _tmunu(cfg, e, u, pi, t2)
    S = torch.cat([(S0[0] + de)[None], S0[1:10], S0[10:14] + dT, S0[14:]])
    tau = cfg.tau0
    for _ in range(c["steps"]):
        S = checkpoint(_step, G, S, tau, par, use_reentrant=False)
        tau += cfg.dtau
    e, u, pi = G.inner(S[0]), G.inner(S[1:5]), G.inner(S[5:10])
    P, _, _ = _eos(cfg, e)
    txx, tyy = (e + P) * u[1] ** 2 + P + pi[0], (e + P) * u[2] ** 2 + P + pi[1]
    eps = (txx - tyy).sum() / (txx + tyy).sum()
    gs, ge, g0, g1 = torch.autograd.grad(eps, [S0, de, *par])
    n = ge.numel()
    return {"eps_p": np.float64(float(eps)), "grad_e0": ge.reshape(n).cpu().numpy(),
            "grad_etas": np.array([float(g0), float(g1)]),
            **{"grad_" + k: v for k, v in _fields(gs.reshape(18, n).cpu().numpy(), False).items()}}


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "freezeout":
        return None  # a list of surface elements
    if kind == "batch":
        sides = _sides(c)
        cfg = _config(c, 64, 64)
        n = len(sides)
        tau = cfg.tau0
        for _ in range(c["steps"]):
            tau += cfg.dtau
        out = {"tau": np.full(n, tau), "steps": None, "state": None, "eps_p": None, "eps_2": None}
        for side in sorted(set(sides)):
            ks = [k for k, v in enumerate(sides) if v == side]
            ecfg = _config(c, side, side)
            G = _Grid(ecfg)
            S = _evolve(G, torch.cat([_inputs(ecfg, seed + 31 * k) for k in ks], 1), cfg.tau0, c["steps"])
            for a, k in enumerate(ks):
                out["event_%02d" % k] = S[:, a].reshape(18, -1)
        return out
    cfg = _config(c)
    G = _Grid(cfg)
    if kind == "adjoint":
        return _exact_adjoint(c, cfg, seed)
    S = _ns_state(cfg, seed) if kind == "start" else _inputs(cfg, seed)
    S = _evolve(G, S, cfg.tau0, c["steps"])
    out = {"tmax": _tmax(G, S)} if kind == "start" or c["read"] else {}
    return {**out, **_fields(S.reshape(18, -1), False)}
