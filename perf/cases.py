"""The work that users of this package have it do, as cases that can be timed.

A case is one of three kinds:

* ``run``: one mesh advanced by some cycles, in one of the three precisions,
  through ``Hydro.run`` (``"step": False``, a captured run between two reports) or
  ``Hydro.cycle`` (``"step": True``, a driver that looks at every cycle's scalars).
  Every pass restarts from the same state (``copy_state_from``), so a pass is the
  same work however often it is made.
* ``batch``: independent meshes of uneven size advanced together (``Batch.run``),
  then read back.  A batch has no restart: it goes on from pass to pass.
* ``train``: Adam steps of the closure network from given weights
  (``Closure.set``, ``Closure.train``, ``Closure.get``).

The start states of ``run`` are self-similar flows in mid-course rather than the
decks' initial states, in which nearly all zones are at rest: a blast wave that has
crossed part of the mesh (Sedov), a shock tube with its fan, contact and shock
apart (Leblanc), and an implosion with its standing shock (Noh).
"""
import functools
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "pennant-legion_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import pennant_b200 as pb  # noqa: E402

GAMMA = 5.0 / 3.0
SSMIN = 0.1
ALFA = 0.5
CFL, CFLV, DTFAC = 0.6, 0.1, 1.2
# steps larger than this would let the smallest instances of a batch run away
# from the largest ones, whose steps are about as long
BATCH_DTMAX = 5.0e-5
CLOSURE = os.path.join(_PKG, "closure", "qcs_mlp.bin")
FIELDS = ("px", "pu", "zr", "ze", "zp", "zetot")
BATCH_FIELDS = ("px", "pu", "zr", "ze")


def listed():
    return [
        # the CPU-sized blast of the decks: a few launches of a few blocks each, so latency
        {"name": "sedov48_fp64", "kind": "run", "mesh": "rect", "flow": "sedov", "nx": 48, "ny": 48, "precision": "fp64", "cycles": 256, "step": False},
        # the drop-in size: the whole state fits the L2 cache
        {"name": "sedov480_fp64", "kind": "run", "mesh": "rect", "flow": "sedov", "nx": 480, "ny": 480, "precision": "fp64", "cycles": 64, "step": False},
        # the headline mesh in each of the three precisions
        {"name": "sedov1920_fp64", "kind": "run", "mesh": "rect", "flow": "sedov", "nx": 1920, "ny": 1920, "precision": "fp64", "cycles": 16, "step": False},
        {"name": "sedov1920_mixed", "kind": "run", "mesh": "rect", "flow": "sedov", "nx": 1920, "ny": 1920, "precision": "mixed", "cycles": 16, "step": False},
        {"name": "sedov1920_learned", "kind": "run", "mesh": "rect", "flow": "sedov", "nx": 1920, "ny": 1920, "precision": "learned", "cycles": 16, "step": False},
        # the shock tube: long rows, and a large share of compressing corners for the network
        {"name": "leblanc2880_mixed", "kind": "run", "mesh": "rect", "flow": "leblanc", "nx": 2880, "ny": 288, "precision": "mixed", "cycles": 16, "step": False},
        {"name": "leblanc2880_learned", "kind": "run", "mesh": "rect", "flow": "leblanc", "nx": 2880, "ny": 288, "precision": "learned", "cycles": 16, "step": False},
        # a mesh with triangles and without the rectangle's numbering: the general kernels
        {"name": "noh_pie_fp64", "kind": "run", "mesh": "pie", "flow": "noh", "nx": 313, "ny": 801, "precision": "fp64", "cycles": 16, "step": False},
        # a driver that steps cycle by cycle, on a ragged mesh
        {"name": "noh_square_step", "kind": "run", "mesh": "rect", "flow": "noh", "nx": 131, "ny": 77, "precision": "mixed", "cycles": 64, "step": True},
        # parameter studies: many meshes of uneven size at once
        {"name": "batch12_fp64", "kind": "batch", "count": 12, "nmin": 32, "nmax": 512, "precision": "fp64", "cycles": 128},
        {"name": "batch12_mixed", "kind": "batch", "count": 12, "nmin": 48, "nmax": 384, "precision": "mixed", "cycles": 128},
        # the closure network's training
        {"name": "train_closure", "kind": "train", "rows": 32768, "steps": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    what = rng.random()
    if what < 0.1:
        return {"kind": "train", "rows": _log(rng, 1024, 65536), "steps": rng.randint(4, 16)}
    if what < 0.25:
        nmin = _log(rng, 24, 96)
        return {"kind": "batch", "count": rng.randint(2, 12), "nmin": nmin, "nmax": nmin * rng.randint(2, 5), "precision": rng.choice(["fp64", "mixed"]), "cycles": 128}
    if what < 0.4:
        nx, ny = _log(rng, 12, 600), _log(rng, 24, 1200)
        case = {"kind": "run", "mesh": "pie", "flow": "noh", "nx": nx, "ny": ny, "precision": "fp64"}
    else:
        flow = rng.choice(["sedov", "sedov", "leblanc", "noh"])
        nx = _log(rng, 32, 1700)
        ny = max(4, nx // rng.randint(6, 14)) if flow == "leblanc" else max(16, int(nx * rng.uniform(0.5, 1.2)))
        if flow == "leblanc":
            nx, ny = nx + 200, ny + 20
        case = {"kind": "run", "mesh": "rect", "flow": flow, "nx": nx, "ny": ny, "precision": rng.choice(["fp64", "mixed", "learned"])}
    zones = case["nx"] * case["ny"]
    case["cycles"] = 256 if zones < 5000 else 64 if zones < 250000 else 16
    case["step"] = zones < 50000 and rng.random() < 0.3
    return case


# --------------------------------------------------------------------------
# Meshes and start states
# --------------------------------------------------------------------------

def _lengths(case):
    nx, ny = case["nx"], case["ny"]
    if case["flow"] == "leblanc":
        return 9.0, 9.0 * ny / nx
    side = 1.125 if case["flow"] == "sedov" else 1.0
    return side, side * ny / nx


def _deck_text(case, dt0, precision):
    nx, ny = case["nx"], case["ny"]
    if case["mesh"] == "pie":
        mesh = f"meshtype pie\nmeshparams {nx} {ny}\nbcx 0.0\nbcy 0.0\n"
    else:
        lx, ly = _lengths(case)
        mesh = f"meshtype rect\nmeshparams {nx} {ny} {lx!r} {ly!r}\n"
        mesh += "bcx 0.0\nbcy 0.0\n" if case["flow"] == "noh" else f"bcx 0.0 {lx!r}\nbcy 0.0 {ly!r}\n"
    if case["flow"] == "leblanc":
        mesh += f"subregion 3.0 9.0  0.0 {_lengths(case)[1]!r}\nrinit 1.0\nrinitsub 1.0e-3\n"
    q1, q2 = _viscosity(case)
    return (f"{mesh}tstop 1.0e9\nssmin {SSMIN}\nq1 {q1}\nq2 {q2}\nalfa {ALFA}\ncfl {CFL}\ncflv {CFLV}\ndtfac {DTFAC}\n"
            f"dtinit {dt0!r}\ndtmax {_dtmax(case)!r}\ndtreport 100\nprecision {precision}\n")


def _dtmax(case):
    """A bound on the step that keeps small meshes, whose steps are long, from running the flow on
    until its waves have crossed the mesh several times."""
    return {"sedov": 0.3, "noh": 0.15, "leblanc": 0.8}[case["flow"]] / case["cycles"]


def _viscosity(case):
    return (0.3, 2.0) if case["flow"] == "leblanc" else (0.1, 1.0)


@functools.lru_cache(maxsize=4)
def _mesh(text):
    return pb.Mesh(deck=pb.Deck(text=text))


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _connect(case):
    """Point coordinates [np][2] of the undeformed mesh and its zones, as groups of
    (first zone, points of each zone's sides [n][3 or 4])."""
    dev = _device()
    nx, ny = case["nx"], case["ny"]
    f64 = dict(dtype=torch.float64, device=dev)
    if case["mesh"] == "rect":
        lx, ly = _lengths(case)
        i = torch.arange(nx + 1, **f64) * (lx / nx)
        j = torch.arange(ny + 1, **f64) * (ly / ny)
        x = torch.stack([i[None, :].expand(ny + 1, -1), j[:, None].expand(-1, nx + 1)], -1).reshape(-1, 2).contiguous()
        z = torch.arange(nx * ny, device=dev)
        p = z // nx * (nx + 1) + z % nx
        return x, [(0, torch.stack([p, p + 1, p + nx + 2, p + nx + 1], 1))]
    # pie: the origin, then rings of nx + 1 points from the top down; the inner zones are triangles
    th = (math.pi / 2 / nx) * torch.arange(nx, -1, -1, **f64)
    r = torch.arange(1, ny + 1, **f64) * (1.0 / ny)
    ring = torch.stack([r[:, None] * torch.cos(th)[None], r[:, None] * torch.sin(th)[None]], -1).reshape(-1, 2)
    x = torch.cat([torch.zeros(1, 2, **f64), ring])
    i = torch.arange(nx, device=dev)
    tri = torch.stack([torch.zeros_like(i), i + 2, i + 1], 1)
    z = torch.arange(nx * (ny - 1), device=dev)
    p = z // nx * (nx + 1) + z % nx + 1
    quad = torch.stack([p, p + 1, p + nx + 2, p + nx + 1], 1)
    return x, [(0, tri)] + ([(nx, quad)] if ny > 1 else [])


def _cross(a, b):
    return a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]


def _dot(a, b):
    return (a * b).sum(-1)


def _geometry(x):
    """Centres, side areas and side volumes of zones whose corners are x [n][sides][2]."""
    zx = x.sum(1) / x.shape[1]
    x2 = x.roll(-1, 1)
    sa = 0.5 * _cross(x2 - x, zx[:, None] - x)
    return zx, sa, sa * (x[..., 0] + x2[..., 0] + zx[:, None, 0]) / 3


def _profile(case, seed, x0):
    """Position and velocity of the points, and pressure and a scale of its zones' signal
    speed as functions of the zone centre: a self-similar flow at a time drawn from the seed."""
    rng = np.random.default_rng([int(seed), case["nx"], case["ny"]])
    flow = case["flow"]
    if flow == "leblanc":
        # gamma = 5/3 shock tube: fan, contact and shock of the exact solution
        t, cl, us, shock, tail, ps = float(rng.uniform(1.0, 2.5)), 1.0 / 3.0, 0.62183, 0.8291, 0.4958, 5.154e-4
        X = x0[:, 0] - 3.0
        a = (-X).clamp(min=1e-30)
        ta = a / cl
        xi_head, xi_inf = -cl, 2 * cl / (GAMMA - 1)
        xi = xi_inf + (xi_head - xi_inf) * (t / ta).clamp(min=1.0) ** -0.25
        tb = ta * ((xi_inf - tail) / (xi_inf - xi_head)) ** -4.0   # leaves the fan at its tail
        left = torch.where(t <= ta, X, torch.where(t < tb, xi * t, tail * tb + us * (t - tb)))
        ul = torch.where(t <= ta, torch.zeros_like(X), torch.where(t < tb, 0.75 * (cl + xi), torch.full_like(X, us)))
        ts = X / shock
        right = torch.where(ts < t, X + us * (t - ts), X)
        ur = torch.where(ts < t, torch.full_like(X, us), torch.zeros_like(X))
        x = torch.stack([3.0 + torch.where(X < 0, left, right), x0[:, 1]], 1)
        # the far walls do not move
        u = torch.stack([torch.where(X < 0, ul, ur), torch.zeros_like(X)], 1)

        def pressure(zx, zr):
            s = (zx[:, 0] - 3.0) / t
            fan = (0.75 * (cl + s)).clamp(0.0, us)
            pl = (2.0 / 3.0 * 0.1) * (1 - (GAMMA - 1) / 2 * fan / cl) ** 5
            return torch.where(s < tail, pl, torch.where(s < shock, torch.full_like(s, ps), torch.full_like(s, 2.0 / 3.0 * 1e-10)))
        return x, u, pressure
    r0 = x0.norm(dim=1)
    dirn = x0 / r0.clamp(min=1e-30)[:, None]
    if flow == "noh":
        t = float(rng.uniform(0.1, 0.4))
        amp = float(rng.uniform(0.95, 1.05))
        inside = r0 < 4 * t / 3
        x = dirn * torch.where(inside, r0 / 4, r0 - t)[:, None]
        u = -amp * dirn * (~inside & (r0 > 0))[:, None]

        def pressure(zx, zr):
            return torch.where(zx.norm(dim=1) < t / 3, (GAMMA - 1) * 0.5 * zr, torch.zeros_like(zr))
        return x, u, pressure
    # Sedov: r / R = (r0 / R)^(1/4) is the mapping whose density, rho0 times 4 (r / R)^9, jumps by 4
    lim = min(_lengths(case))
    R, D = float(rng.uniform(0.4, 0.75)) * lim, float(rng.uniform(0.8, 1.2))
    phase = float(rng.uniform(0, 2 * math.pi))
    inside = r0 < R
    x = torch.where(inside[:, None], dirn * (R * (r0 / R) ** 0.25)[:, None], x0)
    rr = x.norm(dim=1) / R
    ang = torch.atan2(x0[:, 1], x0[:, 0])
    u = torch.where(inside[:, None], dirn * (0.75 * D * rr * (1 + 0.03 * torch.cos(4 * ang + phase)))[:, None], torch.zeros_like(x))

    def pressure(zx, zr):
        s = zx.norm(dim=1) / R
        return torch.where(s < 1, 0.75 * D * D * (0.35 + 0.65 * s.clamp(max=1.0) ** 6), torch.zeros_like(s))
    return x, u, pressure


def _start(case, seed):
    """The start state of a ``run`` case and its first step."""
    x0, groups = _connect(case)
    x, u, pressure = _profile(case, seed, x0)
    if case["mesh"] == "pie":   # points on the axes move along them
        axis = x0.abs() < 1e-12
    else:
        lx, ly = _lengths(case)
        far = torch.tensor([lx, ly], dtype=torch.float64, device=x0.device)
        axis = (x0.abs() < 1e-12) | ((x0 - far).abs() < 1e-12) if case["flow"] != "noh" else x0.abs() < 1e-12
    x = torch.where(axis, x0, x)
    u = torch.where(axis, torch.zeros_like(u), u)
    nz = sum(len(g) for _, g in groups)
    zm, zvol = (torch.zeros(nz, dtype=torch.float64, device=x.device) for _ in range(2))
    zx = torch.zeros(nz, 2, dtype=torch.float64, device=x.device)
    smf, edge = [], []
    for z0, P in groups:
        zc, sa, sv = _geometry(x0[P])
        rho = torch.where(zc[:, 0] > 3.0 - 1e-12, 1e-3, 1.0) if case["flow"] == "leblanc" else torch.ones_like(zc[:, 0])
        zm[z0:z0 + len(P)] = rho * sv.sum(1)
        smf.append(sa / sa.sum(1, keepdim=True))
        zc, sa, sv = _geometry(x[P])
        zx[z0:z0 + len(P)] = zc
        zvol[z0:z0 + len(P)] = sv.sum(1)
        edge.append((2 * sa / (x[P].roll(-1, 1) - x[P]).norm(dim=2)).amin(1))
    zr = zm / zvol
    zp = pressure(zx, zr)
    ze = zp / ((GAMMA - 1) * zr)
    speed = torch.sqrt((GAMMA * zp / zr).clamp(min=SSMIN ** 2)).amax() + u.norm(dim=1).amax()
    dt0 = min(float(0.2 * torch.cat(edge).amin() / speed), _dtmax(case))
    return {"groups": groups, "x0": x0, "px": x, "pu": u, "zm": zm, "zr": zr, "ze": ze, "zp": zp, "zetot": ze * zm, "zvol": zvol,
            "zwrate": torch.zeros_like(zm), "smf": smf, "dt": dt0, "time": 0.0, "cycle": 0}


# --------------------------------------------------------------------------
# What a user's program has in hand, and one pass
# --------------------------------------------------------------------------

class _DeviceArray:
    """A field of a hydro object where it lies, for torch.as_tensor.  The tensor holds this object,
    and this one the hydro object, whose memory goes with it."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (ptr, False), "version": 3, "strides": None}


def _view(h, name):
    shape = (h.mesh.nump, 2) if name in ("px", "pu") else (h.mesh.numz,)
    return torch.as_tensor(_DeviceArray(h, h.device_ptr(name), shape), device="cuda")


def _batch_decks(case, seed):
    """Deck parameters of a batch's instances, Sedov blasts and square Noh implosions: the sizes are
    spread over the range by the case alone, energies and gammas come from the seed."""
    rng = np.random.default_rng([int(seed), case["count"], case["nmin"], case["nmax"]])
    out = []
    for k in range(case["count"]):
        f = (k + 0.5) / case["count"]
        n = int(round(case["nmin"] * (case["nmax"] / case["nmin"]) ** f))
        out.append({"n": n, "e0": float(rng.uniform(0.1, 1.0)), "gamma": float(rng.uniform(1.4, 5.0 / 3.0)), "noh": k % 3 == 2})
    return out


def _batch_deck_text(d, precision):
    n = d["n"]
    h = 1.125 / n
    text = f"tstop 1.0e9\nmeshtype rect\nmeshparams {n} {n} 1.125 1.125\nrinit 1.0\neinit 0.0\ngamma {d['gamma']!r}\n"
    if d["noh"]:
        text += f"uinitradial -1.0\nbcx 0.0\nbcy 0.0\ndtinit {0.05 * h!r}\n"
    else:
        einit = d["e0"] / (math.pi * h ** 3)
        text += (f"subregion 0.0 {h!r} 0.0 {h!r}\nrinitsub 1.0\neinitsub {einit!r}\nbcx 0.0 1.125\nbcy 0.0 1.125\n"
                 f"dtinit {_batch_dtinit(d)!r}\n")
    return text + (f"dtmax {BATCH_DTMAX!r}\nssmin {SSMIN}\nq1 0.1\nq2 1.0\nalfa {ALFA}\ncfl {CFL}\ncflv {CFLV}\n"
                   f"dtfac {DTFAC}\nprecision {precision}\n")


def _batch_dtinit(d):
    if d["noh"]:
        return 0.05 * (1.125 / d["n"])
    return min(1e-4, 1e-4 * (48.0 / d["n"]) ** 2.5 * math.sqrt(0.25 / d["e0"]))


def _train_data(case, seed):
    """Normalised inputs [n][16] (two columns of padding) and the targets of a smooth function of them."""
    g = torch.Generator(device=_device()).manual_seed(int(seed))
    n = case["rows"] * case["steps"]
    x = torch.randn(n, 16, generator=g, device=_device())
    x[:, 14:] = 0
    x = x.to(torch.bfloat16)
    a = torch.randn(14, 4, generator=g, device=_device()) * 0.4
    f = x[:, :14].float()
    t = torch.tanh(f @ a) + 0.2 * (f[:, :4] * f[:, 4:8])
    r = np.random.default_rng(int(seed))
    params = np.concatenate([(r.uniform(-1, 1, s) * math.sqrt(6.0 / w)).astype(np.float32)
                             for s, w in ((64 * 14, 78), (64, 1e9), (64 * 64, 128), (64, 1e9), (4 * 64, 68), (4, 1e9))])
    return x.contiguous(), t.contiguous(), params


LEARNING_RATE = 1.0e-3


def prepare(case, seed):
    if case["kind"] == "train":
        x, t, params = _train_data(case, seed)
        return {"case": case, "closure": pb.Closure(seed=1), "x": x, "t": t, "params": params}
    if case["kind"] == "batch":
        decks = [pb.Deck(text=_batch_deck_text(d, case["precision"])) for d in _batch_decks(case, seed)]
        return {"case": case, "batch": pb.Batch([pb.Mesh(deck=d) for d in decks], [d.params() for d in decks])}
    s = _start(case, seed)
    mesh = _mesh(_deck_text({**case, "cycles": 1}, 1.0, "fp64"))   # the mesh depends on neither the steps nor their number
    ref = pb.Hydro(mesh, pb.Deck(text=_deck_text(case, s["dt"], "fp64")).params())
    for name in ("px", "pu", "zm", "zr", "ze", "zp", "zetot", "zvol", "zwrate"):
        ref.upload(name, s[name].cpu().numpy())
    h = pb.Hydro(mesh, pb.Deck(text=_deck_text(case, s["dt"], case["precision"])).params())
    if case["precision"] == "learned":
        h.set_closure(pb.Closure(path=CLOSURE))
    return {"case": case, "start": ref, "hydro": h}


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        c = state["closure"]
        c.set(params=state["params"])
        n = case["rows"] * case["steps"]
        losses = c.train(state["x"].data_ptr(), state["t"].data_ptr(), n, 0, case["steps"], case["rows"], LEARNING_RATE)
        return {"params": c.get()[0], "losses": losses}
    if case["kind"] == "batch":
        b = state["batch"]
        b.run(case["cycles"])
        return [{name: b.download(i, name) for name in BATCH_FIELDS} for i in range(len(b.meshes))]
    h = state["hydro"]
    h.copy_state_from(state["start"])
    if case["step"]:
        for _ in range(case["cycles"]):
            sc = h.cycle()
    else:
        sc = h.run(case["cycles"])
    out = {name: _view(h, name) for name in FIELDS}
    out["time"], out["dt"], out["cycle"] = sc["time"], sc["dt"], sc["cycle"]
    return out


def work(case):
    """Bytes: per cycle each point's position and velocity and each zone's mass, volume, work rate,
    energy and side mass fractions read once, and the new state (with density, specific energy and
    pressure) written once.  Operations: about 900 a zone and cycle (predictor 600, corrector 200,
    points 50, and their share of divisions and roots as one each)."""
    if case["kind"] == "train":
        n = case["rows"] * case["steps"]
        return {"bytes": n * (16 * 2 + 4 * 4), "flops": n * 6 * (14 * 64 + 64 * 64 + 64 * 4)}
    if case["kind"] == "batch":
        zones = sum(d["n"] ** 2 for d in _batch_decks(case, 0))
        points = sum((d["n"] + 1) ** 2 for d in _batch_decks(case, 0))
        sides = 4 * zones
    else:
        nx, ny = case["nx"], case["ny"]
        zones = nx * ny
        points = (nx + 1) * (ny + 1) if case["mesh"] == "rect" else (nx + 1) * ny + 1
        sides = 4 * zones - (nx if case["mesh"] == "pie" else 0)
    cycles = case["cycles"]
    return {"bytes": cycles * (64 * points + 80 * zones + 8 * sides), "flops": cycles * 900 * zones}


# --------------------------------------------------------------------------
# The same in plain torch and 64 bits
# --------------------------------------------------------------------------

def _cycle(s, planes, c):
    """One cycle of the staggered-grid Lagrangian scheme: predictor, point update, corrector, next dt."""
    dt, dth = s["dt"], 0.5 * s["dt"]
    px0, pu0 = s["px"], s["pu"]
    pxp = px0 + dth * pu0
    mass, force = torch.zeros_like(px0[:, 0]), torch.zeros_like(px0)
    gm1 = c["gamma"] - 1
    zp_new, total, dtn = s["zp"].clone(), [], math.inf
    for (z0, P), mf in zip(s["groups"], s["smf"]):
        z = slice(z0, z0 + len(P))
        n = P.shape[1]
        x, u = pxp[P], pu0[P]
        zx, sa, sv = _geometry(x)
        zu = u.sum(1) / n
        xn, un = x.roll(-1, 1), u.roll(-1, 1)
        area, vol = sa.sum(1), sv.sum(1)
        elen = (xn - x).norm(dim=2)
        zdl = (n * sa / elen).amin(1)
        zr, zm = s["zr"][z], s["zm"][z]
        e = s["ze"][z].clamp(min=0)
        p, per = gm1 * zr * e, gm1 * zr
        csq = (gm1 * e + per * p / zr ** 2).clamp(min=max(SSMIN ** 2, 1e-99))
        ss = csq.sqrt()
        dv = (vol - s["zvol"][z]) / zm
        zp = p + (per * (s["zwrate"][z] * dth / zm) - zr * (zr * csq) * dv) / (1 + 0.5 * per * dv)
        rho = zm / vol
        zp_new[z] = zp
        cm = (rho * area * 0.5)[:, None] * (mf + mf.roll(1, 1))
        ex = 0.5 * (x + xn)
        d = ex - zx[:, None]
        surf = torch.stack([-d[..., 1], d[..., 0]], -1)
        fp = -zp[:, None, None] * surf
        tts = ALFA * ss.clamp(min=SSMIN) ** 2
        ft = -(tts[:, None] * (rho[:, None] * mf * (area[:, None] / sa) - rho[:, None]))[..., None] * surf
        # artificial viscosity at each corner
        zc, zuc = zx[:, None].expand_as(x), zu[:, None].expand_as(u)
        up, xm, uprev = x.roll(1, 1), ex.roll(1, 1), u.roll(1, 1)   # previous point, previous side's middle
        e1, e2 = elen.roll(1, 1), elen
        u1, u3 = 0.5 * (u + un), 0.5 * (uprev + u)
        cvol = 0.5 * _cross(zc - x, xm - ex)
        v1, v2 = xm - x, ex - x
        emin = torch.minimum(e1, e2)
        cc = torch.where(emin < 1e-12, 0.0, 4 * _dot(v1, v2) / (e1 * e2))
        div = (_cross(zuc - u, xm - ex) - _cross(u3 - u1, zc - x)) / (2 * cvol)
        a1, a2 = 0.5 * (ex + zc - x - xm), 0.5 * (zc + xm - x - ex)
        l1, l2 = a1.norm(dim=2), a2.norm(dim=2)
        ua = 0.25 * (u + u1 + zuc + u3)
        first = (_dot(a1, ua) * l2).abs() > (_dot(a2, ua) * l1).abs()
        ev = torch.minimum((4 * cvol * torch.where(first, l1 / l2, l2 / l1)).clamp(min=0).sqrt(), 2 * emin)
        w1, w2 = u1 + zuc - u - u3, zuc + u3 - u - u1
        du = torch.maximum(_dot(w1, w1), _dot(w2, w2)).sqrt()
        k2, k1 = c["q2"] * 0.25 * (5.0 / 3.0 + 1) * du, (c["q1"] * ss)[:, None]
        mu = torch.where(div < 0, (k2 + (k2 * k2 + k1 * k1).sqrt()) * rho[:, None] * ev, 0.0)
        f1, f2 = (mu / e1)[..., None] * (u - uprev), (mu / e2)[..., None] * (un - u)
        sin2 = 1 - cc * cc
        flat = sin2 < 1e-4
        cw = torch.where(flat, 0.0, cvol / torch.where(flat, 1.0, sin2))[..., None]
        cc = torch.where(flat, 0.0, cc)[..., None]
        A, B = cw * (f2 + cc * f1), cw * (f1 + cc * f2)
        fpq = fp + (A + B.roll(-1, 1)) / elen[..., None]
        tot = fpq + ft
        corner = tot - tot.roll(1, 1)
        mass.index_add_(0, P.reshape(-1), cm.reshape(-1))
        force.index_add_(0, P.reshape(-1), corner.reshape(-1, 2))
        dux = torch.where(elen > 0, _dot(un - u, xn - x).abs() / elen, 0.0).amax(1)
        zdu = c["q1"] * ss + 2 * c["q2"] * dux
        dtn = min(dtn, float((zdl * CFL / torch.maximum(zdu, ss.clamp(min=1e-99))).amin()))
        total.append(fpq)
    ub = torch.where(planes, 0.0, pu0)
    acc = torch.where(planes, 0.0, force) / mass.clamp(min=1e-99)[:, None]
    pu = ub + acc * dt
    px = px0 + 0.5 * dt * (ub + pu)
    zvol, zetot, zwrate = s["zvol"].clone(), s["zetot"].clone(), s["zwrate"].clone()
    for (z0, P), f in zip(s["groups"], total):
        z = slice(z0, z0 + len(P))
        vol = _geometry(px[P])[2].sum(1)
        us, xh = (ub + pu)[P], pxp[P][..., 0]
        dw = (-dth * (_dot(f, us) * xh - _dot(f, us.roll(-1, 1)) * xh.roll(-1, 1))).sum(1)
        zwrate[z] = (dw + zp_new[z] * (vol - zvol[z])) / dt
        zetot[z] += dw
        zvol[z] = vol
    dvov = float(((zvol - s["zvol"]) / s["zvol"]).abs().amax())
    rec = min(dtn, dt * CFLV / max(dvov, 1e-99))
    s.update(px=px, pu=pu, zp=zp_new, zvol=zvol, zetot=zetot, zwrate=zwrate, zr=s["zm"] / zvol, ze=zetot / (s["zm"] + 1e-99),
             time=s["time"] + dt, last=dt, dt=min(c["dtmax"], DTFAC * dt, rec), cycle=s["cycle"] + 1)


def _planes(x0, far):
    """Which components of the points' velocities the reflecting walls hold."""
    held = x0.abs() < 1e-12
    return held if far is None else held | ((x0 - torch.tensor(far, dtype=torch.float64, device=x0.device)).abs() < 1e-12)


def exact(case, seed):
    """The same in 64 bits.  The learned cycle stands for the cycle with the plain viscosity, so that is
    what it is compared with."""
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "batch":
        out = []
        for d in _batch_decks(case, seed):
            n, lx = d["n"], 1.125
            flat = {"mesh": "rect", "flow": "sedov", "nx": n, "ny": n}
            x0, groups = _connect(flat)
            _, sa, sv = _geometry(x0[groups[0][1]])
            vol = sv.sum(1)
            ze = torch.zeros_like(vol)
            r = x0.norm(dim=1, keepdim=True)
            pu = torch.where(r > 1e-12, -x0 / r.clamp(min=1e-30), 0.0) if d["noh"] else torch.zeros_like(x0)
            if not d["noh"]:
                ze[0] = d["e0"] / (math.pi * (lx / n) ** 3)
            s = {"groups": groups, "px": x0, "pu": pu, "zm": vol, "zr": torch.ones_like(vol), "ze": ze, "zp": torch.zeros_like(vol),
                 "zetot": ze * vol, "zvol": vol, "zwrate": torch.zeros_like(vol), "smf": [sa / sa.sum(1, keepdim=True)],
                 "dt": min(BATCH_DTMAX, _batch_dtinit(d)), "time": 0.0, "cycle": 0}
            c = {"gamma": d["gamma"], "q1": 0.1, "q2": 1.0, "dtmax": BATCH_DTMAX}
            planes = _planes(x0, None if d["noh"] else (lx, lx))
            for _ in range(case["cycles"]):
                _cycle(s, planes, c)
            out.append({name: s[name] for name in BATCH_FIELDS})
        return out
    s = _start(case, seed)
    q1, q2 = _viscosity(case)
    c = {"gamma": GAMMA, "q1": q1, "q2": q2, "dtmax": _dtmax(case)}
    planes = _planes(s["x0"], None if case["mesh"] == "pie" or case["flow"] == "noh" else _lengths(case))
    for _ in range(case["cycles"]):
        _cycle(s, planes, c)
    out = {name: s[name] for name in FIELDS}
    out["time"], out["dt"], out["cycle"] = s["time"], s["last"], s["cycle"]
    return out


def _exact_train(case, seed):
    x, t, params = _train_data(case, seed)
    dev = x.device
    shapes = [(64, 14), (64,), (64, 64), (64,), (4, 64), (4,)]
    ws, at = [], 0
    for sh in shapes:
        n = math.prod(sh)
        ws.append(torch.tensor(params[at:at + n].reshape(sh), dtype=torch.float64, device=dev, requires_grad=True))
        at += n
    m, v = [torch.zeros_like(w) for w in ws], [torch.zeros_like(w) for w in ws]
    losses = []
    for k in range(case["steps"]):
        rows = slice(k * case["rows"], (k + 1) * case["rows"])
        h = x[rows, :14].double()
        for i in (0, 2):
            h = torch.nn.functional.gelu(h @ ws[i].T + ws[i + 1], approximate="tanh")
        loss = ((h @ ws[4].T + ws[5] - t[rows].double()) ** 2).mean()
        losses.append(float(loss.detach()))
        grads = torch.autograd.grad(loss, ws)
        with torch.no_grad():
            for w, g, a, b in zip(ws, grads, m, v):
                a.mul_(0.9).add_(g, alpha=0.1)
                b.mul_(0.999).addcmul_(g, g, value=0.001)
                w -= LEARNING_RATE * (a / (1 - 0.9 ** (k + 1))) / ((b / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"params": torch.cat([w.detach().reshape(-1) for w in ws]), "losses": torch.tensor(losses, dtype=torch.float64)}
