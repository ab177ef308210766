"""Performance cases of the framework: what is timed when a kernel changes.

Each case is a plain dict; ``listed()`` gives the fixed ones, ``draw(rng)``
one more of the same ranges.  ``prepare`` makes what a program holds before
the call (inputs from the seed, the simulation or the network), ``run`` is one
pass through the public entry points, ``work`` the bytes and operations the
pass cannot do without, ``exact`` the same outputs in 64 bits from plain torch.

Kinds of case:
  steps     NuOsc.step_rk4 / evolve on one grid (FV or FD, both precisions)
  cycle     the driver's loop body: evolve, then analyse and P_ee(v)
  ensemble  many uneven FV simulations advanced together
  forward   one surrogate network on a batch of host rows
  train     one epoch of surrogate training over resident data
"""
import ctypes
import math
import random

import numpy as np
import torch

from cosenu_b200 import NuOsc, make_params
from cosenu_b200 import _lib as L
from cosenu_b200.ensemble import Ensemble, Instance
from cosenu_b200.surrogate import MLP

CFL = 0.4
LR = 2e-4  # late in the surrogate's cosine schedule from 2e-3


def _grid(kind, scheme, nz, nvz, steps, half=600.0, precision="fp64", bc="periodic", omega=0.0,
          mat=False, fd_advec="center", ko=3, tilt=0.3):
    """A simulation case.  tilt: size of the flavour rotation already there
    (0: a fresh start, only the 1e-6 seed noise; else a run resumed from a
    checkpoint in its nonlinear phase, with structure down to single cells)."""
    return {"kind": kind, "scheme": scheme, "nz": nz, "nvz": nvz, "steps": steps, "half": half,
            "precision": precision, "bc": bc, "omega": omega, "mat": mat, "fd_advec": fd_advec,
            "ko": ko, "tilt": tilt}


def listed():
    cases = {
        # the C++ driver's own pattern: one step_rk4() per loop iteration on a
        # small grid; a handful of launches and nothing else
        "fv_one_step": _grid("steps", "fv", 600, 32, 1),
        # the repository's small FV workload, the distance between two analyses
        "fv_1024x64": _grid("steps", "fv", 1024, 64, 100, tilt=0.0),
        # the default job grid with vacuum oscillations, the driver's whole
        # loop body: a stretch of steps, the two tables' rows, P_ee(v)
        "fv_default_cycle": _grid("cycle", "fv", 2400, 32, 50, omega=1e-2),
        # a mid-size FV production run
        "fv_8192x128": _grid("steps", "fv", 8192, 128, 10),
        # the largest FV workload
        "fv_65536x512": _grid("steps", "fv", 65536, 512, 2),
        # the FP32-bulk option on a large FV grid
        "fv_bulk_16384x256": _grid("steps", "fv", 16384, 256, 6, precision="fp32"),
        # a small FD run on ragged sizes (z tiles of 8, odd row count)
        "fd_1000x37": _grid("steps", "fd", 1000, 37, 50, omega=1e-2),
        # FD's other switches: open boundary, matter term, lopsided stencil,
        # KO5, sizes that divide nothing
        "fd_open_4000x100": _grid("steps", "fd", 4000, 100, 20, bc="open", omega=1e-2, mat=True,
                                  fd_advec="lopsided", ko=5),
        # the benchmark grid at its analysis cadence
        "fd_32768x256_cycle": _grid("cycle", "fd", 32768, 256, 40, half=3000.0, omega=1e-3),
        # the same grid with the FP32-bulk option
        "fd_bulk_32768x256": _grid("steps", "fd", 32768, 256, 20, half=3000.0, precision="fp32",
                                   omega=1e-3, tilt=0.0),
        # a share of the ensemble workload: uneven grids run to a common time
        "ensemble_16": {"kind": "ensemble", "members": 16, "nz_max": 4096, "mix": 5,
                        "reach": 3.75},
        # surrogate training: one epoch, minibatches of 64, a ragged last one
        "train_2000": {"kind": "train", "rows": 2000, "batch": 64},
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choices(["fv", "fd", "cycle", "ensemble", "forward", "train"],
                       [5, 4, 2, 1, 1, 1])[0]
    if kind == "ensemble":
        return {"kind": "ensemble", "members": rng.randint(3, 16),
                "nz_max": 256 * rng.randint(4, 16), "mix": rng.randrange(1 << 20),
                "reach": rng.uniform(1.0, 3.75)}
    if kind == "forward":
        return {"kind": "forward", "rows": int(_log(rng, 1, 4096))}
    if kind == "train":
        return {"kind": "train", "rows": rng.randint(200, 2000),
                "batch": rng.choice([32, 50, 64, 128, 256])}
    scheme = kind if kind != "cycle" else rng.choice(["fv", "fd"])
    nz = 8 * int(_log(rng, 16, 8192))
    if rng.random() < 0.5 and nz >= 256:
        nz = nz // 256 * 256
    nvz = int(_log(rng, 8, 512))
    cells = nz * nvz
    # up to the work of the largest listed case
    most = (1 << 26) if scheme == "fv" else (1 << 28)
    steps = max(1, min(rng.choice([1, 5, 20, 50, 100]), most // cells))
    # a cycle is repeated on its own state for long, and its analysis rejects a
    # state that has run away: closed boundary and the stable stencils only
    cycle = kind == "cycle"
    fd = scheme == "fd"
    return _grid("cycle" if cycle else "steps", scheme, nz, nvz, steps,
                 half=min(600.0, nz / 4.0),  # cells of at most half a length unit
                 precision=rng.choice(["fp64", "fp64", "fp32"]),
                 bc="periodic" if cycle else rng.choice(["periodic"] * 3 + ["open"]),
                 omega=rng.choice([0.0, 1e-3, 1e-2]), mat=rng.random() < 0.2,
                 fd_advec=rng.choice(["center"] * 3 + ([] if cycle else ["upwind"]) +
                                     ["lopsided"]) if fd else "center",
                 ko=rng.choice([3, 3, 5]) if fd and not cycle else 3,
                 tilt=0.3 if cycle else rng.choice([0.0, 0.3]))


# -- inputs ---------------------------------------------------------------------

THETA = 37.0  # mixing angle, degrees


def _gauss(v, sigma):
    n = sigma * math.sqrt(math.pi / 2.0) * (math.erf(2.0 / sigma / math.sqrt(2.0)))
    return torch.exp(-(v - 1.0) ** 2 / (2.0 * sigma * sigma)) / n


def _state(nz, nvz, half, tilt, seed, sig=0.6, sigb=0.5, alpha=0.9):
    """Interior state [8][nvz][nz] on the GPU and the two angular profiles:
    Gaussian profiles about v = 1 and per-cell noise of 1e-6, or for tilt > 0 a
    smooth rotation of the flavour vectors over a few wavelengths and noise of
    2e-2."""
    dev = "cuda"
    gen = torch.Generator(device=dev).manual_seed(seed)
    f64 = {"dtype": torch.float64, "device": dev}
    v = -1.0 + (torch.arange(nvz, **f64) + 0.5) * (2.0 / nvz)
    z = -half + (torch.arange(nz, **f64) + 0.5) * (2.0 * half / nz)
    st = torch.empty((8, nvz, nz), **f64)
    amp = 2e-2 if tilt else 1e-6
    profiles = (_gauss(v, sig), alpha * _gauss(v, sigb))
    for s, g in enumerate(profiles):
        ph = torch.rand(6, generator=gen, **f64) * 2.0 * math.pi
        k = math.pi / half
        angle = tilt * (torch.sin(3 * k * z + ph[0]) + 0.5 * torch.sin(11 * k * z + ph[1]))
        angle = angle[None, :] * (1.0 + 0.3 * v[:, None])
        phase = 2.0 * torch.sin(5 * k * z + ph[2])[None, :] + v[:, None] * ph[3]
        noise = torch.rand((2, nvz, nz), generator=gen, **f64).mul_(2 * amp).sub_(amp)
        ex = torch.sin(angle) * torch.cos(phase) + noise[0]
        ey = torch.sin(angle) * torch.sin(phase) + noise[1]
        ez = torch.sqrt(1.0 - ex * ex - ey * ey)
        h = 0.5 * g[:, None]
        st[4 * s + 0] = h * (1.0 + ez)
        st[4 * s + 1] = h * (1.0 - ez)
        st[4 * s + 2] = h * ex
        st[4 * s + 3] = h * ey
    return st, profiles


def _upload(sim, st):
    """Interior state from device memory (cosenu_upload_device)."""
    torch.cuda.synchronize()
    rc = sim.lib.cosenu_upload_device(sim.h, L.DPTR8(*[st[c].data_ptr() for c in range(8)]),
                                      st.shape[2])
    if rc != L.OK:
        raise RuntimeError(f"upload: {rc}")
    sim.synchronize()


class _Device:
    """Device memory of a simulation; whoever holds it keeps the owner alive."""

    def __init__(self, owner, ptr, shape, strides):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False),
                                         "strides": strides, "version": 3}


_STREAM = []


def _stream():
    """The program's one CUDA stream: whatever a program advances next waits
    for what it queued before."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0].cuda_stream


class _View:
    """Zero-copy torch view of a simulation's current state
    (cosenu_device_state); the address may alternate between steps."""

    def __init__(self, sim, owner=None):
        self.sim, self.owner = sim, owner or sim
        self.ptrs, self.ld, self.seen = L.DPTR8(), ctypes.c_int(), {}

    def __call__(self):
        s = self.sim
        s.lib.cosenu_device_state(s.h, self.ptrs, ctypes.byref(self.ld))
        t = self.seen.get(self.ptrs[0])
        if t is None:
            t = torch.as_tensor(_Device(self.owner, self.ptrs[0], (8, s.nvz, s.nz),
                                        (self.ptrs[1] - self.ptrs[0], self.ld.value * 8, 8)),
                                device="cuda")
            self.seen[self.ptrs[0]] = t
        return t


def _members(case):
    """Members of the ensemble workload's distribution, run to a common time
    (steps in proportion to nz)."""
    r = random.Random(case["mix"])
    out = []
    for i in range(case["members"]):
        nz = 256 * max(2, round(_log(r, 512, case["nz_max"]) / 256))
        steps = max(1, math.ceil(case["reach"] * nz / (CFL * 1200.0) - 1e-9))
        out.append(Instance(nz, r.choice((32, 64, 128, 256)), r.uniform(0.6, 1.2),
                            r.uniform(0.4, 0.8), r.uniform(0.3, 0.7), r.uniform(0.5, 2.0),
                            seed=i, nsteps=steps, index=i))
    return out


def _member_state(x, seed, i):
    return _state(x.nz, x.nvz, 600.0, 0.3 * (i % 2), 1000 * seed + i, x.sig_nu, x.sig_nubar,
                  x.alpha)


# surrogate network: 258 -> 3 x 512 -> 128, the library's flat parameter layout
DIMS = [(272, 512), (512, 512), (512, 512), (512, 128)]
NIN = 258


def _net_inputs(rows, seed):
    """Weights U(+-1/sqrt(fan_in)), standardised features, P_ee(v)-like targets
    (float32, host)."""
    r = np.random.default_rng(seed)
    flat = []
    for k, (i, o) in enumerate(DIMS):
        fan = NIN if k == 0 else i
        w = r.uniform(-1.0, 1.0, (o, i)).astype(np.float32) / np.float32(math.sqrt(fan))
        if k == 0:
            w[:, NIN:] = 0.0
        flat += [w.ravel(), np.zeros(o, np.float32)]
    x = r.normal(size=(rows, NIN)).astype(np.float32)
    c = r.normal(size=(NIN, 128)) / math.sqrt(NIN)
    t = (0.6 + 0.3 * np.tanh(x.astype(np.float64) @ c)).astype(np.float32)
    return np.concatenate(flat), x, t


# -- the passes -----------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "train"):
        w, x, t = _net_inputs(case["rows"], seed)
        net = MLP(NIN, 512, 3, 128, seed=0)
        net.set_params(w)
        if kind == "train":
            net.set_data(x, t)
        return {"case": case, "net": net, "x": x, "seed": seed % 1000 + 1}
    if kind == "ensemble":
        xs = _members(case)
        ens = Ensemble(xs)
        ens.set_stream(_stream())
        for i, (m, x) in enumerate(zip(ens.members, xs)):
            st, _ = _member_state(x, seed, i)
            _upload(m, st)
        return {"case": case, "ens": ens, "views": [_View(m, ens) for m in ens.members]}
    sim = NuOsc(_params(case))
    sim.set_stream(_stream())
    st, (g, bg) = _state(case["nz"], case["nvz"], case["half"], case["tilt"], seed)
    _upload(sim, st)
    if kind == "cycle":
        sim.set_profile(*[np.repeat(a.cpu().numpy()[:, None], sim.ld, axis=1) for a in (g, bg)])
        sim.mark_state0()
        sim.synchronize()
    return {"case": case, "sim": sim, "view": _View(sim)}


def _params(case):
    return make_params(nz=case["nz"], nvz=case["nvz"], gz=4, z0=-case["half"], z1=case["half"],
                       cfl=CFL, pmo=1.0, omega=case["omega"], theta_deg=THETA, mu=1.0,
                       scheme=case["scheme"], bc=case["bc"], mat=case["mat"],
                       fd_advec=case["fd_advec"], ko_order=case["ko"],
                       precision=case["precision"])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forward":
        return state["net"].forward(state["x"])
    if kind == "train":
        net = state["net"]
        losses = net.train(epochs=1, batch=case["batch"], lr=LR, seed=state["seed"])
        return {"losses": losses, "params": net.params()}
    if kind == "ensemble":
        state["ens"].run()
        return [v() for v in state["views"]]
    sim = state["sim"]
    if case["steps"] == 1:
        sim.step_rk4()
    else:
        sim.evolve(case["steps"])
    if kind == "steps":
        return state["view"]()
    diag = sim.analyse()
    pee, pbee = sim.pee_v()
    return {"state": state["view"](), "diag": diag, "pee": pee, "pbee": pbee}


def work(case):
    """Bytes: inputs read once, outputs written once (the state in and out, 64
    bytes per cell each way; the analysis reads the initial state too).
    Operations: the right-hand side and the combine of four stages."""
    kind = case["kind"]
    if kind in ("forward", "train"):
        rows = case["rows"]
        macs = sum(i * o for i, o in DIMS)
        if kind == "forward":
            return {"bytes": 4 * rows * (NIN + 128) + 4 * macs, "flops": 2 * rows * macs}
        return {"bytes": 4 * rows * (NIN + 128) + 6 * 4 * macs, "flops": 6 * rows * macs}
    per = {"fv": 4 * 1100, "fd": 4 * 300}
    if kind == "ensemble":
        xs = _members(case)
        return {"bytes": sum(128 * x.cells for x in xs),
                "flops": sum(per["fv"] * x.cells * x.nsteps for x in xs)}
    cells = case["nz"] * case["nvz"]
    return {"bytes": cells * (128 + (64 if kind == "cycle" else 0)),
            "flops": cells * case["steps"] * per[case["scheme"]]}


# -- the same in 64 bits ----------------------------------------------------------

def _pad(u, bc, h=4):
    if bc == "periodic":
        return torch.cat([u[..., -h:], u, u[..., :h]], dim=-1)
    right = [2.0 * u[..., -1:] - u[..., -2:-1]]
    right.append(2.0 * right[0] - u[..., -1:])
    while len(right) < h:
        right.append(2.0 * right[-1] - right[-2])
    return torch.cat([u[..., :1]] * h + [u] + right, dim=-1)


def _weno(a, b, c, d, e, f, g):
    """Seventh-order WENO value at the right face of the stencil's centre d."""
    eps = 1e-6
    s0 = d * (2107 * d - 9402 * e + 7042 * f - 1854 * g) + e * (11003 * e - 17246 * f + 4642 * g) \
        + f * (7043 * f - 3882 * g) + 547 * g * g
    s1 = c * (547 * c - 2522 * d + 1922 * e - 494 * f) + d * (3443 * d - 5966 * e + 1602 * f) \
        + e * (2843 * e - 1642 * f) + 267 * f * f
    s2 = b * (267 * b - 1642 * c + 1602 * d - 494 * e) + c * (2843 * c - 5966 * d + 1922 * e) \
        + d * (3443 * d - 2522 * e) + 547 * e * e
    s3 = a * (547 * a - 3882 * b + 4642 * c - 1854 * d) + b * (7043 * b - 17246 * c + 7042 * d) \
        + c * (11003 * c - 9402 * d) + 2107 * d * d
    w0, w1, w2, w3 = 4 / (eps + s0) ** 2, 18 / (eps + s1) ** 2, 12 / (eps + s2) ** 2, \
        1 / (eps + s3) ** 2
    q0 = 3 * d + 13 * e - 5 * f + g
    q1 = -c + 7 * d + 7 * e - f
    q2 = b - 5 * c + 13 * d + 3 * e
    q3 = -3 * a + 13 * b - 23 * c + 25 * d
    return (w0 * q0 + w1 * q1 + w2 * q2 + w3 * q3) / (12 * (w0 + w1 + w2 + w3))


class _Solver:
    """RK4 with the FV or FD right-hand side in plain torch, float64."""

    def __init__(self, nz, nvz, half, scheme, bc, omega, mat, fd_advec, ko, mu):
        f64 = {"dtype": torch.float64, "device": "cuda"}
        self.nz, self.scheme, self.bc, self.mat = nz, scheme, bc, mat
        self.fd_advec, self.ko, self.mu = fd_advec, ko, mu
        self.dz, self.dv = 2.0 * half / nz, 2.0 / nvz
        self.dt = CFL * self.dz
        self.v = -1.0 + (torch.arange(nvz, **f64) + 0.5) * self.dv
        self.vc = self.v[:, None]
        th = math.radians(THETA)
        self.ct, self.st = 0.5 * omega * math.cos(2 * th), 0.5 * omega * math.sin(2 * th)
        z = -half + (torch.arange(nz, **f64) + 0.5) * self.dz
        self.hm = -1e-3 * (z + 600.0)

    def _advect_fv(self, u):  # one component [nvz][nz]
        p, nz = _pad(u, self.bc), self.nz
        out = torch.empty_like(u)
        up, dn = self.v >= 0, self.v < 0
        for rows, s in ((up, 1), (dn, -1)):
            if not bool(rows.any()):
                continue
            q = p[rows]
            if s > 0:  # faces j + 1/2, j = -1 .. nz - 1
                f = _weno(*[q[:, k:k + nz + 1] for k in range(7)])
                if self.bc == "open":
                    f[:, 0] = f[:, 1]
            else:      # faces j - 1/2, j = 0 .. nz
                f = _weno(*[q[:, 7 - k:7 - k + nz + 1] for k in range(7)])
                if self.bc == "open":
                    f[:, nz] = 2.0 * f[:, nz - 1] - f[:, nz - 2]
            out[rows] = -self.v[rows][:, None] / self.dz * (f[:, 1:] - f[:, :-1])
        return out

    def _advect_fd(self, u):
        p, nz, h = _pad(u, self.bc), self.nz, 4

        def at(k):
            return p[:, h + k:h + k + nz]
        if self.fd_advec == "center":
            adv = -self.vc / (12 * self.dz) * ((at(-2) - at(2)) - 8.0 * (at(-1) - at(1)))
        else:
            pos = self.vc > 0
            if self.fd_advec == "upwind":
                w = {-3: -4.0, -2: 18.0, -1: -36.0, 0: 22.0}
                fac = -self.vc.abs() / (12 * self.dz)
            else:
                w = {-3: 1.0, -2: -6.0, -1: 18.0, 0: -10.0, 1: -3.0}
                fac = self.vc.abs() / (12 * self.dz)
            zero = self.vc == 0
            adv = sum(c * torch.where(zero, at(0), torch.where(pos, at(k), at(-k)))
                      for k, c in w.items())
            adv = fac * adv
        if self.ko == 5:
            ko = -0.1 / self.dz / 64 * (at(-3) + at(3) - 6 * (at(-2) + at(2)) +
                                        15 * (at(-1) + at(1)) - 20 * at(0))
        else:
            ko = -0.1 / self.dz / 16 * (at(-2) + at(2) - 4 * (at(-1) + at(1)) + 6 * at(0))
        return adv + ko

    def rhs(self, y):
        adv = self._advect_fv if self.scheme == "fv" else self._advect_fd
        o = torch.stack([adv(y[c]) for c in range(8)])
        ee, xx, er, ei, bee, bxx, br, bi = y
        ct, st = self.ct, self.st
        if ct or st:
            o[0] -= 2 * st * ei
            o[1] += 2 * st * ei
            o[2] -= 2 * ct * ei
            o[3] += 2 * ct * er + st * (ee - xx)
            o[4] -= 2 * st * bi
            o[5] += 2 * st * bi
            o[6] -= 2 * ct * bi
            o[7] += 2 * ct * br + st * (bee - bxx)
        if self.mat:
            o[2] += self.hm * ei
            o[3] -= self.hm * er
            o[6] -= self.hm * bi
            o[7] += self.hm * br
        f = self.mu * self.dv

        def moment(x):
            return f * (x.sum(dim=0)[None, :] - self.vc * (self.vc * x).sum(dim=0)[None, :])
        sa, sb, sc = moment(ei + bi), moment(er - br), moment(ee - xx - bee + bxx)
        i = 2 * (er * sa - ei * sb)
        o[0] += i
        o[1] -= i
        o[2] += (xx - ee) * sa + ei * sc
        o[3] -= (xx - ee) * sb + er * sc
        i = 2 * (br * sa + bi * sb)
        o[4] += i
        o[5] -= i
        o[6] += (bxx - bee) * sa - bi * sc
        o[7] += (bxx - bee) * sb + br * sc
        return o

    def steps(self, y, n):
        dt = self.dt
        for _ in range(n):
            k = self.rhs(y)
            acc = k.clone()
            k = self.rhs(y + 0.5 * dt * k)
            acc += 2 * k
            k = self.rhs(y + 0.5 * dt * k)
            acc += 2 * k
            k = self.rhs(y + dt * k)
            y = y + dt / 6 * (acc + k)
        return y

    def analysis(self, y, y0, g, bg):
        g, bg = g[:, None].expand_as(y[0]), bg[:, None].expand_as(y[0])

        def pol(s):
            return ((2 * s[2] / g, -2 * s[3] / g, (s[0] - s[1]) / g),
                    (2 * s[6] / bg, 2 * s[7] / bg, (s[4] - s[5]) / bg))

        def norm(p):
            return torch.sqrt(p[0] ** 2 + p[1] ** 2 + p[2] ** 2)
        p, b = pol(y)
        q, c = pol(y0)
        dp, db = (norm(p) - norm(q)).abs(), (norm(b) - norm(c)).abs()
        da = self.dz * self.dv
        e = [float((g * p[k] - bg * b[k]).sum() * da) for k in range(3)]
        diag = {"dP_max": max(float(dp.max()), float(db.max())),
                "avdP": float((dp * g).sum() / g.sum()),
                "avbdP": float((db * bg).sum() / bg.sum())}
        diag.update(M0=math.sqrt(sum(x * x for x in e)), M0_e1=e[0], M0_e2=e[1], M0_e3=e[2],
                    Pee=float(y[0].sum() / y0[0].sum()), Pbee=float(y[4].sum() / y0[4].sum()),
                    trace=float((y[0] + y[1]).sum() * da), btrace=float((y[4] + y[5]).sum() * da),
                    eln=float((y[0] - y[4]).sum() * da))
        pee = (y[0].sum(dim=1) / y0[0].sum(dim=1)).cpu().numpy()
        pbee = (y[4].sum(dim=1) / y0[4].sum(dim=1)).cpu().numpy()
        return diag, pee, pbee


def _layers(flat):
    """The flat parameter vector as float64 (W, b) pairs."""
    out, at = [], 0
    for i, o in DIMS:
        w = torch.tensor(flat[at:at + i * o].reshape(o, i), dtype=torch.float64, device="cuda")
        at += i * o
        b = torch.tensor(flat[at:at + o], dtype=torch.float64, device="cuda")
        at += o
        out.append((w, b))
    return out


def _net(layers, x):
    for k, (w, b) in enumerate(layers):
        x = x @ w.T + b
        if k < len(layers) - 1:
            x = torch.nn.functional.gelu(x)
    return x


def _padded(x):
    h = torch.zeros((x.shape[0], DIMS[0][0]), dtype=torch.float64, device="cuda")
    h[:, :NIN] = torch.tensor(x, dtype=torch.float64, device="cuda")
    return h


def _shuffled(n, seed):
    """Row order of an epoch: Fisher-Yates driven by a 64-bit LCG."""
    a, c, m = 6364136223846793005, 1442695040888963407, (1 << 64) - 1
    st = (seed * a + c) & m
    perm = list(range(n))
    for i in range(n - 1, 0, -1):
        st = (st * a + c) & m
        j = (st >> 33) % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]
    return perm


def _train_exact(case, seed):
    w, x, t = _net_inputs(case["rows"], seed)
    ps = [p.requires_grad_() for pair in _layers(w) for p in pair]
    decay = [1e-4, 0.0] * len(DIMS)
    m1, m2 = [torch.zeros_like(p) for p in ps], [torch.zeros_like(p) for p in ps]
    xs, ts = _padded(x), torch.tensor(t, dtype=torch.float64, device="cuda")
    order = torch.tensor(_shuffled(case["rows"], seed % 1000 + 1), device="cuda")
    total, step = 0.0, 0
    for at in range(0, case["rows"], case["batch"]):
        idx = order[at:at + case["batch"]]
        y = _net(list(zip(ps[::2], ps[1::2])), xs[idx])
        loss = ((y - ts[idx]) ** 2).mean()
        total += float(loss) * y.numel()
        grads = torch.autograd.grad(loss, ps)
        step += 1
        with torch.no_grad():
            for p, g, a, b, wd in zip(ps, grads, m1, m2, decay):
                a.mul_(0.9).add_(g, alpha=0.1)
                b.mul_(0.999).addcmul_(g, g, value=0.001)
                u = (a / (1 - 0.9 ** step)) / (torch.sqrt(b / (1 - 0.999 ** step)) + 1e-8)
                p.sub_(LR * (u + wd * p))
    flat = torch.cat([p.detach().ravel() for p in ps])
    return {"losses": np.array([total / (case["rows"] * 128)]), "params": flat.cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train_exact(case, seed)
    if kind == "forward":
        w, x, _ = _net_inputs(case["rows"], seed)
        return _net(_layers(w), _padded(x)).cpu().numpy()
    if kind == "ensemble":
        out = []
        for i, x in enumerate(_members(case)):
            st, _ = _member_state(x, seed, i)
            s = _Solver(x.nz, x.nvz, 600.0, "fv", "periodic", 0.0, False, "center", 3, x.mu)
            out.append(s.steps(st, x.nsteps))
        return out
    st, (g, bg) = _state(case["nz"], case["nvz"], case["half"], case["tilt"], seed)
    s = _Solver(case["nz"], case["nvz"], case["half"], case["scheme"], case["bc"], case["omega"],
                case["mat"], case["fd_advec"], case["ko"], 1.0)
    y = s.steps(st, case["steps"])
    if kind == "steps":
        return y
    diag, pee, pbee = s.analysis(y, st, g, bg)
    return {"state": y, "diag": diag, "pee": pee, "pbee": pbee}
