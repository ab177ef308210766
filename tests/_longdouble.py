"""RK4 steps of the FV scheme in numpy's long double (64-bit mantissa), for
comparisons below the oracle's own rounding: on data with O(0.1) differences
between neighbours the quadratic forms of its smoothness indicators cancel,
and its results are up to 1.2e-12 from these."""
import math

import numpy as np

LD = np.longdouble


def _face(a, b, c, d, e, f, g):
    eps = LD(1e-6)
    A, B, C, E, F, G = a - d, b - d, c - d, e - d, f - d, g - d
    s0 = E * (11003 * E - 17246 * F + 4642 * G) + F * (7043 * F - 3882 * G) + 547 * G * G
    s1 = C * (547 * C + 1922 * E - 494 * F) + E * (2843 * E - 1642 * F) + 267 * F * F
    s2 = B * (267 * B - 1642 * C - 494 * E) + C * (2843 * C + 1922 * E) + 547 * E * E
    s3 = A * (547 * A - 3882 * B + 4642 * C) + B * (7043 * B - 17246 * C) + 11003 * C * C
    w = [4 / (eps + s0) ** 2, 18 / (eps + s1) ** 2, 12 / (eps + s2) ** 2, 1 / (eps + s3) ** 2]
    q = [13 * E - 5 * F + G, -C + 7 * E - F, B - 5 * C + 3 * E, -3 * A + 13 * B - 23 * C]
    return d + sum(x * y for x, y in zip(w, q)) / (12 * sum(w))


def fill(case, x):
    """Interior state with four ghost cells each side."""
    if case.bc == "periodic":
        return np.concatenate([x[..., -4:], x, x[..., :4]], -1)
    right = [2 * x[..., -1:] - x[..., -2:-1]]
    right.append(2 * right[0] - x[..., -1:])
    while len(right) < 4:
        right.append(2 * right[-1] - right[-2])
    return np.concatenate([x[..., :1]] * 4 + [x] + right, -1)


def _rhs(case, y):
    nz, dz = case.nz, LD(case.dz)
    v = LD(case.v0) + (np.arange(case.nvz, dtype=LD) + LD(0.5)) * LD(case.dv)
    p = fill(case, y)
    o = np.zeros_like(y)
    for rows, up in ((v >= 0, True), (v < 0, False)):
        if not rows.any():
            continue
        f = _face(*[p[:, rows, (k if up else 7 - k):][..., :nz + 1] for k in range(7)])
        if case.bc == "open" and up:
            f[..., 0] = f[..., 1]
        if case.bc == "open" and not up:
            f[..., nz] = 2 * f[..., nz - 1] - f[..., nz - 2]
        o[:, rows] = -(v[rows] / dz)[None, :, None] * (f[..., 1:] - f[..., :-1])
    th = case.theta_deg * math.pi / 180.0
    ct, st = LD(0.5 * case.omega * math.cos(2 * th)), LD(0.5 * case.omega * math.sin(2 * th))
    hm = LD(-1e-3) * (LD(case.z0) + (np.arange(nz, dtype=LD) + LD(0.5)) * dz + 600)
    vc = v[:, None]

    def moment(x):
        return LD(case.mu) * LD(case.dv) * (x.sum(0)[None] - vc * (vc * x).sum(0)[None])
    sa = moment(y[3] + y[7])
    sb = moment(y[2] - y[6])
    sc = moment(y[0] - y[1] - y[4] + y[5])
    for k, s in ((0, 1), (4, -1)):
        e, x, r, i = y[k:k + 4]
        c = 2 * (r * sa - s * i * sb)
        o[k] += -2 * st * i + c
        o[k + 1] += 2 * st * i - c
        o[k + 2] += -2 * ct * i + (x - e) * sa + s * i * sc
        o[k + 3] += 2 * ct * r + st * (e - x) - s * (x - e) * sb - s * r * sc
        if case.mat:
            o[k + 2] += s * hm * i
            o[k + 3] -= s * hm * r
    return o


def step(case, interior, n):
    """n RK4 steps of the FV scheme; the state with its ghost cells (gz 4)."""
    y, dt = interior.astype(LD), LD(case.dt)
    for _ in range(n):
        k1 = _rhs(case, y)
        k2 = _rhs(case, y + dt / 2 * k1)
        k3 = _rhs(case, y + dt / 2 * k2)
        k4 = _rhs(case, y + dt * k3)
        y = y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    return fill(case, y)
