"""Measured workloads of the shallow-water time step, through the package's public API.

A case is a dict: kind, cube size N, precision, members, RK4 steps per pass, and what the
kind needs besides (operator, SBP order, staggering, diffusion).  Kinds:

  apply    one evaluation of the linear operator (operator%apply), the call of a host
           program that has its own time scheme
  steps    `steps` RK4 steps of one context, continuing from the state of the pass before
  members  the same with a time step per member, part of them frozen (served pools)
  output   the driver's loop between two outputs: steps, mass and energy, the state on the host

Outputs are the state's fields h, u, v as views of the device storage (the host arrays and
the integrals for `output`).  `exact` restates the linear operator on Ch in SBP 4-2 with
dense one-dimensional operators in 64 bits; other operators have no restatement here.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ch_swe_b200.swm import (create_domain, create_stvec_swm, create_swm_diff_operator, create_swm_operator,
                             create_timescheme)

RADIUS, GRAV = 0.6371229e7, 9.80616
OMEGA = 2.0 * math.pi / (23 * 60 * 60 + 56 * 60 + 4)
MARGIN = 4              # zero points around every panel box of the device storage


def _case(name, kind, N, precision, members, steps, **more):
    c = {"name": name, "kind": kind, "N": N, "precision": precision, "members": members, "steps": steps,
         "operator": "linear", "staggering": "Ch", "order": 42, "diffusion": 0, "test": "bumps", "tuned": True}
    c.update(more)
    return c


def listed():
    return [
        # a host model's own scheme calling the operator on a small cube: launch latency
        _case("apply-c24-fp64", "apply", 24, "fp64", 1, 0, tuned=False),
        # the small validation run of the linear equations (C32, FP64), a stretch of its loop
        _case("linear-c32-fp64", "steps", 32, "fp64", 1, 24, tuned=False),
        # an hour of the C192 day, reduced and full precision
        _case("linear-c192-fp32", "steps", 192, "fp32", 1, 24),
        _case("linear-c192-fp64", "steps", 192, "fp64", 1, 24),
        # the high-resolution linear run
        _case("linear-c384-fp32", "steps", 384, "fp32", 1, 8),
        # 256 members of a small cube advanced together
        _case("ensemble-c48x256-fp32", "steps", 48, "fp32", 256, 8),
        # the driver's loop with hourly output: integrals and the state on the host
        _case("output-c192-fp64", "output", 192, "fp64", 1, 24),
        # the other SBP orders on a cube that fits no tile evenly
        _case("linear63-c101x2-fp32", "steps", 101, "fp32", 2, 8, order=63),
        # the Ah comparison runs: dynamics and the fourth-order diffusion after each step
        _case("ah-diffusion-c192-fp32", "steps", 192, "fp32", 1, 8, staggering="Ah", diffusion=42),
        # the nonlinear steady zonal flow about a tilted axis
        _case("advective-c384-fp32", "steps", 384, "fp32", 1, 4, operator="advective", test="zonal"),
        # flow over a mountain, full precision, an ordinary cube
        _case("advective-c96-fp64", "steps", 96, "fp64", 1, 8, operator="advective", test="mountain"),
        # a served pool of nonlinear requests: a time step per slot, a quarter of the slots free
        _case("pool-c48x16-fp32", "members", 48, "fp32", 16, 16, operator="advective", test="zonal"),
    ]


def _dofs(case):
    n = case["N"] + 1
    return 18 * n * n if case["staggering"] == "Ah" else 6 * n * n + 12 * case["N"] * n


def work(case):
    """An operator evaluation reads a state and writes one; a step of the scheme reads its
    state and writes it; the output also brings it to the host.  Operations per degree of
    freedom and stage: about 25 (linear), 80 (advective); a diffusion step about 100."""
    size = 8 if case["precision"] == "fp64" else 4
    dof = _dofs(case) * case["members"]
    passes = 1 if case["kind"] == "apply" else case["steps"]
    stages = 1 if case["kind"] == "apply" else 4 * case["steps"]
    per = 80 if case["operator"] == "advective" else 25
    return {"bytes": 2.0 * size * dof * passes + (8.0 * dof if case["kind"] == "output" else 0.0),
            "flops": float(per * dof * stages + (100 * dof * passes if case["diffusion"] else 0))}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["apply", "steps", "steps", "steps", "ah", "order", "advective", "advective", "members", "output"])
        precision = rng.choice(["fp32", "fp64"])
        if kind == "apply":
            c = _case("", "apply", _log(rng, 16, 96), precision, 1, 0, tuned=False)
        elif kind == "steps":
            c = _case("", "steps", _log(rng, 24, 384), precision, _log(rng, 1, 256), rng.randint(4, 24))
        elif kind == "ah":
            c = _case("", "steps", _log(rng, 24, 256), precision, _log(rng, 1, 4), rng.randint(4, 8), staggering="Ah",
                      order=rng.choice([21, 42, 63]))
            c["diffusion"] = rng.choice([0, c["order"]])
        elif kind == "order":
            c = _case("", "steps", _log(rng, 24, 192), precision, _log(rng, 1, 4), rng.randint(4, 12),
                      order=rng.choice([21, 63]))
        elif kind == "advective":
            c = _case("", "steps", _log(rng, 24, 384), precision, _log(rng, 1, 4), rng.randint(4, 8),
                      operator="advective", test=rng.choice(["zonal", "mountain"]))
        elif kind == "members":
            c = _case("", "members", _log(rng, 24, 192), precision, _log(rng, 4, 64), rng.randint(4, 16))
            if rng.random() < 0.5:
                c.update(operator="advective", test="zonal")
        else:
            c = _case("", "output", _log(rng, 48, 192), "fp64", 1, rng.randint(8, 24))
        del c["name"]
        if work(c)["flops"] <= most:
            return c


# --- geometry and initial states --------------------------------------------------------------

_EX = [[-1, 0, 0], [0, 0, -1], [1, 0, 0], [0, 0, 1], [1, 0, 0], [1, 0, 0]]
_EY = [[0, 1, 0], [0, 1, 0], [0, 1, 0], [0, 1, 0], [0, 0, 1], [0, 0, -1]]
_EN = [[0, 0, 1], [-1, 0, 0], [0, 0, -1], [1, 0, 0], [0, 1, 0], [0, -1, 0]]


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _mesh(N, si, sj):
    """Positions r and the panel basis a1, a2, b1, b2 of a mesh, (6, ny, nx, 3), with the
    determinant J and inverse metric Q11, Q12, Q22, (ny, nx): the equiangular gnomonic panels."""
    dev = _dev()
    f64 = dict(dtype=torch.float64, device=dev)
    hx = 0.5 * math.pi / N
    X = torch.tan(-0.25 * math.pi + (torch.arange(N + 1 if si == 0 else N, **f64) + si) * hx)[None, :]
    Y = torch.tan(-0.25 * math.pi + (torch.arange(N + 1 if sj == 0 else N, **f64) + sj) * hx)[:, None]
    X, Y = torch.broadcast_tensors(X, Y)
    d2 = 1 + X * X + Y * Y
    s = d2.sqrt()
    cx, cy = 1 + X * X, 1 + Y * Y
    ex, ey, en = (torch.tensor(v, **f64)[:, None, None, :] for v in (_EX, _EY, _EN))

    def real(x, y, z):
        return x[None, ..., None] * ex + y[None, ..., None] * ey - z[None, ..., None] * en

    r = real(X / s, Y / s, 1 / s)
    a1 = real(cx * cy / s ** 3, -X * Y * cx / s ** 3, -X * cx / s ** 3)
    a2 = real(-X * Y * cy / s ** 3, cx * cy / s ** 3, -Y * cy / s ** 3)
    Q = d2 / cx, d2 * X * Y / (cx * cy), d2 / cy
    b1 = Q[0][..., None] * a1 + Q[1][..., None] * a2
    b2 = Q[1][..., None] * a1 + Q[2][..., None] * a2
    return {"r": r, "a1": a1, "a2": a2, "b1": b1, "b2": b2, "J": cx * cy / s ** 3, "Q": Q}


def _meshes(case):
    N = case["N"]
    xy = _mesh(N, 0, 0)
    return (xy, xy, xy) if case["staggering"] == "Ah" else (xy, _mesh(N, 0.5, 0), _mesh(N, 0, 0.5))


def _axis(rng):
    v = rng.normal(size=3)
    return v / np.linalg.norm(v)


def _initial(case, seed):
    """Seeded (h, u, v), each (members, 6, ny, nx) on the device, the mean depths and the
    orography: bumps on a weak rotation (linear), a balanced zonal flow about a tilted axis
    with bumps, or the flow over an isolated mountain (advective)."""
    rng = np.random.default_rng([int(seed), case["N"], case["members"]])
    mh, mu, mv = _meshes(case)
    dev = _dev()
    hs, us, vs, H = [], [], [], []
    surf = None
    for _ in range(case["members"]):
        depth = float(rng.uniform(500.0, 2000.0))
        x = mh["r"]
        h = torch.zeros(x.shape[:-1], dtype=torch.float64, device=dev)
        amp = 2.0 if case["test"] == "bumps" else 20.0
        for _ in range(int(rng.integers(1, 5))):
            c = torch.tensor(_axis(rng), device=dev)
            width, a = rng.uniform(0.05, 0.3), rng.uniform(-amp, amp)
            h = h + a * torch.exp(-(torch.arccos((x @ c).clamp(-1, 1)) / width) ** 2)
        axis = torch.tensor(_axis(rng), device=dev)
        if case["test"] == "bumps":
            u0 = float(rng.uniform(0.05, 0.2))
        else:
            mountain = case["test"] == "mountain"
            u0 = 20.0 if mountain else 2.0 * math.pi * RADIUS / (12 * 86400)
            depth = 5960.0 if mountain else 2.94e4 / GRAV
            if mountain:
                axis = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device=dev)
                top = torch.tensor([0.0, 0.5 * math.sqrt(3.0), 0.5], dtype=torch.float64, device=dev)
                surf = 2000.0 * (1 - torch.arccos((x @ top).clamp(-1, 1)) / (math.pi / 9)).clamp(min=0)
            h = h + depth - (RADIUS * OMEGA * u0 + 0.5 * u0 * u0) / GRAV * (x @ axis) ** 2
            if mountain:
                h = h - surf
        us.append((u0 * torch.cross(axis.expand_as(mu["r"]), mu["r"], dim=-1) * mu["a1"]).sum(-1))
        vs.append((u0 * torch.cross(axis.expand_as(mv["r"]), mv["r"], dim=-1) * mv["a2"]).sum(-1))
        hs.append(h)
        H.append(depth)
    dts = rng.uniform(0.5, 1.0, case["members"])
    dts[rng.permutation(case["members"])[: case["members"] // 4]] = 0.0   # free slots
    return torch.stack(hs), torch.stack(us), torch.stack(vs), H, surf, dts * _dt(case)


def _dt(case):
    """150 s at C192 for the linear runs and as bench.py's for the advective ones (75 s at C384)."""
    return 150.0 * 192.0 / case["N"]


# --- the calls --------------------------------------------------------------------------------

class _Device:
    """A state's device storage as torch sees it; the tensors made from it keep the state."""

    def __init__(self, state, ptr, shape, typestr):
        self.state = state
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _fields(case, state):
    """h, u, v of a state as strided views of its device storage."""
    ptr, nbytes, precision, pitch = state.device_view()
    N, rows = case["N"], case["N"] + 1 + 2 * MARGIN
    size = 8 if precision == 0 else 4
    shape = (case["members"], 3, 6, rows, pitch)
    assert math.prod(shape) * size == nbytes
    box = torch.as_tensor(_Device(state, ptr, shape, "<f%d" % size), device="cuda")
    ah = case["staggering"] == "Ah"
    ext = [(N + 1, N + 1), (N + 1, N + 1 if ah else N), (N + 1 if ah else N, N + 1)]
    return [box[:, f, :, MARGIN:MARGIN + ny, MARGIN:MARGIN + nx] for f, (ny, nx) in enumerate(ext)]


def prepare(case, seed):
    h, u, v, H, surf, dts = _initial(case, seed)
    dom = create_domain(case["N"], precision=case["precision"], n_members=case["members"], h_mean=H[0],
                        horizontal_staggering=case["staggering"], operator=case["operator"], sbp_order=case["order"])
    if case["tuned"]:
        dom.autotune()
    if case["operator"] == "advective":
        op = create_swm_operator(GRAV, {"swm_operator_type": "advective_swm_operator"}, dom)
        if surf is not None:
            op.set_orography(surf.cpu().numpy())
    else:
        op = create_swm_operator(GRAV, {"swm_operator_type": "linear_swm_operator", "h_mean": H[0]}, dom)
        for k, hk in enumerate(H):
            op.set_member_h_mean(k, hk)
    if case["diffusion"]:
        o = case["diffusion"]
        dom.set_diffusion(create_swm_diff_operator(
            {"hordiff_uv_name": "hordiff_vec_xyz_Ah_sbp_%d_narrow" % o, "uv_diff_coeff": 0.03,
             "hordiff_h_name": "hordiff_scalar_Ah_sbp_%d_narrow" % o, "h_diff_coeff": 0.01}, dom))
    state = create_stvec_swm(dom)
    state.upload(h.cpu().numpy(), u.cpu().numpy(), v.cpu().numpy(), member=None)
    s = {"kind": case["kind"], "domain": dom, "operator": op, "state": state, "scheme": create_timescheme(state, "rk4"),
         "steps": case["steps"], "dt": _dt(case), "dts": dts}
    if case["kind"] == "apply":
        s["tendency"] = create_stvec_swm(dom)
        s["out"] = _fields(case, s["tendency"])
    elif case["kind"] != "output":
        s["out"] = _fields(case, state)
    return s


def run(s):
    kind = s["kind"]
    if kind == "apply":
        s["operator"].apply(s["tendency"], s["state"], s["domain"])
        return s["out"]
    if kind == "members":
        s["scheme"].steps_members(s["state"], s["operator"], s["dts"], s["steps"])
        return s["out"]
    s["scheme"].steps(s["state"], s["operator"], s["domain"], s["dt"], s["steps"])
    if kind == "output":
        return [s["operator"].integrals(s["state"]), s["state"].download()]
    return s["out"]


# --- the linear operator on Ch, SBP 4-2, in 64 bits -------------------------------------------

def _sbp42(N):
    """The four one-dimensional operators as dense matrices (nodes 1..N+1, centres 1..N):
    differences and interpolations, nodes to centres and centres to nodes."""
    a, b = 0.1264926207034815, -0.029892648949074313
    di = [[-79 / 78, 27 / 26, -1 / 26, 1 / 78], [2 / 21, -9 / 7, 9 / 7, -2 / 21], [1 / 75, 0, -27 / 25, 83 / 75, -1 / 25]]
    dc = [[-2, 3, -1], [-1, 1], [1 / 24, -9 / 8, 9 / 8, -1 / 24], [-1 / 71, 6 / 71, -83 / 71, 81 / 71, -3 / 71]]
    ii = [[1 / 2 + a + 2 * b, 1 / 2 - 2 * a - 3 * b, a, b],
          [-8 / 63 - 52 / 21 * a - 104 / 21 * b, 29 / 42 + 104 / 21 * a + 52 / 7 * b, 1 / 2 - 52 / 21 * a,
           -4 / 63 - 52 / 21 * b],
          [-1 / 25 + 26 / 25 * a + 52 / 25 * b, -1 / 50 - 52 / 25 * a - 78 / 25 * b, 3 / 5 + 26 / 25 * a,
           13 / 25 + 26 / 25 * b, -3 / 50]]
    ic = [[39 / 28 + 39 / 14 * a + 39 / 7 * b, -2 / 7 - 39 / 7 * a - 78 / 7 * b, -3 / 28 + 39 / 14 * a + 39 / 7 * b],
          [13 / 27 - 52 / 27 * a - 26 / 9 * b, 29 / 54 + 104 / 27 * a + 52 / 9 * b, -1 / 54 - 52 / 27 * a - 26 / 9 * b],
          [13 / 12 * a, 7 / 16 - 13 / 6 * a, 5 / 8 + 13 / 12 * a, -1 / 16],
          [78 / 71 * b, -4 / 71 - 156 / 71 * b, 39 / 71 + 78 / 71 * b, 81 / 142, -9 / 142]]

    def matrix(rows, cols, closure, inner, shift, sign):
        M = np.zeros((rows, cols))
        for k in range(len(closure), rows - len(closure)):
            M[k, k + shift:k + shift + 4] = inner
        for k, w in enumerate(closure):
            M[k, :len(w)] = w
            M[rows - 1 - k, cols - len(w):] = sign * np.array(w[::-1])
        return torch.tensor(M, device=_dev())

    diff, mean = [1 / 24, -9 / 8, 9 / 8, -1 / 24], [-1 / 16, 9 / 16, 9 / 16, -1 / 16]
    return (matrix(N, N + 1, di, diff, -1, -1), matrix(N + 1, N, dc, diff, -2, -1),
            matrix(N, N + 1, ii, mean, -1, 1), matrix(N + 1, N, ic, mean, -2, 1))


def _sides():
    """[panel][side] -> (neighbour, its side, reversed, sign of the flux), sides left, right,
    bottom, top: matched by the positions of four vertices of a coarse panel."""
    r = _mesh(4, 0, 0)["r"].cpu().numpy()

    def line(p, s):
        return (r[p, :, 0], r[p, :, -1], r[p, 0], r[p, -1])[s]

    out = {}
    for p in range(6):
        for s in range(4):
            for q in range(6):
                for t in range(4):
                    for rev in (0, 1):
                        w = line(q, t)[::-1] if rev else line(q, t)
                        if q != p and np.abs(w - line(p, s)).max() < 1e-12:
                            out[p, s] = q, t, rev, (1 if s in (1, 3) else -1) * (1 if t in (0, 2) else -1)
    return out


def _linear42(N, H):
    """The linear tendency as a function of (h, u, v)."""
    Di, Dc, Ii, Ic = _sbp42(N)
    xy, my, mx = _mesh(N, 0, 0), _mesh(N, 0.5, 0), _mesh(N, 0, 0.5)
    hx = 0.5 * math.pi / N
    sides = _sides()
    f = 2 * OMEGA * xy["r"][..., 2]
    H = torch.tensor(H, dtype=torch.float64, device=_dev())[:, None, None, None]
    r1 = (15 / 8, -5 / 4, 3 / 8)
    satw = [0.5 * r / w for r, w in zip(r1, (13 / 12, 7 / 8, 25 / 24))]
    satc = 0.5 / (7 / 18)

    def X(M, q):
        return q @ M.T

    def Y(M, q):
        return M @ q

    def edge(q, p, s, d=0):
        """Line at depth d of side s of panel p: (members, along)."""
        return (q[:, p, :, d], q[:, p, :, -1 - d], q[:, p, d], q[:, p, -1 - d])[s]

    def across(q, p, s):
        n, t, rev, _ = sides[p, s]
        v = edge(q, n, t)
        return v.flip(-1) if rev else v

    def average(q):
        """The mean of the copies of every panel-edge vertex; q (members, 6, n, n)."""
        total, count = q.clone(), torch.ones_like(q[:1])
        for p in range(6):
            for s in range(4):
                edge(total, p, s).add_(across(q, p, s))
                edge(count, p, s).add_(1)
        return total / count

    def tendency(h, u, v):
        gx, gy = X(Di, h), Y(Di, h)
        for p in range(6):
            for k, w in enumerate(satw):
                gx[:, p, :, k] += w * (h[:, p, :, 0] - across(h, p, 0))
                gx[:, p, :, -1 - k] += w * (across(h, p, 1) - h[:, p, :, -1])
                gy[:, p, k] += w * (h[:, p, 0] - across(h, p, 2))
                gy[:, p, -1 - k] += w * (across(h, p, 3) - h[:, p, -1])
        J12 = xy["J"] * xy["Q"][1]
        ut = my["Q"][0] * u + X(Ii, J12 * Y(Ic, v)) / my["J"]
        vt = mx["Q"][2] * v + Y(Ii, J12 * X(Ic, u)) / mx["J"]
        fu, fv = my["J"] * ut, mx["J"] * vt
        dx, dy = X(Dc, fu), Y(Dc, fv)
        for p in range(6):
            for s in range(4):
                n, t, rev, sign = sides[p, s]
                jump = 0
                for k, w in enumerate(r1):
                    o = edge(fu if t < 2 else fv, n, t, k)
                    jump = jump + w * (edge(fu if s < 2 else fv, p, s, k) - sign * (o.flip(-1) if rev else o))
                edge(dx if s < 2 else dy, p, s).add_((satc if s in (0, 2) else -satc) * jump)
        div = average((dx + dy) / (hx * RADIUS * xy["J"]))
        fJ = f * xy["J"] ** 2
        cu, cv = fJ * Y(Ic, vt), -fJ * X(Ic, ut)
        # the rotated wind is averaged as a vector: Cartesian, then back on this panel's basis
        W = [average(cu * xy["b1"][..., d] + cv * xy["b2"][..., d]) for d in range(3)]
        cu = sum(W[d] * xy["a1"][..., d] for d in range(3))
        cv = sum(W[d] * xy["a2"][..., d] for d in range(3))
        return (-H * div, -GRAV * gx / (hx * RADIUS) + X(Ii, cu) / my["J"],
                -GRAV * gy / (hx * RADIUS) + Y(Ii, cv) / mx["J"])

    return tendency


def exact(case, seed):
    if case["operator"] != "linear" or case["staggering"] != "Ch" or case["order"] != 42:
        return None
    h, u, v, H, _, dts = _initial(case, seed)
    y = [h, u, v]
    A = _linear42(case["N"], H)
    if case["kind"] == "apply":
        return list(A(*y))
    dt = torch.tensor(dts if case["kind"] == "members" else np.full(case["members"], _dt(case)),
                      device=_dev())[:, None, None, None]
    for _ in range(case["steps"]):
        k1 = A(*y)
        k2 = A(*(a + 0.5 * dt * k for a, k in zip(y, k1)))
        k3 = A(*(a + 0.5 * dt * k for a, k in zip(y, k2)))
        k4 = A(*(a + dt * k for a, k in zip(y, k3)))
        y = [a + dt / 6 * (p + 2 * q + 2 * r + s) for a, p, q, r, s in zip(y, k1, k2, k3, k4)]
    if case["kind"] == "output":
        return [None, tuple(a[0].cpu().numpy() for a in y)]
    return y
