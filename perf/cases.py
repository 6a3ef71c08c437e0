"""Performance cases of the level-set transport library, through its public entry points.

Three ways in which programs use it:

  step     a flow solver advances phi by one physical time step of its own grid in FP64
           (`LevelSet.levelsetmethod`, the drop-in for the Fortran routine): volume, WENO3 TVD-RK3
           advection and one of the three reinitialisations, with the arrays on the GPU or, as the
           Fortran caller has them, on the host;
  bands    the bookkeeping such a solver does between steps: water volume with the AdvectionNodes
           band, the narrow band and the ghost-fluid node list;
  rollout  an ensemble of independent grids of uneven sizes goes some steps forward in one batch
           (`LevelSetBatch`, FP32): new phi and velocities in, volumes and phi out;
  gradient forward steps and the reverse sweep for gradients of phi0 and the velocity, through the
           batch's calls or through `transport` (torch.autograd).

Inputs follow the analytic descriptions of the repository's workloads (a sphere in the LeVeque
deformation field, free surfaces with a solitary wave on a stretched curvilinear grid, sheared boxes
with Fourier surfaces), with amplitudes, places and phases from the seed.  `exact` restates the
step in plain torch FP64.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ns-lsm-single-phase_gb300"))

from nslsm import Grid, LevelSet, LsmParams  # noqa: E402
from nslsm.batch import LevelSetBatch, transport  # noqa: E402

DEV = "cuda"
PI = math.pi


# ------------------------------------------------------------------ cases
def _step(name, ni, nj, nk, shape, reinit, iters, host=False):
    return {"name": name, "kind": "step", "ni": ni, "nj": nj, "nk": nk, "shape": shape, "reinit": reinit,
            "iters": iters, "host": host}


def _rollout(name, count, lo, hi, steps, sizes, iters=5):
    return {"name": name, "kind": "rollout", "count": count, "lo": lo, "hi": hi, "steps": steps, "sizes": sizes,
            "iters": iters}


def _gradient(name, ni, nj, nk, shape, iters, steps, every, precision="fp32", mode="store", mass=False, autograd=False,
              count=1):
    return {"name": name, "kind": "gradient", "ni": ni, "nj": nj, "nk": nk, "shape": shape, "iters": iters,
            "steps": steps, "every": every, "precision": precision, "mode": mode, "mass": mass, "autograd": autograd,
            "count": count}


def listed():
    return [
        # the smallest call: a coarse test grid, where launches and waits count
        _step("step_small", 16, 16, 16, "sphere", "godunov", 5),
        # the plain FP64 configuration: 64^3 sphere in the deformation field, 5 pseudo-steps
        _step("step_sphere", 64, 64, 64, "sphere", "godunov", 5),
        # the curvilinear solitary wave at its stated size, 10 pseudo-steps
        _step("step_wave", 256, 128, 96, "wave", "godunov", 10),
        # the same solver called from the host (Fortran) side, odd sizes
        _step("step_wave_host", 101, 67, 53, "wave", "godunov", 10, host=True),
        # the reference's live reinitialisation (ENO2 gradient, RK3 in pseudo-time)
        _step("step_sussman", 192, 96, 72, "wave", "sussman", 10),
        # the reference deck's hybrid branch: band advection + geometric reinitialisation
        _step("step_hybrid", 128, 64, 48, "wave", "hybrid", 10),
        # volume and bands of a solver's grid between its steps
        {"name": "bands", "kind": "bands", "ni": 256, "nj": 128, "nk": 96, "shape": "wave"},
        # a few small grids: latency of the batch's step
        _rollout("rollout_small", 3, 12, 24, 10, 1),
        # the batched configuration: 64 sheared boxes with 32..96 nodes an axis, 5 pseudo-steps
        _rollout("rollout_64", 64, 32, 96, 10, 2),
        # gradient check in FP64: uneven grids, recomputed coefficients
        _gradient("gradient_fp64", 45, 38, 33, "sphere", 3, 4, 2, precision="fp64", mode="recompute", count=2),
        # velocity and phi0 training through torch.autograd, a checkpoint every 5 steps
        _gradient("gradient_train", 128, 128, 128, "sphere", 5, 10, 5, autograd=True),
        # the large free surface: 10 pseudo-steps, mass correction, checkpoints
        _gradient("gradient_large", 512, 256, 256, "wave", 10, 3, 2, mass=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sizes(rng, nodes, least=12):
    """Three sizes of about `nodes` nodes, the axes up to a factor 3 apart."""
    a = [rng.uniform(0.6, 1.7) for _ in range(3)]
    r = (nodes / (a[0] * a[1] * a[2])) ** (1.0 / 3.0)
    return [max(least, int(r * f)) for f in a]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "bands", "rollout", "gradient", "gradient"])
    if kind == "step":
        reinit = rng.choice(["godunov", "godunov", "sussman", "hybrid"])
        host = rng.random() < 0.25
        top = {"godunov": 3.2e6, "sussman": 1.4e6, "hybrid": 4.0e5}[reinit] * (0.2 if host else 1.0)
        ni, nj, nk = _sizes(rng, _log(rng, 4096, top))
        c = _step("", ni, nj, nk, rng.choice(["sphere", "wave"]), reinit, rng.choice([3, 5, 10]), host)
    elif kind == "bands":
        ni, nj, nk = _sizes(rng, _log(rng, 8000, 3.2e6))
        c = {"kind": kind, "ni": ni, "nj": nj, "nk": nk, "shape": rng.choice(["sphere", "wave"])}
    elif kind == "rollout":
        lo = rng.randint(10, 40)
        c = _rollout("", _log(rng, 1, 64), lo, lo + rng.randint(4, 56), rng.choice([5, 10]), rng.randint(0, 10 ** 6),
                     rng.choice([3, 5, 10]))
    else:
        precision = rng.choice(["fp32", "fp32", "fp32", "fp64"])
        count = rng.choice([1, 1, 2, 5])
        ni, nj, nk = _sizes(rng, _log(rng, 2.0e4, 8.0e6 if precision == "fp32" else 2.0e5) / count)
        steps = rng.choice([2, 4, 6])
        c = _gradient("", ni, nj, nk, rng.choice(["sphere", "wave"]), rng.choice([3, 5, 10]), steps,
                      rng.choice([2, steps]), precision, rng.choice(["store", "store", "recompute"]),
                      rng.random() < 0.4, rng.random() < 0.5, count)
        if c["autograd"]:
            c["mass"] = False
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs
def _mesh(ni, nj, nk):
    """(nk, nj, ni) computational coordinates in [0, 1]."""
    ax = [torch.arange(n, dtype=torch.float64, device=DEV) / (n - 1) for n in (nk, nj, ni)]
    ze, et, xi = torch.meshgrid(*ax, indexing="ij")
    return xi, et, ze


def _field(shape, ni, nj, nk, rnd):
    """One grid: coordinates, phi, q, smoothing width, pseudo time step and CFL number."""
    xi, et, ze = _mesh(ni, nj, nk)
    q = torch.zeros((nk, nj, ni, 4), dtype=torch.float64, device=DEV)
    if shape == "sphere":
        x, y, z = xi.clone(), et.clone(), ze.clone()
        c = [0.35 + rnd.uniform(-0.05, 0.05) for _ in range(3)]
        r = 0.15 * rnd.uniform(0.9, 1.3)
        phi = r - torch.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2)
        amp = rnd.uniform(0.7, 1.0)
        s = [torch.sin(PI * a) ** 2 for a in (x, y, z)]
        d = [torch.sin(2 * PI * a) for a in (x, y, z)]
        q[..., 1] = amp * 2.0 * s[0] * d[1] * d[2]
        q[..., 2] = -amp * d[0] * s[1] * d[2]
        q[..., 3] = -amp * d[0] * d[1] * s[2]
        steps = [1.0 / (n - 1) for n in (ni, nj, nk)]
        return x, y, z, phi, q, 1.5 * max(steps), 0.5 * min(steps), 0.5
    if shape == "wave":
        # the solitary wave on its 8 x 2 x 1 domain, the surface also uneven in y
        x = 8.0 * xi + 0.05 * torch.sin(2 * PI * et)
        y, z = 2.0 * et, ze ** 1.3
        amp, depth = 0.1 * rnd.uniform(0.8, 1.2), 0.5 + rnd.uniform(-0.02, 0.02)
        k, x0 = math.sqrt(3.0 * amp / (4.0 * depth ** 3)), 2.0 + rnd.uniform(-0.5, 0.5)
        sech2 = 1.0 / torch.cosh(k * (x - x0)) ** 2
        phi = z - depth - amp * sech2 * (1.0 + 0.2 * torch.cos(PI * y + rnd.uniform(0, 2 * PI)))
        c = amp * math.sqrt(9.81 * depth)
        q[..., 1] = 1.0 + c * sech2
        q[..., 3] = c * sech2
        h = max(8.0 / (ni - 1), 2.0 / (nj - 1))
        return x, y, z, phi, q, 1.5 * h, 0.5 * min(h, 2.0 / (nj - 1), (1.0 / (nk - 1)) ** 1.3), 0.4
    # sheared box, a surface of Fourier modes, the curl of a random vector potential
    sh = [[1.0 if r == c else rnd.uniform(-0.1, 0.1) for c in range(3)] for r in range(3)]
    x, y, z = (sh[r][0] * xi + sh[r][1] * et + sh[r][2] * ze for r in range(3))
    phi = z - 0.5
    for _ in range(4):
        phi = phi - rnd.uniform(0.0, 0.05) * torch.cos(2 * PI * (rnd.randint(1, 4) * x + rnd.randint(1, 4) * y)
                                                       + rnd.uniform(0, 2 * PI))
    for _ in range(8):
        a, k = [rnd.gauss(0.0, 0.2) for _ in range(3)], [rnd.randint(1, 4) for _ in range(3)]
        c = 2 * PI * torch.cos(2 * PI * (k[0] * x + k[1] * y + k[2] * z) + rnd.uniform(0, 2 * PI))
        q[..., 1] += c * (k[1] * a[2] - k[2] * a[1])
        q[..., 2] += c * (k[2] * a[0] - k[0] * a[2])
        q[..., 3] += c * (k[0] * a[1] - k[1] * a[0])
    steps = [1.0 / (n - 1) for n in (ni, nj, nk)]
    return x.contiguous(), y.contiguous(), z.contiguous(), phi, q, 1.5 * max(steps), 0.5 * min(steps), 0.5


def _metrics(x, y, z):
    """csi, eta, zet (nk, nj, ni, 3) and the inverse volume aj, by the metric relations."""
    dx = [[None] * 3 for _ in range(3)]  # dx[axis][coordinate]
    for m in range(3):
        for c, a in enumerate((x, y, z)):
            n, dim = a.shape[2 - m], 2 - m
            d = torch.empty_like(a)
            d.narrow(dim, 1, n - 2).copy_(0.5 * (a.narrow(dim, 2, n - 2) - a.narrow(dim, 0, n - 2)))
            d.narrow(dim, 0, 1).copy_(a.narrow(dim, 1, 1) - a.narrow(dim, 0, 1))
            d.narrow(dim, n - 1, 1).copy_(a.narrow(dim, n - 1, 1) - a.narrow(dim, n - 2, 1))
            dx[m][c] = d

    def cross(a, b):
        return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]

    rows = [cross(dx[1], dx[2]), cross(dx[2], dx[0]), cross(dx[0], dx[1])]
    aj = 1.0 / sum(dx[0][c] * rows[0][c] for c in range(3))
    return [torch.stack([aj * v for v in r], dim=-1).contiguous() for r in rows] + [aj]


def _dt(q, met, cfl):
    return cfl / max(float((m * q[..., 1:]).sum(-1).abs().max()) for m in met[:3])


def _rng(case, seed):
    return random.Random("%d %s" % (int(seed), case["kind"]))


def _one(case, seed):
    """The grid of a `step` or `bands` case."""
    x, y, z, phi, q, eps, dtau, cfl = _field(case["shape"], case["ni"], case["nj"], case["nk"], _rng(case, seed))
    met = _metrics(x, y, z)
    reinit = case.get("reinit", "godunov")
    if reinit == "hybrid":
        # the geometric branch leaves +-9.9 four nodes away from the surface
        far = 4.0 * eps / 1.5
        phi = torch.where(phi.abs() <= far, phi, 9.9 * torch.sign(phi))
    p = LsmParams(epslsm=eps, numiter_lsm=1, delti_lsm=_dt(q, met, cfl), RNitermax=case.get("iters", 5),
                  RNtimestep=dtau, RNfreq=1, isnarrow=1, narrowcoef=4.0, BigPhi=5.0,
                  reinit_scheme=1 if reinit == "sussman" else 0, hybrid_reinitialisation=reinit == "hybrid")
    return (x, y, z), phi.contiguous(), q, met, p


def _instances(case, seed):
    """The grids of a `rollout` or `gradient` case."""
    rnd = _rng(case, seed)
    if case["kind"] == "rollout":
        sz = random.Random(case["sizes"])
        dims = [[sz.randint(case["lo"], case["hi"]) for _ in range(3)] for _ in range(case["count"])]
        shape = "box"
    else:
        dims = [[case["ni"] - 3 * k, case["nj"] + k, case["nk"] - 2 * k] for k in range(case["count"])]
        dims = [[max(8, n) for n in d] for d in dims]
        shape = case["shape"]
    got = []
    for ni, nj, nk in dims:
        x, y, z, phi, q, eps, dtau, cfl = _field(shape, ni, nj, nk, rnd)
        met = _metrics(x, y, z)
        got.append({"n": (ni, nj, nk), "xyz": (x, y, z), "phi": phi.contiguous(), "q": q, "met": met, "eps": eps,
                    "dtau": dtau, "dt": _dt(q, met, cfl)})
    if case["kind"] == "gradient":
        for g in got:
            gen = torch.Generator(device=DEV)
            gen.manual_seed(rnd.randrange(1 << 40))
            g["seed"] = torch.randn(g["phi"].shape, generator=gen, dtype=torch.float64, device=DEV)
    return got


# ------------------------------------------------------------------ prepare / run
def _fortran(t):
    return np.asfortranarray(t.cpu().numpy().T)


def prepare(case, seed):
    if case["kind"] in ("step", "bands"):
        xyz, phi, q, met, p = _one(case, seed)
        ls = LevelSet(device=0)
        arrays = [q, met[0], met[1], met[2], met[3], phi, phi.clone(), *xyz]
        if case.get("host"):
            arrays = [_fortran(a) for a in arrays]
        s = {"case": case, "ls": ls, "grid": Grid(case["ni"], case["nj"], case["nk"]), "p": p, "a": arrays}
        if case["kind"] == "bands":
            # the solver's ghost-fluid list, allocated once for any number of nodes
            s["list"] = np.zeros((phi.numel(), 3), dtype=np.int32)
        return s
    inst = _instances(case, seed)
    forward = case["kind"] == "rollout"
    b = LevelSetBatch([(*g["n"], g["dt"], g["dtau"], g["eps"]) for g in inst], RNitermax=case["iters"], BigPhi=5.0,
                      precision="fp32" if forward else case["precision"],
                      adjoint_mode="store" if forward else case["mode"], mass_correction=not forward and case["mass"])
    for k, g in enumerate(inst):
        b.set_geometry(k, *g["xyz"], *g["met"][:3])
        b.set_velocity(k, g["q"])
        b.set_phi(k, g["phi"])
    s = {"case": case, "batch": b, "phi": [g["phi"] for g in inst], "q": [g["q"] for g in inst]}
    if not forward and case["mass"]:
        for k, v in enumerate(b.water_volume()[:, 3]):
            b.set_mass_target(k, float(v))
    b.step(0, volumes=False)  # the batch's plan: tile shape and graph, once before the program's loop
    if forward:
        # the fields of all instances in one array, as an ensemble keeps them
        s["flat"] = torch.empty(sum(p.numel() for p in s["phi"]), dtype=torch.float64, device=DEV)
        s["outs"] = [v.view(p.shape) for v, p in zip(s["flat"].split([p.numel() for p in s["phi"]]), s["phi"])]
    else:
        s["seed"] = [g["seed"] for g in inst]
        if case["autograd"] and case["precision"] == "fp32":
            # FP32 parameters of a training program: autograd returns their gradients in FP32
            s["phi"] = [p.float() for p in s["phi"]]
            s["q"] = [q.float() for q in s["q"]]
            s["seed"] = [w.float() for w in s["seed"]]
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "step":
        q, csi, eta, zet, aj, phi, phi_n, x, y, z = s["a"]
        # the caller's time loop sets phi = phi_n before each step
        if case["host"]:
            phi[...] = phi_n
        else:
            phi.copy_(phi_n)
        v = s["ls"].levelsetmethod(s["grid"], s["p"], q, csi, eta, zet, aj, phi, phi_n, x, y, z, 1)
        return {"phi": phi, "volumes": v}
    if case["kind"] == "bands":
        _, _, _, _, _, phi, _, x, y, z = s["a"]
        ls, g, p = s["ls"], s["grid"], s["p"]
        v, nodes = ls.total_water_volume(g, phi, x, y, z, with_nodes=True)
        band, found = ls.narrowband(g, p, phi), ls.get_gfm_list(g, p, phi)
        s["list"][:len(found)] = found
        return {"volumes": v, "nodes": nodes, "band": band, "list": s["list"], "listed": len(found)}
    b = s["batch"]
    n = range(b.ninst)
    if case["kind"] == "rollout":
        b.set_velocities(s["q"])
        for k in n:
            b.set_phi(k, s["phi"][k])
        v = b.step(case["steps"])
        b.get_phis(s["outs"])
        # an FP32 batch computes FP32 numbers: the program keeps them as such
        return {"phi": s["flat"].float(), "volumes": v}
    if case["autograd"]:
        phi = [t.detach().requires_grad_() for t in s["phi"]]
        q = [t.detach().requires_grad_() for t in s["q"]]
        out = transport(b, case["steps"], [t.double() for t in phi], [t.double() for t in q],
                        checkpoint_every=case["every"])
        out = [o.to(t.dtype) for o, t in zip(out, phi)]
        torch.autograd.backward(out, s["seed"])
        return {"phi": [o.detach() for o in out], "grad_phi": [t.grad for t in phi], "grad_q": [t.grad for t in q]}
    for k in n:
        b.set_phi(k, s["phi"][k])
        b.set_velocity(k, s["q"][k])
    b.forward_record(case["steps"], case["every"])
    out = [b.get_phi(k, like=s["phi"][k]) for k in n]
    for k in n:
        b.set_grad_phi(k, s["seed"][k])
    b.backward()
    gp = [b.get_grad_phi0(k, like=s["phi"][k]) for k in n]
    gq = [b.get_grad_velocity(k, like=s["phi"][k]) for k in n]
    if case["precision"] == "fp32":
        out, gp, gq = ([t.float() for t in v] for v in (out, gp, gq))
    return {"phi": out, "grad_phi": gp, "grad_q": gq}


def work(case):
    """Bytes: each input read and each output written once.  Operations: one value per WENO face and axis
    (~20), Godunov norm (~40) or ENO2 norm (~50) per pseudo-step, and the rest of a step (~150)."""
    if case["kind"] == "step":
        n = case["ni"] * case["nj"] * case["nk"]
        r = {"godunov": 40 * case["iters"], "sussman": 4 * 60 * case["iters"], "hybrid": 200}[case["reinit"]]
        return {"bytes": n * 8 * (3 + 9 + 1 + 2 + 3 + 1), "flops": n * (3 * 75 + r + 150)}
    if case["kind"] == "bands":
        n = case["ni"] * case["nj"] * case["nk"]
        return {"bytes": n * (8 * 4 + 4 * 2), "flops": n * 60}
    if case["kind"] == "rollout":
        sz = random.Random(case["sizes"])
        n = 0
        for _ in range(case["count"]):
            n += sz.randint(case["lo"], case["hi"]) * sz.randint(case["lo"], case["hi"]) * sz.randint(case["lo"], case["hi"])
        per = 8 * (3 + 1) + 12  # velocity and phi in, phi out in both precisions
        # each step: the state, the metrics and the velocity are read and phi written at least once
        return {"bytes": n * (per + case["steps"] * 4 * (1 + 9 + 3 + 1)),
                "flops": n * case["steps"] * (3 * 75 + 40 * case["iters"] + 50)}
    n = case["ni"] * case["nj"] * case["nk"] * case["count"]
    e = 4 if case["precision"] == "fp32" else 8
    step = e * (1 + 9 + 3 + 1)
    return {"bytes": n * (8 * (1 + 3 + 1) + e * (1 + 1 + 4) + case["steps"] * (2 * step + 3 * e)),
            "flops": 3 * n * case["steps"] * (3 * 75 + 40 * case["iters"] + 50)}


# ------------------------------------------------------------------ exact (plain torch, FP64)
def _sh(a, o, dim):
    """a at index + o along dim, edges repeated."""
    n = a.shape[dim]
    if o > 0:
        return torch.cat([a.narrow(dim, o, n - o)] + [a.narrow(dim, n - 1, 1)] * o, dim)
    if o < 0:
        return torch.cat([a.narrow(dim, 0, 1)] * (-o) + [a.narrow(dim, 0, n + o)], dim)
    return a


def _at(a, dim):
    shape = [1, 1, 1]
    shape[dim] = a.shape[dim]
    return torch.arange(a.shape[dim], device=a.device).view(shape)


def _weno(left, mid, right):
    a0 = (2.0 / 3.0) / (1.0e-6 + (mid - right) ** 2) ** 2
    a1 = (1.0 / 3.0) / (1.0e-6 + (left - mid) ** 2) ** 2
    return (a0 * (0.5 * mid + 0.5 * right) + a1 * (1.5 * mid - 0.5 * left)) / (a0 + a1)


def _advect_rhs(f, w):
    r = torch.zeros_like(f)
    inner = torch.ones_like(f, dtype=torch.bool)
    for m in range(3):
        dim = 2 - m
        n, at = f.shape[dim], _at(f, dim)
        s = {o: _sh(f, o, dim) for o in range(-2, 3)}
        up = w[m] > 0
        plus = torch.where(up | (at == n - 2), _weno(s[-1], s[0], s[1]), _weno(s[2], s[1], s[0]))
        minus = torch.where(up & (at != 1), _weno(s[-2], s[-1], s[0]), _weno(s[1], s[0], s[-1]))
        r = r + w[m] * (plus - minus)
        inner = inner & (at > 0) & (at < n - 1)
    return torch.where(inner, r, torch.zeros_like(r))


def _faces(f, big=5.0):
    """First-order extrapolation onto the six faces, or the neighbour's value where |phi| is large."""
    for face in range(6):
        dim = 2 - face // 2
        n = f.shape[dim]
        b, n1, n2 = (0, 1, 2) if face % 2 == 0 else (n - 1, n - 2, n - 3)
        v1, v2 = f.select(dim, n1), f.select(dim, n2)
        v = torch.where(v2.abs() >= big, v1, 4.0 / 3.0 * v1 - 1.0 / 3.0 * v2).unsqueeze(dim)
        f = torch.cat([v, f.narrow(dim, 1, n - 1)] if b == 0 else [f.narrow(dim, 0, n - 1), v], dim)
    return f


def _advect(f0, w):
    f = f0
    for a, b, c in ((1.0, 0.0, 1.0), (0.75, 0.25, 0.25), (1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0)):
        f = _faces(a * f0 + b * f - c * _advect_rhs(f, w))
    return f


def _godunov(d, met, s):
    fwd, bwd = [], []
    for m in range(3):
        dim = 2 - m
        at = _at(d, dim)
        p, q = _sh(d, 1, dim) - d, d - _sh(d, -1, dim)
        fwd.append(torch.where(at < d.shape[dim] - 1, p, q))
        bwd.append(torch.where(at > 0, q, p))
    acc = torch.zeros_like(d)
    sg = torch.where(s > 0, 1.0, -1.0)
    for c in range(3):
        p = torch.clamp(sg * sum(met[m][..., c] * bwd[m] for m in range(3)), min=0.0)
        q = torch.clamp(sg * sum(met[m][..., c] * fwd[m] for m in range(3)), max=0.0)
        acc = acc + torch.where(p * p >= q * q, p * p, q * q)
    return torch.where(acc > 0, torch.sqrt(torch.where(acc > 0, acc, torch.ones_like(acc))), torch.zeros_like(acc))


def _smooth_sign(f, eps):
    return torch.where(f.abs() >= eps, torch.sign(f), f / eps - torch.sin(PI * f / eps) / PI)


def _redistance(f0, met, eps, dtau, iters):
    with torch.no_grad():
        # the correction returns the nodes within eps of the surface to their value
        pinned = (f0.abs() < eps) & (_godunov(f0, met, f0) > 0)
        s = torch.where(pinned, torch.zeros_like(f0), _smooth_sign(f0, eps))
    d = f0
    for _ in range(iters):
        d = torch.where(s == 0, d, d - dtau * s * (_godunov(d, met, s) - 1.0))
    return d


def _eno_norm(d, f0, met):
    shape = d.shape
    face = []
    for m in range(3):
        at = _at(d, 2 - m)
        face.append(((at == 0) | (at == shape[2 - m] - 1)).expand(shape))
    f = torch.where(face[0] & ~face[1] & ~face[2], f0[-2, -2, -2], f0)
    sg = torch.where(f.abs() > 2.0 ** -52, torch.where(f >= 0, 1.0, -1.0), 0.0)
    der = []
    for m in range(3):
        dim = 2 - m
        at, n = _at(d, dim), shape[dim]
        ll, l, r, rr = (_sh(d, o, dim) for o in (-2, -1, 1, 2))
        a, b, c = r - 2.0 * d + l, rr - 2.0 * r + d, d - 2.0 * l + ll
        mp = torch.where((b.abs() < a.abs()) & (at != n - 2), b, a)
        mm = torch.where((c.abs() < a.abs()) & (at != 1), c, a)
        dp, dm = r - d - 0.5 * mp, d - l + 0.5 * mm
        v = torch.where((sg * (r - d) < 0) & (sg * (d - l) < -sg * (r - d)), dp,
                        torch.where((sg * (d - l) > 0) & (sg * (r - d) > -sg * (d - l)), dm, 0.5 * (dp + dm)))
        der.append(torch.where(at == 0, r - d, torch.where(at == n - 1, d - l, v)))
    return torch.sqrt(sum(sum(met[m][..., c] * der[m] for m in range(3)) ** 2 for c in range(3)))


def _live_redistance(f0, met, eps, dtau, iters, tol):
    s = torch.where(f0.abs() > eps, torch.sign(f0), f0 / eps - torch.sin(PI * f0 / eps) / PI)
    d, g = f0, _eno_norm(f0, f0, met)
    for _ in range(iters):
        if abs(float(g.max()) - 1.0) < tol and abs(float(g.min()) - 1.0) < tol:
            break
        d0 = d
        move = _eno_norm(d, f0, met) - 1.0 > tol
        for a, b, c in ((1.0, 0.0, 1.0), (0.75, 0.25, 0.25), (1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0)):
            g = _eno_norm(d, f0, met)
            delta = torch.where(d.abs() > eps, 0.0, (1.0 + torch.cos(PI * d / eps)) / (2.0 * eps))
            den = delta * delta * g
            lam = torch.where(den.abs() < 2.0 ** -52, 0.0, -delta * s * (1.0 - g) / torch.where(den == 0, 1.0, den))
            d = torch.where(move, a * d0 + b * d - c * dtau * (s * (g - 1.0) - lam * delta * g), d)
    return d


_CELL = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))
_TETS = ((0, 5, 1, 6), (0, 1, 2, 6), (0, 2, 3, 6), (0, 3, 7, 6), (0, 7, 4, 6), (0, 4, 5, 6))


def _share(p):
    """The part of a tetrahedron where the linear function with the vertex values p (4, n) is positive."""
    p = torch.sort(p, dim=0).values
    up = (p > 0).sum(0)

    def cut(a, b):  # share of the edge from a on a's side
        d = a - b
        return a / torch.where(d == 0, 1.0, d)

    one = cut(p[3], p[0]) * cut(p[3], p[1]) * cut(p[3], p[2])
    three = 1.0 - cut(p[0], p[1]) * cut(p[0], p[2]) * cut(p[0], p[3])
    ac, ad, bc, bd = cut(p[3], p[0]), cut(p[3], p[1]), cut(p[2], p[0]), cut(p[2], p[1])
    two = ac * ad * (1.0 - bd) + ac * bd * (1.0 - bc) + bc * bd
    zero = torch.zeros_like(one)
    return torch.where(up == 0, zero, torch.where(up == 1, one, torch.where(up == 2, two, torch.where(
        up == 3, three, zero + 1.0))))


def _volumes(phi, xyz):
    """Water volume in cut tetrahedra, whole tetrahedra of cut cells, whole cells, and all of it."""
    def corner(a, c):
        i, j, k = c
        return a[k:a.shape[0] - 1 + k, j:a.shape[1] - 1 + j, i:a.shape[2] - 1 + i]

    tiny = 2.0 ** -52
    p = torch.stack([corner(phi, c) for c in _CELL])
    water, air = (p > tiny).all(0), (p < -tiny).all(0)
    bulk = _hexahedra([torch.stack([corner(a, c)[water] for a in xyz]) for c in _CELL])
    cut = ~water & ~air
    p = p[:, cut]
    v = [torch.stack([corner(a, c)[cut] for a in xyz]) for c in _CELL]
    k = s = 0.0
    for t in _TETS:
        tp = torch.stack([p[q] for q in t])
        a, b, c = (v[q] - v[t[0]] for q in t[1:])
        vol = (torch.linalg.cross(a, b, dim=0) * c).sum(0).abs() / 6.0
        whole = (tp > tiny).all(0)
        mixed = ~whole & ~(tp < -tiny).all(0)
        k = k + float((vol * _share(tp))[mixed].sum())
        s = s + float(vol[whole].sum())
    bulk = float(bulk.sum())
    return np.array([k, s, bulk, k + s + bulk])


def _hexahedra(v):
    """Volume of hexahedra with bilinear faces."""
    def det(a, b, c):
        return (a * torch.linalg.cross(b, c, dim=0)).sum(0)

    # each face's cone over vertex 6 with the face's mean of its two diagonal splits
    faces = ((0, 3, 2, 1), (4, 5, 6, 7), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7))
    vol = 0.0
    for a, b, c, d in faces:
        a, b, c, d = (v[q] - v[6] for q in (a, b, c, d))
        vol = vol + det(a, b, c) + det(a, c, d) + det(a, b, d) + det(b, c, d)
    return vol / 12.0


def _batch_step(f, w, g, iters):
    f = _advect(f, w)
    return _faces(_redistance(f, g["met"], g["eps"], g["dtau"], iters)) if iters else f


def _velocity(q, met, dt):
    return [dt * (m * q[..., 1:]).sum(-1) for m in met[:3]]


def exact(case, seed):
    if case["kind"] == "step":
        if case["reinit"] == "hybrid":
            return None  # the distances to the surface's triangles
        xyz, f, q, met, p = _one(case, seed)
        v = _volumes(f, xyz)
        f = _advect(f, _velocity(q, met, p.delti_lsm))
        if case["reinit"] == "sussman":
            f = _live_redistance(f, met, p.epslsm, p.RNtimestep, p.RNitermax, p.epsReinitialisation)
        else:
            f = _redistance(f, met, p.epslsm, p.RNtimestep, p.RNitermax)
        f = _faces(f)
        return {"phi": _fortran(f) if case["host"] else f, "volumes": v}
    if case["kind"] == "bands":
        xyz, f, _, _, _ = _one(case, seed)
        return {"volumes": _volumes(f, xyz), "nodes": None, "band": None, "list": None, "listed": None}
    if case["kind"] == "rollout":
        fs, vs = [], []
        for g in _instances(case, seed):
            f, w = g["phi"], _velocity(g["q"], g["met"], g["dt"])
            for _ in range(case["steps"]):
                last, f = f, _batch_step(f, w, g, case["iters"])
            fs.append(f.reshape(-1))
            vs.append(_volumes(last, g["xyz"]))
        return {"phi": torch.cat(fs), "volumes": np.stack(vs)}
    nodes = case["ni"] * case["nj"] * case["nk"] * case["count"]
    if case["mass"] or nodes * case["steps"] * case["iters"] > 1.2e8:
        return None
    from torch.utils.checkpoint import checkpoint
    out = {"phi": [], "grad_phi": [], "grad_q": []}
    for g in _instances(case, seed):
        f0, q = g["phi"].clone(), g["q"].clone()
        if case["autograd"] and case["precision"] == "fp32":
            f0, q, g["seed"] = f0.float().double(), q.float().double(), g["seed"].float().double()
        f0.requires_grad_()
        q.requires_grad_()
        w = _velocity(q, g["met"], g["dt"])
        f = f0
        for _ in range(case["steps"]):
            f = checkpoint(lambda t, a, b, c, g=g: _batch_step(t, (a, b, c), g, case["iters"]), f, *w,
                           use_reentrant=False)
        f.backward(g["seed"])
        out["phi"].append(f.detach())
        out["grad_phi"].append(f0.grad)
        out["grad_q"].append(q.grad)
    return out
