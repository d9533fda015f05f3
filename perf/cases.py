"""The work that programs using this library have it do, as timed cases.

Every case is one pass of such a program through the public entry points
(preprocess_src_b200.step.Simulation / Batch, preprocess_src_b200.adjoint, and the
C ABI behind them where the caller keeps page-locked buffers): an output interval
of a run (the steps, then the fields and the cells read back in the reference's
layouts), the same for many independent capillaries stepped together, one gradient
of an optimisation, or a state moved in and out.  The inputs are a developed flow with
slightly stretched cells, made from the seed, so that no term of the step
vanishes.  ``exact`` restates the step in FP64 with plain torch.

A case is a dict of plain values:
  kind      "step", "batch", "adjoint" or "io"
  flow      "duct" (square or rectangular), "tube" (circular, interpolated
            bounce-back) or "shear" (moving y walls, periodic x)
  L, W, H   periodic length along z and the lattice's x and y extents
  cells     red cells, subdiv their icosphere refinement, radius their size
  white     white cells (a second population of spheres), storage the population type ("f32",
            "f16"), tau, br (bending), M (sub-cycling), lam (viscosity ratio,
            > 0 tracks the volume fraction every vofk steps)
  steps     steps of one pass, monitor: the cells' volume, area and centroid are
            read back after every step
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from preprocess_src_b200 import configs, mesh
from preprocess_src_b200.adjoint import InitialState, ShapeRun, shape_loss
from preprocess_src_b200.step import Batch, Simulation

F64 = torch.float64


def _case(name=None, **kw):
    c = dict(kind="step", flow="duct", L=64, W=32, H=32, cells=1, subdiv=3, radius=7.82, white=0, storage="f32", tau=1.0,
             br=0.0, M=1, lam=0.0, vofk=50, steps=20, monitor=False)
    c.update(kw)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # the smallest coupled run: a test-sized duct with one coarse cell (162 vertices), where every step is a
        # handful of short kernels
        _case("duct_small_162v", L=32, W=20, H=20, subdiv=2, radius=5.0, steps=40),
        # the single-cell duct of the parity and precision studies (642 vertices), stepped one by one with the
        # cell's shape logged at every step
        _case("duct_single_642v_monitor", steps=40, monitor=True),
        # an odd-sized duct at another relaxation time: none of its extents suits a tile or a warp
        _case("duct_odd_97x45x51", L=97, W=45, H=51, cells=9, subdiv=3, radius=6.1, tau=0.83, steps=40),
        # an ordinary suspension: red cells and stiffer white cells on their own mesh, sub-cycled
        # (two lattice steps per membrane step)
        _case("duct_mid_red_white_m2", L=160, W=64, H=64, cells=20, subdiv=4, white=4, M=2, steps=30),
        # the dense suspension, the library's headline workload
        _case("dense_200x2562v_f32", L=256, W=128, H=128, cells=200, subdiv=4, steps=60),
        # the same with half-precision populations, monitored at every step as a production run is
        _case("dense_200x2562v_f16_monitor", L=256, W=128, H=128, cells=200, subdiv=4, storage="f16", steps=60, monitor=True),
        # shear flow between moving walls with bending resistance: cells tank-tread across both periodic boundaries
        _case("shear_bending_6x642v", flow="shear", L=64, W=52, H=44, cells=6, subdiv=3, radius=6.0, br=0.02, steps=40),
        # cells with a more viscous interior: the volume fraction is advected every step and solved for once per pass
        _case("duct_viscosity_ratio", L=96, W=48, H=48, cells=8, subdiv=3, radius=6.5, lam=5.0, vofk=50, steps=50),
        # the plasma alone in a circular vessel
        _case("tube_plasma_220", flow="tube", L=220, W=77, H=77, cells=0, steps=60),
        # uneven capillaries with one cell each, stepped together (a parameter study)
        _case("capillaries_96", kind="batch", cells=96, L=128, W=32, H=32, steps=40),
        # one gradient of a shape fit: forward with checkpoints and the reverse sweep
        _case("gradient_single_642v", kind="adjoint", steps=60),
        # a state taken over from the reference's arrays and handed back (restart, coupling)
        _case("state_in_out_128x64x64", kind="io", L=128, W=64, H=64, cells=12, subdiv=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["duct", "duct", "duct", "dense", "shear", "vof", "tube", "batch", "adjoint", "io"])
    W, H = _log(rng, 20, 72), _log(rng, 20, 72)
    L, subdiv = _log(rng, 24, 200), rng.choice([2, 3, 3, 4])
    radius = round(min(7.82, (min(W, H) - 8.5) / 2.3), 2)
    most = lambda w, h, r: max(1, int(0.09 * L * w * h / (4.19 * (r + 0.6) ** 3)))  # noqa: E731
    c = dict(L=L, W=W, H=H, radius=radius, subdiv=subdiv, storage=rng.choice(["f32", "f32", "f16"]),
             tau=rng.choice([1.0, 1.0, round(rng.uniform(0.75, 1.2), 2)]), monitor=rng.random() < 0.4, steps=rng.randint(10, 40))
    if kind == "dense":
        W, H = _log(rng, 60, 126), _log(rng, 60, 126)
        c.update(L=_log(rng, 96, 250), W=W, H=H, radius=7.82, subdiv=4, cells=0)
        L = c["L"]
        c["cells"] = rng.randint(1, min(190, most(W, H, 7.82)))
        return _case(**c)
    if kind == "duct":
        n = rng.randint(1, min(100, most(W, H, radius)))
        white = rng.choice([0, 0, min(3, n - 1)])
        return _case(**dict(c, cells=n - white, white=white, M=rng.choice([1, 1, 2, 3]), br=rng.choice([0.0, 0.0, 0.02])))
    if kind == "shear":
        H, W, L = max(H, 24), max(W, 32), max(L, 32)
        radius = round(min(7.0, (min(H, 72) - 10) / 2.6), 2)
        room = int(0.05 * L * W * H / (4.19 * (radius + 0.6) ** 3))
        return _case(**dict(c, flow="shear", L=L, W=W, H=H, radius=radius, cells=rng.randint(1, max(1, min(60, room))), br=rng.choice([0.0, 0.02])))
    if kind == "vof":
        return _case(**dict(c, L=min(L, 128), storage="f32", lam=round(rng.uniform(2.0, 6.0), 1), vofk=c["steps"], subdiv=3,
                            cells=rng.randint(1, min(20, most(W, H, radius)))))
    if kind == "tube":
        return _case(**dict(c, flow="tube", W=W | 1, H=W | 1, cells=0, monitor=False))
    if kind == "batch":
        return _case(kind="batch", cells=rng.randint(3, 90), L=128, W=32, H=32, steps=rng.randint(15, 40), storage=c["storage"])
    if kind == "adjoint":
        return _case(kind="adjoint", L=_log(rng, 32, 72), W=rng.randint(26, 36), H=rng.randint(26, 36), subdiv=rng.choice([2, 3]),
                     steps=rng.randint(20, 70))
    return _case(**dict(c, kind="io", cells=rng.randint(1, min(60, most(W, H, radius))), steps=0, monitor=False, tau=1.0))


# ---- inputs -------------------------------------------------------------------


def _storage(case):
    return 1 if case["storage"] == "f16" else 0


def _place(rng, n, r, lo, hi, periods):
    """n sphere centres in [lo, hi] at least 2 r + 1 apart (minimum image along the axes with a period)."""
    got = np.empty((0, 3))
    for _ in range(200000):
        if len(got) == n:
            return got
        c = lo + (hi - lo) * rng.random(3)
        d = got - c
        for k, p in enumerate(periods):
            if p:
                d[:, k] -= p * np.round(d[:, k] / p)
        if not (np.einsum("ij,ij->i", d, d) < (2 * r + 1) ** 2).any():
            got = np.vstack([got, c])
    raise RuntimeError("the cells of %r do not fit" % (n,))


def _spec(case, seed):
    """The configs.Case of a single simulation and, with white cells, theirs."""
    rng = np.random.default_rng(seed)
    kw = dict(tau=case["tau"], storage=_storage(case), br=case["br"], M=case["M"])
    if case["lam"] > 0:
        kw.update(lambda1=case["lam"], vof_k=case["vofk"], vof_residual=1e-10)
    L, W, H, r = case["L"], case["W"], case["H"], case["radius"]
    shape, tri = mesh.rbc_shape(case["subdiv"])
    n, nw = case["cells"], case["white"]
    rb = r * mesh.bounding_radius(shape)
    if case["flow"] == "shear":
        base = configs.shear_case("shear", W - 4, H - 4, L, sr=4e-3, **kw)
        hy = (H - 4) / 2 - rb - 1.5
        centers = _place(rng, n, rb, np.array([-(W - 4) / 2, -hy, -L / 2]), np.array([(W - 4) / 2, hy, L / 2]), (W - 4, 0, L))
    elif case["flow"] == "tube":
        return configs.tube_case("tube", L, (W - 4) / 2.0 + 0.3, **kw), None
    else:
        base = configs.duct_case("duct", L, W, H, **kw)
        hx, hy = (W - 1) / 2 - 1 - rb - 2.0, (H - 1) / 2 - 1 - rb - 2.0
        if n + nw == 1 or min(hx, hy) <= 0:
            centers = np.array([[0.4, -0.3, L * (k + 0.5) / max(1, n + nw) - L / 2] for k in range(n + nw)]).reshape(-1, 3)
        else:
            centers = _place(rng, n + nw, rb, np.array([-hx, -hy, -L / 2]), np.array([hx, hy, L / 2]), (0, 0, L))
    cells = [mesh.place(shape, mesh.random_rotation(rng), r, c) for c in centers[:n]]
    spec = configs.Case(name="case", params=base.params, bc=base.bc, tri=tri.astype(np.int32),
                        xr=np.concatenate(cells).reshape(-1) if n else np.zeros(0), ncell=n, vertex=len(shape), element=len(tri))
    return spec, configs.sphere_cells(spec, centers[n:], subdiv=2, radius=0.6 * r, seed=seed) if nw else None


def _deformed(spec, rng):
    """The cells of spec stretched by 0.5 to 1.5 % along a random axis at constant volume, wrapped into the periodic range, [3][nv]."""
    p = spec.params
    x = spec.xr.reshape(spec.ncell, spec.vertex, 3).copy()
    for c in range(spec.ncell):
        R, a = mesh.random_rotation(rng), 1.0 + rng.uniform(0.005, 0.015)
        m = x[c].mean(axis=0)
        x[c] = (x[c] - m) @ (R @ np.diag([a, 1 / math.sqrt(a), 1 / math.sqrt(a)]) @ R.T) + m
    gx = x.mean(axis=1)
    x = x.reshape(-1, 3).T.copy()
    for k, lo, hi, len_ in ((0, "xmin", "xmax", "LX"), (2, "zmin", "zmax", "LZ")):
        if k == 2 or p["flow"] == 1:
            for a in (x[k], gx[:, k]):
                a[a < p[lo]] += p[len_]
                a[a > p[hi]] -= p[len_]
    return x, gx


E = torch.tensor([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0], [-1, -1, 0], [-1, 1, 0], [1, -1, 0],
                  [0, 1, 1], [0, -1, -1], [0, -1, 1], [0, 1, -1], [1, 0, 1], [-1, 0, -1], [1, 0, -1], [-1, 0, 1]])  # the reference's slots
WT = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
OPP = [0] + [q + 1 if q % 2 else q - 1 for q in range(1, 19)]


def _populations(spec, rng, dev):
    """A developed flow's equilibrium populations [nz][ny][nx][19] (FP64, on dev): the duct's or tube's profile with
    a weak swirl, or the shear profile."""
    p = spec.params
    nx, ny, nz = p["nx"], p["ny"], p["nz"]
    X = torch.arange(nx, dtype=F64, device=dev) - (nx - 1) / 2
    Y = (torch.arange(ny, dtype=F64, device=dev) - (ny - 1) / 2)[:, None]
    Z = (torch.arange(nz, dtype=F64, device=dev) - 2)[:, None, None] * (2 * math.pi / (nz - 4))
    um = float(rng.uniform(0.8, 1.2)) * 4e-3
    if p["flow"] == 1:
        w = (p["sr"] * Y).expand(ny, nx)
        s = torch.clamp(1 - (Y / ((ny - 4) / 2)) ** 2, min=0).expand(ny, nx)
    else:
        s = torch.clamp(1 - (X / ((nx - 2) / 2)) ** 2, min=0) * torch.clamp(1 - (Y / ((ny - 2) / 2)) ** 2, min=0)
        w = um * s
    k = um * 0.05
    u = torch.stack([k * s * torch.sin(Z), k * s * torch.cos(Z), w.expand(nz, ny, nx) * (1 + 0.02 * torch.cos(Z))])
    rho = 1 + 1e-4 * s * torch.sin(Z + 0.3)
    eu = torch.einsum("qk,kzyx->zyxq", E.to(dev, F64), u)
    f = torch.tensor(WT, dtype=F64, device=dev) * (rho[..., None] * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * (u * u).sum(0)[..., None]))
    return torch.where((torch.from_numpy(spec.bc.reshape(nz, ny, nx)).to(dev) == configs.COMP)[..., None], f, torch.zeros((), dtype=F64, device=dev))


def _device():
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")


def _pinned(*shape):
    return torch.empty(*shape, dtype=F64, pin_memory=torch.cuda.is_available())


def _p(t, *index):
    if t is None:
        return None
    return ctypes.cast((t[index] if index else t).data_ptr(), ctypes.POINTER(ctypes.c_double))


def _rows(t):
    return [_p(t, k) for k in range(3)]


def _buffers(n, nv):
    """Page-locked buffers for the fields and, with cells, for their positions, velocities and forces."""
    out = {"density": _pinned(n), "velocity": _pinned(3, n)}
    if nv:
        out.update({k: _pinned(3, nv) for k in ("x", "u", "force")})
    return out


class _Sim:
    """A handle with the buffers its program reads results into."""

    def __init__(self, spec, white, rng, dev, out=None):
        self.sim = sim = Simulation(spec, device=dev.index or 0)
        self.spec, self.white = spec, white
        self.out = out if out is not None else _buffers(spec.n, spec.ncell * spec.vertex)
        fn = _pinned(spec.n * 19)
        fn.copy_(_populations(spec, rng, dev).reshape(-1))
        sim.import_lattice(fn.numpy())
        if spec.ncell:
            x, gx = _deformed(spec, rng)
            sim.import_cells(x=x[0], y=x[1], z=x[2], xd=x.T.reshape(-1), gx=gx.reshape(-1))
        if white is not None:
            sim.add_wbc(white, rgs=2.5, br=0.0)
            self.out.update({"white_" + k: _pinned(3, white.ncell * white.vertex) for k in ("x", "u", "force")})
            x, gx = _deformed(white, rng)
            sim.import_wbc(x=x[0], y=x[1], z=x[2], xd=x.T.reshape(-1), gx=gx.reshape(-1))

    def read(self):
        sim, o = self.sim, self.out
        if self.spec.ncell:
            sim._call("rbc_export_ref_cells", *_rows(o["x"]), None, *_rows(o["u"]), *_rows(o["force"]), None)
        if self.white is not None:
            sim._call("rbc_export_ref_wbc", *_rows(o["white_x"]), None, *_rows(o["white_u"]), *_rows(o["white_force"]), None)
        sim._call("rbc_export_ref_lattice", None, _p(o["density"]), *_rows(o["velocity"]))


def _batch_specs(case, seed):
    """Capillaries of the batch study: 32 x 32 ducts of lengths 48 ... 128 in turn, Gs log-uniform in [1e-4, 2e-3], g uniform in [5e-7, 2e-6]."""
    rng = np.random.default_rng(seed)
    return [configs.duct_case("capillary", L, 32, 32, centers_duct=[(L / 2.0, 16.0, 16.0)], subdiv=3, seed=int(rng.integers(1 << 31)),
                              g=float(rng.uniform(5e-7, 2e-6)), Gs=float(np.exp(rng.uniform(np.log(1e-4), np.log(2e-3)))), storage=_storage(case))
            for L in (48 + 16 * (i % 6) for i in range(case["cells"]))]


def prepare(case, seed):
    dev = _device()
    rng = np.random.default_rng([seed, 1])
    s = {"case": case}
    if case["kind"] == "batch":
        specs = _batch_specs(case, seed)
        # one buffer per quantity, the capillaries one after another
        nv, n = [c.ncell * c.vertex for c in specs], [c.n for c in specs]
        s["out"] = _buffers(sum(n), sum(nv))
        ov, on = np.cumsum([0] + nv), np.cumsum([0] + n)
        part = lambda t, i: t[on[i]:on[i + 1]] if t.dim() == 1 else t.view(-1)[3 * on[i]:3 * on[i + 1]].view(3, -1) if t.size(1) == on[-1] \
            else t.view(-1)[3 * ov[i]:3 * ov[i + 1]].view(3, -1)  # noqa: E731
        s["sims"] = [_Sim(c, None, rng, dev, {k: part(t, i) for k, t in s["out"].items()}) for i, c in enumerate(specs)]
        s["batch"] = Batch([x.sim for x in s["sims"]])
        return s
    spec, white = _spec(case, seed)
    s["spec"] = spec
    if case["kind"] == "io":
        s["sim"] = Simulation(spec, device=dev.index or 0)
        s["fn"], s["out"] = _pinned(spec.n * 19), _pinned(spec.n * 19)
        s["fn"].copy_(_populations(spec, rng, dev).reshape(-1))
        x, gx = _deformed(spec, rng)
        nv = spec.ncell * spec.vertex
        s["x"], s["xd"], s["gx"], s["nd"] = _pinned(3, nv), _pinned(3 * nv), _pinned(3 * spec.ncell), _pinned(4 * spec.ncell * spec.element)
        s["x"].copy_(torch.from_numpy(x))
        s["xd"].copy_(torch.from_numpy(x.T.reshape(-1).copy()))
        s["gx"].copy_(torch.from_numpy(gx.reshape(-1).copy()))
        v = spec.xr.reshape(spec.ncell, spec.vertex, 3)[:, spec.tri]
        a, b = v[:, :, 1] - v[:, :, 0], v[:, :, 2] - v[:, :, 0]
        g11, g12, g22 = (a * a).sum(-1), (a * b).sum(-1), (b * b).sum(-1)
        s["nd"].copy_(torch.from_numpy((np.stack([g22, -g12, -g12, g11], -1) / (g11 * g22 - g12 * g12)[..., None]).reshape(-1)))
        s["outx"], s["outxd"] = _pinned(3, nv), _pinned(3 * nv)
        return s
    if case["kind"] == "adjoint":
        x = _Sim(spec, white, rng, dev)
        s["sim"], s["init"] = x.sim, InitialState(x.sim)
        s["x0"] = torch.from_numpy(_deformed(spec, rng)[0]).requires_grad_()
        s["theta"] = torch.tensor([5e-4, 100.0, 1e-6], dtype=F64, requires_grad=True)
        s["target"] = s["x0"].detach() + 0.1 * torch.from_numpy(rng.standard_normal((3, spec.vertex)))
        return s
    s["sim"] = _Sim(spec, white, rng, dev)
    if case["lam"] > 0:
        s["sim"].sim.front_tracking()
        s["vf"] = _pinned(spec.n)
    if case["monitor"]:
        s["log"] = _pinned(case["steps"], 5 * spec.ncell)
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "batch":
        s["batch"].step(case["steps"])
        for x in s["sims"]:
            x.read()
        return s["out"]
    if case["kind"] == "io":
        sim = s["sim"]
        sim._call("rbc_import_ref_lattice", _p(s["fn"]))
        sim._call("rbc_import_ref_cells", *[_p(s["x"], k) for k in range(3)], _p(s["xd"]), _p(s["nd"]), None, _p(s["gx"]))
        sim._call("rbc_export_ref_lattice", _p(s["out"]), None, None, None, None)
        sim._call("rbc_export_ref_cells", *[_p(s["outx"], k) for k in range(3)], _p(s["outxd"]), *[None] * 7)
        return {"fn": s["out"], "x": s["outx"], "xd": s["outxd"]}
    if case["kind"] == "adjoint":
        spec, sim = s["spec"], s["sim"]
        s["theta"].grad = s["x0"].grad = None
        final = ShapeRun.apply(s["theta"], s["x0"], sim, s["init"], case["steps"], 20)
        loss = shape_loss(final, s["target"], spec.params["LX"], spec.params["LZ"])
        loss.backward()
        return {"loss": loss.detach(), "final": final.detach(), "dGs": s["theta"].grad[0], "dC": s["theta"].grad[1], "dg": s["theta"].grad[2],
                "dx0": s["x0"].grad}
    x = s["sim"]
    sim = x.sim
    if case["monitor"]:
        for k in range(case["steps"]):
            sim.step(1)
            sim._call("rbc_cell_metrics_async", _p(s["log"], k))
    else:
        sim.step(case["steps"])
    x.read()
    out = dict(x.out)
    if case["monitor"]:
        out["log"] = s["log"]
    if case["lam"] > 0:
        sim._call("rbc_export_ref_vof", _p(s["vf"]), None)
        out["vf"] = s["vf"]
    return out


# ---- what a pass cannot do without -----------------------------------------


def _sizes(case):
    """(fluid nodes, lattice nodes with the reference's BUFF planes, vertices, elements) of one simulation."""
    L, W, H = case["L"], case["W"], case["H"]
    fluid = L * ((W - 4) * (H - 4) if case["flow"] == "shear" else math.pi * (W - 4) ** 2 / 4 if case["flow"] == "tube" else (W - 2) * (H - 2))
    nodes = (L + 4) * W * H
    V, T = 10 * 4 ** case["subdiv"] + 2, 20 * 4 ** case["subdiv"]
    return fluid, nodes, case["cells"] * V + case["white"] * 162, case["cells"] * T + case["white"] * 320


def work(case):
    if case["kind"] == "batch":
        one = work(dict(case, kind="step", cells=1, L=88, subdiv=3))
        return {k: v * case["cells"] for k, v in one.items()}
    fluid, nodes, nv, ne = _sizes(case)
    if case["kind"] == "io":
        # the FP64 lattice and cells cross the host link both ways and the FP32 or FP16 lattice is written and read once
        return {"bytes": 2 * (8 * 19 * nodes + 48 * nv) + 32 * ne + 2 * 19 * fluid * (2 if case["storage"] == "f16" else 4), "flops": 19 * 2 * fluid}
    # populations in and out, density and velocity; positions, metric and forces of the membrane, the positions of the
    # spread, the advection and the volume correction
    per_node = (104 if case["storage"] == "f16" else 180) - 12
    b = fluid * per_node * case["steps"] + (24 * nv + 32 * ne + 12 * nv + 36 * nv + 84 * nv + 48 * nv) * (case["steps"] // case["M"])
    fl = fluid * 250.0 * case["steps"] + (ne * 120 + nv * (16 * 60 + 64 * 10 + 4 * 64 * 7 + 200)) * (case["steps"] / case["M"])
    if case["lam"] > 0:
        b += fluid * (3 * 32 + 8) * case["steps"] + 10 * 130 * fluid
        fl += fluid * 400.0 * case["steps"]
    if case["br"]:
        fl += ne * 3 * 250.0 * case["steps"] / case["M"]
    if case["kind"] == "adjoint":   # forward, recomputation, reverse (reading the stored step once)
        return {"bytes": 3 * b + case["steps"] * (19 * 8 + 64) * fluid, "flops": 4.5 * fl}
    return {"bytes": b + 8 * 4 * nodes + 72 * nv, "flops": fl}


def tolerance(case):
    """About four times the largest error of any output against ``exact`` over the listed cases and 22 drawn ones: FP32 populations
    1e-5 (the membrane force of the largest suspension; velocities 2e-6, positions 2e-8), FP16 populations 8e-4 (force; velocities 1.5e-4),
    gradients 4e-6; a state moved in and out keeps its storage type's rounding (5e-11 and 1e-6 of the populations)."""
    half = case["storage"] == "f16"
    if case["kind"] == "io":
        return {"rel": 4e-6 if half else 2e-10}
    if case["kind"] == "adjoint":
        return {"rel": 2e-5}
    return {"rel": 3e-3 if half else 4e-5}


# ---- the step in FP64 ---------------------------------------------------------


class _Pop:
    """One cell population in FP64: positions X (after the volume correction) and Xd (before), [ncell][V][3]."""

    def __init__(self, spec, x, gx, rgs, br, dev):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        self.n, self.V, self.tri = spec.ncell, spec.vertex, t(spec.tri).long()
        self.X = x if torch.is_tensor(x) else t(x.T.reshape(self.n, self.V, 3))
        self.Xd, self.gx, self.rgs, self.br = self.X, t(gx), rgs, br
        ref = t(spec.xr.reshape(self.n, self.V, 3))
        e1, e2 = self.edges(ref, None)
        self.G = [(e1 * e1).sum(-1), (e1 * e2).sum(-1), (e2 * e2).sum(-1)]
        self.V0 = self.measure(ref)[0]
        self.deg = torch.zeros(self.V, dtype=F64, device=dev).index_add_(0, self.tri.reshape(-1), torch.ones(3 * len(self.tri), dtype=F64, device=dev))
        # the four vertices about every edge (the edge's ends in the middle), each edge from both of its triangles
        last, pairs = {}, []
        for a, b, c in spec.tri.tolist():
            for i, j, k in ((a, b, c), (b, c, a), (c, a, b)):
                last[(i, j)] = k
        for (i, j), k in last.items():
            if i < j:
                pairs.append((k, i, j, last[(j, i)]))
        self.quads = t(np.array(pairs)).long()

    def edges(self, X, L):
        a, b, c = (X[:, self.tri[:, k]] for k in range(3))
        e1, e2 = b - a, c - a
        return (e1, e2) if L is None else (e1 - L * torch.round(e1 / L), e2 - L * torch.round(e2 / L))

    def scatter(self, per, base=None):
        """Element values per[k] [n][E][...] of vertex k summed at the vertices."""
        out = torch.zeros(self.n, self.V, *per[0].shape[2:], dtype=F64, device=per[0].device)
        for k in range(3):
            out = out.index_add(1, self.tri[:, k], per[k])
        return out

    def forces(self, C, L):
        e1, e2 = self.edges(self.Xd, L)
        g11, g12, g22 = (e1 * e1).sum(-1), (e1 * e2).sum(-1), (e2 * e2).sum(-1)
        G11, G12, G22 = self.G
        det, detG = g11 * g22 - g12 * g12, G11 * G22 - G12 * G12
        I1 = (G22 * g11 - 2 * G12 * g12 + G11 * g22) / detG - 2
        I2 = det / detG - 1
        Js = torch.sqrt(I2 + 1)
        ca, cb = self.rgs * (I1 + 1) / Js, (C * I2 - 1) * Js
        t00, t01, t11 = ca * G22 / detG + cb * g22 / det, -ca * G12 / detG - cb * g12 / det, ca * G11 / detG + cb * g11 / det
        gab = torch.sqrt(det)
        lb = 0.5 * gab[..., None] * (t00[..., None] * e1 + t01[..., None] * e2)
        lc = 0.5 * gab[..., None] * (t01[..., None] * e1 + t11[..., None] * e2)
        b = self.scatter([-lb - lc, lb, lc])
        area = self.scatter([gab, gab, gab])
        # the P1 mass matrix, gab / 12 on and gab / 24 off the diagonal, by Chebyshev iteration on [1/2, 2] of its Jacobi scaling
        dg = (area / 12)[..., None]
        mul = lambda q: self.scatter([gab[..., None] / 24 * (q[:, self.tri].sum(2) + q[:, self.tri[:, k]]) for k in range(3)]) / dg  # noqa: E731
        r, x, sigma = b / dg, torch.zeros_like(b), 1.25 / 0.75
        d, rho = r / 1.25, 1 / sigma
        for _ in range(34):
            x = x + d
            r = r - mul(d)
            rn = 1 / (2 * sigma - rho)
            d, rho = rn * rho * d + 2 * rn / 0.75 * r, rn
        return -x * (area / 6)[..., None]

    def bending(self, L):
        with torch.enable_grad():
            X = self.X.detach().requires_grad_()
            p = [X[:, self.quads[:, k]] for k in range(4)]
            mi = lambda d: d - L * torch.round(d.detach() / L)  # noqa: E731
            a, b, c = mi(p[1] - p[0]), mi(p[2] - p[0]), mi(p[3] - p[0])
            xi, ze = torch.linalg.cross(a, b), torch.linalg.cross(b - c, a - c)
            cos = (xi * ze).sum(-1) / (xi.norm(dim=-1) * ze.norm(dim=-1))
            (g,) = torch.autograd.grad(torch.where(1 - cos * cos < 1e-6, cos.detach(), cos).sum(), X)
        return 2 / math.sqrt(3) * self.br * g

    def measure(self, p):
        a, b, c = (p[:, self.tri[:, k]] for k in range(3))
        n = torch.linalg.cross(b - a, c - a)
        return ((a + b + c) * n).sum((1, 2)) / 18, n.norm(dim=-1).sum(1) / 2

    def correct(self, box):
        L, lo, hi = box
        p = self.X - L * torch.round((self.X - self.gx[:, None]) / L)
        vol, area = self.measure(p)
        for _ in range(1000):
            move = (vol.detach() - self.V0).abs() / self.V0 * 100 >= 1e-3
            if not move.any():
                break
            e = torch.linalg.cross(*self.edges(p, None))
            n = e / e.norm(dim=-1, keepdim=True)
            n = self.scatter([n, n, n]) / self.deg[:, None]
            p = p + torch.where(move, -18 * (vol - self.V0) / area / 6 * 0.1, torch.zeros_like(vol))[:, None, None] * n
            vol, area = self.measure(p)
        wrap = lambda q: q + torch.where(q < lo, L, 0 * L) - torch.where(q > hi, L, 0 * L)  # noqa: E731
        self.X, self.gx, self.vol, self.area = wrap(p), wrap(p.mean(1).detach()), vol, area


class _Exact:
    def __init__(self, spec, case, pops, fn, dev, P=None, B=None, C=None):
        p = spec.params
        self.p, self.dev, self.pops = p, dev, pops
        self.P, self.B, self.C = (p["P"] if P is None else P), (p["B"] if B is None else B), (p["C"] if C is None else C)
        self.shear = p["flow"] == 1
        xb = 2 if self.shear else 0
        nx, ny, nz = p["nx"], p["ny"], p["nz"]
        self.xb, self.dims = xb, (nz - 4, ny, nx - 2 * xb)
        bc = torch.from_numpy(spec.bc.reshape(nz, ny, nx)).to(dev)[2, :, xb:nx - xb]
        self.fluid = bc == configs.COMP
        self.f = fn.reshape(nz, ny, nx, 19)[2:nz - 2, :, xb:nx - xb].permute(3, 0, 1, 2)   # before collision, [19][z][y][x]
        self.src = [torch.roll(self.fluid, (int(E[q, 1]), int(E[q, 0])), (0, 1)) for q in range(19)]
        inf = float("inf")
        t = lambda *a: torch.tensor(a, dtype=F64, device=dev)  # noqa: E731
        self.edgeL = t(p["LX"], 1e300, p["LZ"])   # 1e300: not periodic
        self.vcbox = (t(p["LX"] if self.shear else 1e300, 1e300, p["LZ"]), t(p["xmin"] if self.shear else -inf, -inf, p["zmin"]),
                      t(p["xmax"] if self.shear else inf, inf, p["zmax"]))
        self.lo, self.hi, self.Lw = t(p["xmin"], -inf, p["zmin"]), t(p["xmax"], inf, p["zmax"]), t(p["LX"], 0, p["LZ"])
        self.off = t((nx - 1) / 2 - xb, (ny - 1) / 2, (nz - 1) / 2 - 2)
        self.vf = None
        self.tube = None
        if p["tube_r"] > 0:
            X, Y = torch.meshgrid(torch.arange(nx, dtype=F64) - (nx - 1) / 2, torch.arange(ny, dtype=F64) - (ny - 1) / 2, indexing="xy")
            X, Y, self.tube = X.to(dev), Y.to(dev), []
            for q in range(19):
                dx, dy = -int(E[q, 0]), -int(E[q, 1])
                a, b, c = dx * dx + dy * dy, X * dx + Y * dy, X * X + Y * Y - p["tube_r"] ** 2
                disc = torch.clamp(b * b - a * c, min=0).sqrt()
                ts = [(-b + disc) / max(a, 1), (-b - disc) / max(a, 1)]
                ok = [(v > 0) & (v < 1) & (b * b >= a * c) for v in ts]
                frac = torch.where(ok[0], ts[0], torch.where(ok[1], ts[1], torch.full_like(X, -1.0)))
                two = ~self.src[q] & ~self.src[OPP[q]]
                self.tube.append(torch.where(self.fluid & ~self.src[q] & ~two & (frac > 0) & (a > 0), frac, torch.full_like(X, -1.0)))
        self.iter = 0
        self.cycle_u = self.cycle_r = self.F = None

    def node(self, X):
        """The 64 stencil nodes [N][64] and weights of positions X [N][3]."""
        l = X + self.off
        base = torch.floor(l.detach())
        f = l - base
        s, c = torch.sin(0.5 * math.pi * f), torch.cos(0.5 * math.pi * f)
        w = 0.25 * torch.stack([1 - s, 1 + c, 1 + s, 1 - c], -1)             # [N][3][4]
        i = base.long()[..., None] + torch.arange(-1, 3, device=self.dev)     # [N][3][4]
        nz, ny, nx = self.dims
        ix = i[:, 0] % nx if self.shear else i[:, 0].clamp(0, nx - 1)
        iy, iz = i[:, 1].clamp(0, ny - 1), i[:, 2] % nz
        idx = (iz[:, :, None, None] * ny + iy[:, None, :, None]) * nx + ix[:, None, None, :]
        ww = w[:, 2, :, None, None] * w[:, 1, None, :, None] * w[:, 0, None, None, :]
        return idx.reshape(len(X), 64), ww.reshape(len(X), 64)

    def spread(self):
        nz, ny, nx = self.dims
        F = torch.zeros(nz * ny * nx, 3, dtype=F64, device=self.dev)
        for g in self.pops:
            idx, w = self.node(g.X.reshape(-1, 3))
            F = F.index_add(0, idx.reshape(-1), (w[..., None] * g.Fv.reshape(-1, 1, 3)).reshape(-1, 3))
        return F.reshape(nz, ny, nx, 3) * self.fluid[..., None]

    def interp(self, X, u):
        idx, w = self.node(X)
        return torch.stack([(u[..., k].reshape(-1)[idx] * w).sum(1) for k in range(3)], -1)

    def walls(self):
        """The walls' z velocity beside each row (shear mode)."""
        ny, LY = self.dims[1], self.dims[1] - 4.0
        uw = torch.zeros(ny, dtype=F64, device=self.dev)
        uw[ny - 3], uw[2] = self.p["sr"] * LY / 2, -self.p["sr"] * LY / 2
        return uw[None, :, None]

    def collide(self, F):
        p, Cr = self.p, self.p["Cr"]
        e = E.to(self.dev).tolist()
        f, fl = self.f, self.fluid
        w = torch.tensor(WT, dtype=F64, device=self.dev)[:, None, None, None]
        g = (f - w) * fl
        j = [sum(e[q][k] * g[q] for q in range(19) if e[q][k]) for k in range(3)]
        drho = g.sum(0)
        r = 1 + drho
        G = [r * self.B * F[..., 0], r * self.B * F[..., 1], r * (self.P + self.B * F[..., 2])]
        u = [(j[k] + G[k]) / (r * Cr) for k in range(3)]
        om = 1 / p["tau"] if self.vf is None else 1 / ((p["tau"] - 0.5) * (1 + (p["lambda1"] - 1) * self.vf) + 0.5)
        fo = 2 - om
        A = om * (drho - 1.5 * Cr * Cr * r * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)) - 3 * Cr * fo * (u[0] * G[0] + u[1] * G[1] + u[2] * G[2])
        post = []
        for q in range(19):
            if q == 0:
                post.append((1 - om) * g[0] + WT[0] * A)
                continue
            eu = sum(e[q][k] * u[k] for k in range(3) if e[q][k])
            eG = sum(e[q][k] * G[k] for k in range(3) if e[q][k])
            post.append((1 - om) * g[q] + WT[q] * (A + 3 * Cr * om * r * eu + 4.5 * Cr * Cr * om * r * eu * eu + fo * eG * (3 + 9 * Cr * eu)))
        new = []
        for q in range(19):
            back = post[OPP[q]]
            if self.shear and e[q][2]:
                back = back + 6 * WT[q] * r * Cr * e[q][2] * self.walls()
            if self.tube is not None and bool((self.tube[q] > 0).any()):
                t = self.tube[q]
                f2 = torch.roll(back, (-e[q][2], -e[q][1], -e[q][0]), (0, 1, 2))
                ts = torch.where(t > 0, t, torch.ones_like(t))
                back = torch.where(t > 0, torch.where(ts < 0.5, 2 * ts * back + (1 - 2 * ts) * f2, back / (2 * ts) + (2 * ts - 1) / (2 * ts) * post[q]), back)
            new.append(torch.where(self.src[q], torch.roll(post[q], (e[q][2], e[q][1], e[q][0]), (0, 1, 2)), back) + WT[q])
        self.f = torch.stack(new) * fl
        z = torch.zeros((), dtype=F64, device=self.dev)
        return torch.stack([torch.where(fl, k, z) for k in u], -1), torch.where(fl, r, z + 1)

    def step(self):
        p, M = self.p, self.p["M"]
        self.iter += 1
        ph = (self.iter - 1) % M
        if ph == 0:
            for g in self.pops:
                g.Fv = g.forces(self.C, self.edgeL)
                if g.br:
                    g.Fv = g.Fv + g.bending(self.edgeL)
            self.F = self.spread()
        u, r = self.collide(self.F)
        self.u, self.rho = (u, r) if ph == 0 else (self.u + u, torch.where(self.fluid, self.rho + r, r))
        if ph != M - 1:
            return
        self.u = self.u / M
        for g in self.pops:
            X = g.X.reshape(-1, 3)
            k1 = self.interp(X, self.u)
            k2 = self.interp(X + 0.5 * M * k1, self.u)
            k3 = self.interp(X + 0.5 * M * k2, self.u)
            k4 = self.interp(X + M * k3, self.u)
            um = (k1 + 2 * k2 + 2 * k3 + k4) / 6
            X = X + M * um
            X = X + torch.where(X < self.lo, self.Lw, 0 * self.Lw)
            X = X - torch.where(X > self.hi, self.Lw, 0 * self.Lw)
            g.U = um.reshape(g.n, g.V, 3)
            g.X = g.Xd = X.reshape(g.n, g.V, 3)
        if self.vf is not None:
            self.thinc()
            if self.iter % p["vof_k"] == 0:
                self.front_tracking()
        for g in self.pops:
            g.correct(self.vcbox)

    # volume fraction: THINC/WLIC sweeps and the Poisson problem of the indicator
    def shift(self, a, axis, d):
        return torch.roll(a, -d, 2 - axis)

    def thinc(self):
        nz, ny, nx = self.dims
        fl = self.fluid.expand(nz, ny, nx)
        ok = torch.zeros(ny, nx, dtype=torch.bool, device=self.dev)
        ok[2:ny - 1, 2:nx - 1] = True   # the reference gives the outermost layers' faces no flux
        for d in range(3):
            v = self.vf
            n = []
            for k in range(3):
                a = self.shift(v, k, 1) - self.shift(v, k, -1)
                for m in range(3):
                    if m != k:
                        a = self.shift(a, m, 1) + 2 * a + self.shift(a, m, -1)
                n.append(a / 32)
            uc = (self.u[..., d] + self.shift(self.u[..., d], d, -1)) / 2
            up = lambda a: torch.where(uc <= 0, a, self.shift(a, d, -1))  # noqa: E731
            s, vu, nd = (uc > 0).to(F64), up(v), [up(k) for k in n]
            nn = nd[0].abs() + nd[1].abs() + nd[2].abs()
            al = torch.where(up(self.shift(v, d, -1)) <= up(self.shift(v, d, 1)), 1.0, -1.0).to(F64)
            mixed = (vu < 1 - 1e-6) & (vu > 1e-6) & (nn > 1e-6)
            vs = torch.where(mixed, vu, torch.full_like(vu, 0.5))
            a1, a3 = torch.exp(2 * (2 * vs - 1) * al), math.exp(2.0)
            xc = 0.25 * torch.log((a3 * a3 - a1 * a3) / (a1 * a3 - 1))
            ft = 0.5 * (uc - al / 2 * torch.log(torch.cosh(2 * (s - uc - xc)) / torch.cosh(2 * (s - xc))))
            w = nd[d].abs() / torch.where(mixed, nn, torch.ones_like(nn))
            fx = torch.where(mixed, ft * w + vu * uc * (1 - w), vu * uc)
            fx = torch.where(ok & fl & self.shift(fl, d, -1), fx, torch.zeros_like(fx))
            self.vf = (v - (self.shift(fx, d, 1) - fx)) * fl

    def front_tracking(self):
        nz, ny, nx = self.dims
        G = torch.zeros(nz * ny * nx, 3, dtype=F64, device=self.dev)
        g = self.pops[0]
        e1, e2 = g.edges(g.X, self.edgeL)
        c = (g.X[:, g.tri[:, 0]] + (e1 + e2) / 3).reshape(-1, 3)
        idx, w = self.node(c)
        G.index_add_(0, idx.reshape(-1), (w[..., None] * (-torch.linalg.cross(e1, e2) / 2).reshape(-1, 1, 3)).reshape(-1, 3))
        G = G.reshape(nz, ny, nx, 3)
        fl = self.fluid.to(F64)
        b = sum(self.shift(G[..., k], k, 1) - self.shift(G[..., k], k, -1) for k in range(3)) / 2 / -6.0 * fl
        mul = lambda q: (q - sum(self.shift(q, k, d) for k in range(3) for d in (1, -1)) / 6) * fl  # noqa: E731
        x = torch.zeros_like(b)
        r = b.clone()
        d, rr, bb = r, (r * r).sum(), (b * b).sum()
        for k in range(4000):
            q = mul(d)
            a = rr / (d * q).sum()
            x, r = x + a * d, r - a * q
            rn = (r * r).sum()
            if k % 10 == 9 and rn < 1e-26 * bb:
                break
            d, rr = r + rn / rr * d, rn
        self.vf = x

    def field(self):
        """Density and velocity in the reference's layout, [4][n]."""
        p = self.p
        z = (torch.arange(p["nz"], device=self.dev) - 2) % self.dims[0]
        x = (torch.arange(p["nx"], device=self.dev) - self.xb) % self.dims[2] if self.shear else torch.arange(p["nx"], device=self.dev)
        a = torch.cat([self.rho[None], self.u.permute(3, 0, 1, 2)])
        return a[:, z][..., x].reshape(4, -1)

    def results(self):
        f = self.field()
        out = {"density": f[0], "velocity": f[1:]}
        for name, g in zip(("", "white_"), self.pops):
            out.update({name + "x": _flat(g.X), name + "u": _flat(g.U), name + "force": _flat(g.Fv)})
        return out

    def whole(self, a):
        z = (torch.arange(self.p["nz"], device=self.dev) - 2) % self.dims[0]
        return a[z].reshape(-1)


def _flat(a):
    return a.reshape(-1, 3).T


def _exact_sim(spec, white, rng, case, dev):
    fn = _populations(spec, rng, dev)
    pops = []
    if spec.ncell:
        pops.append(_Pop(spec, *_deformed(spec, rng), spec.params["rgs"], spec.params["br"], dev))
    if white is not None:
        pops.append(_Pop(white, *_deformed(white, rng), 2.5, 0.0, dev))
    return _Exact(spec, case, pops, fn, dev)


def exact(case, seed):
    dev = _device()
    rng = np.random.default_rng([seed, 1])
    if case["kind"] == "batch":
        got = []
        with torch.no_grad():
            for spec in _batch_specs(case, seed):
                x = _exact_sim(spec, None, rng, case, dev)
                for _ in range(case["steps"]):
                    x.step()
                got.append(x.results())
        return {k: torch.cat([r[k].reshape(-1) for r in got]).reshape(got[0][k].dim() == 1 and (-1,) or (3, -1)) for k in got[0]}
    spec, white = _spec(case, seed)
    if case["kind"] == "io":
        fn = _populations(spec, rng, dev)
        x = torch.from_numpy(_deformed(spec, rng)[0])
        return {"fn": fn.reshape(-1), "x": x, "xd": x.T.reshape(-1).contiguous()}
    if case["kind"] == "adjoint":
        fn = _populations(spec, rng, dev)
        _, gx = _deformed(spec, rng)
        x0 = torch.from_numpy(_deformed(spec, rng)[0]).requires_grad_()
        th = torch.tensor([5e-4, 100.0, 1e-6], dtype=F64, requires_grad=True)
        target = x0.detach() + 0.1 * torch.from_numpy(rng.standard_normal((3, spec.vertex)))
        td = th.to(dev)
        pop = _Pop(spec, x0.T.reshape(1, -1, 3).to(dev), gx, 1.0, 0.0, dev)
        x = _Exact(spec, case, [pop], fn, dev, P=td[2] / 2, B=td[0] / 2, C=td[1])
        for _ in range(case["steps"]):
            x.step()
        final = _flat(pop.X)
        d = final.cpu() - target
        L = torch.tensor([spec.params["LX"], 1e300, spec.params["LZ"]], dtype=F64)[:, None]
        d = d - L * torch.round(d.detach() / L)
        loss = (d * d).sum(0).mean()
        loss.backward()
        return {"loss": loss.detach(), "final": final.detach(), "dGs": th.grad[0], "dC": th.grad[1], "dg": th.grad[2], "dx0": x0.grad}
    with torch.no_grad():
        x = _exact_sim(spec, white, rng, case, dev)
        log = []
        if case["lam"] > 0:
            x.front_tracking()
        for _ in range(case["steps"]):
            x.step()
            if case["monitor"]:
                g = x.pops[0]
                log.append(torch.cat([g.vol, g.area, g.gx.T.reshape(-1)]))
        out = x.results()
        if case["monitor"]:
            out["log"] = torch.stack(log)
        if case["lam"] > 0:
            out["vf"] = x.whole(x.vf)
    return out
