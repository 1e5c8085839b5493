"""Workloads of the Kohn-Sham hot path, as a program that uses this package runs them.

Each case is a dict of plain values; ``kind`` names the call:

* ``hpsi``     H psi of an orbital block on a monitor A-grid or the legacy grid (``ops.apply_hamiltonian_block``)
* ``kinetic``  T psi of one orbital (``ops.apply_kinetic_operator``)
* ``poisson``  the open-boundary Hartree solve of one SCF step (``poisson.solve_poisson_device``)
* ``lsda``     exchange-correlation energy and potentials (``xc.lsda_device``)
* ``density``  spin density of a block of occupied orbitals, renormalised (``density``)
* ``subspace`` the block algebra of one eigensolver iteration: two Gram products of the stacked basis and residual
  block and the rotations to the next basis (``ks.BlockLA``)
* ``eigen``    a whole fixed-potential eigensolve (``ks.solve_fixed_potential_static_local_eigenproblem``)
"""

import math
from collections import OrderedDict
from dataclasses import replace

import numpy as np
import torch

from isogriddft_gb300 import density, ks, ops, poisson, xc
from isogriddft_gb300.config import H2_BENCHMARK_CASE
from isogriddft_gb300.device import device_grid
from isogriddft_gb300.grid import (build_default_h2_grid_spec, build_grid_geometry, build_monitor_grid_for_case,
                                   build_two_peak_element_parameters)

DT = {"fp32": torch.float32, "fp64": torch.float64}


def listed():
    return [
        # the operator benchmark of this repository: a 16-orbital block on the 128^3 A-grid, FP32
        dict(name="hpsi_f32_128x16", kind="hpsi", grid="monitor", nx=128, ny=128, nz=128, nb=16, closure="trial_fix",
             dtype="fp32"),
        # the default A-grid of the H2 runs (67x67x81, odd rows) with the eigensolver's working block for one
        # state (12k + 8 = 20) and the eigensolver's default closure
        dict(name="hpsi_f32_67x67x81x20", kind="hpsi", grid="monitor", nx=67, ny=67, nz=81, nb=20,
             closure="production", dtype="fp32"),
        # the same grid and block in the default precision of the drop-in functions
        dict(name="hpsi_f64_67x67x81x20", kind="hpsi", grid="monitor", nx=67, ny=67, nz=81, nb=20,
             closure="trial_fix", dtype="fp64"),
        # the largest: the 32-column block of the C6H6 study on its 192^3 A-grid
        dict(name="hpsi_f32_192x32", kind="hpsi", grid="monitor", nx=192, ny=192, nz=192, nb=32, closure="trial_fix",
             dtype="fp32"),
        # the smallest call: T psi of one orbital on the 51^3 legacy grid (latency and launches)
        dict(name="kinetic_f64_legacy51", kind="kinetic", grid="legacy", nx=51, ny=51, nz=51, dtype="fp64"),
        # Hartree solve of the 128^3 benchmark (Gaussian charge), mixed precision
        dict(name="poisson_mixed_128", kind="poisson", grid="monitor", nx=128, ny=128, nz=128, precision="mixed",
             tolerance=1e-11),
        # Hartree solve on the default A-grid in the default precision
        dict(name="poisson_f64_67x67x81", kind="poisson", grid="monitor", nx=67, ny=67, nz=81, precision="fp64",
             tolerance=1e-11),
        # LSDA on the 128^3 grid in the default precision: energy, potentials, energy per particle and density
        dict(name="lsda_f64_128", kind="lsda", grid="monitor", nx=128, ny=128, nz=128, math="fp64",
             functional="lda,vwn"),
        # density of the benchmark's 16 orbitals
        dict(name="density_f32_128x16", kind="density", grid="monitor", nx=128, ny=128, nz=128, nb=16, dtype="fp32"),
        # block algebra of one iteration: the FP64 drop-in (m = 20, k = 1) on the default A-grid
        dict(name="subspace_f64_67x67x81_20_1", kind="subspace", grid="monitor", nx=67, ny=67, nz=81, m=20, k=1,
             dtype="fp64"),
        # block algebra of one iteration of the C6H6 study: block of 32, 15 states, FP32
        dict(name="subspace_f32_192_32_15", kind="subspace", grid="monitor", nx=192, ny=192, nz=192, m=32, k=15,
             dtype="fp32"),
        # a whole eigensolve, as the drop-in runs it by default, one state on the default A-grid
        dict(name="eigen_f64_67x67x81", kind="eigen", grid="monitor", nx=67, ny=67, nz=81, k=1, closure="trial_fix",
             precision="fp64"),
    ]


def _edge(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hpsi", "hpsi", "hpsi", "kinetic", "poisson", "lsda", "density", "subspace", "subspace",
                       "eigen"])
    legacy = rng.random() < 0.2
    grid = "legacy" if legacy else "monitor"
    lo, hi = {"poisson": (17, 128), "eigen": (21, 70), "lsda": (13, 128)}.get(kind, (13, 192))
    n = [_edge(rng, lo, hi) for _ in range(3)]
    c = dict(kind=kind, grid=grid, nx=n[0], ny=n[1], nz=n[2])
    points = n[0] * n[1] * n[2]
    if kind == "hpsi":
        c["dtype"] = rng.choice(["fp32", "fp32", "fp64"])
        most = min(32, max(1, (16 * 128**3 if c["dtype"] == "fp64" else 32 * 192**3) // points))
        c["nb"] = min(most, _edge(rng, 1, 32))
        c["closure"] = rng.choice(["trial_fix", "production"])
    elif kind == "kinetic":
        c["dtype"] = rng.choice(["fp32", "fp64"])
    elif kind == "poisson":
        c["precision"] = rng.choice(["mixed", "fp64"])
        c["tolerance"] = 1e-11
    elif kind == "lsda":
        c["math"] = rng.choice(["fp64", "fp64", "fp32"])
        c["functional"] = rng.choice(["lda,vwn", "lda,vwn", "lda,pw92"])
    elif kind == "density":
        c["dtype"] = rng.choice(["fp32", "fp64"])
        c["nb"] = _edge(rng, 1, 32)
    elif kind == "subspace":
        c["dtype"] = rng.choice(["fp32", "fp32", "fp64"])
        c["k"] = _edge(rng, 1, 15)
        c["m"] = c["k"] + _edge(rng, 3, 20)
        if c["dtype"] == "fp64" and points > 10**6:  # the FP64 algebra of large grids costs more than any listed case
            c["dtype"] = "fp32"
    elif kind == "eigen":
        c.update(k=rng.choice([1, 1, 2]), closure=rng.choice(["trial_fix", "production"]),
                 precision=rng.choice(["fp64", "fp32"]))
        if legacy:
            c["closure"] = "production"
    return c


# ------------------------------------------------------------------ inputs
_GRIDS = OrderedDict()


def _geometry(c):
    """The grid of a case; a program builds it once for a molecule and keeps it for all its calls."""
    key = (c["grid"], c["nx"], c["ny"], c["nz"])
    g = _GRIDS.get(key)
    if g is None:
        shape = key[1:]
        if c["grid"] == "legacy":
            g = build_grid_geometry(replace(build_default_h2_grid_spec(H2_BENCHMARK_CASE), nx=shape[0], ny=shape[1],
                                            nz=shape[2]))
        else:
            g = build_monitor_grid_for_case(H2_BENCHMARK_CASE, shape=shape, box_half_extents=(8.0, 8.0, 10.0),
                                            element_parameters=build_two_peak_element_parameters(("H",), 4.0, 0.5),
                                            device=True)
        _GRIDS[key] = g
        while len(_GRIDS) > 2:
            _GRIDS.popitem(last=False)
    _GRIDS.move_to_end(key)
    return g


def _points(geom, dev):
    return [torch.as_tensor(np.ascontiguousarray(p), device=dev).reshape(-1)
            for p in (geom.x_points, geom.y_points, geom.z_points)]


def _to_atoms(geom, dev):
    x, y, z = _points(geom, dev)
    return [torch.sqrt((x - a.position[0])**2 + (y - a.position[1])**2 + (z - a.position[2])**2)
            for a in H2_BENCHMARK_CASE.geometry.atoms]


def _inputs(c, seed, dev):
    """(geometry, generator, the case's tensors): everything from the seed."""
    geom = _geometry(c)
    g = torch.Generator(device=dev).manual_seed(seed)
    n = c["nx"] * c["ny"] * c["nz"]
    kind = c["kind"]

    def rand(*s, dtype=torch.float64):
        return torch.randn(s, generator=g, device=dev, dtype=dtype)

    if kind in ("hpsi", "kinetic"):
        dt = DT[c["dtype"]]
        nb = c.get("nb", 1)
        w = torch.as_tensor(np.ascontiguousarray(geom.cell_volumes), device=dev).reshape(-1)
        psi = rand(nb, n, dtype=dt)
        for o in range(nb):  # unit norm in the cell-volume metric
            psi[o] /= torch.sqrt(torch.dot(psi[o].double()**2, w)).to(dt)
        depth = 2.0 + 0.1 * rand(1)
        v = sum(-depth / torch.sqrt(r * r + 0.1) for r in _to_atoms(geom, dev)).to(dt)
        shape = (c["nx"], c["ny"], c["nz"])
        return geom, dict(psi=psi.reshape((nb,) + shape), v=v.reshape(shape))
    if kind == "poisson":
        s = 0.8 + 0.02 * rand(1)
        x, y, z = _points(geom, dev)
        d = 0.1 * rand(3)
        rho = torch.exp(-0.5 * ((x - d[0])**2 + (y - d[1])**2 + (z - d[2])**2) / (s * s))
        w = torch.as_tensor(np.ascontiguousarray(geom.cell_volumes), device=dev).reshape(-1)
        return geom, dict(rho=rho * (2.0 / torch.dot(rho, w)))
    if kind == "lsda":
        r = _to_atoms(geom, dev)
        up = sum(torch.exp(-1.8 * q) for q in r) * (0.3 + 0.2 * torch.rand(n, generator=g, device=dev,
                                                                          dtype=torch.float64))
        dn = sum(torch.exp(-2.1 * q) for q in r) * (0.3 + 0.2 * torch.rand(n, generator=g, device=dev,
                                                                          dtype=torch.float64))
        return geom, dict(up=up, dn=dn)
    if kind == "density":
        return geom, dict(psi=rand(c["nb"], n, dtype=DT[c["dtype"]]) * 0.02,
                          occ=(0.5 + np.random.default_rng(seed).random(c["nb"])).tolist())
    if kind == "subspace":
        dt, mk, m = DT[c["dtype"]], c["m"] + c["k"], c["m"]
        return geom, dict(X=rand(mk, n, dtype=dt), Y=rand(mk, n, dtype=dt), C=rand(mk, m) / math.sqrt(mk))
    depth = 1.0 + 0.05 * float(rand(1))
    r = _to_atoms(geom, dev)
    v = sum(-depth / torch.sqrt(q * q + 0.3) for q in r).cpu().numpy().reshape(tuple(geom.spec.shape))
    return geom, dict(vloc=v)


def prepare(case, seed):
    c = case
    geom, t = _inputs(c, seed, torch.device("cuda"))
    s = dict(t, c=c, geom=geom)
    if c["kind"] == "eigen":
        zero = np.zeros(tuple(geom.spec.shape))
        s["context"] = ks.prepare_fixed_potential_static_local_operator(
            geom, zero, zero, "up", H2_BENCHMARK_CASE, t["vloc"], zero, zero, kinetic_version=c["closure"])
        ks.operator_for(s["context"], c["precision"])
    dg = s["dg"] = device_grid(geom)
    if c["kind"] == "subspace":
        s["la"] = ks.BlockLA(dg)
    return s


def run(s):
    c, dg, geom = s["c"], s["dg"], s["geom"]
    kind = c["kind"]
    if kind == "hpsi":
        return ops.apply_hamiltonian_block(s["psi"], geom, s["v"], kinetic_version=c["closure"], precision=c["dtype"])
    if kind == "kinetic":
        return ops.apply_kinetic_operator(s["psi"][0], geom)
    if kind == "poisson":
        sol = poisson.solve_poisson_device(dg, geom, s["rho"], tolerance=c["tolerance"], max_iterations=4000,
                                           precision=c["precision"])
        return {"potential": sol.potential, "moments": sol.moments}
    if kind == "lsda":
        return xc.lsda_device(s["up"], s["dn"], functional=c["functional"], math=c["math"], w=dg.cell_volumes)
    if kind == "density":
        integral = torch.zeros(1, dtype=torch.float64, device=dg.device)
        rho = density.build_density_device(dg, s["psi"], s["occ"], integral=integral)
        return density.renormalize_device(dg, rho, float(c["nb"]), integral)
    if kind == "subspace":
        la, X, Y, C, m = s["la"], s["X"], s["Y"], s["C"], c["m"]
        h, o = la.gram(X, Y), la.gram(X, X)
        b = la.rotate(X[:m], C[:m], X[m:], C[m:])
        hb = la.rotate(Y[:m], C[:m], Y[m:], C[m:])
        return {"XHX": h, "XX": o, "B": b, "HB": hb}
    r = ks.solve_fixed_potential_static_local_eigenproblem(
        geom, None, None, "up", c["k"], H2_BENCHMARK_CASE, operator_context=s["context"], max_iterations=400,
        tolerance=1e-3, kinetic_version=c["closure"], precision=c["precision"])
    # the orbitals' densities: an eigenvector's sign is free
    return {"eigenvalues": r.eigenvalues, "overlap": r.weighted_overlap, "density": r.orbitals**2}


def work(case):
    c = case
    n = c["nx"] * c["ny"] * c["nz"]
    geo = 7 if c["grid"] == "monitor" else 0
    es = 8 if c.get("dtype", c.get("precision", "fp64")) == "fp64" else 4
    if c["kind"] in ("hpsi", "kinetic"):
        nb = c.get("nb", 1)
        return {"bytes": n * es * (2 * nb + geo + (c["kind"] == "hpsi")),
                "flops": n * nb * (26 if geo else 18)}
    if c["kind"] == "poisson":  # the charge in, the potential out: how often the rest is read is the method's
        return {"bytes": n * (16 + 8 * geo), "flops": n * 52}
    if c["kind"] == "lsda":
        return {"bytes": n * 8 * 7, "flops": n * 150}
    if c["kind"] == "density":
        return {"bytes": n * (c["nb"] * es + 16), "flops": n * 3 * c["nb"]}
    if c["kind"] == "subspace":
        mk, m = c["m"] + c["k"], c["m"]
        return {"bytes": n * (2 * mk * es + 2 * m * es + 8), "flops": 2 * n * mk * (2 * mk + 2 * m)}
    return {"bytes": n * es * (geo + 3), "flops": n * 26}


# ------------------------------------------------------------------ 64-bit values
def _diff(f, a, h, production):
    """Centred derivative along axis a: zero beyond the faces, or one-sided second order there."""
    f = f.movedim(a, 0)
    d = torch.empty_like(f)
    d[1:-1] = (f[2:] - f[:-2]) / (2 * h)
    if production:
        d[0] = (-3 * f[0] + 4 * f[1] - f[2]) / (2 * h)
        d[-1] = (3 * f[-1] - 4 * f[-2] + f[-3]) / (2 * h)
    else:
        d[0], d[-1] = f[1] / (2 * h), -f[-2] / (2 * h)
    return d.movedim(0, a)


def _laplacian(c, geom, closure, dev):
    def t(a):
        return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=dev)

    if c["grid"] == "legacy":
        parts = []
        for p, u in ((geom.x_point_jacobian, geom.x_logical), (geom.y_point_jacobian, geom.y_logical),
                     (geom.z_point_jacobian, geom.z_logical)):
            p, du = t(p), float(u[1] - u[0])
            parts.append((p, torch.cat([p[:1], 0.5 * (p[1:] + p[:-1]), p[-1:]]), du))

        def lap(f):
            out = torch.zeros_like(f)
            for a, (p, face, du) in enumerate(parts):
                q = f.movedim(a, 0)
                pad = torch.cat([torch.zeros_like(q[:1]), q, torch.zeros_like(q[:1])])
                flux = (pad[1:] - pad[:-1]) / (du * face)[:, None, None]
                out += ((flux[1:] - flux[:-1]) / (du * p)[:, None, None]).movedim(0, a)
            return out

        return lap
    jac, inv = t(geom.jacobian), t(geom.inverse_metric_tensor)
    h = [float(u[1] - u[0]) for u in (geom.logical_x, geom.logical_y, geom.logical_z)]
    prod = closure == "production"

    def lap(f):
        g = [_diff(f, a, h[a], prod) for a in range(3)]
        out = torch.zeros_like(f)
        for a in range(3):
            out += _diff(jac * sum(inv[..., a, b] * g[b] for b in range(3)), a, h[a], prod)
        return out / jac

    return lap


def _lsda(up, dn, functional):
    """Slater exchange with VWN5 or PW92 correlation and its derivatives, in 64 bits."""
    up, dn = up.clamp_min(0.0), dn.clamp_min(0.0)
    live = up + dn >= 1e-15
    u = torch.where(live, up, 1.0).requires_grad_()
    d = torch.where(live, dn, 1.0).requires_grad_()
    with torch.enable_grad():
        r = u + d
        ex = -0.75 * (6 / math.pi)**(1 / 3) * (u**(4 / 3) + d**(4 / 3))
        rs = (3 / (4 * math.pi * r))**(1 / 3)
        z = (u - d) / r
        if functional == "lda,vwn":
            x = torch.sqrt(rs)

            def g(A, b, c, x0):
                X, X0, Q = x * x + b * x + c, x0 * x0 + b * x0 + c, math.sqrt(4 * c - b * b)
                at = torch.atan(Q / (2 * x + b))
                return A * (torch.log(x * x / X) + 2 * b / Q * at - b * x0 / X0 * (
                    torch.log((x - x0)**2 / X) + 2 * (b + 2 * x0) / Q * at))

            p, f, al = (g(0.0310907, 3.72744, 12.9352, -0.10498), g(0.01554535, 7.06042, 18.0578, -0.325),
                        g(-1 / (6 * math.pi**2), 1.13107, 13.0045, -0.0047584))
        else:

            def g(A, a1, b1, b2, b3, b4):
                s = torch.sqrt(rs)
                return -2 * A * (1 + a1 * rs) * torch.log1p(1 / (2 * A * (b1 * s + b2 * rs + b3 * rs * s
                                                                         + b4 * rs * rs)))

            p, f, al = (g(0.031091, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294),
                        g(0.015545, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517),
                        -g(0.016887, 0.11125, 10.357, 3.6231, 0.88026, 0.49671))
        fz = ((2 * u / r)**(4 / 3) + (2 * d / r)**(4 / 3) - 2) / (2**(4 / 3) - 2)
        fpp = 4 / (9 * (2**(1 / 3) - 1))
        ec = p + al * fz * (1 - z**4) / fpp + (f - p) * fz * z**4
        e = ex + r * ec
        vu, vd = torch.autograd.grad(e.sum(), (u, d))
    out = {k: torch.where(live, v.detach(), 0.0) for k, v in
           (("eps", e / r), ("v_up", vu), ("v_down", vd), ("edens", e))}
    return out


def exact(case, seed):
    c = case
    if c["kind"] in ("poisson", "eigen"):  # iterative solves: no short way to their 64-bit values
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    geom, t = _inputs(c, seed, dev)
    w = torch.as_tensor(np.ascontiguousarray(geom.cell_volumes), device=dev).reshape(-1)
    if c["kind"] in ("hpsi", "kinetic"):
        lap = _laplacian(c, geom, c.get("closure", "production"), dev)
        if c["kind"] == "kinetic":
            return -0.5 * lap(t["psi"][0].double())
        v = t["v"].double()
        return torch.stack([-0.5 * lap(p.double()) + v * p.double() for p in t["psi"]])
    if c["kind"] == "lsda":
        out = _lsda(t["up"], t["dn"], c["functional"])
        out["energy"] = torch.dot(out["edens"], w).reshape(1)
        return out
    if c["kind"] == "density":
        rho = sum(o * p.double()**2 for o, p in zip(t["occ"], t["psi"]))
        return rho * (c["nb"] / torch.dot(rho, w))
    m, C = c["m"], t["C"]
    mk, n = t["X"].shape
    out = {"XHX": torch.zeros(mk, mk, dtype=torch.float64, device=dev),
           "XX": torch.zeros(mk, mk, dtype=torch.float64, device=dev),
           "B": torch.empty(m, n, dtype=torch.float64, device=dev),
           "HB": torch.empty(m, n, dtype=torch.float64, device=dev)}
    for a in range(0, n, 1 << 20):
        at = slice(a, min(n, a + (1 << 20)))
        X, Y = t["X"][:, at].double(), t["Y"][:, at].double()
        out["XHX"] += (X * w[at]) @ Y.T
        out["XX"] += (X * w[at]) @ X.T
        out["B"][:, at] = C.T @ X
        out["HB"][:, at] = C.T @ Y
    return out
