"""Performance cases of the framework: the work its users have it do, through
the public entry points of `dpgpu`, over the range of sizes, precisions and
directions (forward, gradient, inversion) in which it is used.

A case is a dict of plain values; `kind` selects the entry point:

  point    compute_flux_gradient: the flux and d flux / d density of one history
  samples  csda_flux_samples: CSDA histories from the caller's own samples
  mc       run_backward_mc: stochastic transport of one line of sight with the
           CSDA gradient, samples drawn on the device
  los      backward_mc_batch: many lines of sight in one call
  dir      DirBatch.run: fixed-path stochastic MC over prepared directions
  wcsda    CsdaBatch.run: water-fraction CSDA flux and its sparse Jacobian
  tomo     TomoModel.vjp / .forward: voxel tomography from host arrays
  eval     TomoPaths.eval: the same on traced rays and device tensors
  solve    TomoPaths.solve: an inversion loop on the device

Sizes are those of the benchmark workloads, the tests and the reference's
defaults, and the range between them.
"""
import math
import os
import sys
from functools import lru_cache

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "diffpumas.jl_gb300"))

import dpgpu as dp  # noqa: E402
from dpgpu.workloads import directional_config, tomography_config  # noqa: E402

MASS, CTAU = 0.10565839, 658.654
AIR0, SCALE_H = 1.205, 12e3


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: one history's flux and density gradient, as a
        # density fit on a single line of sight evaluates it; latency alone
        {"name": "point_gradient_fp64", "kind": "point", "thickness": 100.0, "elevation": 45.0},
        # the deterministic backward MC of the reference's own test size:
        # 10^4 CSDA histories with their gradient, default precision
        {"name": "csda_samples_fp64_1e4", "kind": "samples", "n": 10000, "precision": "fp64",
         "thickness": 100.0, "elevation": 45.0, "emax": 100.0},
        # run_backward_mc as its defaults have it (straggling, scattering,
        # 10^4 samples, FP64), with the gradient
        {"name": "backward_mc_fp64_1e4", "kind": "mc", "n": 10000, "precision": "fp64",
         "thickness": 100.0, "elevation": 45.0, "emax": 100.0},
        # the largest stochastic batch: 10^6 straggled and scattered histories
        # through a runtime mixture, geometry drawn per history
        {"name": "los_mixed_1e6", "kind": "los", "lines": 1, "n_min": 1000000, "n_max": 1000000,
         "precision": "mixed", "mixture": True, "scattering": True, "gradient": False},
        # an ordinary survey: a few hundred lines of sight of 64 to 1024
        # histories, mixed transport, gradient per line
        {"name": "los_mixed_survey", "kind": "los", "lines": 400, "n_min": 64, "n_max": 1024,
         "precision": "mixed", "mixture": False, "scattering": False, "gradient": True},
        # one direction at the default precision of compute_directional_flux_mc
        {"name": "direction_mc_fp64", "kind": "dir", "dirs": 1, "n": 256, "precision": "fp64",
         "surface": 150.0, "emin": 1.0, "emax": 1e6},
        # a detector's sky: hundreds of directions over the reference's energy range
        {"name": "directions_mc_mixed", "kind": "dir", "dirs": 512, "n": 512, "precision": "mixed",
         "surface": 600.0, "emin": 1e-3, "emax": 1e9},
        # the water-fraction forward model and Jacobian at the default precision
        {"name": "wcsda_jacobian_fp64", "kind": "wcsda", "dirs": 192, "nodes": 32,
         "precision": "fp64", "jacobian": True, "surface": 600.0},
        # the same in the precision that calibrations and large skies use
        {"name": "wcsda_jacobian_mixed", "kind": "wcsda", "dirs": 1024, "nodes": 32,
         "precision": "mixed", "jacobian": True, "surface": 600.0},
        # tomography flux and J^T r from host arrays, default precision, rays
        # traced in the call
        {"name": "tomo_vjp_fp64", "kind": "tomo", "nx": 64, "ny": 64, "nz": 32, "rays": 1024,
         "nodes": 32, "precision": "fp64", "vjp": True},
        # the same on resident rays and densities in mixed precision: the inner
        # step of an iterative reconstruction
        {"name": "tomo_eval_mixed", "kind": "eval", "nx": 64, "ny": 64, "nz": 32, "detectors": 4,
         "rays": 1024, "nodes": 32, "precision": "mixed", "vjp": True},
        # a Gauss-Newton inversion of 10^6 cells from 65,536 rays
        {"name": "solve_gn_mixed", "kind": "solve", "nx": 128, "ny": 128, "nz": 64,
         "detectors": 8, "rays": 8192, "precision": "mixed", "method": "gn", "iters": 10},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """A case of the ranges above; FP64 stochastic ones stay thin, since their
    time grows with the rock and not with the number of histories."""
    kind = rng.choice(["point", "samples", "mc", "los", "los", "dir", "dir", "wcsda", "wcsda",
                       "tomo", "eval", "solve"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "point":
        return {"kind": kind, "thickness": round(_log(rng, 5.0, 500.0), 3),
                "elevation": round(rng.uniform(20.0, 90.0), 2)}
    if kind == "samples":
        return {"kind": kind, "n": int(_log(rng, 1, 60000)), "precision": prec,
                "thickness": round(_log(rng, 5.0, 500.0), 3),
                "elevation": round(rng.uniform(20.0, 90.0), 2),
                "emax": round(_log(rng, 20.0, 1e4), 1)}
    if kind == "mc":
        return {"kind": kind, "n": int(_log(rng, 100, 10000)), "precision": prec,
                "thickness": round(_log(rng, 4.0, 25.0 if prec == "fp64" else 300.0), 3),
                "elevation": round(rng.uniform(30.0, 90.0), 2),
                "emax": round(_log(rng, 20.0, 100.0 if prec == "fp64" else 1e4), 1)}
    if kind == "los":
        grad = rng.random() < 0.5
        lines = int(_log(rng, 1, 1500))
        n = int(_log(rng, 32, 2000))
        return {"kind": kind, "lines": lines, "n_min": max(1, n // 4), "n_max": n,
                "precision": "mixed", "mixture": not grad, "scattering": rng.random() < 0.5,
                "gradient": grad}
    if kind == "dir":
        if prec == "fp64":
            return {"kind": kind, "dirs": rng.randint(1, 5), "n": int(_log(rng, 8, 100)),
                    "precision": prec, "surface": round(rng.uniform(20.0, 60.0), 1),
                    "emin": 1.0, "emax": round(_log(rng, 100.0, 1e6), 1)}
        return {"kind": kind, "dirs": int(_log(rng, 1, 512)), "n": int(_log(rng, 16, 512)),
                "precision": prec, "surface": round(rng.uniform(100.0, 600.0), 1),
                "emin": round(_log(rng, 1e-3, 1.0), 6), "emax": round(_log(rng, 1e3, 1e9), 1)}
    if kind == "wcsda":
        return {"kind": kind, "dirs": int(_log(rng, 1, 192 if prec == "fp64" else 1024)),
                "nodes": rng.choice([8, 17, 32, 32, 48]), "precision": prec,
                "jacobian": rng.random() < 0.7, "surface": round(rng.uniform(100.0, 600.0), 1)}
    nx = int(_log(rng, 6, 64))
    # the detectors stand a quarter of the x extent off the centre, inside the grid
    grid = {"nx": nx, "ny": int(nx * rng.uniform(0.7, 1.5)), "nz": int(_log(rng, 3, 32))}
    if kind == "tomo":
        return {"kind": kind, **grid, "rays": int(_log(rng, 8, 1024)),
                "nodes": rng.choice([5, 16, 32, 40]), "precision": prec,
                "vjp": rng.random() < 0.7}
    if kind == "eval":
        return {"kind": kind, **grid, "detectors": rng.choice([4, 8]),
                "rays": int(_log(rng, 16, 4096 if prec == "mixed" else 512)),
                "nodes": rng.choice([5, 16, 32, 40]), "precision": prec,
                "vjp": rng.random() < 0.7}
    return {"kind": kind, **grid, "detectors": rng.choice([4, 8]),
            "rays": int(_log(rng, 32, 2048 if prec == "mixed" else 256)), "precision": prec,
            "method": rng.choice(["gn", "gn", "sart"]), "iters": rng.randint(1, 8)}


# ------------------------------------------------------------------ inputs
@lru_cache(maxsize=None)
def _physics():
    """The tables a program builds once: rock, air and water."""
    return dp.create_physics(materials=(dp.STANDARD_ROCK, dp.AIR, dp.WATER))


@lru_cache(maxsize=None)
def _media():
    ph = _physics()
    return (dp.MaterialMixture(ph, 1), dp.MaterialMixture(ph, 2),
            dp.MaterialMixture(ph, [1, 3, 2], [0.70, 0.25, 0.05]))


def _cuda(a):
    return torch.tensor(np.ascontiguousarray(a, np.float64).ravel(), device="cuda")


def _triples(rng, n, emax):
    """Log-uniform final energies above 1 GeV, charges and their weights."""
    energy = np.exp(rng.uniform(0.0, math.log(emax), n))
    return energy, np.where(rng.random(n) > 0.5, 1.0, -1.0), 2.0 * energy * math.log(emax)


def _density(rng):
    return float(rng.uniform(2400.0, 2800.0))


def _sky(case, seed=2026):
    """Directions through cells of rock and wet rock (0 or 30 % water, as the
    reference's runs have them) under a flat surface."""
    h = case["surface"]
    nz = max(2, min(16, int(h / 20.0)))
    raw, wf = directional_config(case["dirs"], nz=nz, surface=max(h, 20.0 * nz), seed=seed)
    paths = [dp.DirectionalPath(z, a, [dp.CellSegment(c, l) for c, l in segs], tin, slant, rem, sz,
                                True) for z, a, segs, tin, slant, rem, sz in raw]
    return (dp.MaterialConfig(1, 3, 2, -1, 2710.0, 1000.0, 0.0, 0.0),
            dp.SiteConfig(963.0, 30000.0), paths, wf)


def _voxels(case, seed):
    n_det = case.get("detectors", 4)
    return tomography_config(nx=case["nx"], ny=case["ny"], nz=case["nz"], n_detectors=n_det,
                             rays_per_detector=case["rays"], n_nodes=case.get("nodes", 32),
                             seed=seed)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    ph = _physics()
    kind = case["kind"]
    s = {"case": case, "seed": int(seed)}
    if kind == "point":
        s["energy"] = float(_log_np(rng, 1.0, 100.0))
        s["charge"] = 1.0 if rng.random() > 0.5 else -1.0
        s["density"] = _density(rng)
    elif kind == "samples":
        s["triples"] = _triples(rng, case["n"], case["emax"])
        s["density"] = _density(rng)
    elif kind == "mc":
        s["density"] = _density(rng)
    elif kind == "los":
        n = rng.integers(case["n_min"], case["n_max"] + 1, case["lines"])
        if case["mixture"]:
            # geometry drawn per history on the device
            s["los"] = dp.make_los(n, thickness=20.0, thickness_max=500.0,
                                   density=rng.uniform(1900.0, 2100.0, case["lines"]),
                                   density_max=2800.0, elevation=30.0, elevation_max=90.0,
                                   air_height=1000.0, energy_min=1.0, energy_max=1e4)
        else:
            s["los"] = dp.make_los(n, thickness=np.exp(rng.uniform(math.log(50.0),
                                                                   math.log(2000.0),
                                                                   case["lines"])),
                                   density=rng.uniform(2400.0, 2800.0, case["lines"]),
                                   elevation=90.0, energy_min=1.0, energy_max=1e4)
    elif kind == "dir":
        cfg, site, paths, wf = _sky(case, seed)
        mats, dens = dp.build_cell_properties_for_mc(ph, np.zeros(len(wf), bool), wf, cfg)
        s["batch"] = dp.DirBatch(ph, cfg, site, paths, mats, dens, None, n_samples=case["n"],
                                 energy_min=case["emin"], energy_max=case["emax"])
    elif kind == "wcsda":
        # one detector's directions, another water field for every seed
        cfg, site, paths, wf = _sky(case)
        nodes = [dp.EnergySample(*x)
                 for x in zip(*dp.csda_energy_quadrature(case["nodes"], 1.0, 1e6))]
        s["wf"] = np.clip(wf + rng.uniform(0.0, 0.2, len(wf)), 0.0, 1.0)
        s["batch"] = dp.CsdaBatch(ph, np.zeros(len(wf), bool), cfg, site, paths,
                                  nodes).to_device()
    elif kind == "tomo":
        grid, rho, rays, nodes = _voxels(case, seed)
        s["model"] = dp.TomoModel(ph, grid, nodes, side_density=2500.0,
                                  precision=case["precision"])
        s["rho"], s["rays"] = rho, rays
        s["cot"] = rng.uniform(0.5, 1.5, len(rays))
    elif kind in ("eval", "solve"):
        grid, rho, rays, nodes = _voxels(case, seed)
        s["paths"] = dp.TomoPaths(ph, grid, rays, nodes, side_density=2500.0)
        s["rho"] = _cuda(rho)
        s["cot"] = _cuda(rng.uniform(0.5, 1.5, len(rays)))
        if kind == "solve":
            # Poisson counts of ~10^3 per ray, inverse-variance weights, a flat start
            flux = s["paths"].eval(s["rho"], precision="fp64")[0].cpu().numpy()
            tau = 1e3 / np.median(flux)
            counts = rng.poisson(tau * flux)
            s["obs"], s["weight"] = _cuda(counts / tau), _cuda(tau * tau / np.maximum(counts, 1))
            s["rho0"] = torch.full_like(s["rho"], 2650.0)
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return s


def _log_np(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


# ------------------------------------------------------------------ one pass
def run(s):
    case, ph = s["case"], _physics()
    kind = case["kind"]
    if kind == "point":
        return dp.compute_flux_gradient(ph, s["density"], case["thickness"], case["elevation"],
                                        s["energy"], s["charge"])
    if kind == "samples":
        return dp.csda_flux_samples(ph, *s["triples"], rock_thickness=case["thickness"],
                                    rock_density=s["density"], elevation=case["elevation"],
                                    precision=case["precision"])
    if kind == "mc":
        r = dp.run_backward_mc(ph, rock_thickness=case["thickness"], rock_density=s["density"],
                               elevation=case["elevation"], energy_min=1.0,
                               energy_max=case["emax"], n_samples=case["n"],
                               compute_gradient=True, seed=s["seed"],
                               precision=case["precision"])
        return {"flux": r.flux, "sigma": r.sigma, "gradient": r.gradient,
                "gradient_flux": r.gradient_flux}
    if kind == "los":
        rock, air, mix = _media()
        return dp.backward_mc_batch(ph, s["los"], rock=mix if case["mixture"] else rock, air=air,
                                    seed=s["seed"], scattering=case["scattering"],
                                    energy_threshold_low=100.0 if case["mixture"] else 1.0,
                                    precision=case["precision"],
                                    compute_gradient=case["gradient"])
    if kind == "dir":
        return s["batch"].run(s["seed"], precision=case["precision"], return_histories=True)
    if kind == "wcsda":
        return s["batch"].run(s["wf"], jacobian=case["jacobian"], precision=case["precision"])
    if kind == "tomo":
        if case["vjp"]:
            return s["model"].vjp(s["rho"], s["rays"], s["cot"])
        return s["model"].forward(s["rho"], s["rays"])
    if kind == "eval":
        return s["paths"].eval(s["rho"], s["cot"] if case["vjp"] else None,
                               precision=case["precision"])
    return s["paths"].solve(s["obs"], s["rho0"], method=case["method"], n_iter=case["iters"],
                            weight=s["weight"], precision=case["precision"],
                            prior_weight=1e-5 if case["method"] == "gn" else 1.0)


# ------------------------------------------------------------------ work
def _csda_steps(thickness, elevation):
    """Steps of a CSDA history: the range grows by 1 % per step in the rock
    (from about 10 m of rock at these energies), then the air's step limit."""
    slant = thickness / max(math.sin(math.radians(elevation)), 0.05)
    return 100.0 * math.log1p(slant / 3.0) + 100.0


def work(case):
    """Inputs and outputs once; the arithmetic of the physics steps the path
    cannot skip (a table step with its tangent about 60 operations, a
    straggled and scattered step about 300, a differential cross-section sum
    of 52 quadrature points about 5000)."""
    kind = case["kind"]
    if kind == "point":
        return {"bytes": 8 * 2 + 6 * 200 * 8,
                "flops": 60.0 * _csda_steps(case["thickness"], case["elevation"])}
    if kind == "samples":
        return {"bytes": 40.0 * case["n"],
                "flops": 60.0 * case["n"] * _csda_steps(case["thickness"], case["elevation"])}
    if kind == "mc":
        steps = _csda_steps(case["thickness"], case["elevation"])
        return {"bytes": 24.0 * case["n"], "flops": case["n"] * (360.0 * steps + 5e3 * 5)}
    if kind == "los":
        n = case["lines"] * 0.5 * (case["n_min"] + case["n_max"])
        step = 300.0 if case["scattering"] else 150.0
        return {"bytes": 24.0 * n + 150.0 * case["lines"],
                "flops": n * (step * 300.0 + 5e3 * 20 + (60.0 * 300.0 if case["gradient"] else 0))}
    if kind == "dir":
        n = case["dirs"] * float(case["n"])
        return {"bytes": 28.0 * n + 60 * 16.0 * case["dirs"], "flops": n * (150.0 * 300 + 5e3 * 20)}
    if kind == "wcsda":
        lanes = case["dirs"] * float(case["nodes"])
        per = 300.0 if case["jacobian"] else 120.0
        return {"bytes": case["dirs"] * (40.0 + 45 * 28.0),
                "flops": lanes * 800.0 * per}
    rays = case["rays"] * case.get("detectors", 4)
    segs = rays * 0.75 * (case["nx"] + case["ny"] + case["nz"]) * 0.6
    cells = case["nx"] * case["ny"] * case["nz"]
    nodes = case.get("nodes", 32)
    if kind in ("tomo", "eval"):
        vjp = case["vjp"]
        return {"bytes": segs * 24.0 + rays * 72.0 + cells * (16.0 if vjp else 8.0),
                "flops": segs * nodes * (70.0 if vjp else 30.0)}
    it = case["iters"]
    products = 20 if case["method"] == "gn" else 4
    return {"bytes": it * (segs * (24.0 + 12.0 * products) + cells * 8.0 * 5 * products),
            "flops": it * segs * (nodes * 70.0 + 2.0 * products)}


# ------------------------------------------------------------------ 64-bit values
# The same quantities written out in torch on 64-bit tensors.  The tables are
# the caller's inputs (log-linear in energy, ranges inverted log-linearly).
class _Table:
    def __init__(self, name, device):
        ph = _physics()
        m = ph.materials[name]
        T = lambda c: torch.tensor(ph.column(m, c), device=device)
        self.E, self.lE, self.R, self.S = T("E"), T("logE"), T("csda_R"), T("csda_S")

    def at(self, col, E):
        lE = torch.log(E)
        i = (torch.searchsorted(self.lE, lE.detach(), right=True) - 1).clamp(0, len(self.E) - 2)
        y = col[i] + (lE - self.lE[i]) / (self.lE[i + 1] - self.lE[i]) * (col[i + 1] - col[i])
        y = torch.where(E <= self.E[0], col[0], y)
        return torch.where(E >= self.E[-1], col[-1], y)

    def energy(self, X):
        R, lE = self.R, self.lE
        i = (torch.searchsorted(R, X.detach(), right=True) - 1).clamp(0, len(R) - 2)
        e = torch.exp(lE[i] + (X - R[i]) / (R[i + 1] - R[i]) * (lE[i + 1] - lE[i]))
        e = torch.where(X <= R[0], self.E[0], e)
        return torch.where(X >= R[-1], self.E[-1], e)


def _star(c):
    p0, p1, p2, p3, p4 = 0.102573, -0.068287, 0.958633, 0.0407253, 0.817285
    v = (c * c + p0 * p0 + p1 * c ** p2 + p3 * c ** p4) / (1.0 + p0 * p0 + p1 + p3)
    return torch.sqrt(v.clamp(min=0.0))


def _surface_flux(cs, E, q):
    """The GCCLY sea-level spectrum with the charge ratio 1.2766."""
    Emu = E + MASS
    ec = 1.1 * Emu * cs
    h = 1.0 / (1.0 + ec / 115.0) + 0.054 / (1.0 + ec / 850.0)
    r = 1.2766
    frac = torch.where(q < 0, 1.0 / (1.0 + r), torch.where(q > 0, r / (1.0 + r), 1.0 + 0.0 * q))
    return (1.0 + 3.64 / (Emu * cs ** 1.29)) ** -2.7 * 1.4e3 * Emu ** -2.7 * h * frac


def _time_of_flight(L, E):
    """Proper length of a path at the mean kinetic energy E."""
    g = 1.0 + E / MASS
    return L / (torch.sqrt((1.0 - 1.0 / (g * g)).clamp(min=1e-12)) * g)


def _exact_samples(energy, charge, weight, thickness, density, elevation, device):
    """CSDA histories with d/d density carried forward."""
    import torch.autograd.forward_ad as fw
    rock, air = _Table("StandardRock", device), _Table("Air", device)
    T = lambda a: torch.as_tensor(np.atleast_1d(a), dtype=torch.float64, device=device)
    E, q, w = T(energy), T(charge), T(weight)
    c = math.cos((90.0 - elevation) * math.pi / 180.0)
    H, eps, one = 3e4, 2.220446049250313e-16, torch.ones_like(E)
    with fw.dual_level():
        rho = fw.make_dual(density * one, one.clone())
        zero = 0.0 * rho
        E, z, tau, ws = E + zero, zero, zero, 1.0 + zero
        while True:
            on = (E < 1e9 - eps) & (z >= 0.0) & (z < H - eps)
            if not bool(on.any()):
                break
            top = z >= thickness
            X = torch.where(top, air.at(air.R, E), rock.at(rock.R, E))
            dens = torch.where(top, AIR0 * torch.exp(z / -SCALE_H), rho)
            ahead = (torch.where(top, H + zero, thickness + zero) - z) / c
            lim = 0.01 * X / dens
            cap = 0.05 * SCALE_H / max(abs(c), 0.05)
            lim = torch.where(top & (lim > cap), cap + zero, lim)
            step = torch.where(lim < ahead + 1e-7, lim, ahead + 1e-7)
            step = torch.where(step < 1e-7, 1e-7 + zero, torch.where(step > 1e3, 1e3 + zero, step))
            Y = X + step * dens
            En = torch.where(top, air.energy(Y), rock.energy(Y))
            S0 = torch.where(top, air.at(air.S, E), rock.at(rock.S, E))
            S1 = torch.where(top, air.at(air.S, En), rock.at(rock.S, En))
            tau = torch.where(on, tau + _time_of_flight(step, 0.5 * (E + En)), tau)
            ws = torch.where(on, ws * S1 / S0, ws)
            z = torch.where(on, z + step * c, z)
            E = torch.where(on, En, E)
        cs = _star(torch.tensor(c, dtype=torch.float64, device=device))
        f = w * ws * torch.exp(-tau / CTAU) * _surface_flux(cs, E, q)
        f = torch.where((z >= H - 1.0) & (E < 1e9), f, 0.0 * f)
        v, d = fw.unpack_dual(f)
    return v, d


def _trace(rays, grid, device):
    """Cells and lengths of every ray by the march that defines the model
    (position-based steps to the nearest face more than 1e-10 m ahead, a
    nudge of 1 cm where there is none), and the way left to the top plane."""
    n, o, d = np.array([grid.nx, grid.ny, grid.nz]), np.array(grid.origin), np.array(grid.pitch)
    hi = o + n * d
    p, u, rows = rays[:, :3].copy(), rays[:, 3:6], np.arange(len(rays))
    on, z_exit = np.ones(len(rays), bool), rays[:, 2].copy()
    cells, lens = [], []
    for _ in range(1000):
        on &= ((p >= o) & (p <= hi)).all(1)
        if not on.any():
            break
        c = np.clip(np.floor((p - o) / d).astype(int) + 1, 1, n)
        with np.errstate(divide="ignore", invalid="ignore"):
            t = (o + np.where(u > 0, c, c - 1) * d - p) / u
        t = np.where((np.abs(u) > 1e-10) & (t > 1e-10), t, np.inf)
        a = np.argmin(t, axis=1)
        dist = t[rows, a]
        go = on & (dist > 1e-10) & np.isfinite(dist)
        dist = np.where(go, dist, 0.0)
        cells.append(np.where(go, c[:, 0] - 1 + grid.nx * (c[:, 1] - 1 + grid.ny * (c[:, 2] - 1)), 0))
        lens.append(dist)
        move = np.where(go, dist, np.where(on, 0.01, 0.0))
        p = p + u * move[:, None]
        z_exit = np.where(go, p[:, 2], z_exit)
        on &= ~(go & np.where(u[rows, a] > 0, c[rows, a] + 1 > n[a], c[rows, a] - 1 < 1))
    top = grid.origin[2] + grid.nz * grid.pitch[2]
    side = np.where(z_exit < top, (top - z_exit) / np.maximum(np.abs(rays[:, 6]), 0.01), 0.0)
    T = lambda x: torch.tensor(np.array(x), device=device)
    return T(cells), T(lens), T(side), top


def _exact_tomo(case, seed, device):
    s = np.random.default_rng(seed)
    grid, rho, rays, nodes = _voxels(case, seed)
    cot = s.uniform(0.5, 1.5, len(rays))
    rock, air = _Table("StandardRock", device), _Table("Air", device)
    cells, lens, side, top = _trace(rays, grid, device)
    rho = torch.tensor(np.ascontiguousarray(rho, np.float64).ravel(), device=device,
                       requires_grad=True)
    E0, q, w = (torch.tensor(x, device=device)[None, :] for x in nodes)
    E = E0.expand(len(rays), -1)
    logw = torch.zeros_like(E)
    for k in range(len(cells) + 1):
        if k < len(cells):
            L, X = lens[k][:, None], (lens[k] * rho[cells[k]])[:, None]
        else:
            L, X = side[:, None], 2500.0 * side[:, None]
        En = rock.energy(rock.at(rock.R, E) + X)
        En = torch.where(L > 0, En, E)
        logw = logw + torch.log(rock.at(rock.S, En) / rock.at(rock.S, E)) - \
            _time_of_flight(L, 0.5 * (E + En)) / CTAU
        E = En
    c = torch.tensor(rays[:, 6], device=device)[:, None]
    safe = c.abs().clamp(min=0.01)
    gram = (AIR0 * SCALE_H / safe) * (math.exp(-top / SCALE_H) - math.exp(-3e4 / SCALE_H))
    En = air.energy(air.at(air.R, E) + gram)
    logw = logw + torch.log(air.at(air.S, En) / air.at(air.S, E)) - \
        _time_of_flight((3e4 - top) / safe, 0.5 * (E + En)) / CTAU
    f = torch.exp(logw) * _surface_flux(_star(c), En, q.expand_as(En))
    flux = (2.0 * w * f).sum(1) / E0.shape[1]
    if not case["vjp"]:
        return flux.detach(), None
    return flux.detach(), torch.autograd.grad((flux * torch.tensor(cot, device=device)).sum(),
                                              rho)[0]


def _exact_wcsda(case, seed, device):
    """Heun walks of the water-fraction model: reverse mode through the cells,
    forward mode through the rock and the air above them."""
    import torch.autograd.forward_ad as fw
    rng = np.random.default_rng(seed)
    _, site, paths, wf = _sky(case)
    wf = np.clip(wf + rng.uniform(0.0, 0.2, len(wf)), 0.0, 1.0)
    rock, air, water = (_Table(n, device) for n in ("StandardRock", "Air", "Water"))
    nseg = max(len(p.segments) for p in paths)
    cell = np.zeros((len(paths), nseg), int)
    leng = np.zeros((len(paths), nseg))
    for b, p in enumerate(paths):
        for j, (i, l) in enumerate(p.segments):
            cell[b, j], leng[b, j] = i - 1, l
    T = lambda x: torch.tensor(np.asarray(x, np.float64), device=device)[:, None]
    W = torch.tensor(wf[cell], device=device, requires_grad=case["jacobian"])
    E0, q, ew = (torch.tensor(x, device=device)[None, :]
                 for x in dp.csda_energy_quadrature(case["nodes"], 1.0, 1e6))
    ct = T([math.cos(math.radians(p.zenith)) for p in paths])

    def heun(S, s0, ds, dens, E, lw, on):
        gx = ds * dens
        s1 = S(E + s0 * gx)
        En = E + 0.5 * (s0 + s1) * gx
        lw2 = lw + torch.log(S(En) / s0) - _time_of_flight(ds, 0.5 * (E + En)) / CTAU
        return torch.where(on, En, E), torch.where(on, lw2, lw)

    def solid(S, dens, length, E, lw):
        left = length + 0.0 * E
        while bool((left > 1e-8).any()):
            on = left > 1e-8
            s0 = S(E)
            gain = 0.02 * E / s0
            cap = torch.minimum(left * dens, 60.0 * dens)
            ds = torch.where(cap <= gain, cap, gain) / dens
            ds = torch.where(ds < left, ds, left)
            E, lw = heun(S, s0, ds, dens, E, lw, on)
            left = torch.where(on, left - ds, left)
        return E, lw

    E, lw = E0.expand(len(paths), -1), torch.zeros(len(paths), E0.shape[1], dtype=torch.float64,
                                                   device=device)
    for j in range(nseg):
        w = W[:, j:j + 1]
        dens = 1.0 / ((1.0 - w) / 2710.0 + w / 1000.0)
        E, lw = solid(lambda e, w=w: (1.0 - w) * rock.at(rock.S, e) + w * water.at(water.S, e),
                      dens, torch.tensor(leng[:, j:j + 1], device=device), E, lw)
    with torch.no_grad(), fw.dual_level():
        Ed = fw.make_dual(E.detach(), torch.ones_like(E))
        zero = 0.0 * Ed
        Ea, la = solid(lambda e: rock.at(rock.S, e), 2710.0 + zero,
                       T([p.remaining_rock_distance for p in paths]), Ed, zero)
        z0 = T([p.surface_exit_z for p in paths])
        left = (3e4 - z0).clamp(min=0.0) / ct.clamp(min=1e-3) + zero
        done, base = zero, site.detector_elevation + z0
        while bool((left > 1e-8).any()):
            on = left > 1e-8
            s0 = air.at(air.S, Ea)
            half = torch.where(left < 60.0, left, 60.0 + zero)
            rho = AIR0 * torch.exp(-(base + ct * (done + 0.5 * half)) / SCALE_H)
            ds = 0.02 * Ea / s0 / rho
            ds = torch.where(ds < half, ds, half)
            ds = torch.where(ds < 1e-3, 1e-3 + zero, ds)
            rho = AIR0 * torch.exp(-(base + ct * (done + 0.5 * ds)) / SCALE_H)
            Ea, la = heun(lambda e: air.at(air.S, e), s0, ds, rho, Ea, la, on)
            done = torch.where(on, done + ds, done)
            left = torch.where(on, left - ds, left)
        lf = la + torch.log(_surface_flux(_star(ct), Ea, q.expand_as(E)))
        above, slope = fw.unpack_dual(lf)
    f = 2.0 * ew * torch.exp(lw.detach() + above) / E0.shape[1]
    flux = f.sum(1)
    if not case["jacobian"]:
        return flux, None
    jac, = torch.autograd.grad((f * (lw + slope * E)).sum(), W)
    keep = torch.tensor(np.arange(nseg)[None, :] < np.array([[len(p.segments)] for p in paths]),
                        device=device)
    return flux, jac[keep]


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "point":
        e, q = _log_np(rng, 1.0, 100.0), 1.0 if rng.random() > 0.5 else -1.0
        v, d = _exact_samples(e, q, 1.0, case["thickness"], _density(rng), case["elevation"],
                              device)
        return float(v[0]), float(d[0])
    if kind == "samples":
        tri = _triples(rng, case["n"], case["emax"])
        return _exact_samples(*tri, case["thickness"], _density(rng), case["elevation"], device)
    if kind == "tomo" or kind == "eval":
        flux, grad = _exact_tomo(case, seed, device)
        if kind == "eval":
            return flux, grad, None
        return (flux, grad) if case["vjp"] else flux
    if kind == "wcsda":
        return _exact_wcsda(case, seed, device)
    # a stochastic estimate has no value but its own, and an inversion loop
    # takes longer than a comparison should
    return None
