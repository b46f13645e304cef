"""Performance cases of the stepping engine: what a user's program has it do.

Every case is one run of a chain over a batch of candidates (or one value and
gradient of the adjoint loss) through the package's Python entry points.  The
kinds and the ranges of their sizes:

  boris      PropagationBP, fixed step, over a periodic Kolmogorov Grid3f
             (workloads.grid_bp_256 and its smaller relatives);
  cash_karp  PropagationCK with tolerance 1e-4 over the 64^3 grid
             (workloads.grid_ck_64);
  nuclei     PropagationCK of a mixed composition with a maximum length per
             candidate over the 256^3 grid (workloads.grid_ck_nuclei);
  region     adaptive PropagationBP over a grid whose size is not a power of
             two (periodic or reflective), with a maximum length, an observer
             sphere and a spherical boundary: the chain most scripts build;
  waves      PropagationBP in PlaneWaveTurbulence;
  galaxy     backtracking through a galactic field to the 20 kpc sphere
             (workloads.jf12_backtrack and its relatives);
  diffusion  DiffusionSDE in a toroidal field plus PlaneWaveTurbulence
             (workloads.sde_galactic), a bounded number of steps per call;
  adjoint    arrival loss and its gradients (workloads.grid_bp_backtrack_128).
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

from crpropa3_b200 import _abi, plan as P, units as U, workloads as W
from crpropa3_b200.adjoint import arrival_loss
from crpropa3_b200.engine import Plan
from crpropa3_b200.turbulence import grid_turbulence_device

PRECISION = {"fp64": _abi.PRECISION_FP64, "mixed": _abi.PRECISION_MIXED}
GALAXY = {"jf12": lambda: P.JF12Field(), "uf23": lambda: P.UF23Field(_abi.UF23_BASE),
          "pt11": lambda: P.PT11Field(), "tf17": lambda: P.TF17Field()}
TENSORS = ("x", "y", "z", "dx", "dy", "dz", "px", "py", "pz", "trajectory_length", "time",
           "current_step", "next_step", "active", "flags", "step_count")


def listed():
    return [
        # a script's first try: a few hundred protons in host arrays, a short chain
        {"name": "boris_host_257", "kind": "boris", "n": 257, "grid": 64, "steps": 64,
         "precision": "fp64", "host": True},
        # an ordinary run: some 10^4 protons over a 128^3 grid
        {"name": "boris_mixed_20011", "kind": "boris", "n": 20011, "grid": 128, "steps": 1000,
         "precision": "mixed", "host": False},
        # the headline workload: 10^6 protons, 5000 steps, 256^3 grid
        {"name": "boris_mixed_1e6", "kind": "boris", "n": 1000000, "grid": 256, "steps": 5000,
         "precision": "mixed", "host": False},
        # the same field in the reference's own arithmetic, a shorter run
        {"name": "boris_fp64_200001", "kind": "boris", "n": 200001, "grid": 256, "steps": 1000,
         "precision": "fp64", "host": False},
        # 10^4 protons to 10 Mpc with the adaptive Cash-Karp integrator
        {"name": "cash_karp_fp64_1e4", "kind": "cash_karp", "n": 10000, "mpc": 10.0, "precision": "fp64"},
        # a composition with rigidities over 4.5 decades: very uneven step counts
        {"name": "nuclei_mixed_1e5", "kind": "nuclei", "n": 100000, "mpc": 5.0, "precision": "mixed"},
        # adaptive Boris push in a bounded region, a grid of 100^3 cells
        {"name": "region_mixed_50000", "kind": "region", "n": 50000, "grid": 100, "reflective": False,
         "precision": "mixed"},
        # protons in a turbulent field given by its wave modes
        {"name": "waves_mixed_20000", "kind": "waves", "n": 20000, "modes": 200, "steps": 200,
         "precision": "mixed"},
        # a sky map's worth of antiprotons backtracked through the JF12 field
        {"name": "jf12_mixed_200000", "kind": "galaxy", "field": "jf12", "n": 200000, "precision": "mixed"},
        # the events of one data set backtracked through UF23 in the reference's arithmetic
        {"name": "uf23_fp64_5000", "kind": "galaxy", "field": "uf23", "n": 5000, "precision": "fp64"},
        # pseudo-particles of galactic diffusion, 1024 modes, 16 steps per call
        {"name": "diffusion_mixed_32768", "kind": "diffusion", "n": 32768, "modes": 1024, "steps": 16,
         "precision": "mixed"},
        # loss and gradients of 10^5 backtracked antiprotons over a 128^3 grid
        {"name": "adjoint_1e5", "kind": "adjoint", "n": 100000, "grid": 128, "steps": 2000, "every": 100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["boris", "boris", "cash_karp", "nuclei", "region", "waves", "galaxy", "diffusion",
                       "adjoint"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "boris":
        host = rng.random() < 0.35
        return {"kind": kind, "n": _log(rng, 200, 20000 if host else 500000), "grid": rng.choice([64, 128, 256]),
                "steps": _log(rng, 50, 1500), "precision": precision, "host": host}
    if kind == "cash_karp":
        return {"kind": kind, "n": _log(rng, 2000, 20000), "mpc": rng.uniform(2.0, 10.0), "precision": precision}
    if kind == "nuclei":
        return {"kind": kind, "n": _log(rng, 10000, 100000), "mpc": rng.uniform(1.0, 4.0), "precision": "mixed"}
    if kind == "region":
        return {"kind": kind, "n": _log(rng, 2000, 50000), "grid": rng.choice([60, 80, 100, 120]),
                "reflective": rng.random() < 0.5, "precision": precision}
    if kind == "waves":
        return {"kind": kind, "n": _log(rng, 2000, 20000), "modes": rng.randint(50, 300),
                "steps": _log(rng, 50, 200), "precision": "mixed" if rng.random() < 0.7 else "fp64"}
    if kind == "galaxy":
        return {"kind": kind, "field": rng.choice(sorted(GALAXY)), "n": _log(rng, 2000, 100000),
                "precision": precision}
    if kind == "diffusion":
        return {"kind": kind, "n": _log(rng, 4000, 32768), "modes": rng.choice([256, 500, 1024]),
                "steps": rng.randint(6, 16), "precision": "mixed"}
    return {"kind": kind, "n": _log(rng, 5000, 100000), "grid": rng.choice([64, 128]),
            "steps": _log(rng, 300, 2000), "every": rng.choice([20, 50, 100])}


# ------------------------------------------------------------------ inputs
def _grid(n, spacing, brms, lmin, lmax, seed):
    return grid_turbulence_device(_abi.TURBULENCE_GRID, n, spacing, brms, lmin, lmax, seed=seed)


def _field(case, seed):
    """(Grid3f values on the device or None, spacing) of a case."""
    kind = case["kind"]
    if kind == "boris":
        n = case["grid"]
        return _grid(n, 5 * U.kpc, 10 * U.nG, 10 * U.kpc, min(500, 2.5 * n) * U.kpc, 42 + seed), 5 * U.kpc
    if kind == "cash_karp":
        return _grid(64, 10 * U.kpc, 1 * U.nG, 20 * U.kpc, 200 * U.kpc, 42 + seed), 10 * U.kpc
    if kind == "nuclei":
        return _grid(256, 5 * U.kpc, 10 * U.nG, 10 * U.kpc, 500 * U.kpc, 42 + seed), 5 * U.kpc
    if kind == "region":
        n = case["grid"]
        return _grid(n, 10 * U.kpc, 1 * U.nG, 20 * U.kpc, 4 * n * U.kpc, 42 + seed), 10 * U.kpc
    if kind == "adjoint":
        n = case["grid"]
        return _grid(n, 10 * U.kpc, 3 * U.nG, 20 * U.kpc, 10 * n * U.kpc, 42 + seed), 10 * U.kpc
    return None, None


def _candidates(case, seed):
    """Candidates on the device, drawn from the workload's source."""
    kind, n = case["kind"], case["n"]
    H = W.IDS["H"]
    if kind == "nuclei":
        c = W.source_candidates_device(n, [W.IDS[k] for k in ("H", "He", "N", "Fe")], 0.1 * U.EeV, 100 * U.EeV,
                                       -2.0, seed)
        r = np.random.default_rng(seed)
        c.max_length = torch.from_numpy(r.uniform(0.02, 1.0, n) * case["mpc"] * U.Mpc).cuda()
        return c
    if kind == "galaxy":
        return W.source_candidates_device(n, [-H], 5 * U.EeV, 100 * U.EeV, -1.0, seed,
                                          position=(-8.5 * U.kpc, 0.0, 0.0))
    if kind == "diffusion":
        return W.source_candidates_device(n, [H], 1 * U.TeV, 1000 * U.TeV, -1.0, seed,
                                          position=(8.5 * U.kpc, 0.0, 0.0))
    if kind == "adjoint":
        return W.source_candidates_device(n, [-H], 5 * U.EeV, 50 * U.EeV, -1.0, seed)
    return W.source_candidates_device(n, [H], 1 * U.EeV, 100 * U.EeV, -1.0, seed)


def _modes(case, seed):
    if case["kind"] == "waves":
        return (1 * U.nG, 20 * U.kpc, 200 * U.kpc, 200 * U.kpc, 5.0 / 3.0, 4.0), case["modes"], 11 + seed
    return (0.5 * U.muG, 1 * U.pc, 100 * U.pc, 1 * U.pc, 5.0 / 3.0, 4.0), case["modes"], 11 + seed


def _chain(case, seed, grid, spacing):
    kind = case["kind"]
    precision = PRECISION[case["precision"]]
    if kind in ("waves", "diffusion"):
        spectrum, n_modes, mode_seed = _modes(case, seed)
        waves = P.PlaneWaveField(*W.plane_wave_modes(*spectrum, n_modes, mode_seed), spectrum=spectrum,
                                 seed=mode_seed)
    if kind == "boris":
        return P.ChainSpec([P.GridField(grid, (0, 0, 0), (spacing,) * 3)],
                           [P.Propagation(_abi.PROP_BP, 0.42, 1 * U.kpc, 1 * U.kpc),
                            P.MaxTrajectoryLength(case["steps"] * U.kpc)], precision=precision)
    if kind == "cash_karp":
        return P.ChainSpec([P.GridField(grid, (0, 0, 0), (spacing,) * 3)],
                           [P.Propagation(_abi.PROP_CK, 1e-4, 0.1 * U.kpc, 10 * U.kpc),
                            P.MaxTrajectoryLength(case["mpc"] * U.Mpc)], precision=precision)
    if kind == "nuclei":
        return P.ChainSpec([P.GridField(grid, (0, 0, 0), (spacing,) * 3)],
                           [P.Propagation(_abi.PROP_CK, 1e-4, 0.1 * U.kpc, 100 * U.kpc),
                            P.MaxTrajectoryLength(per_candidate=True)], precision=precision)
    if kind == "region":
        size = case["grid"] * spacing
        return P.ChainSpec([P.GridField(grid, (-size / 2,) * 3, (spacing,) * 3, reflective=case["reflective"])],
                           [P.Propagation(_abi.PROP_BP, 1e-4, 0.5 * U.kpc, 5 * U.kpc),
                            P.MaxTrajectoryLength(4 * size),
                            P.ObserverSpec(_abi.OBSERVER_SURFACE_SPHERE, (0.0, 0.0, 0.0), 0.4 * size, True, False),
                            P.BoundarySpec(_abi.BOUNDARY_SPHERICAL, (0.0, 0.0, 0.0), size=0.5 * size)],
                           precision=precision)
    if kind == "waves":
        return P.ChainSpec([waves], [P.Propagation(_abi.PROP_BP, 0.42, 1 * U.kpc, 1 * U.kpc),
                                     P.MaxTrajectoryLength(case["steps"] * U.kpc)], precision=precision)
    if kind == "galaxy":
        return P.ChainSpec([GALAXY[case["field"]]()],
                           [P.Propagation(_abi.PROP_CK, 1e-4, 0.1 * U.pc, 100 * U.pc),
                            P.MaxTrajectoryLength(100 * U.kpc),
                            P.ObserverSpec(_abi.OBSERVER_SURFACE_SPHERE, (0.0, 0.0, 0.0), 20 * U.kpc, True, False)],
                           precision=precision)
    return P.ChainSpec([P.ToroidalField(1 * U.muG), waves],
                       [P.Propagation(_abi.PROP_SDE, 1e-4, 0.1 * U.pc, 100 * U.pc, epsilon=0.1, alpha=1.0 / 3.0,
                                      scale=1.0),
                        P.ObserverSpec(_abi.OBSERVER_SURFACE_SPHERE, (0.0, 0.0, 0.0), 20 * U.kpc, True, False)],
                       precision=precision, seed=seed)


def _adjoint_inputs(case, seed):
    grid, spacing = _field(case, seed)
    c = _candidates(case, seed)
    u = torch.stack([c.dx, c.dy, c.dz], 1)
    gen = torch.Generator("cuda").manual_seed(seed)
    target = torch.randn(case["n"], 3, generator=gen, device="cuda", dtype=torch.float64)
    target /= target.norm(dim=1, keepdim=True)
    return {"grid": grid, "spacing": spacing, "pos": torch.zeros_like(u), "charge": c.charge, "target": target,
            "p0": u * (c.energy / U.c_light)[:, None]}


def prepare(case, seed):
    if case["kind"] == "adjoint":
        s = _adjoint_inputs(case, seed)
        s["p0"].requires_grad_(True)
        s["grid"].requires_grad_(True)
        return {"case": case, **s}
    grid, spacing = _field(case, seed)
    spec = _chain(case, seed, None if grid is None else grid.cpu().numpy(), spacing)
    c = _candidates(case, seed)
    return {"case": case, "plan": Plan(spec), "candidates": c.to_host() if case.get("host") else c,
            "options": {"max_steps": case["steps"]} if case["kind"] == "diffusion" else {}}


def run(s):
    case = s["case"]
    if case["kind"] == "adjoint":
        loss = arrival_loss(s["p0"], s["grid"], s["pos"], s["charge"], s["target"], (0.0, 0.0, 0.0), s["spacing"],
                            1 * U.kpc, case["steps"], case["every"])
        g_p0, g_grid = torch.autograd.grad(loss, (s["p0"], s["grid"]))
        return {"loss": loss.detach(), "grad_p0": g_p0, "grad_grid": g_grid}
    c = s["candidates"].copy()  # a run advances its candidates in place
    s["plan"].run(c, **s["options"])
    return {name: getattr(c, name) for name in TENSORS}


# -------------------------------------------------------------------- work
def work(case):
    """Candidate state in and out and the field once; operations of the steps
    the chain cannot do without (adaptive chains: their mean step count)."""
    kind, n = case["kind"], case["n"]
    state = n * (145 + 121)
    grid = 12 * case["grid"] ** 3 if "grid" in case else 0
    push = 130  # Boris push without its field; an interpolation takes about 90 operations
    if kind == "boris":
        return {"bytes": state + grid, "flops": n * case["steps"] * (push + 90)}
    if kind == "cash_karp":
        return {"bytes": state + 12 * 64 ** 3, "flops": n * case["mpc"] * 110 * (6 * 170 + 60)}
    if kind == "nuclei":
        return {"bytes": state + 12 * 256 ** 3, "flops": n * case["mpc"] * 280 * (6 * 170 + 60)}
    if kind == "region":
        return {"bytes": state + grid, "flops": n * case["grid"] * 2 * 3 * (push + 90)}
    if kind == "waves":
        return {"bytes": state + 72 * case["modes"], "flops": n * case["steps"] * (push + 14 * case["modes"])}
    if kind == "galaxy":
        return {"bytes": state, "flops": n * 250 * (6 * 250 + 60)}
    if kind == "diffusion":
        return {"bytes": state + 72 * case["modes"], "flops": n * case["steps"] * 24 * (60 + 14 * case["modes"])}
    return {"bytes": n * 200 + 24 * case["grid"] ** 3, "flops": n * case["steps"] * 3 * (push + 90)}


# ------------------------------------------- the same in 64 bits, by torch
CORNERS = ((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (0, 1, 1), (1, 1, 0), (1, 1, 1))


def _trilinear(values, origin, spacing, reflective, dtype):
    """B(x) of a Grid3f, its weights in `dtype` as the entry point has them."""
    n = values.shape[0]
    flat = values.reshape(-1, 3)

    def field(x):
        r = (x - (origin + spacing / 2)) / spacing
        if reflective:
            for _ in range(8):
                out = (r < -0.5) | (r > n - 0.5)
                r = torch.where(out, 2 * n * (r > n - 0.5) - r - 1, r)
            lo = r.floor().long()
            hi = torch.where(lo < n - 1, lo + 1, lo)
            hi = torch.where(r < 0, torch.zeros_like(lo), hi)
            f0 = r - r.floor()
            lo = lo.clamp(min=0)
        else:
            fl = r.floor()
            lo = fl.long() % n
            hi = (lo + 1) % n
            f0 = r - fl
        i, f = (lo, hi), ((1 - f0).to(dtype), f0.to(dtype))
        b = 0
        for q in CORNERS:
            index = (i[q[0]][:, 0] * n + i[q[1]][:, 1]) * n + i[q[2]][:, 2]
            w = f[q[0]][:, 0] * f[q[1]][:, 1] * f[q[2]][:, 2]
            b = b + flat[index].to(dtype) * w[:, None]
        return b.double()

    return field


def _wave_sum(case, seed):
    spectrum, n_modes, mode_seed = _modes(case, seed)
    xi, kappa, k, beta, ak = (torch.from_numpy(a).cuda() for a in W.plane_wave_modes(*spectrum, n_modes, mode_seed))
    return lambda x: torch.cos((x @ kappa.T) * k + beta) @ (xi * ak[:, None])


def _boris(field, x, u, step, kq):
    """One Boris step of length `step` (n, 1); kq = q c / 2E."""
    x = x + u * step / 2
    t = field(x) * (kq * step)
    s = t * 2 / (1 + (t * t).sum(1, keepdim=True))
    u = u + torch.linalg.cross(u + torch.linalg.cross(u, t), s)
    return x + u * step / 2, u


A = ((), (1 / 5,), (3 / 40, 9 / 40), (3 / 10, -9 / 10, 6 / 5), (-11 / 54, 5 / 2, -70 / 27, 35 / 27),
     (1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096))
B5 = (37 / 378, 0, 250 / 621, 125 / 594, 0, 512 / 1771)
B4 = (2825 / 27648, 0, 18575 / 48384, 13525 / 55296, 277 / 14336, 1 / 4)


def _cash_karp(field, x, u, step, kq):
    """One Cash-Karp step: end point, direction, error of the direction."""
    h, kx, ku = step / U.c_light, [], []
    for a in A:
        yx, yu = x, u
        for c, vx, vu in zip(a, kx, ku):
            yx, yu = yx + vx * (c * h), yu + vu * (c * h)
        v = yu / yu.norm(dim=1, keepdim=True) * U.c_light
        kx.append(v)
        ku.append(torch.linalg.cross(v, field(yx)) * (2 * kq))
    add = lambda y, k, b: y + sum(v * c for v, c in zip(k, b)) * h  # noqa: E731
    err = sum(v * (p - q) for v, p, q in zip(ku, B5, B4)) * h
    return add(x, kx, B5), add(u, ku, B5), err.norm(dim=1)


def _walk(case, field, c, spec):
    """The chain's candidates stepped to their end in 64 bits: the real-valued members."""
    col = lambda *names: torch.stack([getattr(c, k) for k in names], 1)  # noqa: E731
    x, u, prev = col("x", "y", "z"), col("dx", "dy", "dz"), col("px", "py", "pz")
    kq = (c.charge * U.c_light / (2 * c.energy))[:, None]
    length, time, cur, nxt = c.trajectory_length, c.time, c.current_step, c.next_step
    prop = spec.modules[0]
    end = spec.modules[1].max_length
    adaptive = prop.min_step != prop.max_step
    todo = torch.arange(case["n"], device="cuda")
    while len(todo):
        x0, u0, k = x[todo], u[todo], kq[todo]
        if not adaptive:
            step = torch.full((len(todo),), prop.max_step, dtype=torch.float64, device="cuda")
            x1, u1 = _boris(field, x0, u0, step[:, None], k)
            new = step
        else:
            step = nxt[todo].clamp(prop.min_step, prop.max_step)
            x1, u1, new = torch.empty_like(x0), torch.empty_like(u0), step.clone()
            left = torch.arange(len(todo), device="cuda")
            while len(left):
                s = step[left]
                if prop.propagator == _abi.PROP_CK:
                    xa, ua, err = _cash_karp(field, x0[left], u0[left], s[:, None], k[left])
                    r = err / prop.tolerance
                else:
                    xa, ua = _boris(field, x0[left], u0[left], s[:, None], k[left])
                    xb, ub = _boris(field, x0[left], u0[left], s[:, None] / 2, k[left])
                    xb, ub = _boris(field, xb, ub, s[:, None] / 2, k[left])
                    r = math.sqrt(3.0) * (xa - xb).norm(dim=1) / (s * 0.75) / prop.tolerance
                x1[left], u1[left] = xa, ua
                want = s * 0.95 * r ** -0.2
                bad = (r > 1) & (s != prop.min_step)
                smaller = torch.maximum(torch.maximum(want, 0.1 * s), torch.full_like(s, prop.min_step))
                larger = torch.minimum(want, 5 * s).clamp(max=prop.max_step)
                new[left] = torch.where(r > 1, torch.where(bad, smaller, new[left]),
                                        torch.where(s != prop.max_step, larger, new[left]))
                step[left] = torch.where(bad, smaller, s)
                left = left[bad]
        prev[todo], x[todo], u[todo] = x0, x1, u1 / u1.norm(dim=1, keepdim=True)
        length[todo] += step
        time[todo] += step / U.c_light
        cur[todo], nxt[todo] = step, new
        on = length[todo] < end
        nxt[todo] = torch.where(on, torch.minimum(nxt[todo], end - length[todo]), nxt[todo])
        if case["kind"] == "region":
            r1, r0 = x[todo].norm(dim=1), prev[todo].norm(dim=1)
            d1, d0 = r1 - spec.modules[2].radius, r0 - spec.modules[2].radius
            room = spec.modules[3].size - r1
            nxt[todo] = torch.minimum(nxt[todo], torch.minimum(d1.abs(), room + spec.modules[3].margin))
            on &= ~((d1 * d0 <= 0) & (d0 != 0)) & (room > 0)
        todo = todo[on]
    return {"x": x[:, 0], "y": x[:, 1], "z": x[:, 2], "dx": u[:, 0], "dy": u[:, 1], "dz": u[:, 2],
            "px": prev[:, 0], "py": prev[:, 1], "pz": prev[:, 2], "trajectory_length": length, "time": time,
            "current_step": cur, "next_step": nxt, "active": None, "flags": None, "step_count": None}


def _loss(case, s, p0, grid):
    """The arrival loss by plain torch, in segments that the backward pass recomputes."""
    pn = p0.norm(dim=1, keepdim=True)
    kq = s["charge"][:, None] / (2 * pn)
    step = torch.full_like(pn, 1 * U.kpc)
    field = _trilinear(grid, 0.0, s["spacing"], False, torch.float64)

    def segment(x, u, k):
        for _ in range(k):
            x, u = _boris(field, x, u, step, kq)
            u = u / u.norm(dim=1, keepdim=True)
        return x, u

    x, u, k = s["pos"], p0 / pn, 25
    for i in range(0, case["steps"], k):
        x, u = torch.utils.checkpoint.checkpoint(segment, x, u, min(k, case["steps"] - i), use_reentrant=False)
    return (1 - (u * s["target"]).sum(1)).sum()


def exact(case, seed):
    kind = case["kind"]
    # nuclei: over 20 s of plain torch; diffusion: random displacements have no exact value;
    # galaxy: the fields' models have no 64-bit form outside this package
    if kind in ("nuclei", "diffusion", "galaxy"):
        return None
    # thousands of steps in single-precision increments: the turbulent field
    # separates such trajectories from the 64-bit ones altogether
    if kind == "boris" and case["precision"] == "mixed" and case["steps"] > 1500:
        return None
    if kind == "adjoint":
        s = _adjoint_inputs(case, seed)
        p0, grid = s["p0"].requires_grad_(True), s["grid"].double().requires_grad_(True)
        loss = _loss(case, s, p0, grid)
        g_p0, g_grid = torch.autograd.grad(loss, (p0, grid))
        return {"loss": loss.detach(), "grad_p0": g_p0, "grad_grid": g_grid}
    grid, spacing = _field(case, seed)
    spec = _chain(case, seed, np.zeros((1, 1, 1, 3), np.float32), spacing)
    if kind == "waves":
        field = _wave_sum(case, seed)
    else:
        # the chains' Grid3f interpolation is single precision by definition (Grid.h:571)
        origin = spec.fields[0].origin[0]
        field = _trilinear(grid, origin, spacing, kind == "region" and case["reflective"], torch.float32)
    return _walk(case, field, _candidates(case, seed), spec)
