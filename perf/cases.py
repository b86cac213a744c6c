"""Performance cases of the particle pass: what a program does with this package.

Each case goes through the public entry points on synthetic, seeded inputs with
the shapes of the configurations the package is used on (2-D and 3-D dam breaks
with walls, a periodic shear wave, a liquid column, droplet impacts).

``listed()``  the cases, ``draw(rng)`` one more of the same ranges,
``prepare(case, seed)`` the inputs and handles a program holds before the call,
``run(state)`` one pass, ``work(case)`` the bytes and operations it cannot do
without, ``exact(case, seed)`` the same outputs by plain torch in 64 bits.

Particle order: nothing in the drop-in path reorders particles, so a run's
arrays keep their lattice order while the particles drift apart.  The clouds
are shuffled over short distances of that order; ``mixed`` shuffles all of it,
as a flow that has been stirred for a long time does.
"""
from __future__ import annotations

from dataclasses import replace
import functools
import math

import torch

from tensorsph_b200.dam_break import DamBreakConfig, make_column
from tensorsph_b200.dam_break_3d import mass_3d, rhs_3d
from tensorsph_b200.droplet_impact import lattice_mass_unit, rhs, wall_lattice
from tensorsph_b200.engine import (BatchEngine, DamBreak3DEngine, capacity_for, dam_break_2d_case,
                                   dam_break_3d_host_state, obstacle_case)
from tensorsph_b200.ensemble import draw_ensemble, ensemble_specs
from tensorsph_b200.neighbor_search import PairListCache, cell_linked_pairs
from tensorsph_b200.particle_shifting import shift_positions
from tensorsph_b200.threed import accelerations, periodic_pairs
from tensorsph_b200.threed.csf3 import csf_fields3, surface_tension_acceleration3
from tensorsph_b200.transport_velocity_correction import transport_velocity_correction

DEV = "cuda"
F64 = torch.float64
DX = 0.01           # spacing of the generic clouds
HF = 1.3            # h / dx everywhere, the package's default
G = 9.81


def listed():
    return [
        # one search of a small cloud: a 2-D case's list rebuild, where launches and host reads count
        {"name": "pairs_2d_small", "kind": "pairs", "dim": 2, "n": 2000, "dtype": "float32", "box": False, "mixed": False},
        # the list rebuild of a large 3-D run
        {"name": "pairs_3d_large", "kind": "pairs", "dim": 3, "n": 1000000, "dtype": "float64", "box": False, "mixed": False},
        # one right-hand side of the 2-D dam break with a kept list (the step between two rebuilds), large
        {"name": "rhs_2d_large", "kind": "rhs2d", "n": 1019592, "dtype": "float32", "form": "molteni", "given": True},
        # the 5,000-particle 2-D dam break in FP64 with the psi diffusion, search included (no list kept)
        {"name": "rhs_2d_small", "kind": "rhs2d", "n": 5000, "dtype": "float64", "form": "antuono", "given": False},
        # the 3-D dam break with the obstacle's force read back, search included
        {"name": "rhs_3d", "kind": "rhs3d", "dx": 0.0138, "dtype": "float32", "given": False},
        # one evaluation of the 64^3 periodic shear wave in FP64 with a kept list
        {"name": "shear_3d", "kind": "shear", "edge": 64, "dtype": "float64", "psi": True},
        # particle shifting of a 2-D fluid after the update, search included
        {"name": "shift_2d", "kind": "shift", "dim": 2, "n": 200003, "dtype": "float32", "given": False, "mixed": False},
        # surface tension of a periodic liquid column, FP64
        {"name": "csf_3d", "kind": "csf3", "radius": 32, "length": 150, "dtype": "float64"},
        # transport-velocity correction over a stirred 3-D fluid with walls, FP64
        {"name": "tvc_3d", "kind": "tvc", "edge": 69, "dtype": "float64", "mixed": True},
        # the device engine: 3-D dam break with obstacle and shifting, the package's headline run
        {"name": "dam_3d", "kind": "dam3d", "dx": 0.0069, "steps": 8},
        # the device engine: the 5,000-particle 2-D dam break, where each step is short
        {"name": "dam_2d", "kind": "dam2d", "dx": 0.02, "steps": 20},
        # the device engine: an ensemble of droplet impacts with surface tension in one batch
        {"name": "droplets", "kind": "droplets", "count": 64, "steps": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pairs", "pairs", "rhs2d", "rhs2d", "rhs3d", "shear", "shift", "csf3", "tvc", "dam3d", "dam2d",
                       "droplets"])
    dtype = rng.choice(["float32", "float64"])
    if kind == "pairs":
        dim = rng.choice([2, 3])
        return {"kind": kind, "dim": dim, "n": _log(rng, 2000, 900000), "dtype": dtype, "box": rng.random() < 0.3,
                "mixed": rng.random() < 0.25}
    if kind == "rhs2d":
        return {"kind": kind, "n": _log(rng, 4000, 900000), "dtype": dtype, "form": rng.choice(["molteni", "antuono"]),
                "given": rng.random() < 0.6}
    if kind == "rhs3d":
        return {"kind": kind, "dx": round(math.exp(rng.uniform(math.log(0.0115), math.log(0.04))), 5), "dtype": dtype,
                "given": rng.random() < 0.6}
    if kind == "shear":
        return {"kind": kind, "edge": rng.randint(17, 80), "dtype": dtype, "psi": rng.random() < 0.5}
    if kind == "shift":
        return {"kind": kind, "dim": rng.choice([2, 3]), "n": _log(rng, 3000, 400000), "dtype": dtype,
                "given": rng.random() < 0.5, "mixed": rng.random() < 0.25}
    if kind == "csf3":
        return {"kind": kind, "radius": rng.randint(8, 32), "length": rng.randint(24, 150), "dtype": "float64"}
    if kind == "tvc":
        return {"kind": kind, "edge": rng.randint(14, 90), "dtype": "float64", "mixed": rng.random() < 0.25}
    if kind == "dam3d":
        return {"kind": kind, "dx": round(math.exp(rng.uniform(math.log(0.0085), math.log(0.03))), 5), "steps": 8}
    if kind == "dam2d":
        return {"kind": kind, "dx": round(math.exp(rng.uniform(math.log(0.004), math.log(0.021))), 5), "steps": 20}
    return {"kind": kind, "count": rng.randint(5, 64), "steps": 10}


# ------------------------------------------------------------------ inputs --

def _gen(seed, device=DEV):
    return torch.Generator(device=device).manual_seed(int(seed))


def _jitter(x, dx, gen):
    return x + dx * (2.0 * torch.rand(x.shape, generator=gen, dtype=F64, device=x.device) - 1.0)


def _grid(counts, dx):
    axes = torch.meshgrid(*[(torch.arange(c, dtype=F64, device=DEV) + 0.5) * dx for c in counts], indexing="ij")
    return torch.stack([a.reshape(-1) for a in axes], dim=-1)


def _shuffled(x, gen, mixed):
    n = x.shape[0]
    if mixed:
        return x[torch.randperm(n, generator=gen, device=x.device)]
    drift = 64.0 * torch.rand(n, generator=gen, dtype=F64, device=x.device)
    return x[torch.argsort(torch.arange(n, dtype=F64, device=x.device) + drift)]


def _cloud(dim, n, seed, mixed=False, jitter=0.1):
    """``n`` particles of a jittered lattice block; its edges."""
    side = (n / (2.0 if dim == 2 else 1.1)) ** (1.0 / dim)
    counts = [max(4, round(side)) for _ in range(dim - 1)]
    counts.append(-(-n // math.prod(counts)))
    g = _gen(seed)
    x = _jitter(_grid(counts, DX)[:n], jitter * DX, g)
    return _shuffled(x, g, mixed).contiguous(), [c * DX for c in counts]


def _velocity(x, seed, scale=1.0):
    k = 2.0 * math.pi / float(x.max())
    v = torch.stack([torch.sin(k * x[:, (a + 1) % x.shape[1]]) for a in range(x.shape[1])], dim=1)
    return scale * (v + 0.1 * torch.randn(x.shape, generator=_gen(seed + 77), dtype=F64, device=x.device))


def _default64(f):
    @functools.wraps(f)
    def g(*a, **k):
        saved = torch.get_default_dtype()
        torch.set_default_dtype(F64)
        try:
            return f(*a, **k)
        finally:
            torch.set_default_dtype(saved)
    return g


def _dam_config_2d(dx, form="molteni"):
    c0 = 10.0 * math.sqrt(2.0 * G * 2.0)
    return DamBreakConfig(dx=dx, column_width=1.0, column_height=2.0, pool_width=4.0, tank_height=3.0, sound_speed=c0,
                          viscosity=1.0e-6, dt=0.25 * HF * dx / c0, density_diffusion=0.1, density_diffusion_form=form)


@_default64
def _rhs2d_arrays(case, seed):
    cfg = _dam_config_2d(math.sqrt(2.0 / case["n"]), case["form"])
    x, m = make_column(cfg, DEV)
    wall = wall_lattice(cfg, DEV, top=cfg.tank_top())
    x = _jitter(x, 0.05 * cfg.dx, _gen(seed))
    dt = getattr(torch, case["dtype"])
    return cfg, x.to(dt), _velocity(x, seed).to(dt), m.to(dt), wall.to(dt)


@functools.lru_cache(maxsize=2)
def _dam3d_lattice(dx):
    cfg, obstacle = obstacle_case(dx)
    return cfg, obstacle, dam_break_3d_host_state(cfg, obstacle)


def _rhs3d_arrays(case, seed):
    cfg, _, (x, m, wall, _) = _dam3d_lattice(case["dx"])
    x = _jitter(x.to(DEV), 0.05 * cfg.dx, _gen(seed))
    dt = getattr(torch, case["dtype"])
    return cfg, x.to(dt), _velocity(x, seed).to(dt), m.to(DEV, dt), wall.to(DEV, dt)


def _shear_arrays(case, seed):
    e, dt = case["edge"], getattr(torch, case["dtype"])
    dx = 1.0 / e
    x = _jitter(_grid([e] * 3, dx), 0.05 * dx, _gen(seed)).remainder(1.0)
    v = torch.zeros_like(x)
    v[:, 0] = 1.0e-3 * torch.sin(2.0 * math.pi * x[:, 2])
    m = torch.full((x.shape[0],), mass_3d(dx, HF, 1000.0, True), dtype=F64, device=DEV)
    h = HF * dx
    kw = dict(rho0=1000.0, sound_speed=1.0, viscosity=1.0e-2)
    if case["psi"]:
        kw.update(density_diffusion=0.1, dt=min(0.25 * h, 0.1 * h * h / 1.0e-2))
    return x.to(dt), v.to(dt), m.to(dt), h, kw


def _csf3_arrays(case, seed):
    r, length, dt = case["radius"], case["length"], getattr(torch, case["dtype"])
    x = _grid([2 * r + 1, 2 * r + 1, length], DX)
    x[:, :2] -= (r + 0.5) * DX
    x = x[x[:, 0].square() + x[:, 1].square() <= (r * DX) ** 2]
    x = _jitter(x, 0.05 * DX, _gen(seed))
    box = [4.0 * r * DX, 4.0 * r * DX, length * DX]
    x[:, :2] += 0.5 * box[0]
    x[:, 2] = x[:, 2].remainder(box[2])
    rho = 1000.0 * (1.0 + 0.01 * torch.rand(x.shape[0], generator=_gen(seed + 5), dtype=F64, device=DEV))
    return x.to(dt), torch.full((x.shape[0],), 1000.0 * DX ** 3, dtype=dt, device=DEV), rho.to(dt), box


def _tvc_arrays(case, seed):
    e, dt, g = case["edge"], getattr(torch, case["dtype"]), _gen(seed)
    x = _shuffled(_jitter(_grid([e] * 3, DX), 0.08 * DX, g), g, case["mixed"])
    floor = _grid([e, 3, e], DX)
    floor[:, 1] = -floor[:, 1]
    x = torch.cat((x, floor)).to(dt).contiguous()
    return x, torch.full((x.shape[0],), DX ** 3, dtype=dt, device=DEV), floor.shape[0]


def _dam3d_host(case, seed):
    cfg, obstacle, (x, m, wall, n_ob) = _dam3d_lattice(case["dx"])
    cfg = replace(cfg, pair_skin_factor=0.15)     # the autotuner's choice for this run
    x = _jitter(x.to(DEV), 0.05 * cfg.dx, _gen(seed))
    return cfg, obstacle, (x.cpu(), m, wall, n_ob)


def _dam2d_spec(case, seed):
    spec = dam_break_2d_case(_dam_config_2d(case["dx"]))
    return replace(spec, x=_jitter(spec.x, 0.05 * case["dx"], _gen(seed, "cpu")))


def _droplet_specs(case, seed):
    g = _gen(seed, "cpu")
    return [replace(s, x=_jitter(s.x, 0.02 * s.params.h / HF, g)) for s in ensemble_specs(draw_ensemble(case["count"]))]


# ----------------------------------------------------------------- prepare --

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "pairs":
        # the list cutoff lies between two lattice shells, which this jitter does not cross: every
        # seed has as many pairs
        x, box = _cloud(case["dim"], case["n"], seed, case["mixed"], jitter=0.045)
        s.update(x=x.to(getattr(torch, case["dtype"])).contiguous(), cutoff=2.05 * HF * DX,
                 box=box if case["box"] else None)
    elif kind in ("rhs2d", "rhs3d"):
        cfg, x, v, m, wall = (_rhs2d_arrays if kind == "rhs2d" else _rhs3d_arrays)(case, seed)
        pairs = None
        if case["given"]:
            h = HF * cfg.dx
            pairs, _ = PairListCache(2.0 * h, 0.15 * h, fluid_count=x.shape[0]).get(torch.cat((x, wall)))
        s.update(cfg=cfg, x=x, v=v, m=m, wall=wall, pairs=pairs)
    elif kind == "shear":
        x, v, m, h, kw = _shear_arrays(case, seed)
        s.update(x=x, v=v, m=m, h=h, kw=kw, box=[1.0] * 3, pairs=periodic_pairs(x, [1.0] * 3, 2.1 * h))
    elif kind == "shift":
        x, _ = _cloud(case["dim"], case["n"], seed, case["mixed"])
        x = x.to(getattr(torch, case["dtype"]))
        vol = torch.full((x.shape[0],), DX ** case["dim"], dtype=x.dtype, device=DEV)
        s.update(x=x, vol=vol, pairs=cell_linked_pairs(x, 2.15 * HF * DX) if case["given"] else None)
    elif kind == "csf3":
        x, m, rho, box = _csf3_arrays(case, seed)
        s.update(x=x, m=m, rho=rho, box=box, pairs=periodic_pairs(x, box, 2.0 * HF * DX))
    elif kind == "tvc":
        x, vol, walls = _tvc_arrays(case, seed)
        s.update(x=x, vol=vol, walls=walls, pairs=cell_linked_pairs(x, 2.0 * HF * DX))
    elif kind == "dam3d":
        cfg, obstacle, host = _dam3d_host(case, seed)
        eng = DamBreak3DEngine(cfg, obstacle=obstacle, shift_every=1, host_state=host)
        eng.set_batch(8)                          # the autotuner's choice for this run
        s.update(eng=eng, ids=[eng.case_id])
    elif kind == "dam2d":
        spec = _dam2d_spec(case, seed)
        eng = BatchEngine(**capacity_for([spec], max_neighbors=64))
        s.update(eng=eng, ids=[eng.add(spec)])
    else:
        specs = _droplet_specs(case, seed)
        eng = BatchEngine(**capacity_for(specs, max_neighbors=64))
        s.update(eng=eng, ids=[eng.add(spec) for spec in specs])
    return s


# --------------------------------------------------------------------- run --

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "pairs":
        return cell_linked_pairs(s["x"], s["cutoff"]) if s["box"] is None else periodic_pairs(s["x"], s["box"], s["cutoff"])
    if kind == "rhs2d":
        return rhs(s["x"], s["v"], s["m"], s["cfg"], pairs=s["pairs"], wall=s["wall"])
    if kind == "rhs3d":
        return rhs_3d(s["x"], s["v"], s["m"], s["cfg"], pairs=s["pairs"], wall=s["wall"], return_wall_force=True)
    if kind == "shear":
        return accelerations(s["x"], s["v"], s["m"], s["h"], s["pairs"], box=s["box"], **s["kw"])
    if kind == "shift":
        out, st = shift_positions(s["x"], s["vol"], HF * DX, dt=1.0e-3, v_ref=1.0, pairs=s["pairs"], return_state=True)
        return out, st.concentration, st.grad_c, st.shift
    if kind == "csf3":
        st = csf_fields3(s["x"], s["m"], HF * DX, s["pairs"], rho0=1000.0, box=s["box"])
        acc = surface_tension_acceleration3(st, s["rho"], 0.0728)
        return st.color, st.grad_c, st.normal, st.kappa, st.delta_s, acc
    if kind == "tvc":
        r = transport_velocity_correction(s["x"], s["vol"], HF * DX, pairs=s["pairs"], wall_count=s["walls"],
                                          max_shift=0.05 * HF * DX)
        return r.gradient_integral, r.shift, r.squared_norm
    # a run's chunk of steps and the state it writes out: positions in 64 bits, the fields of the
    # FP32 pair pass in 32 (velocity, density and pressure of a snapshot)
    s["eng"].step(case["steps"])
    got = [s["eng"].read(i) for i in s["ids"]]
    x, v, rho, p = (got[0] if len(got) == 1 else [torch.cat([g[k] for g in got]) for k in range(4)])
    return x, v.float(), rho.float(), p.float()


# -------------------------------------------------------------------- work --

def _per_particle(dim, reach):
    """Pairs per particle of a lattice cloud within ``reach`` spacings."""
    return 0.5 * (math.pi * reach ** 2 if dim == 2 else 4.0 / 3.0 * math.pi * reach ** 3)


def _dam3d_count(dx):
    return 0.66 / dx ** 3, 3.0 * (3.2 * 1.0 + 2 * 1.0 + 2 * 3.2) / dx ** 2


def work(case):
    kind = case["kind"]
    w = 4 if case.get("dtype") == "float32" else 8
    if kind == "pairs":
        p = case["n"] * _per_particle(case["dim"], 2.05 * HF)
        return {"bytes": case["n"] * case["dim"] * w + 16.0 * p, "flops": 9.0 * p}
    if kind == "rhs2d":
        p = case["n"] * _per_particle(2, 2.15 * HF)
        return {"bytes": case["n"] * 9 * w + (16.0 * p if case["given"] else 0.0), "flops": 2 * 110.0 * p}
    if kind == "rhs3d":
        n, nw = _dam3d_count(case["dx"])
        p = n * _per_particle(3, 2.15 * HF)
        return {"bytes": n * 12 * w + nw * 6 * w + (16.0 * p if case["given"] else 0.0), "flops": 2 * 140.0 * p}
    if kind == "shear":
        n = case["edge"] ** 3
        p = n * _per_particle(3, 2.1 * HF)
        return {"bytes": n * 12 * w + 16.0 * p, "flops": 2 * (240.0 if case["psi"] else 130.0) * p}
    if kind == "shift":
        p = case["n"] * _per_particle(case["dim"], 2.15 * HF)
        return {"bytes": case["n"] * (4 * case["dim"] + 2) * w + (16.0 * p if case["given"] else 0.0), "flops": 2 * 60.0 * p}
    if kind == "csf3":
        n = math.pi * case["radius"] ** 2 * case["length"]
        p = n * _per_particle(3, 2.0 * HF)
        return {"bytes": n * 17 * w + 16.0 * p, "flops": 2 * 180.0 * p}
    if kind == "tvc":
        n = case["edge"] ** 3 + 3 * case["edge"] ** 2
        p = n * _per_particle(3, 2.0 * HF)
        return {"bytes": n * 11 * w + 16.0 * p, "flops": 2 * 40.0 * p}
    if kind == "dam3d":
        n, nw = _dam3d_count(case["dx"])
        p = n * _per_particle(3, 2.0 * HF)
        return {"bytes": case["steps"] * (n * 308.0 + nw * 48.0) + n * 44.0, "flops": case["steps"] * 2 * 250.0 * p}
    if kind == "dam2d":
        n = 2.0 / case["dx"] ** 2
        return {"bytes": case["steps"] * n * 268.0 + n * 36.0, "flops": case["steps"] * n * 2 * 170.0 * _per_particle(2, 2 * HF)}
    n = case["count"] * 14000.0
    fit = _per_particle(2, 4 * HF)
    return {"bytes": case["steps"] * n * 600.0 + n * 36.0,
            "flops": case["steps"] * n * 2 * (320.0 * _per_particle(2, 2 * HF) + 40.0 * fit)}


# ------------------------------------------------------------ 64-bit values --
# Plain torch over unordered pairs (i, j), each added to both of its ends.

def _near(x, cutoff, box=None):
    """Unordered pairs within ``cutoff`` and their separations x_i - x_j."""
    n, dim = x.shape
    if box is not None:
        edges = torch.tensor(box, dtype=F64, device=x.device)
        nc = [max(3, int(b / cutoff)) for b in box]
        cell = torch.stack([torch.floor(x[:, k] / (box[k] / nc[k])).long() % nc[k] for k in range(dim)], dim=1)
    else:
        cell = torch.floor(x / cutoff).long()
        cell = cell - cell.min(dim=0).values + 1
        nc = [int(c) + 2 for c in cell.max(dim=0).values]
    stride = [math.prod(nc[k + 1:]) for k in range(dim)]
    key = sum(cell[:, k] * stride[k] for k in range(dim))
    sk, order = torch.sort(key)
    xs, cs = x[order], cell[order]
    left, right = [], []
    for o in range(3 ** dim // 2, 3 ** dim):      # half of the stencil; its first entry is the home cell
        off = [(o // 3 ** (dim - 1 - k)) % 3 - 1 for k in range(dim)]
        nb = [cs[:, k] + off[k] for k in range(dim)]
        if box is not None:
            nb = [c % nc[k] for k, c in enumerate(nb)]
        nk = sum(c * stride[k] for k, c in enumerate(nb))
        lo, hi = torch.searchsorted(sk, nk), torch.searchsorted(sk, nk, right=True)
        home = not any(off)
        if home:
            lo = torch.arange(1, n + 1, device=x.device)
        cnt = (hi - lo).clamp_min(0)
        i = torch.repeat_interleave(torch.arange(n, device=x.device), cnt)
        j = lo[i] + torch.arange(i.numel(), device=x.device) - (torch.cumsum(cnt, 0) - cnt)[i]
        d = xs[i] - xs[j]
        if box is not None:
            d = d - edges * torch.round(d / edges)
        keep = d.square().sum(dim=1) <= cutoff * cutoff
        left.append(order[i[keep]])
        right.append(order[j[keep]])
    i, j = torch.cat(left), torch.cat(right)
    return i, j, _delta(x, i, j, box)


def _delta(x, i, j, box=None):
    d = x[i] - x[j]
    if box is not None:
        edges = torch.tensor(box, dtype=F64, device=x.device)
        d = d - edges * torch.round(d / edges)
    return d


def _cubic(d, h, dim):
    """Distance, W and the scale g with grad_i W = g d."""
    r = d.square().sum(dim=1).sqrt()
    q = r / h
    s = 10.0 / (7.0 * math.pi * h * h) if dim == 2 else 1.0 / (math.pi * h ** 3)
    t = (2.0 - q).clamp_min(0.0)
    w = s * torch.where(q < 1.0, 1.0 - 1.5 * q * q + 0.75 * q ** 3, 0.25 * t ** 3)
    f = torch.where(q < 1.0, -3.0 * q + 2.25 * q * q, -0.75 * t * t)
    return r, w, s * f / (h * r.clamp_min(1e-12)), s


def _add(n, i, vi, j, vj):
    out = torch.zeros((n,) + vi.shape[1:], dtype=vi.dtype, device=vi.device)
    return out.index_add_(0, i, vi).index_add_(0, j, vj)


def _tait(rho, rho0, c0, gamma=7.0):
    return (rho0 * c0 ** 2 / gamma * ((rho / rho0).clamp_min(0.01) ** gamma - 1.0)).clamp_min(0.0)


def _floored(m, g, floor):
    """(V max(l, floor mean l) V^T)^-1 g for symmetric m."""
    vals, vecs = torch.linalg.eigh(m.cpu())
    vals, vecs = vals.to(g.device), vecs.to(g.device)
    mean = (vals.sum(dim=1) / m.shape[1]).clamp_min(1e-30)
    vals = torch.maximum(vals, floor * mean[:, None])
    return torch.einsum("pak,pk->pa", vecs, torch.einsum("pka,pk->pa", vecs, g) / vals)


def _diffusion(rho, m, i, j, d, g, form, floor=0.1):
    """The density diffusion's rate at unit scale."""
    n, d2 = rho.shape[0], d.square().sum(dim=1)
    vi, vj = (m / rho)[i], (m / rho)[j]
    contrast = rho[i] - rho[j]
    if form == "antuono":
        diff = (rho[j] - rho[i])[:, None] * (g[:, None] * d)
        grad = _add(n, i, vj[:, None] * diff, j, vi[:, None] * diff)
        outer = -(g[:, None, None] * d[:, :, None] * d[:, None, :])
        grad = _floored(_add(n, i, vj[:, None, None] * outer, j, vi[:, None, None] * outer), grad, floor)
        contrast = contrast - 0.5 * ((grad[i] + grad[j]) * d).sum(dim=1)
    c = contrast * (-g * d2) / (d2 + 1e-12)
    return _add(n, i, -vj * c, j, vi * c)


def _wcsph(x, v, m, wall, cfg, unit, i, j, diffusion, form="molteni"):
    """rho, p, acc and the reaction on the walls, from pairs of cat(x, wall) without wall-wall pairs."""
    n, nw, dim, h = x.shape[0], wall.shape[0], x.shape[1], HF * cfg.dx
    pos = torch.cat((x, wall))
    mass = torch.cat((m, torch.full((nw,), unit, dtype=F64, device=x.device)))
    d = pos[i] - pos[j]
    r, w, g, s = _cubic(d, h, dim)
    rho = (mass * s + _add(n + nw, i, mass[j] * w, j, mass[i] * w))[:n].clamp_min(0.1 * cfg.rho0)
    ff = (i < n) & (j < n)
    if diffusion > 0.0:
        rate = _diffusion(rho, m, i[ff], j[ff], d[ff], g[ff], form, cfg.density_diffusion_eigenvalue_floor)
        rho = (rho + cfg.dt * 2.0 * diffusion * cfg.sound_speed * h * rate).clamp_min(0.1 * cfg.rho0)
    p = _tait(rho, cfg.rho0, cfg.sound_speed, cfg.gamma)
    cross = ~ff
    fi = torch.where(i < n, i, j)[cross]
    wi = torch.where(i < n, j, i)[cross]
    dy = (pos[wi] - pos[fi])[:, 1]
    num = torch.zeros(n + nw, dtype=F64, device=x.device).index_add_(0, wi, (p[fi] - rho[fi] * cfg.gravity * dy) * w[cross])
    den = torch.zeros(n + nw, dtype=F64, device=x.device).index_add_(0, wi, w[cross])
    pw = (num / den.clamp_min(1e-30))[n:].clamp_min(0.0)
    bulk = cfg.rho0 * cfg.sound_speed ** 2 / cfg.gamma
    pa = torch.cat((p, pw))
    da = torch.cat((rho, cfg.rho0 * (pw / bulk + 1.0) ** (1.0 / cfg.gamma)))
    va = torch.cat((v, torch.zeros_like(wall)))
    f = ((pa[i] / da[i] ** 2 + pa[j] / da[j] ** 2) * g)[:, None] * d
    acc = _add(n + nw, i, -mass[j][:, None] * f, j, mass[i][:, None] * f)
    lw = 2.0 * cfg.viscosity * (-g * r * r).clamp_min(0.0) / (r * r + 0.01 * h * h) * ff
    dv = (va[i] - va[j]) * lw[:, None]
    acc = acc + _add(n + nw, i, -(mass / da)[j][:, None] * dv, j, (mass / da)[i][:, None] * dv)
    acc = acc[:n].clone()
    acc[:, 1] -= cfg.gravity
    sign = torch.where(i < n, 1.0, -1.0)[cross]
    reaction = torch.zeros((n + nw, dim), dtype=F64, device=x.device)
    reaction.index_add_(0, wi, (sign * mass[i[cross]] * mass[j[cross]])[:, None] * f[cross])
    return rho, p, acc, reaction[n:]


def _fluid_pairs(x, wall, cutoff):
    i, j, _ = _near(torch.cat((x, wall)), cutoff)
    keep = torch.minimum(i, j) < x.shape[0]
    return i[keep], j[keep]


def _shifted(x, vol, h, magnitude, i, j):
    d = x[i] - x[j]
    _, w, g, s = _cubic(d, h, 2)                  # the 2-D normalisation in every dimension
    c = vol * s + _add(x.shape[0], i, vol[j] * w, j, vol[i] * w)
    diff = ((c[j] - c[i]) * g)[:, None] * d
    grad = _add(x.shape[0], i, vol[j][:, None] * diff, j, vol[i][:, None] * diff)
    mag = grad.square().sum(dim=1).sqrt()
    normal = -grad / mag.clamp_min(1e-30)[:, None]
    q = 0.95 * (c.numel() - 1)
    cs = torch.sort(c).values
    lo = int(q)
    ref = cs[lo] + (q - lo) * (cs[min(lo + 1, c.numel() - 1)] - cs[lo])
    shift = -magnitude * grad
    free = (c < 0.95 * ref)[:, None]
    shift = torch.where(free, shift - (shift * normal).sum(dim=1, keepdim=True) * normal, shift)
    size = shift.square().sum(dim=1).sqrt()
    shift = shift * torch.where(size > 0.25 * h, 0.25 * h / size.clamp_min(1e-300), 1.0)[:, None]
    return x + shift, c, grad, shift


def _advance(x, v, acc, cfg, box):
    v = v + cfg.dt * acc
    x = x + cfg.dt * v
    tol = 0.25 * cfg.dx
    v = torch.where((x < -tol) | (x > box + tol), 0.0, v)
    return torch.minimum(x.clamp_min(0.0), box), v


def _inverse3(a):
    """Inverse and determinant of 3 x 3 matrices, by cofactors."""
    c = torch.stack([torch.linalg.cross(a[:, 1], a[:, 2]), torch.linalg.cross(a[:, 2], a[:, 0]),
                     torch.linalg.cross(a[:, 0], a[:, 1])], dim=2)
    det = (a[:, 0] * c[:, :, 0]).sum(dim=1)
    return c / det[:, None, None], det


def _lower_median(x):
    return torch.sort(x).values[(x.numel() - 1) // 2]


def _shear_exact(x, v, m, h, kw):
    n = x.shape[0]
    i, j, d = _near(x, 2.1 * h, [1.0] * 3)
    r, w, g, s = _cubic(d, h, 3)
    rho = m * s + _add(n, i, m[j] * w, j, m[i] * w)
    if "density_diffusion" in kw:
        rate = _diffusion(rho, m, i, j, d, g, "antuono")
        rho = (rho + kw["dt"] * 2.0 * kw["density_diffusion"] * kw["sound_speed"] * h * rate).clamp_min(100.0)
    p = (1000.0 / 7.0 * ((rho / 1000.0) ** 7.0 - 1.0)).clamp_min(0.0)
    f = ((p[i] / rho[i] ** 2 + p[j] / rho[j] ** 2) * g)[:, None] * d
    acc = _add(n, i, -m[j][:, None] * f, j, m[i][:, None] * f)
    q = r / h
    fp = torch.where(q < 1.0, -3.0 * q + 2.25 * q * q, -0.75 * (2.0 - q).clamp_min(0.0) ** 2)
    second = torch.where(q < 1.0, -3.0 + 4.5 * q, 1.5 * (2.0 - q).clamp_min(0.0))
    lap = torch.where(q < 2.0, s * (second + 2.0 * fp / q.clamp_min(1e-12)) / (h * h), 0.0)
    rij = 0.5 * (rho[i] + rho[j])
    moment = _add(n, i, r * r * lap * m[j] / rij, j, r * r * lap * m[i] / rij) / 3.0
    weight = m[j] * lap / rij * (2.0 / (0.5 * (moment[i] + moment[j])).clamp_min(1e-12))
    dv = (v[j] - v[i]) * weight[:, None]
    return acc + kw["viscosity"] * _add(n, i, dv, j, -dv), rho, p


def _csf3_exact(x, m, rho, box):
    h, n, vol = HF * DX, x.shape[0], m / 1000.0
    i, j, d = _near(x, 2.0 * h, box)
    _, w, g, s = _cubic(d, h, 3)
    c = vol * s + _add(n, i, vol[j] * w, j, vol[i] * w)
    outer = -(g[:, None, None] * d[:, :, None] * d[:, None, :])
    a = _add(n, i, vol[j][:, None, None] * outer, j, vol[i][:, None, None] * outer)
    _, det = _inverse3(a)
    valid = det.abs() > 1e-6 * _lower_median(det.abs()).clamp_min(1e-30)
    inv, _ = _inverse3(torch.where(valid[:, None, None], a, torch.eye(3, dtype=F64, device=x.device)))
    num = ((c[j] - c[i]) * g)[:, None] * d
    grad = torch.einsum("pab,pb->pa", inv, _add(n, i, vol[j][:, None] * num, j, vol[i][:, None] * num))
    ds = grad.square().sum(dim=1).sqrt()
    normal = -grad / ds.clamp_min(1e-30)[:, None]
    kappa = torch.zeros(n, dtype=F64, device=x.device)
    for k in range(3):                            # trace(S inv), one row of S at a time
        row = ((normal[j, k] - normal[i, k]) * g)[:, None] * d
        row = _add(n, i, vol[j][:, None] * row, j, vol[i][:, None] * row)
        kappa += (row * inv[:, k]).sum(dim=1)
    kappa = torch.where(valid, kappa, 0.0)
    on = ds > 1e-3 * ds.max()
    return c, grad, normal, kappa, ds, -(0.0728 * kappa * ds * on / rho)[:, None] * normal


def _csf2_exact(x, rho, m, h, sigma, rho0):
    """Acceleration of the consistent 2-D scheme with the quadratic curvature fit over 4h."""
    n, vol = x.shape[0], m / rho0
    i, j, d = _near(x, 4.0 * h)
    _, w, g, s = _cubic(d, h, 2)
    gw = g[:, None] * d
    c = (vol * s + _add(n, i, vol[j] * w, j, vol[i] * w)).clamp(0.0, 1.0)
    outer = -(d[:, :, None] * gw[:, None, :])
    a = _add(n, i, vol[j][:, None, None] * outer, j, vol[i][:, None, None] * outer)
    det = (a[:, 0, 0] * a[:, 1, 1] - a[:, 0, 1] * a[:, 1, 0]).abs()
    ok = det > 1e-4 * _lower_median(det).clamp_min(1e-30)
    inv = torch.linalg.inv(torch.where(ok[:, None, None], a, torch.eye(2, dtype=F64, device=x.device)))
    num = (c[j] - c[i])[:, None] * gw
    grad = torch.einsum("pba,pb->pa", inv, _add(n, i, vol[j][:, None] * num, j, vol[i][:, None] * num))
    mag = grad.square().sum(dim=1).sqrt()
    has = (mag > 1e-12)[:, None]
    normal = torch.where(has, -grad / mag.clamp_min(1e-12)[:, None], 0.0)
    sm = normal
    den = (vol * s + _add(n, i, vol[j] * w, j, vol[i] * w)).clamp_min(1e-30)[:, None]
    for _ in range(2):
        sm = _add(n, i, (vol[j] * w)[:, None] * sm[j], j, (vol[i] * w)[:, None] * sm[i]) / den
    normal = torch.where(has, sm / sm.square().sum(dim=1).sqrt().clamp_min(1e-12)[:, None], normal)
    cn = (normal[j] - normal[i])[:, :, None] * gw[:, None, :]
    kappa = (_add(n, i, vol[j][:, None, None] * cn, j, vol[i][:, None, None] * cn) * inv.transpose(1, 2)).sum(dim=(1, 2))
    ds = 2.0 * mag
    node = (ds / ds.max().clamp_min(1e-30)).clamp(0.0, 1.0)
    tangent = torch.stack((-normal[:, 1], normal[:, 0]), dim=1)

    def moments(a_, b_, sgn):
        u, y = (sgn * d * tangent[a_]).sum(dim=1), (sgn * d * normal[a_]).sum(dim=1)
        return torch.stack([torch.ones_like(u), u, y, u * u, u * y, u ** 3, u * u * y, u ** 4], dim=1) * node[b_][:, None]

    z = _add(n, i, moments(i, j, -1.0), j, moments(j, i, 1.0))
    z[:, 0] += node
    mat = torch.stack([z[:, [0, 1, 3]], z[:, [1, 3, 5]], z[:, [3, 5, 7]]], dim=1)
    _, det3 = _inverse3(mat)
    fit = (node > 0.05) & (det3.abs() > 1e-6 * det3.abs().max().clamp_min(1e-30))
    inv3, _ = _inverse3(torch.where(fit[:, None, None], mat, torch.eye(3, dtype=F64, device=x.device)))
    sol = torch.einsum("pab,pb->pa", inv3, z[:, [2, 4, 6]])
    kappa = torch.where(fit, -2.0 * sol[:, 2] / (1.0 + sol[:, 1] ** 2) ** 1.5, kappa)
    ds = torch.where(mag <= 1e-3 * mag.max(), 0.0, ds)
    return (-sigma * kappa * ds)[:, None] * normal / rho[:, None]


def _engine_exact(x, v, m, wall, cfg, unit, box, steps, *, diffusion, shift=False, sigma=0.0):
    h = HF * cfg.dx
    box = torch.tensor(box, dtype=F64, device=DEV)
    i, j = _fluid_pairs(x, wall, 2.1 * h)
    rho = p = None
    for k in range(steps):
        rho, p, acc, _ = _wcsph(x, v, m, wall, cfg, unit, i, j, diffusion)
        if sigma > 0.0:
            acc = acc + _csf2_exact(x, rho, m, h, sigma, cfg.rho0)
        speed = float(v.square().sum(dim=1).sqrt().max())
        x, v = _advance(x, v, acc, cfg, box)
        if shift and k:
            ff = (i < x.shape[0]) & (j < x.shape[0])
            x = _shifted(x, m / rho, h, h * max(speed, 0.05 * cfg.sound_speed) * cfg.dt, i[ff], j[ff])[0]
    return x, v, rho, p


def exact(case, seed):
    kind = case["kind"]
    if kind == "pairs":
        return None
    if kind in ("rhs2d", "rhs3d"):
        cfg, x, v, m, wall = (_rhs2d_arrays if kind == "rhs2d" else _rhs3d_arrays)(case, seed)
        x, v, m, wall = (t.double() for t in (x, v, m, wall))
        # rhs makes the wall masses in the default dtype, rhs_3d in the positions'
        unit = (float(torch.tensor(lattice_mass_unit(cfg), dtype=torch.get_default_dtype())) if kind == "rhs2d"
                else mass_3d(cfg.dx, HF, cfg.rho0, True))
        i, j = _fluid_pairs(x, wall, 2.0 * HF * cfg.dx)
        out = _wcsph(x, v, m, wall, cfg, unit, i, j, cfg.density_diffusion, case.get("form", "molteni"))
        return out if kind == "rhs3d" else out[:3]
    if kind == "shear":
        x, v, m, h, kw = _shear_arrays(case, seed)
        return _shear_exact(x.double(), v.double(), m.double(), h, kw)
    if kind == "shift":
        x, _ = _cloud(case["dim"], case["n"], seed, case["mixed"])
        x = x.to(getattr(torch, case["dtype"])).double()
        vol = torch.full((x.shape[0],), DX ** case["dim"], dtype=F64, device=DEV)
        i, j, _ = _near(x, 2.0 * HF * DX)
        return _shifted(x, vol, HF * DX, HF * DX * 1.0e-3, i, j)
    if kind == "csf3":
        x, m, rho, box = _csf3_arrays(case, seed)
        return _csf3_exact(x.double(), m.double(), rho.double(), box)
    if kind == "tvc":
        x, vol, walls = _tvc_arrays(case, seed)
        h, n = HF * DX, x.shape[0] - walls
        i, j, d = _near(x, 2.0 * h)
        _, _, g, _ = _cubic(d, h, 3)
        f = 2.0 * g[:, None] * d
        grad = -_add(x.shape[0], i, vol[j][:, None] * f, j, -vol[i][:, None] * f)[:n]
        shift = 0.05 * h * h * grad
        size = shift.square().sum(dim=1).sqrt()
        cap = 0.05 * h
        shift = shift * torch.where(size > cap, cap / size.clamp_min(1e-30), 1.0)[:, None]
        return grad, shift, grad.square().sum(dim=1)
    if kind == "dam3d":
        cfg, _, (x, m, wall, _) = _dam3d_host(case, seed)
        x, m, wall = (t.to(DEV) for t in (x, m, wall))
        return _engine_exact(x, torch.zeros_like(x), m, wall, cfg, mass_3d(cfg.dx, HF, cfg.rho0, True),
                             (cfg.pool_width, cfg.tank_height, cfg.tank_depth), case["steps"],
                             diffusion=cfg.density_diffusion, shift=True)
    if kind == "dam2d":
        cfg, spec = _dam_config_2d(case["dx"]), _dam2d_spec(case, seed)
        x, m, wall = (t.to(DEV) for t in (spec.x, spec.mass, spec.wall))
        return _engine_exact(x, torch.zeros_like(x), m, wall, cfg, lattice_mass_unit(cfg),
                             (cfg.pool_width, cfg.tank_height), case["steps"], diffusion=cfg.density_diffusion)
    from tensorsph_b200.droplet_impact import domain_top
    from tensorsph_b200.ensemble import droplet_config
    got = []
    for one, spec in zip(draw_ensemble(case["count"]), _droplet_specs(case, seed)):
        cfg = droplet_config(one)
        x, v, m, wall = (t.to(DEV) for t in (spec.x, spec.v, spec.mass, spec.wall))
        got.append(_engine_exact(x, v, m, wall, cfg, lattice_mass_unit(cfg), (cfg.pool_width, domain_top(cfg)),
                                 case["steps"], diffusion=0.0, sigma=cfg.surface_tension_coefficient))
    return tuple(torch.cat([g[k] for g in got]) for k in range(4))
