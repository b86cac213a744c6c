"""The right-hand sides at the row counts where the lanes per row change, against
the oracle at the tolerances of the fixture tests (FP64 1e-12 of the density
scale; FP32 as in the small cases), and a particle on top of another."""
import numpy as np
import pytest
import torch

from oracle import pairpass as op
from oracle.neighbors import cell_linked_pairs_batched

pytestmark = pytest.mark.gpu


def close(got, want, scale, tol):
    assert float(np.abs(got.cpu().numpy().astype(np.float64) - want).max()) < tol * scale


def pruned(x, wall, cutoff):
    pairs = cell_linked_pairs_batched(np.concatenate((x, wall)), cutoff)
    return pairs[pairs[:, 0] < x.shape[0]]


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 2e-6)])
@pytest.mark.parametrize("n", [49151, 49152, 49153])
def test_rhs_lanes_2d(gpu, dtype, tol, n):
    from tensorsph_b200.dam_break import DamBreakConfig
    from tensorsph_b200.droplet_impact import lattice_mass_unit, rhs
    side = 222
    cfg = DamBreakConfig(dx=0.01, density_diffusion=0.1, sound_speed=20.0, dt=1e-4, viscosity=1e-3)
    g = np.stack(np.meshgrid(np.arange(side), np.arange(side), indexing="ij"), -1).reshape(-1, 2)[:n]
    rng = np.random.default_rng(n)
    x = ((g + 0.5 + 0.05 * rng.uniform(-1, 1, g.shape)) * cfg.dx)
    x[7] = x[6]
    v = rng.normal(0, 0.1, x.shape)
    wall = (np.stack(np.meshgrid(np.arange(side), np.arange(3), indexing="ij"), -1).reshape(-1, 2)
            + [0.5, -2.5]) * cfg.dx
    t = [torch.from_numpy(a).to(gpu, dtype) for a in (x, v, np.full(n, lattice_mass_unit(cfg)), wall)]
    h = cfg.h_factor * cfg.dx
    pairs = pruned(x, wall, 2.0 * h)
    saved = torch.get_default_dtype()
    torch.set_default_dtype(torch.float64)
    try:
        got = rhs(t[0], t[1], t[2], cfg, pairs=torch.from_numpy(pairs).to(gpu), wall=t[3])
    finally:
        torch.set_default_dtype(saved)
    want = op.rhs(*[a.double().cpu().numpy() for a in t[:3]], cfg, pairs=pairs, wall=t[3].double().cpu().numpy())
    bulk = cfg.rho0 * cfg.sound_speed ** 2 / cfg.gamma
    close(got[0], want[0], cfg.rho0, tol)
    close(got[1], want[1], bulk, 20 * tol)          # Tait: gamma (rho / rho0)^gamma times the density's
    close(got[2], want[2], np.abs(want[2]).max(), 100 * tol)


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 2e-6)])
@pytest.mark.parametrize("n", [49152, 49153])
def test_rhs_lanes_3d(gpu, dtype, tol, n):
    from tensorsph_b200.dam_break_3d import DamBreak3DConfig, mass_3d, rhs_3d
    side = 37
    cfg = DamBreak3DConfig(dx=0.01, density_diffusion=0.1, sound_speed=20.0, dt=1e-4, viscosity=1e-3)
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    rng = np.random.default_rng(n)
    x = ((g + 0.5 + 0.05 * rng.uniform(-1, 1, g.shape)) * cfg.dx)
    v = rng.normal(0, 0.1, x.shape)
    wall = (np.stack(np.meshgrid(np.arange(side), np.arange(3), np.arange(side), indexing="ij"), -1).reshape(-1, 3)
            + [0.5, -2.5, 0.5]) * cfg.dx
    m = np.full(n, mass_3d(cfg.dx, cfg.h_factor, cfg.rho0, True))
    t = [torch.from_numpy(a).to(gpu, dtype) for a in (x, v, m, wall)]
    h = cfg.h_factor * cfg.dx
    got = rhs_3d(*t[:3], cfg, wall=t[3], return_wall_force=True)
    d = [a.double().cpu().numpy() for a in t]
    want = op.rhs_3d(*d[:3], cfg, pairs=pruned(d[0], d[3], 2.0 * h), wall=d[3], return_wall_force=True)
    bulk = cfg.rho0 * cfg.sound_speed ** 2 / cfg.gamma
    close(got[0], want[0], cfg.rho0, tol)
    close(got[1], want[1], bulk, 20 * tol)
    close(got[2], want[2], np.abs(want[2]).max(), 100 * tol)
    close(got[3], want[3], np.abs(want[3]).max(), 100 * tol)
