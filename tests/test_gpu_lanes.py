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


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-11), (torch.float32, 2e-4)])
@pytest.mark.parametrize("n", [49152, 49153])
def test_periodic_operators(gpu, dtype, tol, n):
    """accelerations (psi diffusion, order 4, images on every axis) and csf_fields3 on a
    jittered block with a free face in a periodic box."""
    from oracle import csf3 as oc
    from oracle.neighbors import periodic_pairs
    from tensorsph_b200.threed import accelerations
    from tensorsph_b200.threed.csf3 import csf_fields3
    side, dx = 37, 1.0 / 37
    h = 1.3 * dx
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    rng = np.random.default_rng(n)
    x = ((g + 0.1 * rng.uniform(-1, 1, g.shape)) * dx) % 1.0
    v = rng.normal(0, 1e-3, x.shape)
    m = np.full(n, 1000.0 * dx ** 3)
    t = [torch.from_numpy(a).to(gpu, dtype) for a in (x, v, m)]
    d = [a.double().cpu().numpy() for a in t]
    pairs = periodic_pairs(d[0], [1.0] * 3, 2.0 * h)
    kw = dict(rho0=1000.0, sound_speed=1.0, viscosity=1e-2, viscous_order=4, density_diffusion=0.1, dt=1e-4,
              gravity=(0.0, -9.81, 0.0))
    p = torch.from_numpy(pairs).to(gpu)
    got = accelerations(*t, h, p, box=[1.0] * 3, **kw)
    want = op.accelerations(*d, h, pairs, box=[1.0] * 3, **kw)
    close(got[0], want[0], np.abs(want[0]).max(), 10 * tol)
    close(got[1], want[1], 1000.0, tol)
    close(got[2], want[2], 1000.0, 10 * tol)
    got = csf_fields3(t[0], t[2], h, p, rho0=1000.0, box=[1.0] * 3)
    want = oc.csf_fields3(d[0], d[2], h, pairs, rho0=1000.0, box=[1.0] * 3)
    for name in ("color", "grad_c", "delta_s"):
        close(getattr(got, name), want[name], max(np.abs(want[name]).max(), 1.0), tol)
    if dtype == torch.float64:
        close(got.kappa, want["kappa"], np.abs(want["kappa"]).max(), 1e-8)


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 2e-5)])
@pytest.mark.parametrize("dim,n", [(1, 2000), (2, 49152), (2, 49153), (3, 49152), (3, 49153)])
def test_tvc_lanes(gpu, dtype, tol, dim, n):
    from oracle import tvc as ot
    from tensorsph_b200.transport_velocity_correction import kernel_gradient_integral
    side = int(np.ceil(n ** (1.0 / dim)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * dim, indexing="ij"), -1).reshape(-1, dim)[:n]
    rng = np.random.default_rng(n + dim)
    x = (g + 0.1 * rng.uniform(-1, 1, g.shape)) * 0.01
    t = torch.from_numpy(x[rng.permutation(n)]).to(gpu, dtype)
    x = t.double().cpu().numpy()
    vol = np.full(n, 0.01 ** dim)
    pairs = cell_linked_pairs_batched(x, 0.026)
    got = kernel_gradient_integral(t, torch.from_numpy(vol).to(gpu, dtype), 0.013, wall_count=n // 10,
                                   pairs=torch.from_numpy(pairs).to(gpu))
    want = ot.kernel_gradient_integral(x, vol, 0.013, pairs, wall_count=n // 10)
    close(got, want, np.abs(want).max(), tol)


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 2e-5)])
@pytest.mark.parametrize("dim,copies", [(2, 1), (2, 300), (2, 3000), (3, 1), (3, 300)])
def test_short_rows(gpu, dtype, tol, dim, copies):
    """Rows of 0 to 18 entries at each lane count: clusters of 1 to 19 particles, out of reach
    of one another, all pairs of a cluster within the cutoff (the tail of a lane's part of a
    row: no entry, one, an odd number)."""
    from oracle import tvc as ot
    from tensorsph_b200.transport_velocity_correction import kernel_gradient_integral
    rng = np.random.default_rng(dim)
    size = np.tile(np.arange(1, 20), copies)
    n = int(size.sum())
    start = np.concatenate(([0], np.cumsum(size)))
    home = np.repeat(np.arange(size.size), size)
    x = rng.uniform(0.0, 0.9, (n, dim))
    x[:, 0] += 4.0 * (home % 64)
    x[:, 1] += 4.0 * (home // 64)
    pairs = np.concatenate([start[c] + np.stack(np.triu_indices(s, 1), -1) for c, s in enumerate(size)])
    t = torch.from_numpy(x).to(gpu, dtype)
    x, vol = t.double().cpu().numpy(), np.full(n, 0.5)
    got = kernel_gradient_integral(t, torch.from_numpy(vol).to(gpu, dtype), 1.0,
                                   pairs=torch.from_numpy(pairs).to(gpu))
    want = ot.kernel_gradient_integral(x, vol, 1.0, pairs)
    close(got, want, np.abs(want).max(), tol)


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 2e-5)])
@pytest.mark.parametrize("dim,options", [(1, False), (2, True), (3, False), (3, True)])
def test_tvc_without_records(gpu, monkeypatch, dtype, tol, dim, options):
    """Without memory for the packed records the sums come from the caller's arrays."""
    from oracle import tvc as ot
    from tensorsph_b200 import _lib
    from tensorsph_b200.transport_velocity_correction import kernel_gradient_integral
    n = 1331
    rng = np.random.default_rng(dim)
    side = int(np.ceil(n ** (1.0 / dim)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * dim, indexing="ij"), -1).reshape(-1, dim)[:n]
    t = torch.from_numpy(((g + 0.1 * rng.uniform(-1, 1, g.shape)) * 0.01)[rng.permutation(n)]).to(gpu, dtype)
    vol = torch.from_numpy(0.01 ** dim * rng.uniform(0.5, 2.0, n)).to(gpu, dtype)
    kw = dict(wall_count=100) if options else {}
    corr = torch.from_numpy(rng.uniform(0.9, 1.1, n)).to(gpu, dtype) if options else None
    pairs = cell_linked_pairs_batched(t.double().cpu().numpy(), 0.026)
    plain, refused = _lib.workspace, []

    def tight(nbytes, device):
        if nbytes == n * 4 * t.element_size():
            refused.append(nbytes)
            raise torch.OutOfMemoryError("no room")
        return plain(nbytes, device)

    want = ot.kernel_gradient_integral(t.double().cpu().numpy(), vol.double().cpu().numpy(), 0.013, pairs,
                                       correction=None if corr is None else corr.double().cpu().numpy(), **kw)
    for route in (plain, tight):
        monkeypatch.setattr(_lib, "workspace", route)
        got = kernel_gradient_integral(t, vol, 0.013, pairs=torch.from_numpy(pairs).to(gpu), correction=corr, **kw)
        close(got, want, np.abs(want).max(), tol)
    assert refused
