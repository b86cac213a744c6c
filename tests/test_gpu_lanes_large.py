"""The passes at the row counts above which large clouds take fewer lanes per row
(3-D: two above 196,608; 2-D: one above 524,288), against the oracle on the first
layers of the cloud: a row sees four supports at most (density, its gradient,
diffusion, force), so the oracle takes the layers within that of the compared
ones.  Tolerances are those of the smaller sizes."""
import numpy as np
import pytest
import torch

from oracle import pairpass as op
from oracle.neighbors import cell_linked_pairs_batched
from tests.test_gpu_lanes import close

pytestmark = pytest.mark.gpu

DX, H = 0.01, 0.013
RINGS = 11                                  # layers in four supports of 2.6 dx


def layers(dim, n, side, keep, dtype, gpu):
    """A jittered block of n particles, layer after layer along x: the device's arrays, the
    oracle's part in 64 bits (``keep`` layers and four supports), and the rows compared."""
    g = np.stack(np.meshgrid(*[np.arange(side)] * dim, indexing="ij"), -1).reshape(-1, dim)[:n]
    assert g.shape[0] == n
    rng = np.random.default_rng(n)
    x = torch.from_numpy((g + 0.5 + 0.05 * rng.uniform(-1, 1, g.shape)) * DX).to(gpu, dtype)
    v = torch.from_numpy(rng.normal(0, 0.1, g.shape)).to(gpu, dtype)
    part = (keep + RINGS) * side ** (dim - 1)
    d = [t[:part].double().cpu().numpy() for t in (x, v)]
    return x, v, d, part, keep * side ** (dim - 1)


SIZES3 = [196608, 196609]
DTYPES = [(torch.float64, 1e-12), (torch.float32, 2e-6)]


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("n", [524288, 524289])
def test_rhs_2d(gpu, dtype, tol, n):
    from tensorsph_b200.dam_break import DamBreakConfig
    from tensorsph_b200.droplet_impact import lattice_mass_unit, rhs
    cfg = DamBreakConfig(dx=DX, density_diffusion=0.1, sound_speed=20.0, dt=1e-4, viscosity=1e-3)
    x, v, d, part, rows = layers(2, n, 725, 20, dtype, gpu)
    m = torch.full((n,), lattice_mass_unit(cfg), device=gpu, dtype=dtype)
    saved = torch.get_default_dtype()
    torch.set_default_dtype(torch.float64)
    try:
        got = rhs(x, v, m, cfg)
    finally:
        torch.set_default_dtype(saved)
    want = op.rhs(*d, m[:part].double().cpu().numpy(), cfg, pairs=cell_linked_pairs_batched(d[0], 2.0 * H))
    for k, (scale, t) in enumerate(((cfg.rho0, tol), (cfg.rho0 * cfg.sound_speed ** 2 / cfg.gamma, 20 * tol),
                                    (np.abs(want[2][:rows]).max(), 100 * tol))):
        close(got[k][:rows], want[k][:rows], scale, t)


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("n", SIZES3)
def test_rhs_3d(gpu, dtype, tol, n):
    from tensorsph_b200.dam_break_3d import DamBreak3DConfig, mass_3d, rhs_3d
    cfg = DamBreak3DConfig(dx=DX, density_diffusion=0.1, sound_speed=20.0, dt=1e-4, viscosity=1e-3)
    x, v, d, part, rows = layers(3, n, 59, 4, dtype, gpu)
    m = torch.full((n,), mass_3d(cfg.dx, cfg.h_factor, cfg.rho0, True), device=gpu, dtype=dtype)
    got = rhs_3d(x, v, m, cfg)
    want = op.rhs_3d(*d, m[:part].double().cpu().numpy(), cfg, pairs=cell_linked_pairs_batched(d[0], 2.0 * H))
    for k, (scale, t) in enumerate(((cfg.rho0, tol), (cfg.rho0 * cfg.sound_speed ** 2 / cfg.gamma, 20 * tol),
                                    (np.abs(want[2][:rows]).max(), 100 * tol))):
        close(got[k][:rows], want[k][:rows], scale, t)


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-11), (torch.float32, 2e-4)])
@pytest.mark.parametrize("n", SIZES3)
def test_operators_3d(gpu, dtype, tol, n):
    """accelerations (psi diffusion, second-order viscosity) and csf_fields3."""
    from oracle import csf3 as oc
    from tensorsph_b200.neighbor_search import cell_linked_pairs
    from tensorsph_b200.threed import accelerations
    from tensorsph_b200.threed.csf3 import csf_fields3
    x, v, d, part, rows = layers(3, n, 59, 4, dtype, gpu)
    m = torch.full((n,), 1000.0 * DX ** 3, device=gpu, dtype=dtype)
    dm = m[:part].double().cpu().numpy()
    p, q = cell_linked_pairs(x, 2.0 * H), cell_linked_pairs_batched(d[0], 2.0 * H)
    kw = dict(rho0=1000.0, sound_speed=1.0, viscosity=1e-2, density_diffusion=0.1, dt=1e-4,
              gravity=(0.0, -9.81, 0.0))
    got = accelerations(x, v, m, H, p, **kw)
    want = op.accelerations(*d, dm, H, q, **kw)
    close(got[0][:rows], want[0][:rows], np.abs(want[0][:rows]).max(), 10 * tol)
    close(got[1][:rows], want[1][:rows], 1000.0, tol)
    close(got[2][:rows], want[2][:rows], 1000.0, 10 * tol)
    got = csf_fields3(x, m, H, p, rho0=1000.0)
    want = oc.csf_fields3(d[0], dm, H, q, rho0=1000.0)
    for name in ("color", "grad_c", "delta_s"):
        close(getattr(got, name)[:rows], want[name][:rows], max(np.abs(want[name][:rows]).max(), 1.0), tol)
    if dtype == torch.float64:
        close(got.kappa[:rows], want["kappa"][:rows], np.abs(want["kappa"][:rows]).max(), 1e-8)


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 2e-5)])
@pytest.mark.parametrize("dim,n,side", [(2, 524288, 725), (2, 524289, 725), (3, 196608, 59), (3, 196609, 59)])
def test_transport_velocity(gpu, dtype, tol, dim, n, side):
    from oracle import tvc as ot
    from tensorsph_b200.neighbor_search import cell_linked_pairs
    from tensorsph_b200.transport_velocity_correction import kernel_gradient_integral
    x, _, d, part, rows = layers(dim, n, side, 6, dtype, gpu)
    vol = torch.full((n,), DX ** dim, device=gpu, dtype=dtype)
    got = kernel_gradient_integral(x, vol, H, pairs=cell_linked_pairs(x, 2.0 * H))
    want = ot.kernel_gradient_integral(d[0], vol[:part].double().cpu().numpy(), H,
                                       cell_linked_pairs_batched(d[0], 2.0 * H))
    close(got[:rows], want[:rows], np.abs(want[:rows]).max(), tol)
