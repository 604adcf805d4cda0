"""The one-launch driver steps (cavity 3D, Rayleigh-Benard 2D, natural
convection 3D) against the separate kernels they replace.

FP64 is bit-identical.  FP32 on odd Nx is bit-identical too (the separate
forced BGK then takes one node per thread, the same expressions); on even Nx
the separate forced BGK runs two packed lanes, which differ by at most 3 ulp
per population (the bound of the two-lane kernels), so 4 ulp is asked there."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

W9 = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
W19 = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
# 1 x 1, rows shorter and longer than a block (128), walls that share a node
SIZES2 = [(1, 1), (2, 3), (17, 13), (128, 5), (130, 9), (257, 4)]
SIZES3 = [(1, 1, 1), (3, 2, 5), (17, 5, 6), (34, 9, 4), (129, 3, 2)]


def _pop(W, shape, dtype, dev, seed, base=1.0):
    rng = np.random.default_rng(seed)
    w = W.reshape((-1,) + (1,) * len(shape))
    return torch.from_numpy(base * w * (1 + 0.05 * rng.standard_normal((len(W),) + shape))).to(dev, dtype)


def _check(a, b, packed):
    torch.cuda.synchronize()
    a, b = a.cpu().numpy(), b.cpu().numpy()
    if not packed:
        assert np.array_equal(a, b)
    else:
        assert np.all(np.abs(a - b) <= 4 * np.spacing(np.maximum(np.abs(a), np.abs(b))))


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("size", SIZES3)
@pytest.mark.parametrize("with_mask", [False, True])
def test_cavity_step_3d_equals_separate_kernels(cuda, pkg, dtype, size, with_mask):
    Nx, Ny, Nz = size
    shape = (Nz, Ny, Nx)
    fi = _pop(W19, shape, dtype, cuda, 1)
    m = None
    if with_mask:
        m = torch.from_numpy(np.random.default_rng(2).random(shape) < 0.2).to(cuda)
    ref = torch.empty_like(fi)
    pkg.stream_3d_(ref, fi, Nx, Ny, Nz)
    pkg.apply_zou_he_top_3d_(ref, 0.07, Nx, Ny, Nz)
    pkg.collide_3d_(ref, m, 1.3)
    mr = [torch.empty(shape, dtype=dtype, device=cuda) for _ in range(4)]
    pkg.compute_macroscopic_3d_(*mr, ref)
    out = torch.empty_like(fi)
    mo = [torch.empty(shape, dtype=dtype, device=cuda) for _ in range(4)]
    pkg.cavity_step_3d_(out, fi, *mo, m, Nx, Ny, Nz, 1.3, 0.07)
    _check(out, ref, False)
    for a, b in zip(mo, mr):
        _check(a, b, False)
    out2 = torch.empty_like(fi)
    pkg.cavity_step_3d_(out2, fi, None, None, None, None, m, Nx, Ny, Nz, 1.3, 0.07)
    _check(out2, ref, False)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("size", SIZES2)
@pytest.mark.parametrize("vertical", [True, False])
def test_rayleigh_step_equals_separate_kernels(cuda, pkg, dtype, size, vertical):
    Nx, Ny = size
    shape = (Ny, Nx)
    fi, gi = _pop(W9, shape, dtype, cuda, 3), _pop(W9, shape, dtype, cuda, 4, 0.6)
    fr, gr = torch.empty_like(fi), torch.empty_like(gi)
    T, rho, ux, uy = (torch.empty(shape, dtype=dtype, device=cuda) for _ in range(4))
    stream = pkg.stream_periodic_x_wall_y_2d_ if vertical else pkg.stream_2d_
    stream(fr, fi, Nx, Ny)
    stream(gr, gi, Nx, Ny)
    if vertical:
        pkg.apply_fixed_temp_south_2d_(gr, 0.9, Nx)
        pkg.apply_fixed_temp_north_2d_(gr, 0.1, Nx, Ny)
    else:
        pkg.apply_fixed_temp_west_2d_(gr, 0.9, Ny)
        pkg.apply_fixed_temp_east_2d_(gr, 0.1, Nx, Ny)
    pkg.compute_temperature_2d_(T, gr)
    pkg.compute_macroscopic_2d_(rho, ux, uy, fr)
    pkg.collide_thermal_2d_(gr, ux, uy, 1.31)
    pkg.collide_boussinesq_2d_(fr, T, None, 1.21, 3e-3, 0.5)
    fo, go = torch.empty_like(fi), torch.empty_like(gi)
    pkg.rayleigh_step_2d_(fo, fi, go, gi, Nx, Ny, 1.21, 1.31, 3e-3, 0.5, 0.9, 0.1, vertical)
    _check(go, gr, False)
    _check(fo, fr, dtype == torch.float32 and Nx % 2 == 0)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("size", SIZES3)
def test_natconv_step_3d_equals_separate_kernels(cuda, pkg, dtype, size):
    Nx, Ny, Nz = size
    shape = (Nz, Ny, Nx)
    fi, gi = _pop(W19, shape, dtype, cuda, 5), _pop(W19, shape, dtype, cuda, 6, 0.6)
    fr, gr = torch.empty_like(fi), torch.empty_like(gi)
    T, rho, ux, uy, uz = (torch.empty(shape, dtype=dtype, device=cuda) for _ in range(5))
    pkg.stream_3d_(fr, fi, Nx, Ny, Nz)
    pkg.stream_3d_(gr, gi, Nx, Ny, Nz)
    pkg.apply_fixed_temp_west_3d_(gr, 0.9, Ny, Nz)
    pkg.apply_fixed_temp_east_3d_(gr, 0.1, Nx, Ny, Nz)
    pkg.compute_temperature_3d_(T, gr)
    pkg.compute_macroscopic_3d_(rho, ux, uy, uz, fr)
    pkg.collide_thermal_3d_(gr, ux, uy, uz, 1.31)
    pkg.collide_boussinesq_3d_(fr, T, None, 1.21, 3e-3, 0.5)
    fo, go = torch.empty_like(fi), torch.empty_like(gi)
    pkg.natconv_step_3d_(fo, fi, go, gi, Nx, Ny, Nz, 1.21, 1.31, 3e-3, 0.5, 0.9, 0.1)
    _check(go, gr, False)
    _check(fo, fr, dtype == torch.float32 and Nx % 2 == 0)


def test_fused_steps_refuse_bad_arguments(cuda, pkg):
    f = torch.zeros((19, 2, 3, 4), device=cuda)
    g2 = torch.zeros((9, 3, 4), device=cuda)
    with pytest.raises(pkg.KrakenArgumentError):
        pkg.cavity_step_3d_(f, f, None, None, None, None, None, 4, 3, 2, 1.0, 0.1)
    with pytest.raises(pkg.KrakenArgumentError):
        pkg.cavity_step_3d_(f.double(), f, None, None, None, None, None, 4, 3, 2, 1.0, 0.1)
    with pytest.raises(pkg.KrakenArgumentError):
        pkg.natconv_step_3d_(f, f.clone(), f, f.clone(), 4, 3, 2, 1.0, 1.0, 0.0, 0.5, 1.0, 0.0)
    with pytest.raises(pkg.KrakenArgumentError):
        pkg.rayleigh_step_2d_(g2.half(), g2, g2.clone(), g2.clone(), 4, 3, 1.0, 1.0, 0.0, 0.5, 1.0,
                              0.0, True)
