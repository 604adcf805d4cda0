"""Thread mappings of the reference-arithmetic kernels: two nodes per thread
in FP32, and planes numbered through their rows.

The two-node forms of the fused BGK / TRT steps run the one-node kernel's
scalar arithmetic, so they are compared bit for bit with the one-node kernel,
which the same call takes when a buffer starts 4 bytes off an 8-byte boundary.
The two-node natural-convection step runs packed lanes (Lanes2), whose
multiply-adds may round once where the scalar form rounds twice.  A population
collects the products of its equilibrium, its source and its relaxation: at
most 12 of them, each off by at most half an ulp of the population and scaled
by the relaxation rate (1.31 at most), 8 ulp together."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

W9 = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
W19 = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


def _pop(W, shape, dev, seed, base=1.0):
    rng = np.random.default_rng(seed)
    w = W.reshape((-1,) + (1,) * len(shape))
    return torch.from_numpy((base * w * (1 + 0.05 * rng.standard_normal((len(W),) + shape))
                             ).astype(np.float32)).to(dev)


def _off(t):
    """The same tensor one element past an 8-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    v = buf[1:].view(t.shape)
    v.copy_(t)
    assert v.data_ptr() % 8 == 4
    return v


def _mask(shape, dev, seed):
    return torch.from_numpy(np.random.default_rng(seed).random(shape) < 0.2).to(dev)


# one pair, a row inside and past one block of 128 pairs, odd row counts
SIZES2 = [(2, 1), (2, 3), (16, 13), (130, 9), (256, 3), (258, 5)]


@pytest.mark.parametrize("size", SIZES2)
@pytest.mark.parametrize("with_mask", [False, True])
def test_fused_2d_pairs_equal_one_node(cuda, pkg, size, with_mask):
    Nx, Ny = size
    fi = _pop(W9, (Ny, Nx), cuda, 1)
    m = _mask((Ny, Nx), cuda, 2) if with_mask else None
    for step in (lambda o, i, mo: pkg.fused_bgk_step_(o, i, *mo, m, Nx, Ny, 1.3),
                 lambda o, i, mo: pkg.fused_trt_step_(o, i, *mo, m, Nx, Ny, 0.07)):
        a, ma = torch.empty_like(fi), [torch.empty((Ny, Nx), device=cuda) for _ in range(3)]
        b, mb = torch.empty_like(fi), [torch.empty((Ny, Nx), device=cuda) for _ in range(3)]
        step(a, fi, ma)
        step(b, _off(fi), mb)
        assert torch.equal(a, b)
        assert all(torch.equal(x, y) for x, y in zip(ma, mb))


@pytest.mark.parametrize("size", [(2, 1, 1), (2, 3, 2), (16, 5, 6), (34, 9, 4), (256, 3, 2), (258, 2, 3)])
@pytest.mark.parametrize("periodic", range(8))
def test_fused_trt_3d_pairs_equal_one_node(cuda, pkg, size, periodic):
    Nx, Ny, Nz = size
    shape = (Nz, Ny, Nx)
    fi = _pop(W19, shape, cuda, 3)
    m = _mask(shape, cuda, 4) if periodic & 1 else None
    out = []
    for src in (fi, _off(fi)):
        o, mo = torch.empty_like(fi), [torch.empty(shape, device=cuda) for _ in range(4)]
        pkg.fused_trt_step_3d_(o, src, *mo, m, Nx, Ny, Nz, 0.07, 0.25, periodic=periodic)
        out.append([o] + mo)
    assert all(torch.equal(x, y) for x, y in zip(*out))


@pytest.mark.parametrize("size", [(24, 20, 18), (130, 20, 18)])
@pytest.mark.parametrize("periodic", [0, 7])
def test_cut_link_pairs_equal_one_node(cuda, pkg, size, periodic):
    """Pairs with a cut, a solid or two such nodes around a sphere."""
    Nx, Ny, Nz = size
    shape = (Nz, Ny, Nx)
    qw, solid = pkg.libb.precompute_q_wall_sphere_3d_torch(Nx, Ny, Nz, Nx / 2 - 0.3, 9.6, 8.2, 5.3,
                                                           dtype=torch.float32)
    rng = np.random.default_rng(5)
    uw = [torch.from_numpy((1e-3 * rng.standard_normal(qw.shape)).astype(np.float32)).to(cuda)
          for _ in range(3)]
    links = pkg.libb.CutLinks(solid, qw, *uw)
    fi = _pop(W19, shape, cuda, 6)
    out = []
    for src in (fi, _off(fi)):
        o, mo = torch.empty_like(fi), [torch.empty(shape, device=cuda) for _ in range(4)]
        pkg.fused_trt_libb_links_step_3d_(o, src, *mo, links, 0.05, periodic=periodic)
        out.append([o] + mo)
    assert all(torch.equal(x, y) for x, y in zip(*out))
    links.close()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_cut_links_without_planes_left(cuda, pkg, dtype):
    """At 65535 planes the launch has none left for the cut nodes, so the link
    code runs at every node; the dense arrays' step gives the same bits."""
    Nx, Ny, Nz = 4, 3, 65535
    shape = (Nz, Ny, Nx)
    gen = torch.Generator(device=cuda).manual_seed(9)
    rand = lambda *s: torch.rand(s, generator=gen, dtype=dtype, device=cuda)
    w = torch.from_numpy(W19).to(cuda, dtype).view(19, 1, 1, 1)
    fi = w * (1 + 0.1 * (rand(19, *shape) - 0.5))
    qw = rand(19, *shape)
    qw[rand(19, *shape) < 0.9] = 0
    qw[0] = 0
    uw = [0.02 * (rand(19, *shape) - 0.5) for _ in range(3)]
    solid = (rand(*shape) < 0.15).to(torch.uint8)
    links = pkg.libb.CutLinks(solid, qw, *uw)
    a, b = torch.empty_like(fi), torch.empty_like(fi)
    ma, mb = ([torch.empty(shape, dtype=dtype, device=cuda) for _ in range(4)] for _ in range(2))
    pkg.fused_trt_libb_links_step_3d_(a, fi, *ma, links, 0.05, periodic=7)
    pkg.fused_trt_libb_v2_step_3d_(b, fi, *mb, solid, qw, *uw, Nx, Ny, Nz, 0.05,
                                   periodic=(True, True, True))
    assert torch.equal(a, b) and all(torch.equal(x, y) for x, y in zip(ma, mb))
    links.close()


@pytest.mark.parametrize("size", [(2, 2), (2, 3), (16, 13), (130, 9), (256, 3), (258, 5)])
@pytest.mark.parametrize("vt", [False, True])
def test_natconv_pairs_match_one_node(cuda, pkg, size, vt):
    Nx, Ny = size
    fi, gi = _pop(W9, (Ny, Nx), cuda, 7), _pop(W9, (Ny, Nx), cuda, 8, 0.6)
    out = []
    for f, g in ((fi, gi), (_off(fi), gi)):
        fo, go, T = torch.empty_like(fi), torch.empty_like(gi), torch.empty((Ny, Nx), device=cuda)
        if vt:
            pkg.fused_natconv_vt_step_(fo, f, go, g, T, Nx, Ny, 0.05, 0.0, -0.7, 1.31, 3e-3, 0.5, 0.9, 0.1)
        else:
            pkg.fused_natconv_step_(fo, f, go, g, T, Nx, Ny, 1.21, 1.31, 3e-3, 0.5, 0.9, 0.1)
        out.append([x.cpu().numpy() for x in (fo, go, T)])
    for a, b in zip(*out):
        assert np.all(np.abs(a - b) <= 8 * np.spacing(np.maximum(np.abs(a), np.abs(b))))


@pytest.mark.parametrize("Nx,Ny", [(1, 1), (1, 300), (3, 200), (127, 5), (128, 5), (129, 5), (1000, 3),
                                   (65537, 2), (7, 65535)])
def test_row_numbering_covers_the_plane(cuda, pkg, Nx, Ny):
    """Every node is visited, with its own (i, j): a periodic stream against
    rolled copies, in FP64 (one node per thread)."""
    f = torch.rand((9, Ny, Nx), dtype=torch.float64, device=cuda)
    out = torch.full_like(f, -1.0)
    pkg.stream_fully_periodic_2d_(out, f, Nx, Ny)
    cx, cy = (0, 1, 0, -1, 0, 1, -1, -1, 1), (0, 0, 1, 0, -1, 1, 1, -1, -1)
    for q in range(9):
        assert torch.equal(out[q], torch.roll(f[q], (cy[q], cx[q]), (0, 1))), q
