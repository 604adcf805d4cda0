"""Cavity runs in one launch against the same number of step calls.

Both use the same node functions without contraction, so both buffers (the
last two states) and the moments agree bit for bit; the sizes cover one
column, one row, partial tiles in x and y and several tiles each way."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 9), (9, 1), (2, 3), (63, 5), (64, 2), (65, 4), (128, 8), (130, 65), (200, 130)]


def _ws(pkg, moving, Nx, Ny, T):
    n = pkg.ops.cavity_run_bytes_2d(Nx, Ny, moving, T)
    assert n > 0
    return torch.full(((n + 3) // 4,), -1, dtype=torch.int32, device="cuda")


def _pops(Nx, Ny, T, seed, scale=0.05):
    gen = torch.Generator().manual_seed(seed)
    w = torch.tensor([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4, dtype=torch.float64)
    f = w[:, None, None] * (1 + scale * (torch.rand((9, Ny, Nx), generator=gen, dtype=torch.float64) - 0.5))
    return f.to(T).cuda()


@pytest.mark.parametrize("T", [torch.float64, torch.float32])
@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("solid", [False, True])
@pytest.mark.parametrize("Nx,Ny", SIZES)
def test_cavity_run_matches_steps(cuda, pkg, Nx, Ny, solid, moving, T):
    mask = None
    if solid:
        mask = torch.zeros((Ny, Nx), dtype=torch.bool, device="cuda")
        mask[Ny // 2:Ny // 2 + 2, Nx // 3:Nx // 2 + 1] = True
    step = pkg.ops.cavity_movingwall_step_2d_ if moving else pkg.ops.cavity_step_2d_
    for n in (1, 2, 7, 40):
        a = [_pops(Nx, Ny, T, 1), _pops(Nx, Ny, T, 2)]
        b = [t.clone() for t in a]
        ma = [torch.zeros((Ny, Nx), dtype=T, device="cuda") for _ in range(3)]
        mb = [t.clone() for t in ma]
        for s in range(n):
            step(a[1 - (s & 1)], a[s & 1], *ma, mask, Nx, Ny, 1.3, 0.08)
        ws = _ws(pkg, moving, Nx, Ny, T)
        pkg.ops.cavity_run_2d_(b[0], b[1], *mb, mask, Nx, Ny, 1.3, 0.08, moving, n, ws)
        assert int(ws[0]) == 0
        for x, y in zip(a + ma, b + mb):
            assert torch.equal(x, y)


def test_grids_that_do_not_fit_are_refused(cuda, pkg):
    assert pkg.ops.cavity_run_bytes_2d(4096, 4096, False, torch.float64) == 0
    f = [torch.ones((9, 2048, 2048), dtype=torch.float32, device="cuda") for _ in range(2)]
    m = [torch.ones((2048, 2048), dtype=torch.float32, device="cuda") for _ in range(3)]
    ws = torch.zeros(1024, dtype=torch.int32, device="cuda")
    with pytest.raises(pkg.KrakenArgumentError):
        pkg.ops.cavity_run_2d_(*f, *m, None, 2048, 2048, 1.0, 0.1, False, 4, ws)
    small = [t[:, :8, :8].contiguous() for t in f]
    sm = [t[:8, :8].contiguous() for t in m]
    with pytest.raises(pkg.KrakenArgumentError):  # workspace too small
        pkg.ops.cavity_run_2d_(*small, *sm, None, 8, 8, 1.0, 0.1, False, 4, ws[:16])


def test_a_wait_that_gives_up_is_reported(cuda, pkg, monkeypatch):
    """Blocks whose first missed poll gives up set the flag and end the launch,
    and the context stays usable; the driver raises on the flag."""
    import ctypes as C
    from importlib import import_module
    lib = import_module(pkg.__name__ + "._lib")
    drivers = import_module(pkg.__name__ + ".drivers")
    flag = C.c_int(-1)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    lib.call("kb_selftest_cavity_run", C.c_longlong(1 << 21), C.byref(flag), stream)
    assert flag.value == 0
    with pytest.raises(lib.KrakenError) as e:
        lib.call("kb_selftest_cavity_run", C.c_longlong(-1), C.byref(flag), stream)
    assert e.value.code == lib.KB_ERR_TIMEOUT and flag.value == 1
    for bad in (-2, (1 << 21) + 1):
        with pytest.raises(lib.KrakenArgumentError):
            lib.call("kb_selftest_cavity_run", C.c_longlong(bad), C.byref(flag), stream)

    cfg = pkg.LBMConfig.d2q9(70, 6, 0.05, 0.1, 40)
    want = pkg.run_cavity_2d(cfg)
    run = drivers.ops.cavity_run_2d_

    def gave_up(*a):
        run(*a)
        a[-1][0] = 1

    with monkeypatch.context() as m:
        m.setattr(drivers.ops, "cavity_run_2d_", gave_up)
        with pytest.raises(RuntimeError, match="gave up"):
            pkg.run_cavity_2d(cfg)
    assert (pkg.run_cavity_2d(cfg)["ux"] == want["ux"]).all()
