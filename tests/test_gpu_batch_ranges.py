"""The batch's default schedule (each block one run of the tile list, taken a
case at a time) and its collision (multiplied out, two nodes per thread on
even N, one on odd N)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,tol", [("f16", 5e-3), ("f32", 1e-5)])
def test_default_schedule_equals_explicit_tiles(cuda, pkg, storage, tol):
    """The schedule only changes which block updates which nodes.  Sizes: less
    than one tile, odd N, cases that split between blocks; one case converges
    and leaves the list half-way."""
    N = np.array([2, 8, 33, 64, 97, 160, 72, 320], np.int32)
    nu = np.array([0.5, 0.5, 0.05, 0.04, 0.02, 0.1, 0.03, 0.2])
    u = np.full(len(N), 0.05)
    out = []
    for tn in (0, 256, 1024):
        b = pkg.CavityBatch(N, nu, u, storage)
        b.run(max_steps=300, check_every=50, tol=tol, tile_nodes=tn)
        st = b.status()
        assert not st["timed_out"]
        out.append(([b.case(c) for c in range(len(N))], st["updates"]))
        b.close()
    assert any(r["steps"] < 300 for r in out[0][0])
    for other, updates in out[1:]:
        assert updates == out[0][1]
        for a, c in zip(out[0][0], other):
            assert a["steps"] == c["steps"] and a["state"] == c["state"]
            assert np.array_equal(a["ux"], c["ux"]) and np.array_equal(a["uy"], c["uy"])


@pytest.mark.parametrize("N", [32, 33])
def test_sweep_mass_does_not_drift(cuda, pkg, N):
    """Rest population from conservation: the mass of an FP32 cavity stays at
    rest's to the rounding of the stores.  10 000 steps of N^2 nodes round 9
    deviations of at most 0.1 w_q each to 2^-24: a random walk of 3e-9 per
    node and 1e-4 steps^-1/2 (measured: 5e-9 and 1.5e-8); 1e-7 per node bounds
    it with room, while a coefficient error of half an ulp per step would reach
    1e-5."""
    import ctypes as C
    import torch
    b = pkg.CavityBatch(np.array([N], np.int32), np.array([0.05]), np.array([0.1]), "f32")
    b.run(max_steps=10000, check_every=5000, tol=1e-12)
    ptr, dt = C.c_void_p(), C.c_int()
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    pkg._lib.call("kb_batch_populations", b._h, 0, C.byref(ptr), C.byref(dt), s)
    out = C.c_double()
    pkg._lib.call("kb_mass", ptr, 9, N * N, dt.value, C.byref(out), s)
    # the Zou-He lid exchanges mass with the wall: compare with the FP64 run
    st = pkg.initialize_2d(pkg.LBMConfig.d2q9(N, N, 0.05, 0.1))
    x, y = st["f_in"], st["f_out"]
    for _ in range(10000):
        pkg.cavity_mrt_step_2d_(y, x, None, None, None, None, N, N, 0.05, 0.1)
        x, y = y, x
    assert abs(out.value - pkg.ops.mass(x)) / (N * N) < 1e-7
    b.close()


def test_reported_schedules_can_be_asked_for(cuda, pkg):
    """A (tile_nodes, blocks_per_sm) pair names one schedule: the untuned one
    is 256-node tiles at the occupancy limit, so asking for that pair takes its
    time (dealing such tiles out one by one takes 1.7 times as long)."""
    import torch
    N, nu, u, _ = pkg.sweep_cases(48, seed=3)
    b = pkg.CavityBatch(N, nu, u, "f16")
    took = {}
    for tn in (0, 256, 0, 256):
        for _ in range(3):
            b.reset()
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            b.run(max_steps=200, check_every=100, tol=0.0, tile_nodes=tn)
            e[1].record()
            torch.cuda.synchronize()
            took[tn] = min(took.get(tn, 1e9), e[0].elapsed_time(e[1]))
    assert took[256] < 1.25 * took[0]
    b.close()
