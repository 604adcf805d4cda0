"""The stream a graph is captured on belongs to that graph alone."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_capture_stream_is_not_a_pool_stream(cuda, pkg):
    """More streams at once than are kept between captures; they go back and
    are taken again."""
    b = pkg.batch
    pool = {torch.cuda.Stream().cuda_stream for _ in range(64)}
    taken = [b._take_stream() for _ in range(b._IDLE_MOST + 3)]
    own = {s.cuda_stream for s in taken}
    assert len(own) == len(taken) and not pool & own
    for s in taken:
        b._give_back(s)
    assert len(b._idle) == b._IDLE_MOST
    g = pkg.Graph()
    with g:
        assert g.stream.cuda_stream in own
        assert torch.cuda.current_stream().cuda_stream == g.stream.cuda_stream
        assert len(b._idle) == b._IDLE_MOST - 1
    assert len(b._idle) == b._IDLE_MOST
    g.close()


def test_failed_begin_leaves_the_current_stream(cuda, pkg, monkeypatch):
    pkg.batch._give_back(pkg.batch._take_stream())
    g = pkg.Graph()
    before = torch.cuda.current_stream().cuda_stream

    def refuse(*a):
        raise RuntimeError("begin refused")

    with monkeypatch.context() as m:
        m.setattr(pkg.batch, "call", refuse)
        with pytest.raises(RuntimeError):
            with g:
                pass
    assert torch.cuda.current_stream().cuda_stream == before
    g.close()


def test_driver_runs_beside_another_threads_stream(cuda, pkg):
    """Captured driver runs in one thread, and work queued on a pool stream in
    another all the while: both come out as alone."""
    cfg = pkg.LBMConfig.d3q19(12, 9, 7, 0.05, 0.1, 40)
    want = pkg.run_cavity_3d(cfg)["ux"]
    done, sums = threading.Event(), []

    def other():
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            x = torch.zeros(1 << 12, device="cuda")
            n = 0
            while not done.is_set():
                x += 1
                n += 1
                if n % 64 == 0:
                    s.synchronize()
            sums.append((float(x.sum()), n))

    t = threading.Thread(target=other)
    t.start()
    try:
        for _ in range(70):
            assert (pkg.run_cavity_3d(cfg)["ux"] == want).all()
    finally:
        done.set()
        t.join()
    assert sums and sums[0][0] == sums[0][1] * float(1 << 12)
