"""The stream a graph is captured on belongs to that graph alone."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_capture_stream_is_not_a_pool_stream(cuda, pkg):
    pool = {torch.cuda.Stream().cuda_stream for _ in range(64)}
    graphs = [pkg.Graph() for _ in range(33)]
    own = [g.stream.cuda_stream for g in graphs]
    assert len(set(own)) == len(own) and not pool & set(own)
    for g in graphs:
        g.close()


def test_failed_begin_leaves_the_current_stream(cuda, pkg, monkeypatch):
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
