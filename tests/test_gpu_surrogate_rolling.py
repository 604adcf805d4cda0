"""The kernels that roll down the rows of a pixel column (convolutions of
128-pixel row tiles, weight gradients of 64-pixel steps) and the reduction of
their partial sums, bit for bit.

Weights of -1, 0 and 1 with few entries per channel, small whole inputs and
biases, and a loss whose error is a whole number of one power of two make every
product a multiple of one quantum and every sum, of any order, at most 2^24 of
them: FP32 holds the sums exactly, so a kernel that drops, doubles or misplaces
one contribution anywhere is off and a correct one has no error.  The largest
sum of magnitudes over the shapes below is 0.9 x 2^24 quanta (a weight gradient).

A CTA takes a contiguous range of row tiles (592 CTAs where four share an SM),
so the shapes put its seams in the middle of a column, between the columns of an
image and between images: one-row ranges, ranges of one and two rows, ranges of
several rows; H != W; both concatenated inputs; 16 to 128 output channels (N of
an MMA from 48 to 256, one to four CTAs per SM, one and two output-gradient
blocks)."""
import numpy as np
import pytest
import torch

from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu


def _case(C, H, W, n, seed):
    """Parameters, input, and the sparse whole errors of the head."""
    rng = np.random.default_rng(seed)
    table, npar = U.layer_table(C)
    p = np.zeros(npar)
    for cin, cout, wo, bo in table:
        rows = 3 if bo + cout == npar else cout  # the head: the three channels that are read
        w = np.zeros((cout, 9 * cin))
        for c in np.tile(np.arange(cin), 3 if rows == 3 else 1):
            w[rng.integers(rows), rng.integers(9) * cin + c] = rng.choice([1.0, -1.0])
        w[np.arange(rows), rng.integers(9 * cin, size=rows)] = 1.0
        p[wo:bo] = w.ravel()
        p[bo:bo + cout] = rng.integers(0, 2, cout)
    x = rng.integers(0, 2, (n, H, W, U.IN_CH)).astype(np.float64)
    # 2 e / (3 n H W) is a whole multiple of a power of two
    unit = 3 * n * H * W
    while unit % 2 == 0:
        unit //= 2
    few = rng.random((n, 1, H, W)) < min(0.25, 200 / (n * H * W))
    return p, x, rng.integers(-1, 2, (n, 3, H, W)) * few * float(unit)


def _run(model, x, e):
    """Head output and gradients for the errors e."""
    out = model.infer(x).clone()
    model.loss_backward(x, out - e)
    return out, model.grads().clone()


@pytest.fixture
def sur(pkg):
    from importlib import import_module
    return import_module(pkg.__name__ + ".surrogate")


def _model(sur, C, H, W, n, p):
    model = sur.Surrogate(max_batch=n, H=H, W=W, base_channels=C, scale=(1.0, 1.0, 1.0),
                          offset=(0.0, 0.0, 0.0))
    model.set_params(torch.from_numpy(p))
    return model


@pytest.mark.parametrize("C,H,W,n", [(16, 40, 128, 1), (32, 24, 256, 3), (16, 16, 64, 3),
                                     (48, 16, 128, 1), (64, 16, 128, 2), (128, 8, 128, 1)])
def test_rolling_kernels_match_oracle(cuda, sur, C, H, W, n):
    p, x, e = _case(C, H, W, n, seed=C + H)
    out, _ = U.forward(p, x, C, round_bf16=True)
    pred = np.moveaxis(out[..., :3], -1, 1)
    _, want = U.loss_and_grad(p, x, pred - e, (1.0, 1.0, 1.0), (0.0, 0.0, 0.0), C, round_bf16=True)
    model = _model(sur, C, H, W, n, p)
    got, grads = _run(model, torch.from_numpy(x).to("cuda", torch.bfloat16),
                      torch.from_numpy(e).float().cuda())
    assert not model.timed_out()
    assert np.array_equal(got.double().cpu().numpy(), pred)
    g = grads.double().cpu().numpy()
    for cin, cout, wo, bo in U.layer_table(C)[0]:
        assert np.any(want[wo:bo]) and np.array_equal(g[wo:bo + cout], want[wo:bo + cout]), (cin, cout)
    model.close()


@pytest.mark.parametrize("C,H,W,n", [(16, 200, 128, 3), (32, 328, 256, 3), (32, 128, 128, 5),
                                     (64, 64, 256, 3), (128, 48, 128, 2)])
def test_rolling_kernels_equal_per_tile_engine(cuda, pkg, sur, C, H, W, n):
    """Larger grids, against the engine of one CTA per tile."""
    p, x, e = _case(C, H, W, n, seed=C + H)
    model = _model(sur, C, H, W, n, p)
    x = torch.from_numpy(x).to("cuda", torch.bfloat16)
    e = torch.from_numpy(e).float().cuda()
    outs = []
    try:
        for engine in (1, 2):
            pkg.set_umma_engine(engine)
            outs.append(_run(model, x, e))
    finally:
        pkg.set_umma_engine(2)
    assert not model.timed_out()
    assert torch.equal(outs[0][0], outs[1][0])
    for cin, cout, wo, bo in U.layer_table(C)[0]:
        a, b = (o[1][wo:bo + cout] for o in outs)
        assert a.abs().sum() > 0 and torch.equal(a, b), (cin, cout)
    model.close()
