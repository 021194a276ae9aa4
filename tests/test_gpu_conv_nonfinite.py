"""Infinities and NaN in the proposal's convolutions reach what they reach in the general kernels, no more:
not through a tap off the grid, nor through a gradient that is zero.  All other values are small whole numbers,
whose sums are exact in any order, so results are compared bit for bit."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")


def _whole(g, *shape):
    return torch.randint(-2, 3, shape, generator=g).float()


def _p(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _same(a, b):
    assert torch.equal(a.isnan(), b.isnan())
    assert torch.equal(torch.nan_to_num(a, nan=0.0), torch.nan_to_num(b, nan=0.0))


@pytest.mark.parametrize("d", [1, 2, 5, 9])
@pytest.mark.parametrize("where", ["input", "gradient", "both", "masked"])
def test_weight_gradient(dev, d, where):
    """Two output channels (the staged kernel) against one at a time (the general kernel)."""
    from vesper_python_gb300 import _native
    g = torch.Generator().manual_seed(d)
    cin, cout = 3, 2
    x, dout, out = _whole(g, cin, d, d, d), _whole(g, cout, d, d, d), _whole(g, cout, d, d, d)
    dout[torch.rand(dout.shape, generator=g) < 0.4] = 0.0
    if where in ("input", "both"):
        x[0, 0, 0, 0], x[1, d // 2, d - 1, d // 2] = INF, NAN
    if where in ("gradient", "both"):
        dout[0, d - 1, 0, d // 2], dout[1, d // 2, d // 2, 0] = INF, -INF
        out[0] = 1.0
    if where == "masked":               # the activation is infinite where the ReLU lets nothing through
        x[0, 0, 0, 0], x[2, d - 1, d - 1, d - 1] = INF, -INF
        out[:, :, :, :] = -1.0
    W = torch.zeros(cout, cin, 27, dtype=torch.bfloat16)
    x, dout, out, W = (t.to(dev.device) for t in (x, dout, out, W))

    def grads(lo, hi):
        n = hi - lo
        dW, db = torch.ones((n, cin, 27), device=dev.device), torch.ones(n, device=dev.device)
        _native.check(dev.lib.vesper_prop_conv_bwd(_p(dout[lo:hi].contiguous()), _p(out[lo:hi].contiguous()), 1, _p(x),
                                                   _p(W[lo:hi].contiguous()), cin, n, d, None, _p(dW), _p(db), dev.stream))
        return dW, db

    both, one = grads(0, 2), [grads(i, i + 1) for i in range(2)]
    for k in range(2):
        _same(both[k], torch.cat([o[k] for o in one]))
    if where == "masked":
        assert torch.equal(both[0], torch.ones_like(both[0]))


@pytest.mark.parametrize("d", [1, 3, 8, 13])
@pytest.mark.parametrize("nmap", [1, 40])     # one voxel per thread, and four
@pytest.mark.parametrize("relu", [0, 1])
@pytest.mark.parametrize("where", ["weights", "input", "both", "bias"])
def test_forward(dev, d, nmap, relu, where):
    """Four output channels per thread against one (a channel count that four does not divide)."""
    from vesper_python_gb300 import _native
    g = torch.Generator().manual_seed(d)
    cin = 5
    x, W, b = _whole(g, nmap, cin, d, d, d), _whole(g, 8, cin, 27), _whole(g, 8)
    if where in ("weights", "both"):
        W[0, 0, 0], W[1, 2, 14], W[2, 4, 26], W[5, 1, 3] = INF, -INF, NAN, INF
    if where in ("input", "both"):
        x[0, 1, d // 2, 0, d - 1], x[-1, 3, 0, d // 2, 0] = INF, NAN
    if where == "bias":
        b[1], b[6] = INF, NAN
    x, W, b = x.to(dev.device), W.to(torch.bfloat16).to(dev.device), b.to(dev.device)

    def layer(lo, hi):
        o = torch.full((nmap, hi - lo, d, d, d), 7.0, device=dev.device)
        _native.check(dev.lib.vesper_prop_conv_fwd(_p(x), cin, _p(W[lo:hi].contiguous()), _p(b[lo:hi].contiguous()), hi - lo,
                                                   d, relu, nmap, _p(o), dev.stream))
        return o

    fast, plain = layer(0, 8), torch.cat([layer(i, i + 1) for i in range(8)], 1)
    assert torch.equal(fast.isnan(), plain.isnan())
    assert torch.equal(torch.nan_to_num(fast, nan=0.0, posinf=9e9, neginf=-9e9),
                       torch.nan_to_num(plain, nan=0.0, posinf=9e9, neginf=-9e9))
