"""The warm-start network on the tensor cores against its CPU oracle -- GPU."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net(in_dim=22, width=128, hidden=2, out_dim=3, seed=3):
    from morphoshell_b200 import Mlp
    return Mlp(in_dim, width=width, hidden_layers=hidden, out_dim=out_dim, seed=seed)


def _data(n, in_dim=22, out_dim=3, seed=0):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, in_dim)).astype(np.float32)
    t = np.stack([np.sin(x[:, 0]) * np.cos(x[:, 1]), 0.5 * x[:, 2] * x[:, 3], np.tanh(x[:, 4])][:out_dim], 1)
    return x, t.astype(np.float32)


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("n", [128, 300, 1000])
def test_forward_matches_oracle(n):
    from oracle import mlp_ref
    net = _net()
    x, _ = _data(n)
    y = net.forward(x)
    yr = mlp_ref.forward(net.params(), x, 22, 128, 2, 3, bf16_points=True)
    assert _rel(y, yr) < 1e-2
    ye = mlp_ref.forward(net.params(), x, 22, 128, 2, 3, bf16_points=False)
    assert _rel(y, ye) < 5e-2


@pytest.mark.parametrize("width,hidden", [(128, 2), (256, 4)])
def test_gradients_match_oracle(width, hidden):
    """Loss and every layer's weight and bias gradient against the oracle
    with the GPU's bf16 rounding points, and against exact float64."""
    from oracle import mlp_ref
    net = _net(width=width, hidden=hidden)
    x, t = _data(700)
    loss, g = net.loss_grad(x, t)
    lr, gr = mlp_ref.loss_grad(net.params(), x, t, 22, width, hidden, 3, bf16_points=True)
    le, ge = mlp_ref.loss_grad(net.params(), x, t, 22, width, hidden, 3, bf16_points=False)
    assert abs(loss - lr) / lr < 1e-3 and abs(loss - le) / le < 2e-2
    for off, N, K, Np in net.layers():
        w = slice(off, off + N * K)
        b = slice(off + N * K, off + N * K + N)
        assert _rel(g[w], gr[w]) < 2e-2, ("W", off)
        assert _rel(g[b], gr[b]) < 2e-2, ("b", off)
        assert _rel(g[w], ge[w]) < 6e-2
    # padded parameters get no gradient
    off, N, K, Np = net.layers()[-1]
    assert not g[off + N * K + N:off + N * K + Np].any()


def test_training_reduces_loss():
    net = _net(width=128, hidden=2)
    x, t = _data(20000, seed=1)
    net.set_data(x, t)
    losses = net.train(epochs=30, batch=2048, lr=2e-3, seed=0)
    assert np.all(np.isfinite(losses))
    assert losses[-1] < 0.1 * losses[0], losses
    xv, tv = _data(4000, seed=2)
    yv = net.forward(xv)
    assert float(((yv - tv) ** 2).mean()) < 2 * losses[-1] + 1e-3


# Edges of the 128-row tiles and the 512-row gradient splits, of the input
# padding, and every cluster size; tolerances as above (the same rounding
# points, accumulation in FP32 instead of double).
@pytest.mark.parametrize("n,in_dim,width,hidden,out_dim", [
    (1, 1, 128, 1, 1), (127, 16, 128, 7, 3), (129, 17, 256, 2, 16), (512, 22, 384, 3, 3), (513, 256, 128, 2, 3),
    (1025, 255, 512, 2, 2)])
def test_network_shapes(n, in_dim, width, hidden, out_dim):
    from oracle import mlp_ref
    rng = np.random.default_rng(n)
    net = _net(in_dim, width, hidden, out_dim)
    x = rng.standard_normal((n, in_dim)).astype(np.float32)
    t = rng.standard_normal((n, out_dim)).astype(np.float32)
    shape = (in_dim, width, hidden, out_dim)
    assert _rel(net.forward(x), mlp_ref.forward(net.params(), x, *shape, bf16_points=True)) < 1e-2
    loss, g = net.loss_grad(x, t)
    lr, gr = mlp_ref.loss_grad(net.params(), x, t, *shape, bf16_points=True)
    assert abs(loss - lr) / lr < 1e-3
    for off, N, K, Np in net.layers():
        assert _rel(g[off:off + N * K], gr[off:off + N * K]) < 2e-2
        assert _rel(g[off + N * K:off + N * K + N], gr[off + N * K:off + N * K + N]) < 2e-2


def test_new_rows_right_after_others():
    """Rows from pageable memory are in place when the kernels read them: a
    short call right after another one, and new parameters right before one."""
    from oracle import mlp_ref
    net = _net(width=256, hidden=2)
    p = net.params()
    for k in range(20):
        x, t = _data(1000, seed=k)
        net.loss_grad(x[::-1], t)
        net.set_params(p * np.float32(1.0 + 0.01 * k))
        assert _rel(net.forward(x), mlp_ref.forward(net.params(), x, 22, 256, 2, 3, bf16_points=True)) < 1e-2


def _activations(net, first=1.0):
    """A network of one hidden layer whose first 16 hidden units are its
    outputs, and whose hidden pre-activations are its inputs (the first one's
    times `first`)."""
    p = np.zeros(net.num_params(), dtype=np.float32)
    (o0, n0, k0, _), (o1, n1, k1, _) = net.layers()
    w0 = np.eye(n0, k0, dtype=np.float32)
    w0[0, 0] = first
    p[o0:o0 + n0 * k0] = w0.ravel()
    p[o1:o1 + n1 * k1] = np.eye(n1, k1, dtype=np.float32).ravel()
    net.set_params(p)


def test_silu_of_every_bf16_value():
    """Every finite BF16 pre-activation, beside others of every size (a
    reciprocal serves two of them, one test sixteen), against SiLU in double,
    rounded to BF16: rounding is monotone, so the result lies between the
    rounded ends of an interval of FP32's errors around the value.  Those are
    2^-22 of the exponential, of its argument's rounding 1.5 2^-24 times up to
    89, and 2^-23 of the sum and the quotient: together under 2^-16.  Below
    1e-36 the exponential overflows."""
    import torch
    rng = np.random.default_rng(70)
    bits = np.arange(65536, dtype=np.uint32)
    v = (bits[(bits & 0x7f80) != 0x7f80] << 16).view(np.float32)
    x = np.stack([v] + [rng.permutation(v) for _ in range(127)], 1)
    x[:, 64:] = rng.standard_normal((len(v), 64)).astype(np.float16)
    net = _net(128, 128, 1, 16)
    _activations(net)
    z = torch.from_numpy(x[:, :16].astype(np.float64))
    want = z / (1.0 + torch.exp(-z))
    got = torch.from_numpy(net.forward(x)).double()
    ends = [(want * (1.0 + e)).to(torch.float32).to(torch.bfloat16).double() for e in (-2.0 ** -16, 2.0 ** -16)]
    ok = (got >= torch.minimum(*ends)) & (got <= torch.maximum(*ends)) | ((got - want).abs() <= 1e-36)
    assert ok.all(), (z[~ok][:8], got[~ok][:8], want[~ok][:8])


def test_silu_of_an_infinite_preactivation():
    """A pre-activation beyond FP32 is infinite, and so is its SiLU."""
    net = _net(128, 128, 1, 16)
    _activations(net, first=4.0)
    x = np.zeros((200, 128), dtype=np.float32)
    x[::3, 0] = 3e38
    y = net.forward(x)[:, 0]
    assert (y[::3] == np.inf).all()
    assert (np.delete(y, np.s_[::3]) == 0).all()
