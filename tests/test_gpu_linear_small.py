"""Backward of a small Linear layer, whose two products share a launch, against 64-bit products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [
    (1, 1, 1), (64, 10, 256), (64, 256, 784),   # neither, both uncut; dX cut into four ranges
    (33, 65, 31), (200, 40, 70), (257, 33, 129),  # dW cut, ragged everything
    (300, 500, 65), (512, 90, 40),              # both cut, one into more ranges; as many as a cluster holds
    (513, 20, 33), (20, 600, 40),               # longer sums: one launch each
])
@pytest.mark.parametrize("masked,bias", [(False, True), (True, False), (True, True)])
def test_linear_backward(dev, M, N, K, masked, bias):
    rng = np.random.default_rng(M + N + K)
    g, x, w, mask = (rng.standard_normal(s).astype(np.float32) for s in ((M, N), (M, K), (N, K), (M, K)))
    d = [dev.to_device(a) for a in (g, x, w, mask)]
    out = [dev.to_device(np.full(s, np.nan, np.float32)) for s in ((M, K), (N, K), (N,))]
    for _ in range(2):
        dev.linear_bwd_f32_planes(d[0], d[1], d[2], out[0], out[1], out[2] if bias else None, M, N, K,
                                  relu_mask_src=d[3] if masked else None)
    dx, dw, db = (o.numpy() for o in out)
    G = g.astype(np.float64)
    rdx, rdw = G @ w, G.T @ x
    if masked:
        rdx = np.where(mask < 0, 0, rdx)
    # f32 sums of n terms: at most n * 2^-24 of the sum of magnitudes
    assert (np.abs(dx - rdx) <= (N + 2) * 2.0**-24 * (np.abs(G) @ np.abs(w))).all()
    assert (np.abs(dw - rdw) <= (M + 2) * 2.0**-24 * (np.abs(G).T @ np.abs(x))).all()
    if bias:
        assert np.allclose(db, G.sum(axis=0), rtol=2.0**-23, atol=1e-12)
    for b in d + out:
        b.free()


def test_weight_gradient_into_the_weights(dev):
    """dW written over W: dX is still the product with the old weights."""
    M, N, K = 64, 96, 130
    rng = np.random.default_rng(0)
    g, x, w = (rng.standard_normal(s).astype(np.float32) for s in ((M, N), (M, K), (N, K)))
    dg, dxin, dw = (dev.to_device(a) for a in (g, x, w))
    dx = dev.zeros((M, K))
    dev.linear_bwd_f32(dg, dxin, dw, dx, dw, None, M, N, K)
    assert np.allclose(dx.numpy(), g.astype(np.float64) @ w, rtol=1e-4, atol=1e-4)
    assert np.allclose(dw.numpy(), g.T.astype(np.float64) @ x, rtol=1e-4, atol=1e-4)
    for b in (dg, dxin, dw, dx):
        b.free()


@pytest.mark.parametrize("M,N,K", [(256, 512, 600), (256, 256, 2048), (512, 64, 4096), (512, 512, 512), (33, 700, 3001)])
def test_long_products_with_the_limit_that_nobody_set(M, N, K):
    """Forward and backward on either side of the line between CUDA cores and tensor cores."""
    from vtl_b200 import capi
    dev = capi.Device(0)
    rng = np.random.default_rng(K)
    x, w, g = (rng.standard_normal(s).astype(np.float32) for s in ((M, K), (N, K), (M, N)))
    d = [dev.to_device(a) for a in (x, w, g)]
    out = [dev.to_device(np.full(s, np.nan, np.float32)) for s in ((M, N), (M, K), (N, K), (N,))]
    dev.linear_fwd_f32(d[0], d[1], None, out[0], M, N, K)
    dev.linear_bwd_f32(d[2], d[0], d[1], out[1], out[2], out[3], M, N, K)
    assert dev.check_status() == 0
    y, dx, dw, db = (o.numpy() for o in out)
    X, W, G = (a.astype(np.float64) for a in (x, w, g))
    # 3xTF32: 2^-22 a factor, at most 48 truncations of 2^-23 between two exact sums; f32 sums of 256 terms less
    bound = 2 * 2.0**-22 + 48 * 2.0**-23
    assert (np.abs(y - X @ W.T) <= bound * (np.abs(X) @ np.abs(W).T)).all()
    assert (np.abs(dx - G @ W) <= bound * (np.abs(G) @ np.abs(W))).all()
    assert (np.abs(dw - G.T @ X) <= bound * (np.abs(G).T @ np.abs(X))).all()
    assert np.allclose(db, G.sum(axis=0), rtol=2.0**-23, atol=1e-12)
    for b in d + out:
        b.free()
    dev.close()


# 3xTF32: 2^-22 a factor, at most 48 truncations of 2^-23 between two exact sums; f32 sums of 256 terms less
LONG = 2 * 2.0**-22 + 48 * 2.0**-23


def _close(got, a, b):
    a, b = a.astype(np.float64), b.astype(np.float64)
    return (np.abs(got - a @ b) <= LONG * (np.abs(a) @ np.abs(b))).all()


@pytest.mark.parametrize("over", ["x", "w", "pre over x"])
def test_forward_over_an_operand(over):
    """Above the limit of small products the result may lie over an operand."""
    from vtl_b200 import capi
    dev = capi.Device(0)
    M, N, K = (512, 320, 512) if over == "w" else (320, 512, 512)
    rng = np.random.default_rng(1)
    x, w = (rng.standard_normal(s).astype(np.float32) for s in ((M, K), (N, K)))
    n = max(M, N) * 512
    dx, dw, spare = (dev.to_device(np.resize(a, n)) for a in (x, w, np.zeros(1, np.float32)))
    if over == "pre over x":
        y, pre = spare, dx
    else:
        y, pre = (dx if over == "x" else dw), None
    dev.linear_fwd_f32(dx, dw, None, y, M, N, K, False, pre)
    assert dev.check_status() == 0
    for buf in (y, pre):
        assert buf is None or _close(buf.numpy().ravel()[:M * N].reshape(M, N), x, w.T)
    for b in (dx, dw, spare):
        b.free()
    dev.close()


@pytest.mark.parametrize("over", ["dX over G", "dX over W", "dW over X", "dW over G", "db over G"])
def test_backward_over_an_operand(over):
    from vtl_b200 import capi
    dev = capi.Device(0)
    M, N, K = {"dW over X": (512, 320, 512), "dW over G": (512, 512, 320)}.get(over, (320, 512, 512))
    rng = np.random.default_rng(2)
    g, x, w = (rng.standard_normal(s).astype(np.float32) for s in ((M, N), (M, K), (N, K)))
    d = {"G": dev.to_device(g), "X": dev.to_device(x), "W": dev.to_device(w)}
    out = {"dX": dev.zeros((M, K)), "dW": dev.zeros((N, K)), "db": dev.zeros((N,))}
    what, on = over.split(" over ")
    where = {**out, what: d[on]}
    # one output over an operand; another that reads the operand is not asked for
    args = {k: where[k] if k == what or (k, on) in (("dW", "W"), ("dX", "X")) else None for k in out}
    if what == "db":
        args = where
    dev.linear_bwd_f32(d["G"], d["X"], d["W"], args["dX"], args["dW"], args["db"], M, N, K)
    assert dev.check_status() == 0
    flat = lambda b, *s: b.numpy().ravel()[:int(np.prod(s))].reshape(s)  # noqa: E731
    if args["dX"]:
        assert _close(flat(args["dX"], M, K), g, w)
    if args["dW"]:
        assert _close(flat(args["dW"], N, K), g.T, x)
    if args["db"]:
        assert np.allclose(flat(args["db"], N), g.astype(np.float64).sum(axis=0), rtol=2.0**-23, atol=1e-12)
    for b in (*d.values(), *out.values()):
        b.free()
    dev.close()


def test_bias_gradient_over_the_mask(dev):
    """The mask is read before the bias gradient is written, also where both products could share a launch."""
    M, N, K = 64, 96, 130
    rng = np.random.default_rng(3)
    g, x, w, mask = (rng.standard_normal(s).astype(np.float32) for s in ((M, N), (M, K), (N, K), (M, K)))
    d = [dev.to_device(a) for a in (g, x, w, mask)]
    dx, dw = dev.zeros((M, K)), dev.zeros((N, K))
    dev.linear_bwd_f32_planes(d[0], d[1], d[2], dx, dw, d[3], M, N, K, relu_mask_src=d[3])
    assert np.allclose(dx.numpy(), np.where(mask < 0, 0, g.astype(np.float64) @ w), rtol=1e-4, atol=1e-4)
    assert np.allclose(dw.numpy(), g.T.astype(np.float64) @ x, rtol=1e-4, atol=1e-4)
    assert np.allclose(d[3].numpy().ravel()[:N], g.astype(np.float64).sum(axis=0), rtol=2.0**-23, atol=1e-12)
    for b in (*d, dx, dw):
        b.free()
