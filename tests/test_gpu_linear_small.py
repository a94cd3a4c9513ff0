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
