"""Edges of the one-launch losses and BatchNorm: the class counts at which the lanes per row and the values per
lane change, row counts at which the rows per thread change, lengths that no vector divides.  Same oracle and
bounds as test_gpu_elementwise.py and test_gpu_layers_extra.py (f64 sums in another order, rounded once)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C", [(1, 1), (65, 4), (33, 5), (100, 16), (9, 17), (7, 33), (257, 64), (5, 128), (3, 129), (17, 256),
                                 (2, 257), (6, 1000)])
def test_softmax_ce_edges(dev, orc, B, C):
    rng = np.random.default_rng(B * 1000 + C)
    x = (rng.standard_normal((B, C)) * 3).astype(np.float32)
    t = np.eye(C, dtype=np.float32)[rng.integers(0, C, B)]
    dx, dt, dl, dg = dev.to_device(x), dev.to_device(t), dev.zeros(1), dev.zeros((B, C))
    for _ in range(2):  # the second launch needs the block ticket reset by the first
        dev.softmax_ce_fwd_bwd_f32(dx, dt, B, C, B, dl, dg)
    ref = float(orc.softmax_ce_f32(x, t))
    assert abs(float(dl.numpy()[0]) - ref) <= 1e-6 * max(1.0, abs(ref))
    assert np.abs(dg.numpy() - orc.softmax_ce_bwd_f32(x, t)).max() <= 1e-7
    for b in (dx, dt, dl, dg):
        b.free()


@pytest.mark.parametrize("n,offset", [(8192, 0), (8193, 0), (8195, 1), (1 << 20, 0), ((1 << 20) + 3, 0), (300007, 3)])
def test_mse_edges(dev, orc, n, offset):
    rng = np.random.default_rng(n)
    p, t = rng.standard_normal(n + offset).astype(np.float32), rng.standard_normal(n + offset).astype(np.float32)
    dp, dt, dl, dg = dev.to_device(p), dev.to_device(t), dev.zeros(1), dev.zeros(n + offset)
    dev.mse_fwd_bwd_f32(dp.ptr + 4 * offset, dt.ptr + 4 * offset, n, n, dl, dg.ptr + 4 * offset)
    p, t = p[offset:], t[offset:]
    assert np.array_equal(dg.numpy()[offset:].view(np.uint32), orc.mse_bwd_f32(p, t).view(np.uint32))
    assert abs(float(dl.numpy()[0]) - orc.mse_f64(p, t)) <= 1e-6 * orc.mse_f64(p, t)
    for b in (dp, dt, dl, dg):
        b.free()


@pytest.mark.parametrize("B,F", [(1, 1), (32, 9), (128, 7), (129, 8), (256, 33), (257, 512), (512, 1), (1024, 17), (1025, 17),
                                 (1600, 300)])
@pytest.mark.parametrize("params", [True, False])
def test_batchnorm_edges(dev, orc, B, F, params):
    rng = np.random.default_rng(B * 7 + F)
    x = (rng.standard_normal((B, F)) * 2 + 0.5).astype(np.float32)
    g = rng.standard_normal((B, F)).astype(np.float32)
    gamma, beta = rng.uniform(0.5, 1.5, F).astype(np.float32), rng.standard_normal(F).astype(np.float32)
    rm, rv = rng.standard_normal(F).astype(np.float32), rng.uniform(0.5, 2, F).astype(np.float32)
    d = [dev.to_device(a) for a in (x, g, gamma, beta, rm, rv)]
    y, m, v, dx, dg, db = (dev.zeros(s) for s in ((B, F), F, F, (B, F), F, F))
    dev.batchnorm1d_train_f32(d[0], B, F, d[2], d[3], 1e-5, y, m, v, d[4], d[5], 0.1)
    ry, rmean, rvar, rrm, rrv = orc.batchnorm1d_train_f32(x, gamma, beta, 1e-5, rm, rv, 0.1)
    # f32 results of f64 sums: at most one unit in the last place from the oracle's order
    for got, ref in ((m, rmean), (v, rvar), (d[4], rrm), (d[5], rrv)):
        assert np.abs(got.numpy() - ref).max() <= 2.0 ** -23 * max(1e-30, float(np.abs(ref).max()))
    assert np.abs(y.numpy() - ry).max() <= 2e-6 * max(1.0, float(np.abs(ry).max()))
    dm, dv = dev.to_device(rmean), dev.to_device(rvar)
    dev.batchnorm1d_bwd_f32(d[1], d[0], B, F, d[2], dm, dv, 1e-5, dx, dg if params else None, db if params else None)
    rdx, rdg, rdb = orc.batchnorm1d_bwd_f32(g, x, gamma, rmean, rvar, 1e-5)
    assert np.abs(dx.numpy() - rdx).max() <= 2e-6 * max(1.0, float(np.abs(rdx).max()))
    if params:
        assert np.abs(dg.numpy() - rdg).max() <= 1e-6 * max(4 * B ** 0.5, float(np.abs(rdg).max()))
        assert np.abs(db.numpy() - rdb).max() <= 2.0 ** -22 * max(1e-30, float(np.abs(rdb).max()))
    for b in d + [y, m, v, dx, dg, db, dm, dv]:
        b.free()
