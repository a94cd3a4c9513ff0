"""Bit-exact checks of the INT8 Linear where its kernels change over: rows of Y that TMA cannot store, row maxima
from the few-row kernels, more output channels than one wave of tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(q, sa, w, sw, bias, relu):
    """acc -> float(acc) * (sa * sw) + bias -> ReLU, every f32 operation rounded on its own."""
    acc = (q.astype(np.float64) @ w.astype(np.float64).T).astype(np.int32)  # exact: |acc| < 2^53
    y = acc.astype(np.float32) * (sa[:, None] * sw[None, :]).astype(np.float32)
    if bias is not None:
        y = y + bias[None, :]
    if relu:
        y[y < 0] = 0
    return acc, y


@pytest.mark.parametrize("M,N,K,relu", [
    (129, 1, 64, False), (130, 127, 144, True), (255, 1003, 272, False),  # 128 x 64 tiles
    (400, 6001, 160, True),                                               # 128 x 128 tiles
    (300, 12801, 128, False),                                             # 128 x 256 tiles
    (999, 3001, 2047, False), (513, 4999, 144, True),                     # CTA pairs
    (2305, 2303, 1024, True),                                             # CTA pairs, K-split last wave
])
def test_rows_that_tma_cannot_store(dev, M, N, K, relu):
    _check(dev, M, N, K, relu)


@pytest.mark.parametrize("M,N,K,relu", [
    (1, 4097, 272, False), (1, 28672, 128, True),          # dp4a kernel: row maxima over one and several channels a warp
    (2, 130, 2048, False), (16, 128, 4096, True),          # K over four CTAs, one tile
    (8, 19073, 256, True), (17, 18945, 144, False), (33, 28672, 256, True),  # more tiles than SMs
    (64, 38017, 128, False),                               # more tiles than two to an SM
    (65, 18945, 144, True), (128, 18944, 128, False),      # above 64 rows: the general kernel, and one wave
])
def test_few_rows_and_their_maxima(dev, M, N, K, relu):
    _check(dev, M, N, K, relu)


@pytest.mark.parametrize("given", [False, True])
@pytest.mark.parametrize("M,K,offset", [(3, 1, 0), (5, 15, 0), (2, 17, 0), (7, 1023, 0), (600, 1025, 0), (4, 2047, 0),
                                        (3, 4097, 0), (513, 8191, 0), (2, 8192, 1), (3, 1024, 2), (2, 64, 3)])
def test_rows_that_vector_loads_cannot_take(dev, orc, M, K, offset, given):
    A = np.random.default_rng(K).standard_normal((M, K)).astype(np.float32)
    A[0] = 0.0
    amax = (np.abs(A).max(axis=1) * 1.25).astype(np.float32)
    ld = dev.i8_ld(K)
    buf = dev.to_device(np.concatenate([np.zeros(offset, np.float32), A.ravel()]))  # a base `offset` values off
    dM = dev.to_device(amax)
    dQ, dS = dev.to_device(np.full((M, ld), 77, np.int8)), dev.empty((M,), np.float32)
    dev.quant_rows_i8(buf.ptr + 4 * offset, M, K, dQ, dS, dM if given else None)
    q_ref, s_ref = orc.quant_rows_i8_with_amax(A, amax) if given else orc.quant_rows_i8(A)
    q = dQ.numpy()
    assert np.array_equal(q[:, :K], q_ref) and (q[:, K:] == 77).all()
    assert np.array_equal(dS.numpy().view(np.uint32), s_ref.view(np.uint32))
    for b in (buf, dM, dQ, dS):
        b.free()


@pytest.mark.parametrize("M,K", [(1, 8208), (3, 28672), (2, 12293), (513, 8196)])
def test_long_rows_quantised_in_pieces(dev, orc, M, K):
    A = np.random.default_rng(K).standard_normal((M, K)).astype(np.float32)
    amax = np.abs(A).max(axis=1)
    amax[0] = 0.0  # a maximum of zero: scale 0, codes 0
    dA, dM = dev.to_device(A), dev.to_device(amax)
    dQ, dS = dev.zeros((M, dev.i8_ld(K)), np.int8), dev.empty((M,), np.float32)
    dev.quant_rows_i8(dA, M, K, dQ, dS, dM)
    q_ref, s_ref = orc.quant_rows_i8_with_amax(A, amax)
    assert np.array_equal(dQ.numpy()[:, :K], q_ref)
    assert np.array_equal(dS.numpy().view(np.uint32), s_ref.view(np.uint32))
    for b in (dA, dM, dQ, dS):
        b.free()


def _check(dev, M, N, K, relu):
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    ld = dev.i8_ld(K)
    q = rng.integers(-127, 128, (M, ld), dtype=np.int8)  # the padding holds garbage on purpose
    w = rng.integers(-127, 128, (N, ld), dtype=np.int8)
    sa = rng.uniform(1e-3, 1e-2, M).astype(np.float32)
    sw = rng.uniform(1e-4, 1e-3, N).astype(np.float32)
    bias = rng.standard_normal(N).astype(np.float32) if M & 1 else None
    acc, y = _reference(q[:, :K], sa, w[:, :K], sw, bias, relu)
    dq, dw, dsa, dsw = (dev.to_device(t) for t in (q, w, sa, sw))
    db = dev.to_device(bias) if bias is not None else None
    guard = np.full(N, 7.0, np.float32)
    dY = dev.to_device(np.vstack([np.zeros((M, N), np.float32), guard[None, :]]))
    dA = dev.to_device(np.full(M + 1, 9.0, np.float32))  # what an earlier batch left behind
    dC = dev.zeros((M, N), np.int32)
    for _ in range(2):  # the second pass finds the counters and flags of the first
        dev.linear_i8_fwd_amax(dq, 1, dsa, dw, dsw, db, dY, M, N, K, relu, dA)
        dev.gemm_i8_i32(dq, dw, M, N, K, dC)
        assert dev.check_status() == 0
        got, amax = dY.numpy(), dA.numpy()
        assert np.array_equal(dC.numpy(), acc)
        assert np.array_equal(got[:M].view(np.uint32), y.view(np.uint32)), f"max diff {np.abs(got[:M] - y).max()}"
        assert np.array_equal(got[M], guard), "wrote past the last row"
        assert np.array_equal(amax[:M], np.abs(y).max(axis=1)) and amax[M] == 9.0
    dev.linear_i8_fwd(dq, dsa, dw, dsw, db, dY, M, N, K, relu)
    assert np.array_equal(dY.numpy()[:M].view(np.uint32), y.view(np.uint32))
    for b in (dq, dw, dsa, dsw, dY, dA, dC) + ((db,) if db else ()):
        b.free()
