"""f32 products large enough for the CTA-pair kernel on f16 planes, against 64-bit products; and operands that f16
planes cannot hold, which have to come out as well as 3xTF32 does."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _error(C, A, B):
    """Largest error of C against A @ B^T, over |A| @ |B|^T element by element."""
    A, B = torch.from_numpy(A).double().cuda(), torch.from_numpy(B).double().cuda()
    d = (torch.from_numpy(C).double().cuda() - A @ B.T).abs()
    return float((d / (A.abs() @ B.abs().T).clamp_min(1e-300)).max())


# Operands keep 22 bits (2^-22 a factor, twice); an accumulator of tcgen05 truncates, at most 24 times before it is
# closed (8 K steps x 3 products), by less than 2^-23 of the sum of magnitudes each; the closed ones round to nearest.
BOUND = 2 * 2.0**-22 + 24 * 2.0**-23


def _product(dev, ta, tb, A, B):
    M, K = A.shape
    N = B.shape[0]
    dA = dev.to_device(np.ascontiguousarray(A.T if ta else A))
    dB = dev.to_device(np.ascontiguousarray(B if tb else B.T))
    dC = dev.to_device(np.full((M, N), np.nan, np.float32))
    dev.gemm_f32(ta, tb, M, N, K, dA, dB, dC)
    assert dev.check_status() == 0
    C = dC.numpy()
    for b in (dA, dB, dC):
        b.free()
    return C


@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(2048, 1280, 63), (1500, 1800, 255), (1537, 1793, 256), (2049, 1279, 257),
                                   (512, 4868, 1001), (2500, 1003, 516)])
def test_product(dev, ta, tb, M, N, K):
    rng = np.random.default_rng(M + N + K)
    A, B = (rng.standard_normal((r, K)).astype(np.float32) for r in (M, N))
    assert _error(_product(dev, ta, tb, A, B), A, B) < BOUND


def _features(rng, r, K, sign):
    return rng.standard_normal((r, K)) * 10.0 ** (sign * 12 * (np.arange(K) % 7 / 6 - 0.5))


@pytest.mark.parametrize("kind", ["features", "rows", "tiny", "huge", "lognormal", "zeros", "sparse"])
def test_operands_of_any_range(dev, kind):
    M, N, K = 1536, 1792, 600
    rng = np.random.default_rng(3)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((N, K))
    if kind == "features":  # columns on scales 1e-6 .. 1e6, undone by the weights
        A, B = _features(rng, M, K, 1), _features(rng, N, K, -1)
    if kind == "rows":      # every output on a scale of its own, both sides
        A, B = A * 10.0 ** rng.uniform(-8, 8, (M, 1)), B * 10.0 ** rng.uniform(-8, 8, (N, 1))
    if kind == "tiny":
        A, B = A * 1e-25, B * 1e-8
    if kind == "huge":
        A, B = A * 1e30, B * 1e-20
    if kind == "lognormal":
        A, B = A * np.exp(3 * rng.standard_normal(A.shape)), B * np.exp(3 * rng.standard_normal(B.shape))
    if kind == "zeros":
        A[:, 256:512], B[100:200] = 0, 0
    if kind == "sparse":    # a few values a row, on scales of their own
        A = A * (rng.random(A.shape) < 0.01) * 10.0 ** rng.uniform(-9, 0, A.shape)
    A, B = A.astype(np.float32), B.astype(np.float32)
    # 3xTF32 closes an accumulator after 48 products; the operands keep the same 22 bits
    assert _error(_product(dev, False, True, A, B), A, B) < 2 * 2.0**-22 + 48 * 2.0**-23


LIMIT = 2 * 2.0**-22 + 48 * 2.0**-23  # 3xTF32's, element by element


def _pruned(rng, r, K, every, scale=None):
    """Normal values in every `every`-th column: alone there, or `scale` times smaller than the others."""
    x, some = rng.standard_normal((r, K)), np.arange(K) % every == every // 2
    return (x * some if scale is None else np.where(some, x * scale, x)).astype(np.float32)


@pytest.mark.parametrize("ta,tb", [(False, True), (True, False)])
@pytest.mark.parametrize("s", [1e-4, 1e-6, 1e-7, 1e-9, 1e-11, 1e-13, 1e-30])
def test_small_elements_that_meet_the_only_large_ones(dev, s, ta, tb):
    """The elements of one operand that f16 cannot hold beside their neighbours are the ones that count: the other
    operand is zero wherever this one is large."""
    M, N, K = 1536, 1792, 600
    rng = np.random.default_rng(6)
    A, B = _pruned(rng, M, K, 20, s), _pruned(rng, N, K, 20)
    assert _error(_product(dev, ta, tb, A, B), A, B) < LIMIT
    A, B = _pruned(rng, M, K, 20), _pruned(rng, N, K, 20, s)
    assert _error(_product(dev, ta, tb, A, B), A, B) < LIMIT


@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("few", [1, 3, 4, 5, 6, 60])
def test_few_small_elements(dev, ta, tb, few):
    """So few that the product stays on f16 planes (5 in one row of a block, or 60 in all, are too many): planted in both
    operands, at the edges of blocks, groups and the matrices, some of them opposite one another."""
    M, N, K = 1501, 1797, 775
    rng = np.random.default_rng(few)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((N, K))
    ks = np.array([0, 255, 256, 511, 512, 767, 768, 774, 300, 301])
    if few <= 5:  # in one row of one block
        A[5, 256:256 + few] *= 10.0 ** -np.arange(10, 10 + few)
        B[M % 31, 512:512 + few] *= 10.0 ** -np.arange(10, 10 + few)
        B[:, 256:256 + few] *= 1e3
        A[:, 512:512 + few] *= 1e3
    else:
        rows, cols = rng.choice(M, few, replace=False), rng.choice(N, few, replace=False)
        rows[:3], cols[:3] = (0, 31, M - 1), (0, 32, N - 1)
        A[rows, ks[np.arange(few) % 10]] *= 10.0 ** -rng.uniform(9, 18, few)
        B[cols, ks[np.arange(few) % 10]] *= 10.0 ** -rng.uniform(9, 18, few)
        keep = np.zeros(K, bool)  # and nothing else meets them
        keep[ks] = True
        B[:N // 2, ~keep] = 0
        A[M // 2:, ~keep] = 0
    A, B = A.astype(np.float32), B.astype(np.float32)
    assert _error(_product(dev, ta, tb, A, B), A, B) < LIMIT


@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("kind", ["diagonal", "permutation", "sparse"])
def test_sparse_second_operand(dev, kind, tb):
    """32 rows of B share a scale: a row of a single value has to survive beside much larger ones."""
    M, N, K = 1536, 1792, 512
    rng = np.random.default_rng(7)
    A, B = rng.standard_normal((M, K)), np.zeros((N, K))
    at = rng.permutation(K)
    if kind == "diagonal":
        B[at, np.arange(K)] = 10.0 ** -np.linspace(0, 12, K)[rng.permutation(K)]
    if kind == "permutation":
        A *= 10.0 ** rng.uniform(-9, 0, A.shape)
        B[at, np.arange(K)] = 1
    if kind == "sparse":
        B = rng.standard_normal((N, K)) * (rng.random((N, K)) < 0.005) * 10.0 ** rng.uniform(-9, 0, (N, K))
    A, B = A.astype(np.float32), B.astype(np.float32)
    assert _error(_product(dev, False, tb, A, B), A, B) < LIMIT


def test_infinities_and_nans_stay_in_their_rows(dev):
    M, N, K = 1536, 1792, 512
    rng = np.random.default_rng(4)
    A, B = (rng.standard_normal((r, K)).astype(np.float32) for r in (M, N))
    A[3, 300], A[700, 0], B[9, 511] = np.inf, np.nan, -np.inf
    C = _product(dev, False, True, A, B)
    assert not np.isfinite(C[3]).any() and np.isnan(C[700]).all() and not np.isfinite(C[:, 9]).any()
    rows, cols = np.delete(np.arange(M), [3, 700]), np.delete(np.arange(N), 9)
    assert _error(np.ascontiguousarray(C[rows][:, cols]), A[rows], B[cols]) < 2 * 2.0**-22 + 48 * 2.0**-23


@pytest.mark.parametrize("wide", [False, True])
def test_linear_backward(dev, wide):
    """dX masked by the layer below, dW, and the bias gradient that the transposing pass sums on the way."""
    M, N, K = 1300, 1600, 1540
    rng = np.random.default_rng(5)
    g, x, w, mask = (rng.standard_normal(s).astype(np.float32) for s in ((M, N), (M, K), (N, K), (M, K)))
    if wide:  # unfit for f16 planes: the bias gradient still comes from their pass
        g = (g * 10.0 ** rng.uniform(-9, 0, g.shape)).astype(np.float32)
    d = [dev.to_device(a) for a in (g, x, w, mask)]
    out = [dev.to_device(np.full(s, np.nan, np.float32)) for s in ((M, K), (N, K), (N,))]
    dev.linear_bwd_f32_planes(d[0], d[1], d[2], out[0], out[1], out[2], M, N, K, relu_mask_src=d[3])
    assert dev.check_status() == 0
    dx, dw, db = (o.numpy() for o in out)
    assert (dx[mask < 0] == 0).all()
    full = np.where(mask < 0, (g.astype(np.float64) @ w.astype(np.float64)).astype(np.float32), dx)
    assert _error(full, g, np.ascontiguousarray(w.T)) < 2 * 2.0**-22 + 48 * 2.0**-23
    assert _error(dw, np.ascontiguousarray(g.T), np.ascontiguousarray(x.T)) < 2 * 2.0**-22 + 48 * 2.0**-23
    ref = g.astype(np.float64).sum(axis=0)
    assert (np.abs(db - ref) <= 2.0**-24 * np.abs(ref) + 1e-13 * np.abs(g).sum(axis=0)).all()
    for b in d + out:
        b.free()


def test_scratch_of_a_large_product():
    """The context keeps the operands' planes, 8 bytes an element, and little beside them."""
    from vtl_b200.capi import Device
    dev = Device(0)
    M, N, K = 8192, 4096, 4096
    bufs = [dev.to_device(np.zeros(s, np.float32)) for s in ((M, K), (N, K), (M, N))]
    dev.sync()
    free = torch.cuda.mem_get_info()[0]
    dev.gemm_f32(False, True, M, N, K, *bufs)
    dev.sync()
    assert free - torch.cuda.mem_get_info()[0] < 1.25 * 8 * (M + N) * K
    for b in bufs:
        b.free()
    dev.close()


def test_time_of_a_product_that_f16_planes_cannot_hold(dev):
    """The profile brackets the launches of a product, whichever of them does the work."""
    M, N, K = 4096, 4096, 4096
    rng = np.random.default_rng(8)
    A = (rng.standard_normal((M, K)) * 10.0 ** rng.uniform(-9, 0, (M, K))).astype(np.float32)
    B = rng.standard_normal((N, K)).astype(np.float32)
    bufs = [dev.to_device(A), dev.to_device(B), dev.zeros((M, N))]
    dev.gemm_f32(False, True, M, N, K, *bufs)
    dev.sync()
    dev.profile_gemm(True)
    dev.gemm_f32(False, True, M, N, K, *bufs)
    ms, launches, ops = dev.profile_gemm_read()
    dev.profile_gemm(False)
    assert launches == 1 and ops == 2.0 * M * N * K
    assert ops / (ms * 1e-3) < 1.0e15  # three f16 products at 2.25 PFLOP/s are 0.75 of these
    for b in bufs:
        b.free()


def test_switch_that_keeps_products_on_single_ctas():
    """VTLB_F32_PAIR=0: two split passes and one product; else the f16 planes' two more launches."""
    import os
    import subprocess
    import sys
    code = """
import numpy as np
from vtl_b200.capi import Device
dev = Device(0)
bufs = [dev.zeros(s) for s in ((2048, 256), (2048, 256), (2048, 2048))]
n = dev.launch_count()
dev.gemm_f32(False, True, 2048, 2048, 256, *bufs)
dev.sync()
print(dev.launch_count() - n)
"""
    got = {}
    for pair in ("0", "1"):
        root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
        p = subprocess.run([sys.executable, "-c", code], cwd=root, env={**os.environ, "VTLB_F32_PAIR": pair},
                           capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stderr
        got[pair] = int(p.stdout)
    assert got == {"0": 3, "1": 5}
