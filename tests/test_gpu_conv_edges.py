"""Convolution against 64-bit sums (torch on the CPU) where its kernels change over."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bound(terms, a, b):
    # three TF32 products per f32 product leave 2^-21 of each term, sums of `terms` of them round to f32
    return 1e-5 * np.sqrt(terms) * float(np.abs(a).max()) * float(np.abs(b).max())


def _check(dev, B, C, H, W, O, k, pad, stride, relu=True, bias=True):
    rng = np.random.default_rng(B + 10 * C + 100 * H + O + k)
    x = rng.standard_normal((B, C, H, W)).astype(np.float32)
    w = (rng.standard_normal((O, C, k, k)) * (2.0 / (C * k * k)) ** 0.5).astype(np.float32)
    b = rng.standard_normal(O).astype(np.float32) if bias else None
    t = lambda a: torch.from_numpy(a).double()  # noqa: E731
    pre = torch.nn.functional.conv2d(t(x), t(w), t(b) if bias else None, stride, pad).numpy()
    OH, OW = pre.shape[2:]
    g = rng.standard_normal(pre.shape).astype(np.float32)
    rdx = torch.nn.grad.conv2d_input(x.shape, t(w), t(g), stride, pad).numpy()
    rdw = torch.nn.grad.conv2d_weight(t(x), w.shape, t(g), stride, pad).numpy()
    rdb = g.astype(np.float64).sum(axis=(0, 2, 3))
    d = [dev.to_device(a) for a in (x, w, g)]
    db_in = dev.to_device(b) if bias else None
    out = [dev.to_device(np.full(s, np.nan, np.float32)) for s in (pre.shape, pre.shape, x.shape, w.shape, (O,))]
    dims = (B, C, H, W, O, k, k, pad, pad, stride, stride)
    dev.conv2d_fwd_f32(d[0], d[1], db_in, out[0], *dims, relu, out[1])
    dev.conv2d_bwd_f32(d[2], d[0], d[1], out[2], out[3], out[4], *dims)
    assert dev.check_status() == 0
    y, p, dx, dw, db = (o.numpy() for o in out)
    fwd = _bound(C * k * k, x, w) + (2e-7 * np.abs(b).max() if bias else 0)
    assert np.abs(p - pre).max() <= fwd
    assert np.array_equal(y, np.where(p < 0, np.float32(0), p) if relu else p)
    assert np.abs(dx - rdx).max() <= _bound(O * k * k, g, w)
    assert np.abs(dw - rdw).max() <= _bound(B * OH * OW, g, x)
    assert np.abs(db - rdb).max() <= 1e-6 * max(1.0, np.abs(g).sum(axis=(0, 2, 3)).max())
    for o in d + out + ([db_in] if bias else []):
        o.free()


@pytest.mark.parametrize("B,C,H,W,O,k,pad,stride", [
    (2, 3, 11, 14, 5, 3, 0, 2), (3, 4, 12, 9, 6, 3, 1, 2), (1, 2, 7, 7, 3, 3, 2, 2),   # window rows and columns left over
    (2, 5, 15, 16, 4, 5, 2, 2), (1, 1, 5, 5, 2, 5, 0, 2), (2, 3, 13, 40, 9, 5, 1, 2),
    (2, 3, 10, 11, 4, 4, 1, 2), (2, 3, 11, 10, 4, 3, 1, 3), (2, 6, 9, 9, 7, 1, 0, 2),  # any window, any stride
])
def test_strided_windows(dev, B, C, H, W, O, k, pad, stride):
    _check(dev, B, C, H, W, O, k, pad, stride)


@pytest.mark.parametrize("B,C,H,W,O,k,pad", [
    (1, 1, 5, 5, 1, 5, 0), (65, 1, 28, 28, 8, 3, 1),              # one pixel; more images than a wave
    (3, 3, 9, 7, 5, 3, 0), (2, 2, 13, 11, 9, 5, 2), (2, 4, 6, 6, 13, 1, 0),   # nothing divides
    (2, 3, 8, 126, 12, 3, 2), (1, 2, 3, 127, 6, 3, 2), (1, 3, 4, 300, 4, 3, 1),  # rows of 128, 129 and 300 outputs
    (4, 2, 7, 9, 6, 3, 3), (2, 3, 6, 5, 4, 1, 2), (2, 1, 4, 4, 3, 5, 6),      # more padding than the window covers
    (16, 8, 28, 28, 16, 5, 0), (2, 64, 14, 14, 3, 5, 2), (2, 70, 5, 5, 2, 5, 0),  # slices and stages of channels
    (50, 20, 12, 12, 50, 5, 0), (16, 3, 32, 32, 33, 3, 1),        # CTAs that share the channels
])
@pytest.mark.parametrize("relu,bias", [(True, True), (False, False)])
def test_small_products_on_cuda_cores(dev, B, C, H, W, O, k, pad, relu, bias):
    _check(dev, B, C, H, W, O, k, pad, 1, relu, bias)


@pytest.mark.parametrize("B,C,H,O,k,pad", [
    (300, 3, 8, 512, 5, 0), (300, 3, 3, 2048, 3, 0), (512, 3, 4, 512, 5, 2), (320, 64, 1, 2048, 3, 1),   # forward
    (512, 512, 4, 3, 5, 2), (320, 2048, 1, 64, 3, 1),                                                    # input gradient
])
def test_many_channels_on_tiny_planes(dev, B, C, H, O, k, pad):
    """The weights of all the channels that a CTA's threads could hold are more than a stage of shared memory."""
    _check(dev, B, C, H, H, O, k, pad, 1)


# layer, and whether forward and input gradient may run on CUDA cores (a sum has at most 1600 terms there)
FORCED = [
    ((1, 1, 5, 5, 1, 5, 0), True, True), ((3, 3, 9, 7, 5, 3, 0), True, True), ((2, 2, 13, 11, 9, 5, 2), True, True),
    ((2, 4, 6, 6, 13, 1, 0), True, True), ((2, 3, 8, 126, 12, 3, 2), True, True), ((1, 2, 3, 127, 6, 3, 2), False, True),
    ((2, 3, 6, 5, 4, 1, 2), True, True), ((2, 1, 4, 4, 3, 5, 6), True, True), ((2, 64, 5, 5, 2, 5, 0), True, True),
    ((2, 65, 5, 5, 2, 5, 0), False, True), ((16, 64, 14, 14, 80, 3, 1), True, True), ((40, 96, 28, 28, 70, 1, 0), True, True),
]


def forced(dev):
    """Every layer of FORCED on the CUDA-core kernels (VTLB_CONV_DIRECT=2), which are one launch forward, one for the
    input gradient; the tensor-core kernels have one more, which regroups the weights."""
    for (B, C, H, W, O, k, pad), fwd, dx in FORCED:
        _check(dev, B, C, H, W, O, k, pad, 1)
        OH, OW = H + 2 * pad - k + 1, W + 2 * pad - k + 1
        bufs = [dev.zeros(s) for s in ((B, C, H, W), (O, C, k, k), (B, O, OH, OW))]
        dims = (B, C, H, W, O, k, k, pad, pad, 1, 1)
        n = dev.launch_count()
        dev.conv2d_fwd_f32(bufs[0], bufs[1], None, bufs[2], *dims)
        assert (dev.launch_count() - n == 1) == fwd, (B, C, H, W, O, k, pad)
        n = dev.launch_count()
        dev.conv2d_bwd_f32(bufs[2], bufs[0], bufs[1], bufs[0], None, None, *dims)
        assert (dev.launch_count() - n == 1) == dx, (B, C, H, W, O, k, pad)
        for b in bufs:
            b.free()


def test_every_window_on_cuda_cores():
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = ("import sys; sys.path.insert(0, 'tests'); import test_gpu_conv_edges as t; from vtl_b200.capi import Device; "
            "d = Device(0); t.forced(d); d.close()")
    p = subprocess.run([sys.executable, "-c", code], cwd=root, env={**os.environ, "VTLB_CONV_DIRECT": "2"},
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]


@pytest.mark.parametrize("layer,direct", [
    ((256, 3, 32, 32, 32, 3, 1), True), ((50, 1, 28, 28, 20, 5, 0), True), ((2, 4, 6, 6, 13, 1, 0), True),
    ((50, 104, 18, 18, 214, 1, 0), False), ((31, 107, 28, 28, 189, 1, 0), False), ((125, 31, 14, 14, 54, 1, 0), False),
    ((256, 32, 32, 32, 64, 3, 1), False),
])
def test_which_kernel_runs_forward(dev, layer, direct):
    """1 x 1 layers that took up to three times as long on CUDA cores; first layers that take half as long there."""
    B, C, H, W, O, k, pad = layer
    bufs = [dev.zeros(s) for s in ((B, C, H, W), (O, C, k, k), (B, O, H + 2 * pad - k + 1, W + 2 * pad - k + 1))]
    n = dev.launch_count()
    dev.conv2d_fwd_f32(bufs[0], bufs[1], None, bufs[2], B, C, H, W, O, k, k, pad, pad, 1, 1)
    assert (dev.launch_count() - n == 1) == direct
    for b in bufs:
        b.free()


@pytest.mark.parametrize("B,C,H,W,O,k,pad", [
    (2, 3, 11, 10, 4, 7, 3), (1, 2, 9, 8, 3, 7, 0), (2, 1, 7, 20, 5, 7, 6),   # 49 taps: more than the gathered kernel takes
    (1, 2, 6, 7, 260, 3, 1), (2, 5, 5, 4, 90, 5, 2),                          # more (channel, tap) pairs than it takes
])
def test_unit_stride_on_the_lowered_route(dev, B, C, H, W, O, k, pad):
    _check(dev, B, C, H, W, O, k, pad, 1)
