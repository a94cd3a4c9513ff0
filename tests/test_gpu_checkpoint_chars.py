"""Every byte in every place of a base64 group: accepted with its value, or refused."""
import base64

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ALPHABET = b"ABCDEFGHIJKLMNOPQRSTUVWXYZabcdefghijklmnopqrstuvwxyz0123456789+/"


@pytest.mark.parametrize("place", [0, 1, 2, 3, 18, 31])
def test_every_byte(dev, place):
    from vtl_b200 import capi
    good = np.frombuffer(base64.b64encode(np.arange(1.0, 97.0).astype(">f8").tobytes()), np.uint8)  # one warp's values
    dst = dev.empty(96)
    for byte in range(256):
        text = good.copy()
        text[5 * 32 + place] = byte
        d = dev.to_device(text)
        if byte in ALPHABET:
            dev.ckpt_decode_f32(d, text.size, dst, 96)
            ref = np.frombuffer(base64.b64decode(text.tobytes()), ">f8")
            with np.errstate(over="ignore", invalid="ignore"):
                ref = ref.astype(np.float32)
            got = dst.numpy()
            assert np.array_equal(got.view(np.uint32)[~np.isnan(ref)], ref.view(np.uint32)[~np.isnan(ref)])
            assert np.array_equal(np.isnan(got), np.isnan(ref))
        else:
            with pytest.raises(capi.VtlbError):
                dev.ckpt_decode_f32(d, text.size, dst, 96)
        d.free()
    dst.free()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 95, 96, 97, 98, 767, 768, 769, 100003])
def test_ends_of_warps_and_grids(dev, n):
    x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    text = np.frombuffer(base64.b64encode(x.astype(">f8").tobytes()), np.uint8)
    dt, dst = dev.to_device(text), dev.to_device(np.full(n + 64, 5.0, np.float32))
    dev.ckpt_decode_f32(dt, text.size, dst, n)
    got = dst.numpy()
    assert np.array_equal(got[:n].view(np.uint32), x.view(np.uint32)) and (got[n:] == 5.0).all()
    dt.free()
    dst.free()
