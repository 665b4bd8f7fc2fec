"""The forward and backward-data convolutions with tiles of 4 and 8 image rows on
images wider than a tile: every quarter of the 128-pixel tile, the second and third
segment and the periodic wrap between them, for every kind of layer; small
integers, so the results equal the float64 oracle's.  And the weight gradient's
fp32 sums on Gaussian data at the size of a training batch."""
import ctypes

import numpy as np
import pytest

from test_learned_gpu import C, _bf, _conv, _ints

pytestmark = pytest.mark.gpu


def _tiles(shape, rows):
    b, h, w = shape
    return b * -(-h // rows) * -(-w // 128)


# (shape, rows a tile gets on 148 SMs: the fewest of 2, 4, 8 that leave every tile an SM)
SHAPES = [((5, 75, 129), 8), ((5, 67, 257), 8), ((3, 66, 129), 4), ((2, 61, 257), 4)]


@pytest.mark.parametrize("max_ctas", [0, 2])
@pytest.mark.parametrize("shape,rows", SHAPES)
def test_wide_images_at_every_tile_height(pmhd_lib, monkeypatch, shape, rows, max_ctas):
    assert _tiles(shape, rows // 2) > 148 and (rows == 8 or _tiles(shape, rows) <= 148)
    monkeypatch.setenv("PMHD_CONV_MAX_CTAS", str(max_ctas))
    rng = np.random.default_rng(31)
    x = _ints(rng, shape + (32,))
    b = rng.integers(-3, 4, 32).astype(np.float64)
    W = _ints(rng, (32, 9, 32), 0.2)
    z, _ = _conv(pmhd_lib, pmhd_lib.CONV_GELU, x, W, b, 32)
    np.testing.assert_array_equal(z, C.conv3x3(x, W, b))
    o, _ = _conv(pmhd_lib, pmhd_lib.CONV_LINEAR, x, W[:16], b[:16], 16)
    np.testing.assert_array_equal(o, C.conv3x3(x, W[:16], b[:16]))
    zp = _bf(rng.normal(0, 1.0, shape + (32,)))
    for cin in (16, 32):
        dz = _ints(rng, shape + (cin,))
        Wl = _ints(rng, (cin, 9, 32), 0.3)
        d, _ = _conv(pmhd_lib, pmhd_lib.CONV_DGELU, dz, np.ascontiguousarray(Wl.transpose(2, 1, 0)), None, 32, zprev=zp)
        ref = _bf((C.conv3x3_backward_input(dz, Wl) * C.gelu_grad(zp)).astype(np.float32))
        np.testing.assert_allclose(d, ref, rtol=2.0 ** -7, atol=0)  # gelu' in fp32: one bf16 ulp


@pytest.mark.parametrize("co", [16, 32])
def test_weight_gradient_sums_of_a_training_batch(pmhd_lib, co):
    """8 x 512^2 Gaussian data against binary64 sums.  A CTA's accumulator takes
    at most 28 tiles of 16 MMAs, 448 additions in fp32 that may truncate: each loses at
    most 2^-23 of the running sum, so a sum is off by less than 448 * 2^-23 = 5.4e-5
    of itself (all of one sign); the atomics and the bias sums (28 tiles of 8 rows a
    thread, then a tree) add less."""
    import torch

    B, H, W = 8, 512, 512
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn((B, H, W, 32), generator=g, device="cuda").to(torch.bfloat16)
    dz = torch.randn((B, H, W, co), generator=g, device="cuda").to(torch.bfloat16)
    dw, db = torch.zeros((co, 9, 32), device="cuda"), torch.zeros((co,), device="cuda")
    fp = ctypes.POINTER(ctypes.c_float)
    assert pmhd_lib.load().pmhd_conv3x3_wgrad(x.data_ptr(), dz.data_ptr(), B, H, W, 32, co, ctypes.cast(dw.data_ptr(), fp),
                                              ctypes.cast(db.data_ptr(), fp), None) == pmhd_lib.OK
    D = dz.double().reshape(-1, co)
    ref = torch.stack([D.T @ torch.roll(x.double(), (-dy, -dx), (1, 2)).reshape(-1, 32)
                       for dy in (-1, 0, 1) for dx in (-1, 0, 1)], 1)
    bound = 448 * 2.0 ** -23
    assert ((dw.double() - ref).norm() / ref.norm()).item() < bound
    assert ((db.double() - D.sum(0)).norm() / D.sum(0).norm()).item() < bound
