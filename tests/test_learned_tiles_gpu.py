"""The tiled convolution kernels (pmhd_conv3x3, pmhd_conv3x3_wgrad) at the
edges of their tiles -- 2, 4 or 8 x 128 pixels forward and backward, 8 x 64 for
the weight gradient -- against the float64 oracle: small integers, so every product
and partial sum is exact in the fp32 accumulators and the results are equal."""
import ctypes

import numpy as np
import pytest

from test_learned_gpu import C, _bf, _conv, _ints, _wgrad

pytestmark = pytest.mark.gpu

# One pixel; one less than, at and one more than a tile in each direction;
# narrower than a halo; several segments; images that take tiles of 4 and 8 rows
# (more than 148 of the next smaller ones).
SHAPES = [(1, 1, 1), (1, 2, 3), (2, 7, 63), (1, 9, 65), (1, 8, 127), (1, 15, 129), (1, 17, 64), (2, 8, 257), (8, 39, 65), (20, 33, 20)]


@pytest.mark.parametrize("max_ctas", [0, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_forward_and_backward_data_at_tile_edges(pmhd_lib, monkeypatch, shape, max_ctas):
    monkeypatch.setenv("PMHD_CONV_MAX_CTAS", str(max_ctas))
    rng = np.random.default_rng(3)
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


@pytest.mark.parametrize("max_ctas", [0, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_weight_gradient_at_tile_edges(pmhd_lib, monkeypatch, shape, max_ctas):
    monkeypatch.setenv("PMHD_CONV_MAX_CTAS", str(max_ctas))
    rng = np.random.default_rng(4)
    x = _ints(rng, shape + (32,))
    for co in (16, 32):
        dz = _ints(rng, shape + (co,))
        dw, db = _wgrad(pmhd_lib, x, dz)
        dwr, dbr = C.conv3x3_backward_weight(x, dz)
        np.testing.assert_array_equal(dw, dwr)
        np.testing.assert_array_equal(db, dbr)


@pytest.mark.parametrize("offset", [0, 8])
def test_outputs_aligned_to_16_bytes_only(pmhd_lib, offset):
    """Outputs and z_prev 16 but not 32 bytes aligned take the 16-byte accesses."""
    import torch

    rng = np.random.default_rng(5)
    shape = (1, 9, 130)
    n = int(np.prod(shape)) * 32
    x = _ints(rng, shape + (32,))
    W = _ints(rng, (32, 9, 32), 0.2)
    xd = torch.from_numpy(x.astype(np.float32)).to(torch.bfloat16).cuda()
    wd = torch.from_numpy(W.astype(np.float32)).to(torch.bfloat16).cuda()
    bd = torch.zeros(32, device="cuda")
    bufs = [torch.zeros(n + 16, dtype=torch.bfloat16, device="cuda")[offset:offset + n] for _ in range(3)]
    L = pmhd_lib.load()
    fp = ctypes.POINTER(ctypes.c_float)
    assert L.pmhd_conv3x3(pmhd_lib.CONV_GELU, xd.data_ptr(), *shape, 32, wd.data_ptr(), ctypes.cast(bd.data_ptr(), fp),
                          32, None, bufs[0].data_ptr(), bufs[1].data_ptr(), None) == pmhd_lib.OK
    z = bufs[0].float().cpu().numpy().reshape(shape + (32,))
    np.testing.assert_array_equal(z, C.conv3x3(x, W, np.zeros(32)))
    assert L.pmhd_conv3x3(pmhd_lib.CONV_DGELU, xd.data_ptr(), *shape, 32, wd.data_ptr(), None, 32, bufs[0].data_ptr(),
                          bufs[2].data_ptr(), None, None) == pmhd_lib.OK
    d = bufs[2].float().cpu().numpy().reshape(shape + (32,))
    da = C.conv3x3_backward_input(x, np.ascontiguousarray(W.transpose(2, 1, 0)))
    np.testing.assert_allclose(d, _bf((da * C.gelu_grad(z)).astype(np.float32)), rtol=2.0 ** -7, atol=0)
