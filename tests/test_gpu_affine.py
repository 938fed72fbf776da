"""The per-channel affine at the edges of how its launch is cut: fewer pixels than a thread takes, quarters that end inside the last
one, channel counts that end inside a vector, prefixes, slices, several images."""
import ctypes as C

import pytest

from paella_b200 import capi

pytestmark = pytest.mark.gpu


def _launch(kind, p, x, y):
    import torch
    L = capi.load()
    p.x, p.y = x.data_ptr(), y.data_ptr()
    capi.check(L.pb_op_launch(kind, C.byref(p), None, 0, None), "pb_op_launch")
    torch.cuda.synchronize()


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("shape", [
    # C, Cs of the input, H, W, images
    (8, 8, 1, 1, 1),          # one vector: three of a thread's four pixels do not exist
    (8, 16, 1, 3, 1),         # three pixels
    (40, 64, 5, 7, 3),        # a prefix; 105 pixels, a quarter is 27 (the last one 24)
    (61, 64, 9, 4, 1),        # channels end inside a vector
    (1024, 1024, 14, 14, 2),
])
def test_affine(shape, act, dtype):
    """One fused multiply-add and one rounding to the element type: 2^-8 (bf16) or 2^-23 relative."""
    import torch
    c, cs, h, w, n = shape
    dt, vec = (torch.bfloat16, 8) if dtype else (torch.float32, 4)
    gen = torch.Generator(device="cuda").manual_seed(c + h)
    x = torch.randn((n, h, w, cs), generator=gen, device="cuda").to(dt)
    scale, bias = torch.randn(c, generator=gen, device="cuda"), torch.randn(c, generator=gen, device="cuda")
    ks = (c + vec - 1) // vec * vec + 8
    y = torch.full((n, h, w, ks), 7.0, device="cuda", dtype=dt)
    p = capi.OpParams()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks, p.out_c_off = dtype, c, h, w, cs, c, h, w, ks, 8
    p.R, p.S, p.stride_h, p.stride_w, p.groups, p.batch, p.act = 1, 1, 1, 1, 1, n, act
    p.w, p.bias = scale.data_ptr(), bias.data_ptr()
    _launch(capi.STAGE_AFFINE, p, x, y)
    want = x[..., :c].double() * scale.double() + bias.double()
    want = torch.relu(want) if act else want
    got = y[..., 8:8 + c].double()
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** (-8 if dtype else -23) + 1e-30).all())
    assert bool((y[..., 8 + c:] == 0).all()) and bool((y[..., :8] == 7.0).all())
