"""The input stage in patch form: every output value is one input value (or zero) converted once, so the result is compared
bit for bit with torch's unfold, in both element types and on both sides of the tiled kernel's limits."""
import ctypes as C

import pytest

from paella_b200 import capi

pytestmark = pytest.mark.gpu

CASES = [
    # C, H, W, R, S, stride, pad, extra zero k, images
    (3, 224, 224, 7, 7, 2, 3, 0, 2),       # a stem of 147 values of k
    (3, 75, 61, 3, 3, 2, 0, 0, 3),         # 27 values: ragged tiles in both directions
    (1, 5, 3, 3, 3, 1, 1, 0, 1),           # a map smaller than a tile, 9 values: a vector with one value
    (3, 90, 300, 11, 5, 4, 2, 0, 1),       # windows of more than 96 columns: a second round of loads
    (4, 33, 65, 3, 3, 1, 1, 220, 1),       # 256 values of k, the most of the tiled kernel: vectors of zeros only
    (4, 20, 20, 9, 9, 1, 4, 0, 2),         # 324: past the tiled kernel
]


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("case", CASES)
def test_input_patches_are_the_unfolded_image(case, dtype):
    import torch
    L = capi.load()
    c, h, w, r, s, stride, pad, extra, n = case
    p_, q_ = (h + 2 * pad - r) // stride + 1, (w + 2 * pad - s) // stride + 1
    vec, dt = (8, torch.bfloat16) if dtype else (4, torch.float32)
    k = r * s * c
    ks = (k + extra + vec - 1) // vec * vec
    x = torch.randn((n, c, h, w), device="cuda")
    y = torch.full((n, p_, q_, ks), 7.0, device="cuda", dtype=dt)
    p = capi.OpParams()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks = dtype, c, h, w, c, k, p_, q_, ks
    p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.batch = r, s, stride, stride, pad, pad, 1, n
    p.x, p.y = x.data_ptr(), y.data_ptr()
    capi.check(L.pb_op_launch(capi.STAGE_INPUT, C.byref(p), None, 0, None), "pb_op_launch")
    torch.cuda.synchronize()
    cols = torch.nn.functional.unfold(x, (r, s), padding=pad, stride=stride)            # [n][(c, r, s)][pixels]
    want = torch.zeros((n, p_ * q_, ks), device="cuda")
    want[:, :, :k] = cols.view(n, c, r * s, -1).permute(0, 3, 2, 1).reshape(n, -1, k)   # k = (r, s, c)
    assert torch.equal(y.view(n, p_ * q_, ks), want.to(dt))
