"""2 x 2 pooling at the edges of how its launch is cut: rows around a block's 512 vectors, odd maps whose last row and column are
dropped, channel counts that end inside a vector, several images, slices, NaN and infinities."""
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


POOL_CASES = [
    # C, H, W, images, out channels, slice offset
    (192 * 8, 2, 2, 1, 192 * 8, 0),      # one row of 192 vectors (bf16): the shortest this kernel takes
    (64, 9, 129, 2, 64, 0),              # 64 x 8 = 512 vectors, an odd map
    (72, 8, 130, 3, 96, 8),              # 65 x 9 = 585: a second block of 73
    (61, 6, 200, 1, 64, 0),              # channels end inside a vector
    (256, 28, 28, 2, 256, 0),
    (16, 4, 10, 1, 16, 0),               # short rows: the general kernel
]


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("op", ["max", "avg"])
@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("case", POOL_CASES)
def test_pool2(case, dtype, op, special):
    import torch
    c, h, w, n, total, off = case
    dt, vec = (torch.bfloat16, 8) if dtype else (torch.float32, 4)
    cs = (c + vec - 1) // vec * vec
    gen = torch.Generator(device="cuda").manual_seed(c + h)
    x = torch.zeros((n, h, w, cs), device="cuda", dtype=dt)
    x[..., :c] = torch.randn((n, h, w, c), generator=gen, device="cuda").to(dt)
    if special:
        pick = torch.rand((n, h, w, c), generator=gen, device="cuda")
        for lo, value in ((0.0, float("nan")), (0.2, float("inf")), (0.4, float("-inf")), (0.6, -0.0)):
            x[..., :c][(pick >= lo) & (pick < lo + 0.2)] = value
    P, Q = h // 2, w // 2
    bias, act = (torch.randn(c, generator=gen, device="cuda"), 1) if op == "avg" and not special else (None, 0)
    y = torch.full((n, P, Q, total), 7.0, device="cuda", dtype=dt)
    p = capi.OpParams()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks, p.out_c_off = dtype, c, h, w, cs, c, P, Q, total, off
    p.R, p.S, p.stride_h, p.stride_w, p.groups, p.batch, p.act = 2, 2, 2, 2, 1, n, act
    if bias is not None:
        p.bias = bias.data_ptr()
    _launch(capi.STAGE_MAXPOOL if op == "max" else capi.STAGE_AVGPOOL, p, x, y)
    v = x[:, :2 * P, :2 * Q, :c].float().view(n, P, 2, Q, 2, c)
    taps = [v[:, :, r, :, s] for r in range(2) for s in range(2)]
    want = torch.full_like(taps[0], float("-inf")) if op == "max" else torch.zeros_like(taps[0])
    if op == "max":
        for t in taps:                   # a maximum ignores NaN
            want = torch.where(t > want, t, want)
    else:                                # the columns of a row first
        want = (want + (taps[0] + taps[1]) + (taps[2] + taps[3])) / 4
        if bias is not None:
            want = torch.relu(want + bias)
    got = y[..., off:off + c]
    assert torch.equal(torch.nan_to_num(got.float(), nan=123.0), torch.nan_to_num(want.to(dt).float(), nan=123.0))
    pad = y[..., off + c:off + cs]
    assert bool((pad == 0).all())
    assert bool((y[..., :off] == 7.0).all()) and bool((y[..., off + cs:] == 7.0).all())
