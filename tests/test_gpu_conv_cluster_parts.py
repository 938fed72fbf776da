"""Split reductions of the tensor-core convolution: the parts that the ranks of a cluster send each other, beside the pipeline and in its
buffers, at two, four and eight ranks and every width a part can have (8 to 64 columns), launch after launch.

Reference: the convolution of the bf16 operands in 64 bits.  n products of bf16 values, exact in fp32, summed in fp32 in any order differ
from the exact sum by at most n * 2^-23 * sum|products| (every addition truncating); the result is rounded to bf16 once."""
import ctypes as C

import pytest

from paella_b200 import capi
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

CASES = [
    # N, C, H, K, R                     columns of a tile, ranks (as chosen when this was written)
    (1, 64, 14, 16, 3),             # 16, 2: the narrowest part
    (2, 128, 28, 256, 3),           # 64, 2
    (8, 256, 17, 256, 3),           # 96, 2
    (8, 256, 17, 384, 3),           # 128, 2: the widest part, in the pipeline's buffers
    (2, 256, 28, 512, 3),           # 112, 2
    (1, 64, 7, 16, 3),              # 32, 4: 49 rows
    (1, 256, 28, 384, 3),           # 96, 4: parts of 24 columns, in the buffers
    (1, 256, 28, 512, 3),           # 128, 4: in the buffers
    (8, 256, 14, 256, 3),           # 128, 4: tiles straddle images
    (1, 256, 7, 64, 3),             # 64, 8
    (1, 128, 17, 512, 3),           # 64, 4 or 128, 8
    (1, 520, 8, 72, 3),             # channels and columns past whole boxes and tiles
]


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("case", CASES)
def test_parts(case, residual):
    import torch
    L = capi.load()
    n, c, h, k, r = case
    gen = torch.Generator(device="cuda").manual_seed(c + k)
    rnd = lambda *s: torch.randn(s, generator=gen, device="cuda")
    x, res, b = rnd(n, h, h, c).relu().to(torch.bfloat16), rnd(n, h, h, k).to(torch.bfloat16), rnd(k) * 0.1
    w = (rnd(k, c, r, r) * (2.0 / (c * r * r)) ** 0.5).to(torch.bfloat16)
    p = capi.OpParams()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks = 1, c, h, h, c, k, h, h, k
    p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.act, p.batch = r, r, 1, 1, r // 2, r // 2, 1, 1, n
    wd, scratch = gu.pack_weights(capi.STAGE_CONV_UMMA, p, w.float().cpu().numpy()), torch.zeros(4096, dtype=torch.uint8, device="cuda")
    ys = torch.full((6, n, h, h, k), 7.0, dtype=torch.bfloat16, device="cuda")
    p.x, p.w, p.bias, p.scratch, p.scratch_bytes = x.data_ptr(), wd.data_ptr(), b.data_ptr(), scratch.data_ptr(), 4096
    if residual:
        p.residual, p.res_Cs = res.data_ptr(), k
    p.y = ys.data_ptr()
    li = capi.LaunchInfo()
    capi.check(L.pb_op_info(capi.STAGE_CONV_UMMA, C.byref(p), C.byref(li)), "pb_op_info")
    assert li.scratch_bytes > 0                       # it does split
    for y in ys:                                      # back to back: a block's memory is the next one's
        p.y = y.data_ptr()
        capi.check(L.pb_op_launch(capi.STAGE_CONV_UMMA, C.byref(p), None, 0, None), "pb_op_launch")
    gu.sync()
    assert gu.error_flag() == 0
    for y in ys[1:]:
        assert torch.equal(y, ys[0])
    conv = lambda a, b2: torch.nn.functional.conv2d(a.permute(0, 3, 1, 2).double(), b2.double(), None, 1, r // 2).permute(0, 2, 3, 1)
    ref, mass = conv(x, w) + b.double(), conv(x.abs(), w.abs())
    if residual:
        ref = ref + res.double()
    ref = ref.relu()
    assert ((ys[0].double() - ref).abs() <= (c * r * r + 4) * 2.0 ** -23 * (mass + ref) + 2.0 ** -8 * ref).all()
