"""How large the windows of a pooling launch are cut: for four blocks an SM (54 KB) or for three (74 KB), where each was measured faster (B200)."""
import ctypes as C

import pytest

from paella_b200 import capi

# kind, N, C, H, W, stride, pad: us with windows for three and for four blocks
MEASURED = [
    ("max", 97, 192, 56, 30, 2, 0, 8.30, 8.97), ("max", 292, 64, 56, 30, 2, 0, 8.29, 8.84), ("avg", 97, 192, 56, 30, 2, 0, 10.07, 10.65),
    ("max", 78, 192, 56, 30, 2, 0, 7.37, 7.00), ("avg", 234, 64, 56, 30, 2, 0, 8.95, 8.70),
    ("max", 182, 64, 24, 90, 2, 0, 8.45, 6.80), ("avg", 60, 192, 24, 90, 2, 0, 9.78, 8.22), ("max", 109, 192, 60, 20, 2, 0, 9.62, 8.44),
    ("max", 453, 192, 17, 17, 1, 1, 21.06, 17.91), ("avg", 83, 192, 28, 28, 1, 1, 12.44, 10.83), ("max", 160, 64, 35, 35, 1, 1, 9.69, 8.43),
]


@pytest.mark.parametrize("what,n,c,h,w,stride,pad,three,four", MEASURED)
def test_the_faster_one(what, n, c, h, w, stride, pad, three, four):
    p, li = capi.OpParams(), capi.LaunchInfo()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.Ks = 1, c, h, w, c, c, c
    p.P, p.Q = (h + 2 * pad - 3) // stride + 1, (w + 2 * pad - 3) // stride + 1
    p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.batch, p.flags = 3, 3, stride, stride, pad, pad, 1, n, 1
    capi.check(capi.load().pb_op_info(capi.STAGE_MAXPOOL if what == "max" else capi.STAGE_AVGPOOL, C.byref(p), C.byref(li)), "pb_op_info")
    assert (li.smem_per_block <= 54 * 1024) == (four < three)
