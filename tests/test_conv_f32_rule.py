"""Which fp32 layers of up to 32 output channels run on the tensor cores: on either side of the line the faster of the two measured times."""
import ctypes as C

import pytest

from paella_b200 import capi

# N, C, H = W, K, R, S: us a launch in a chain on the fp32 units, on the tensor cores (B200)
MEASURED = [
    (2, 128, 56, 32, 3, 3, 31.3, 11.8), (1, 256, 112, 24, 3, 3, 76.7, 30.2), (1, 64, 112, 24, 1, 7, 20.9, 10.2), (8, 512, 56, 16, 1, 7, 142.8, 72.9),
    (1, 256, 112, 8, 1, 7, 48.4, 25.4), (2, 96, 112, 8, 5, 5, 99.7, 55.0), (8, 512, 14, 8, 5, 5, 39.7, 23.5), (2, 32, 56, 16, 5, 5, 16.1, 10.2),
    (2, 48, 112, 24, 3, 3, 32.8, 21.9), (8, 32, 56, 32, 3, 3, 22.6, 15.7), (8, 512, 14, 16, 1, 7, 15.1, 10.9), (2, 32, 56, 32, 3, 3, 9.6, 7.2),
    (8, 48, 112, 8, 3, 3, 83.1, 64.2), (1, 96, 56, 8, 3, 3, 10.1, 8.4), (8, 96, 7, 32, 5, 5, 10.6, 9.2), (1, 48, 14, 8, 1, 7, 8.8, 7.9),
    (1, 48, 56, 16, 1, 7, 8.9, 8.1), (1, 256, 28, 8, 3, 3, 8.6, 9.3), (1, 64, 28, 8, 5, 5, 7.6, 8.4), (1, 64, 7, 16, 5, 5, 7.2, 8.4),
    (1, 96, 14, 32, 3, 3, 6.9, 8.1), (2, 48, 7, 24, 3, 3, 6.1, 7.4), (1, 64, 28, 32, 3, 3, 6.1, 7.5), (1, 96, 14, 16, 3, 3, 6.4, 8.1),
]


@pytest.mark.parametrize("n,c,h,k,r,s,units,split", MEASURED)
def test_the_faster_one(n, c, h, k, r, s, units, split):
    p, li = capi.OpParams(), capi.LaunchInfo()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks = 0, c, h, h, c, k, h, h, k
    p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.batch = r, s, 1, 1, r // 2, s // 2, 1, n
    capi.check(capi.load().pb_op_info(capi.STAGE_CONV_SIMT, C.byref(p), C.byref(li)), "pb_op_info")
    assert li.threads_per_block == (832 if split < units else 256)
