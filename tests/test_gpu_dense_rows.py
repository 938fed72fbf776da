"""The matrix-vector kernel at the row lengths where its steps of eight, four and one loads meet, against a float64 product.
A lane adds n / 32 products with fused multiply-adds, five levels of shuffles add the lanes and the bias comes last, each
rounding at most 2^-24 of what has been added so far: (n / 32 + 6) x 2^-24 x the sum of magnitudes (a lost product is
hundreds of times that)."""
import ctypes as C

import numpy as np
import pytest

from oracle import graph as og
from paella_b200 import capi
from tests import gpu_util as gu
from tests.test_gpu_ops import RNG, _params

pytestmark = pytest.mark.gpu


# a step is 256 bf16 or 128 fp32 elements of a row: below, at and above 4 and 8 of them, then several of each
@pytest.mark.parametrize("n_in", [8, 512, 1016, 1024, 1032, 2040, 2048, 2056, 5384])
@pytest.mark.parametrize("dtype", [0, 1])
def test_dense_row_lengths(dtype, n_in):
    import torch
    L = capi.load()
    k = 13                                                    # one full block and five warps of the next
    t = torch.float32 if dtype == 0 else torch.bfloat16
    rb = (lambda v: v) if dtype == 0 else og.round_bf16
    x, w = rb(RNG.standard_normal(n_in, dtype=np.float32)), rb(RNG.standard_normal((k, n_in), dtype=np.float32))
    b = RNG.standard_normal(k, dtype=np.float32)
    xd, wd, bd = torch.from_numpy(x).cuda().to(t), torch.from_numpy(w).cuda().to(t), torch.from_numpy(b).cuda()
    y = torch.full((k + 3,), 7.0, device="cuda")
    p = _params(dtype, (n_in, 1, 1), k, 1, 1, k, Cs=n_in)
    p.flags = 2                                               # fp32 results
    p.x, p.w, p.bias, p.y = xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), y.data_ptr()
    capi.check(L.pb_op_launch(capi.STAGE_DENSE, C.byref(p), None, 0, None), "dense")
    gu.sync()
    got = y.cpu().numpy()
    ref = w.astype(np.float64) @ x.astype(np.float64) + b
    size = np.abs(w).astype(np.float64) @ np.abs(x).astype(np.float64) + np.abs(b)
    assert (np.abs(got[:k] - ref) <= (np.ceil(n_in / 32) + 6) * 2.0 ** -24 * size).all()
    assert (got[k:] == 7.0).all()
