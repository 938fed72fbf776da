"""The tiled 3x3 window kernel on batches, whose tiles are fitted to the map: widths and heights around a strip, a band and a
tile, channel counts off the slab and off the vector, pooling with the bias + activation tail.  Bit for bit the strip kernels
(PB_WINDOW_TILE=0) on the same launch."""
import ctypes as C

import numpy as np
import pytest

from paella_b200 import capi
from tests import gpu_util as gu
from tests.test_gpu_ops import _params

pytestmark = pytest.mark.gpu

CASES = [
    # N, C, H, W, stride, pad
    (2, 64, 35, 35, 1, 1), (3, 72, 17, 17, 1, 1), (2, 8, 8, 8, 1, 1), (2, 200, 4, 3, 1, 1), (2, 64, 41, 81, 1, 1), (2, 128, 14, 1, 1, 1),
    (2, 64, 71, 71, 2, 0), (3, 40, 35, 36, 2, 1), (2, 64, 7, 7, 2, 1), (2, 24, 3, 90, 2, 1), (2, 16, 64, 40, 1, 0),
    # channels past the last vector (stored as zeros): one, two and three of four missing, past a slab
    (2, 20, 9, 10, 1, 1), (3, 69, 17, 17, 1, 1), (2, 131, 12, 40, 1, 1), (2, 67, 15, 15, 2, 1), (1, 133, 40, 33, 1, 1),
]


@pytest.mark.parametrize("case", CASES)
def test_tiles_of_a_batch_equal_the_strip_kernels(case, monkeypatch):
    import torch
    L = capi.load()
    nb, c, h, w, st, pad = case
    P, Q = (h + 2 * pad - 3) // st + 1, (w + 2 * pad - 3) // st + 1
    if P < 1 or Q < 1:
        pytest.skip("no output")
    gen = torch.Generator(device="cuda").manual_seed(c * 1000 + h)
    cs = gu.round_up(c, 8)
    x = torch.zeros((nb, h, w, cs), device="cuda", dtype=torch.bfloat16)
    x[..., :c] = torch.randn((nb, h, w, c), generator=gen, device="cuda").to(torch.bfloat16)
    wt = np.random.default_rng(c).standard_normal((c, 1, 3, 3), dtype=np.float32)
    bd = torch.randn(c, generator=gen, device="cuda")
    for kind, flags, act, bias in ((capi.STAGE_DWCONV, 0, 2, True), (capi.STAGE_DWCONV, 0, 0, False), (capi.STAGE_MAXPOOL, 0, 0, False),
                                   (capi.STAGE_AVGPOOL, 1, 0, False), (capi.STAGE_AVGPOOL, 0, 0, False), (capi.STAGE_AVGPOOL, 1, 1, True),
                                   (capi.STAGE_MAXPOOL, 0, 1, True)):
        p = _params(1, (c, h, w), c, P, Q, cs + 16, 3, 3, st, st, pad, pad, groups=c if kind == capi.STAGE_DWCONV else 1, act=act, flags=flags,
                    out_c_off=8, Cs=cs)
        p.batch = nb
        if kind == capi.STAGE_DWCONV:
            wd = gu.pack_weights(kind, p, wt)
            p.w = wd.data_ptr()
        p.x, p.bias = x.data_ptr(), bd.data_ptr() if bias else None
        outs, blocks = [], []
        for tile in ("1", "0"):
            monkeypatch.setenv("PB_WINDOW_TILE", tile)
            monkeypatch.setenv("PB_WINDOW_TILE_MIN_BLOCKS", "1")
            y = torch.full((nb, P, Q, cs + 16), 3.0, device="cuda", dtype=torch.bfloat16)
            p.y = y.data_ptr()
            li = capi.LaunchInfo()
            capi.check(L.pb_op_info(kind, C.byref(p), C.byref(li)), "pb_op_info")
            blocks.append(li.threads_per_block)
            capi.check(L.pb_op_launch(kind, C.byref(p), None, 0, None), "pb_op_launch")
            gu.sync()
            outs.append(y.float().cpu().numpy())
        assert blocks[0] <= 160 and blocks[1] == 256
        np.testing.assert_array_equal(outs[0], outs[1], err_msg=str((kind, flags, act, bias)))
        assert (outs[0][..., :8] == 3.0).all() and (outs[0][..., 8 + cs:] == 3.0).all() and (outs[0][..., 8 + c: 8 + cs] == 0.0).all()
