"""3x3 depthwise convolutions of stride 1 whose rows are shared out over a fixed number of blocks, the window in a ring of
rows: ranges that begin and end anywhere in a map, maps narrower and shorter than a range, widths around a strip and a column tile,
channel counts off the slab and off the vector, a slice on a 4-byte boundary, values that are not finite.
Bit for bit the strip kernels (PB_WINDOW_TILE=0) on the same launch."""
import ctypes as C

import numpy as np
import pytest

from paella_b200 import capi
from tests import gpu_util as gu
from tests.test_gpu_ops import _params

pytestmark = pytest.mark.gpu

CASES = [
    # N, C, H, W, pad             (rows of all units: at least 24 for each of 444 blocks)
    (130, 136, 30, 31, 1),        # three slabs, the last one of eight channels; 24 to 27 rows a block: most ranges cross a map's end
    (60, 24, 200, 25, 1),         # seven strips, one column of the last
    (100, 64, 110, 34, 0),        # no padding: 32 columns
    (1, 200, 600, 300, 1),        # one image, ten column tiles, four slabs
    (600, 16, 19, 27, 1),         # more maps than blocks
    (1400, 8, 9, 32, 1),          # a range holds several maps
    (90, 67, 64, 58, 1),          # channels past the last vector are stored as zeros; the second tile hangs over the edge
]


@pytest.mark.parametrize("case", CASES)
def test_ring_equals_the_strip_kernels(case, monkeypatch):
    import torch
    L, kind = capi.load(), capi.STAGE_DWCONV
    nb, c, h, w, pad = case
    P, Q = h + 2 * pad - 2, w + 2 * pad - 2
    gen = torch.Generator(device="cuda").manual_seed(c * 1000 + h)
    cs = gu.round_up(c, 8)
    x = torch.zeros((nb, h, w, cs), device="cuda", dtype=torch.bfloat16)
    x[..., :c] = torch.randn((nb, h, w, c), generator=gen, device="cuda").to(torch.bfloat16)
    x[0, 1, 2, 3], x[-1, -1, -1, 1], x[nb // 2, h // 2, 0, 0] = float("inf"), float("nan"), -float("inf")
    wt = np.random.default_rng(c).standard_normal((c, 1, 3, 3), dtype=np.float32)
    bd = torch.randn(c, generator=gen, device="cuda")
    for act, bias in ((2, True), (0, False), (1, True)):
        for moved in (0, 4):                       # bytes
            p = _params(1, (c, h, w), c, P, Q, cs + 16, 3, 3, 1, 1, pad, pad, groups=c, act=act, out_c_off=8, Cs=cs)
            wd = gu.pack_weights(kind, p, wt)
            p.batch, p.x, p.w, p.bias = nb, x.data_ptr(), wd.data_ptr(), bd.data_ptr() if bias else None
            outs, infos = [], []
            for tile in ("1", "0"):
                if moved and tile == "0":
                    continue
                monkeypatch.setenv("PB_WINDOW_TILE", tile)
                y = torch.full((nb * P * Q * (cs + 16) + 8,), 3.0, device="cuda", dtype=torch.bfloat16)
                p.y = y.data_ptr() + moved
                li = capi.LaunchInfo()
                capi.check(L.pb_op_info(kind, C.byref(p), C.byref(li)), "pb_op_info")
                infos.append((li.num_blocks, li.threads_per_block))
                capi.check(L.pb_op_launch(kind, C.byref(p), None, 0, None), "pb_op_launch")
                gu.sync()
                assert gu.error_flag() == 0
                outs.append(y[moved // 2: moved // 2 + nb * P * Q * (cs + 16)].view(nb, P, Q, cs + 16).view(torch.int16))
            assert infos[0][0] == 444 // -(-cs // 64) * -(-cs // 64) and infos[0][1] <= 160 and (moved or infos[1][1] == 256)
            if not moved:
                ref = outs[1]
            same = outs[0] == ref
            if not bool(same.all()):               # NaN may carry other bits
                a, b = outs[0].view(torch.bfloat16)[~same], ref.view(torch.bfloat16)[~same]
                assert bool(torch.isnan(a).all()) and bool(torch.isnan(b).all()), (act, bias, moved, int((~same).sum()))
