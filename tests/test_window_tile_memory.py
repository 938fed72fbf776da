"""The shared memory the tiled 3x3 window kernel asks for: three blocks have to fit an SM (228 KB, of which each block costs 1 KB
of its own), whatever the map of a batch."""
import ctypes as C

import pytest

from paella_b200 import capi


@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("batch", [1, 2])
def test_three_blocks_fit_an_sm(monkeypatch, batch, stride):
    monkeypatch.setenv("PB_WINDOW_TILE_MIN_BLOCKS", "1")
    L = capi.load()
    li = capi.LaunchInfo()
    for h in list(range(1, 50)) + [56, 71, 112, 149, 300]:
        for w in list(range(1, 50)) + [56, 71, 79, 80, 81, 112, 121, 149, 300]:
            p = capi.OpParams()
            p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.Ks = 1, 64, h, w, 64, 64, 64
            p.P, p.Q = (h - 1) // stride + 1, (w - 1) // stride + 1
            p.R = p.S = 3
            p.stride_h = p.stride_w = stride
            p.pad_h, p.pad_w, p.groups, p.batch = 1, 1, 1, batch
            capi.check(L.pb_op_info(capi.STAGE_MAXPOOL, C.byref(p), C.byref(li)), "pb_op_info")
            assert li.threads_per_block <= 160 and 3 * (li.smem_per_block + 1024) <= 228 * 1024, (h, w, li.smem_per_block)
            rows = li.num_blocks // batch
            assert 1 <= rows <= h * w
