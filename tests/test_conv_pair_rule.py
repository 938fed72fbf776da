"""Which large convolutions run on pairs of blocks, by what pb_op_info declares: the pair kernel holds half of a tile's weights per block,
so its shared memory or its even number of row tiles tells it from a launch of lone blocks (not with 256 columns and an even
number)."""
import ctypes as C

import pytest

from paella_b200 import capi


def _info(monkeypatch, mode, c, k, r, row_tiles, scratch=True):
    monkeypatch.setenv("PB_CONV_PAIR", mode)
    p, li = capi.OpParams(), capi.LaunchInfo()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks = 1, c, 8, 16, c, k, 8, 16, k      # 128 pixels an image
    p.R = p.S = r
    p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.batch = 1, 1, r // 2, r // 2, 1, row_tiles
    p.x = p.y = p.w = 4096
    if scratch:
        p.scratch, p.scratch_bytes = 4096, 1 << 20
    capi.check(capi.load().pb_op_info(capi.STAGE_CONV_UMMA, C.byref(p), C.byref(li)), "pb_op_info")
    return li.num_blocks, li.smem_per_block, li.scratch_bytes


@pytest.mark.parametrize("pair, c, k, r, row_tiles", [
    (False, 256, 224, 3, 94), (True, 256, 224, 3, 95),           # 48 pairs
    (True, 256, 224, 3, 148), (False, 256, 224, 3, 149),         # 74 pairs
    (False, 256, 224, 3, 278), (True, 256, 224, 3, 279),         # 140 pairs
    (True, 256, 224, 3, 300), (True, 256, 224, 3, 390),          # 150 and 195: a second wave of few pairs, and of few lone blocks
    (False, 960, 224, 1, 100), (True, 1024, 224, 1, 100),        # 16 k-blocks
    (False, 256, 160, 3, 100), (True, 256, 168, 3, 100),         # 192 columns
    (False, 512, 384, 3, 49), (True, 512, 384, 3, 50),           # 147 lone blocks of 128 columns; 150 do not fit a round
    (False, 192, 512, 3, 49), (True, 256, 512, 3, 49),           # 147 of 176 columns against 256: from 36 k-blocks on
    (False, 512, 576, 3, 37), (True, 512, 576, 3, 39),
    (True, 1024, 1024, 1, 27), (False, 1024, 1024, 1, 24),       # five tiles of 208 columns; six of 176
    (False, 512, 768, 3, 197), (True, 512, 768, 3, 199),         # 297 pairs of which the last are half empty
    (True, 512, 768, 3, 345),
    (False, 256, 640, 3, 99), (True, 512, 640, 3, 99), (True, 256, 576, 3, 99), (False, 256, 768, 3, 99),
    (True, 288, 384, 3, 613),
])
def test_which_launches_are_pairs(monkeypatch, pair, c, k, r, row_tiles):
    lone, forced, got = (_info(monkeypatch, mode, c, k, r, row_tiles) for mode in ("0", "1", ""))
    assert forced[:2] != lone[:2]
    assert got[:2] == (forced if pair else lone)[:2]


def test_pairs_ask_for_no_scratch(monkeypatch):
    """A reduction that lone blocks would split (144 k-blocks on 100 row tiles) and pairs do not: the scratch memory
    that allows the split is asked for only where it would be used."""
    lone, forced, got = (_info(monkeypatch, mode, 1024, 192, 3, 100) for mode in ("0", "1", ""))
    assert lone[2] > 0 and lone[0] > 100
    assert got == forced and got[2] == 0
    assert _info(monkeypatch, "", 1024, 192, 3, 100, scratch=False) == got
