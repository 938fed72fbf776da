"""Which depthwise 3x3 launches of many rows walk behind a ring of window rows: where that was measured faster than tiles by 3 % and
more, and not where it was slower (B200)."""
import ctypes as C

import pytest

from paella_b200 import capi

# N, C, H, W: us of tiles and ring
MEASURED = [
    (3780, 64, 8, 26, 52.4, 58.9), (2457, 64, 10, 32, 36.7, 40.7), (1404, 64, 5, 112, 56.6, 63.8), (2006, 64, 14, 28, 45.1, 46.9), (1755, 64, 8, 56, 50.2, 53.6),
    (702, 64, 10, 112, 42.2, 46.8), (351, 64, 20, 112, 42.1, 45.9), (877, 64, 16, 56, 41.5, 43.1), (1400, 8, 9, 32, 21.7, 24.3), (1903, 16, 7, 26, 21.4, 25.3),
    (1478, 64, 19, 28, 49.7, 42.5), (1591, 64, 19, 26, 52.9, 45.8), (460, 64, 28, 61, 46.3, 39.0), (438, 64, 56, 32, 40.2, 35.5), (125, 64, 56, 112, 42.7, 40.5),
    (1003, 64, 28, 28, 43.7, 41.7), (805, 64, 16, 61, 48.1, 40.6), (1, 128, 1024, 1024, 104.0, 98.6), (32, 64, 224, 224, 83.6, 71.9), (64, 200, 57, 57, 50.6, 45.7),
]


@pytest.mark.parametrize("n,c,h,w,tiles,ring", MEASURED)
def test_the_faster_one(n, c, h, w, tiles, ring, monkeypatch):
    monkeypatch.delenv("PB_WINDOW_TILE", raising=False)
    p, li = capi.OpParams(), capi.LaunchInfo()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks = 1, c, h, w, c, c, h, w, c
    p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.batch = 3, 3, 1, 1, 1, 1, c, n
    rings = 444 // -(-c // 64) * -(-c // 64)
    for switch, want in ((None, ring < tiles), ("1", True)):
        if switch:
            monkeypatch.setenv("PB_WINDOW_TILE", switch)
        capi.check(capi.load().pb_op_info(capi.STAGE_DWCONV, C.byref(p), C.byref(li)), "pb_op_info")
        assert (li.num_blocks == rings) == want
