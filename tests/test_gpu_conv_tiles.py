"""The tiled convolution kernels at the sizes where a tiling can go wrong: row and column counts around a tile, k ranges
around a stage and a split, the smallest and largest tiles of the dispatch, a batch whose tiles straddle images.  Against
the CPU oracle, with the tolerances of the other operator tests (derived there)."""
import ctypes as C

import numpy as np
import pytest

from oracle import graph as og
from paella_b200 import capi
from tests import gpu_util as gu
from tests.test_gpu_ops import RNG, _assert_close, _params, _run_conv

pytestmark = pytest.mark.gpu

F32_CASES = [
    # C, H, W, K, R, S, sh, sw, ph, pw        what it exercises (tiles of 64 rows x 64 / 32 / 16 columns, stages of 32 k)
    (16, 8, 8, 8, 1, 1, 1, 1, 0, 0),          # smallest layer it takes: one tile, one half-filled stage, half a 16-column tile
    (32, 13, 5, 64, 1, 1, 1, 1, 0, 0),        # 65 rows: one row in the second tile; exactly one stage
    (33, 9, 7, 65, 1, 1, 1, 1, 0, 0),         # 63 rows, channels past a stage (36 with padding), one column in the second tile
    (7, 12, 12, 30, 3, 3, 1, 1, 1, 1),        # channel padding inside every tap; 30 columns: rows of weights padded to 32
    (20, 11, 11, 17, 3, 3, 2, 2, 0, 0),       # 17 columns of a 32-column tile, stride 2
    (3, 40, 40, 64, 7, 7, 2, 2, 3, 3),        # stem: a tap per chunk of four channels
    (256, 7, 7, 512, 3, 3, 1, 1, 1, 1),       # 49 rows, 72 stages: split over a cluster of 8
    (128, 14, 14, 128, 3, 3, 1, 1, 1, 1),     # 36 stages, 8 tiles: split
    (64, 30, 30, 128, 1, 1, 1, 1, 0, 0),      # two stages: no split
]


@pytest.mark.parametrize("case", F32_CASES)
def test_conv_f32(case):
    _run_conv(capi.STAGE_CONV_SIMT, 0, *case, act=1, residual=(case[3] % 4 == 0), bias=case[3] != 30)


def test_conv_f32_slice_and_dilation():
    _run_conv(capi.STAGE_CONV_SIMT, 0, 24, 9, 9, 40, 3, 3, 1, 1, 1, 1, out_total=64, off=8, act=2)
    _run_conv(capi.STAGE_CONV_SIMT, 0, 24, 9, 9, 24, 3, 3, 1, 1, 1, 1, out_total=40, off=3)            # unaligned slice
    _run_conv(capi.STAGE_CONV_SIMT, 0, 16, 19, 23, 16, 3, 3, 1, 1, 2, 3, dilation=(2, 3))


@pytest.mark.parametrize("cols", [16, 24, 72])
def test_conv_f32_weights_on_a_4_byte_boundary(cols):
    """Weights that do not start on a 16-byte boundary take another instance of each of the three tile widths (16, 32, 64
    columns): same order of additions, so the bits of the aligned ones."""
    import torch
    L = capi.load()
    c, h = 20, 11
    x = torch.randn((h, h, c), device="cuda")
    w = RNG.standard_normal((cols, c, 3, 3), dtype=np.float32)
    p = _params(0, (c, h, h), cols, h, h, cols, 3, 3, 1, 1, 1, 1, 1, 1, 0, 0, c)
    packed = gu.pack_weights(capi.STAGE_CONV_SIMT, p, w).view(torch.float32)
    outs = []
    for shift in (0, 1, 3):
        wd = torch.full((packed.numel() + 4,), float("nan"), device="cuda")
        wd[shift: shift + packed.numel()] = packed
        y = torch.full((h, h, cols), 7.0, device="cuda")
        p.x, p.w, p.y = x.data_ptr(), wd.data_ptr() + 4 * shift, y.data_ptr()
        capi.check(L.pb_op_launch(capi.STAGE_CONV_SIMT, C.byref(p), None, 0, None), "pb_op_launch")
        gu.sync()
        outs.append(y)
    ref = og.conv2d(np.ascontiguousarray(x.permute(2, 0, 1).cpu().numpy()), w, None, (1, 1), (1, 1), 1, 1, None)
    _assert_close(gu.from_device_cl(outs[0], cols), ref, 0)
    assert torch.equal(outs[1], outs[0]) and torch.equal(outs[2], outs[0])


UMMA_SPLITS = [
    # C, H, W, K, R, S, sh, sw, ph, pw, blocks     (tiles of 128 rows; a k-block is 64 channels of one tap)
    (64, 28, 28, 16, 3, 3, 1, 1, 1, 1, 14),       # 2 ranks on each of 7 row tiles, 8 columns each; 9 k-blocks: 4 and 5
    (128, 70, 70, 40, 3, 3, 1, 1, 1, 1, 78),      # 2 ranks on 39 row tiles, 24 columns each: an odd number of octets
    (64, 8, 16, 16, 3, 3, 1, 1, 1, 1, 4),         # 4 ranks on exactly one row tile; 9 k-blocks
    (192, 56, 56, 80, 3, 3, 1, 1, 1, 1, 100),     # 4 ranks on 25 row tiles, 24 columns each
    (256, 7, 7, 16, 3, 3, 1, 1, 1, 1, 8),         # 8 ranks on one tile, 8 columns each
    (128, 3, 43, 40, 3, 3, 1, 1, 1, 1, 16),       # 129 rows, 40 columns: the last tile is mostly outside
    (448, 8, 8, 384, 3, 3, 1, 1, 1, 1, 48),       # 63 k-blocks: ranks with unequal shares
    (512, 7, 7, 512, 3, 3, 1, 1, 1, 1, 64),       # 72 k-blocks on half a row tile
    (192, 17, 17, 200, 1, 7, 1, 1, 0, 3, 84),     # 21 k-blocks, 200 columns
]


@pytest.mark.parametrize("act", [0, 1, 2])
@pytest.mark.parametrize("case", UMMA_SPLITS)
def test_conv_umma_cluster_split(case, act):
    """Split over a cluster (scratch allows it), with a residual and an output slice."""
    L = capi.load()
    L.pb_set_conv_split_gain_us(0.0)
    try:
        _run_conv(capi.STAGE_CONV_UMMA, 1, *case[:10], act=act, residual=True, scratch=True, split_blocks=case[10], out_total=case[3] + 24, off=16)
    finally:
        L.pb_set_conv_split_gain_us(-1.0)


WIDE = [
    # N, C, H, K, R                            the tile leaves through TMA stores
    (13, 64, 40, 64, 1),                       # 163 row tiles, the last one half empty
    (20, 32, 35, 96, 3),                       # 96 columns: three boxes of 32
    (20, 64, 33, 200, 1),                      # 200 columns: the last box is cut
    (40, 16, 29, 136, 3),                      # tiles straddle images
    (30, 64, 40, 24, 1),                       # the narrowest box: 24 columns of 32
    (8, 32, 14, 1024, 1),                      # 13 row tiles, wide: no width that only direct stores can take
]


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("case", WIDE)
def test_conv_umma_many_tiles(case, residual):
    import torch
    L = capi.load()
    nb, C_, H, K, R = case
    x = og.round_bf16(RNG.standard_normal((nb, C_, H, H), dtype=np.float32))
    w = og.round_bf16(RNG.standard_normal((K, C_, R, R), dtype=np.float32) * np.float32(np.sqrt(2.0 / (C_ * R * R))))
    b = RNG.standard_normal(K, dtype=np.float32) * np.float32(0.1)
    res = og.round_bf16(RNG.standard_normal((nb, K, H, H), dtype=np.float32)) if residual else None
    cl = lambda t: torch.from_numpy(np.ascontiguousarray(np.transpose(t, (0, 2, 3, 1)))).cuda().to(torch.bfloat16)
    total, off = K + 16, 8
    p = _params(1, (C_, H, H), K, H, H, total, R, R, 1, 1, R // 2, R // 2, 1, 1, 0, off, C_)
    xd, y = cl(x), torch.full((nb, H, H, total), 7.0, device="cuda", dtype=torch.bfloat16)
    wd, bd = gu.pack_weights(capi.STAGE_CONV_UMMA, p, w), torch.from_numpy(b).cuda()
    p.batch, p.x, p.w, p.bias, p.y = nb, xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), y.data_ptr()
    if residual:
        rd = cl(res)
        p.residual, p.res_Cs = rd.data_ptr(), K
    capi.check(L.pb_op_launch(capi.STAGE_CONV_UMMA, C.byref(p), None, 0, None), "pb_op_launch")
    gu.sync()
    assert gu.error_flag() == 0
    got = np.transpose(y.float().cpu().numpy(), (0, 3, 1, 2))
    for i in (0, nb // 2, nb - 1):
        _assert_close(got[i, off:off + K], og.conv2d(x[i], w, b, (1, 1), (R // 2, R // 2), 1, 1, res[i] if residual else None), 1)
    assert (got[:, :off] == 7.0).all() and (got[:, off + K:] == 7.0).all()


@pytest.mark.parametrize("c,cs,k,r", [(7, 8, 16, 3), (24, 40, 24, 3), (33, 36, 72, 1), (5, 32, 64, 5)])
def test_conv_f32_reads_its_own_channels_only(c, cs, k, r):
    """Channels from C to the stride Cs belong to nobody (padding) or to another layer (a prefix of a concatenation): whatever they
    hold, NaN included, the result is that of zeros there."""
    import torch
    L = capi.load()
    h = 9
    gen = torch.Generator(device="cuda").manual_seed(c)
    x = torch.full((h, h, cs), float("nan"), device="cuda")
    x[..., :c] = torch.randn((h, h, c), generator=gen, device="cuda")
    w = RNG.standard_normal((k, c, r, r), dtype=np.float32) * np.float32(np.sqrt(2.0 / (c * r * r)))
    p = _params(0, (c, h, h), k, h, h, k, r, r, 1, 1, r // 2, r // 2, 1, 0, 0, 0, cs)
    wd = gu.pack_weights(capi.STAGE_CONV_SIMT, p, w)
    outs = []
    for t in (x, torch.nan_to_num(x)):
        y = torch.full((h, h, k), 7.0, device="cuda")
        p.x, p.w, p.y = t.data_ptr(), wd.data_ptr(), y.data_ptr()
        capi.check(L.pb_op_launch(capi.STAGE_CONV_SIMT, C.byref(p), None, 0, None), "pb_op_launch")
        gu.sync()
        outs.append(y)
    ref = og.conv2d(np.ascontiguousarray(x[..., :c].permute(2, 0, 1).cpu().numpy()), w, None, (1, 1), (r // 2, r // 2), 1, 0, None)
    _assert_close(gu.from_device_cl(outs[1], k), ref, 0)
    assert torch.equal(outs[0], outs[1])
