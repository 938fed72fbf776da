"""The tiled 3x3 window kernel where its values, pointers or surroundings are unusual.  Bit for bit the strip kernels
(PB_WINDOW_TILE=0), which it stands in for on launches that fill the GPU."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from paella_b200 import capi
from tests import gpu_util as gu
from tests.test_gpu_ops import _params

pytestmark = pytest.mark.gpu

KINDS = [(kind, flags, act, bias) for kind, flags, biases in ((capi.STAGE_DWCONV, 0, (True, False)), (capi.STAGE_MAXPOOL, 0, (True, False)),
                                                              (capi.STAGE_AVGPOOL, 1, (True, False)), (capi.STAGE_AVGPOOL, 0, (True, False)))
         for act in (0, 1, 2) for bias in biases]


def _both(monkeypatch, L, kind, p, y):
    """Output of the strip kernels and of the tiled kernel for the same parameters, as raw 16-bit words."""
    import torch
    outs = []
    for tile in ("0", "1"):
        monkeypatch.setenv("PB_WINDOW_TILE", tile)
        monkeypatch.setenv("PB_WINDOW_TILE_MIN_BLOCKS", "1")
        y.fill_(3.0)
        li = capi.LaunchInfo()
        capi.check(L.pb_op_info(kind, C.byref(p), C.byref(li)), "pb_op_info")
        assert (li.threads_per_block == 256) == (tile == "0")
        capi.check(L.pb_op_launch(kind, C.byref(p), None, 0, None), "pb_op_launch")
        gu.sync()
        assert gu.error_flag() == 0
        outs.append(y.view(torch.int16).cpu().numpy().view(np.uint16).copy())
    return outs


def _same_values(a, b, what):
    """Equal words, any NaN equal to any other, and -0 equal to +0 (the sign of a zero sum is not specified)."""
    fa, fb = ((v.astype(np.uint32) << 16).view(np.float32) for v in (a, b))
    np.testing.assert_array_equal(fa, fb, err_msg=str(what))


@pytest.mark.parametrize("stride,pad", [(1, 1), (2, 1), (1, 0)])
@pytest.mark.parametrize("nb", [1, 3])
def test_special_values_give_what_the_strip_kernels_give(monkeypatch, nb, stride, pad):
    """NaN, infinities, the largest finite values and whole windows of NaN: a maximum passes over NaN, ReLU makes zero of it,
    an average keeps it."""
    import torch
    L = capi.load()
    c, h, w = 72, 21, 19
    P, Q = (h + 2 * pad - 3) // stride + 1, (w + 2 * pad - 3) // stride + 1
    rng = np.random.default_rng(5)
    x = rng.standard_normal((nb, h, w, c)).astype(np.float32)
    pick = rng.random(x.shape)
    for lo, v in ((0.00, np.nan), (0.02, np.inf), (0.04, -np.inf), (0.06, 3.3e38), (0.08, -3.3e38), (0.10, 0.0), (0.13, -0.0)):
        x[(pick >= lo) & (pick < lo + 0.02)] = v
    x[:, 4:10, 4:12, :20] = np.nan                        # windows with nothing but NaN
    x[:, 12:18, 4:12, 8:30] = -np.inf
    xd = torch.from_numpy(x).cuda().to(torch.bfloat16)
    wt = rng.standard_normal((c, 1, 3, 3)).astype(np.float32)
    bd = torch.randn(c, device="cuda")
    y = torch.zeros((nb, P, Q, c + 16), device="cuda", dtype=torch.bfloat16)
    for kind, flags, act, bias in KINDS:
        p = _params(1, (c, h, w), c, P, Q, c + 16, 3, 3, stride, stride, pad, pad, groups=c if kind == capi.STAGE_DWCONV else 1, act=act, flags=flags,
                    out_c_off=8, Cs=c)
        p.batch = nb
        if kind == capi.STAGE_DWCONV:
            wd = gu.pack_weights(kind, p, wt)
            p.w = wd.data_ptr()
        p.x, p.bias, p.y = xd.data_ptr(), bd.data_ptr() if bias else None, y.data_ptr()
        strip, tile = _both(monkeypatch, L, kind, p, y)
        _same_values(tile, strip, (kind, flags, act, bias))


@pytest.mark.parametrize("nb", [1, 2])
def test_pointers_aligned_to_a_pair_of_channels(monkeypatch, nb):
    """Output and filter that start on a 4-byte boundary give the bits of aligned ones, and nothing beside the output is touched."""
    import torch
    L = capi.load()
    c, h, w = 72, 20, 37
    x = torch.randn((nb, h, w, c), device="cuda").to(torch.bfloat16)
    wt = np.random.default_rng(9).standard_normal((c, 1, 3, 3)).astype(np.float32)
    bd = torch.randn(c, device="cuda")
    monkeypatch.setenv("PB_WINDOW_TILE_MIN_BLOCKS", "1")
    for kind, flags in ((capi.STAGE_DWCONV, 0), (capi.STAGE_MAXPOOL, 0), (capi.STAGE_AVGPOOL, 0)):
        outs = []
        for shift in (0, 2):                              # elements of two bytes
            p = _params(1, (c, h, w), c, h, w, c, 3, 3, 1, 1, 1, 1, groups=c if kind == capi.STAGE_DWCONV else 1, act=1, flags=flags, Cs=c)
            p.batch = nb
            if kind == capi.STAGE_DWCONV:
                packed = gu.pack_weights(kind, p, wt).view(torch.bfloat16)
                wd = torch.zeros(packed.numel() + 8, device="cuda", dtype=torch.bfloat16)
                wd[shift: shift + packed.numel()] = packed
                p.w = wd.data_ptr() + 2 * shift
            y = torch.full((nb * h * w * c + 8,), 3.0, device="cuda", dtype=torch.bfloat16)
            p.x, p.bias, p.y = x.data_ptr(), bd.data_ptr(), y.data_ptr() + 2 * shift
            li = capi.LaunchInfo()
            capi.check(L.pb_op_info(kind, C.byref(p), C.byref(li)), "pb_op_info")
            assert li.threads_per_block <= 160
            capi.check(L.pb_op_launch(kind, C.byref(p), None, 0, None), "pb_op_launch")
            gu.sync()
            assert gu.error_flag() == 0
            assert (y[:shift] == 3.0).all() and (y[shift + nb * h * w * c:] == 3.0).all()
            outs.append(y[shift: shift + nb * h * w * c].clone())
        assert torch.equal(outs[0], outs[1]), kind


CAPTURED = """
import ctypes as C, torch
from paella_b200 import capi
L = capi.load()
torch.manual_seed(1)
x = torch.randn((1, 128, 64, 512), device="cuda").to(torch.bfloat16)
y = torch.zeros((1, 128, 64, 512), device="cuda", dtype=torch.bfloat16)
p = capi.OpParams()
p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks = 1, 512, 128, 64, 512, 512, 128, 64, 512
p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.batch = 3, 3, 1, 1, 1, 1, 1, 1
p.x, p.y = x.data_ptr(), y.data_ptr()
li = capi.LaunchInfo()
capi.check(L.pb_op_info(capi.STAGE_MAXPOOL, C.byref(p), C.byref(li)), "pb_op_info")
assert li.threads_per_block <= 160, "the tiled kernel"
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    rc = L.pb_op_launch(capi.STAGE_MAXPOOL, C.byref(p), torch.cuda.current_stream().cuda_stream, 0, None)
assert rc == 0, L.pb_last_error()
g.replay()
torch.cuda.synchronize()
want = torch.nn.functional.max_pool2d(x.float().permute(0, 3, 1, 2), 3, 1, 1).permute(0, 2, 3, 1)
assert torch.equal(y.float(), want)
flag = C.c_uint32(7)
capi.check(L.pb_device_error_flag(0, C.byref(flag), 1), "flag")
assert flag.value == 0
print("captured")
"""


def test_a_first_launch_may_be_captured():
    """A program whose first call into the library is a pooling launch inside a stream capture: nothing may be allocated there."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CAPTURED], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]
