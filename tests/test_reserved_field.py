"""pb_op_params.reserved is the caller's to leave unset: whatever it holds, every public entry point does what it does with a
zero there.  Run in a child process, which a fault would end."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HOST = """
import ctypes as C, numpy as np
from paella_b200 import capi
L = capi.load()
def params(reserved):
    p = capi.OpParams()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks = 1, 512, 7, 7, 512, 64, 7, 7, 64
    p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.reserved = 3, 3, 1, 1, 1, 1, 1, reserved
    return p
w = np.random.default_rng(1).standard_normal((64, 512, 3, 3)).astype(np.float32)
def packed(reserved):
    p = params(reserved)
    n = L.pb_op_pack_weights(capi.STAGE_CONV_UMMA, C.byref(p), w.ctypes.data, None)
    assert n > 0, n
    buf = np.zeros(n, np.uint8)
    assert L.pb_op_pack_weights(capi.STAGE_CONV_UMMA, C.byref(p), w.ctypes.data, buf.ctypes.data) == n
    return buf
def info(reserved):
    li = capi.LaunchInfo()
    capi.check(L.pb_op_info(capi.STAGE_CONV_UMMA, C.byref(params(reserved)), C.byref(li)), "pb_op_info")
    return bytes(li)
want, want_info = packed(0), info(0)
for r in (1, 2, 3, 5, 8, 0x100, 0x103, 255, -1):
    assert (packed(r) == want).all() and info(r) == want_info, r
print("same")
"""

DEVICE = """
import ctypes as C, torch
from paella_b200 import capi
L = capi.load()
x = torch.randn((1, 14, 14, 512), device="cuda").to(torch.bfloat16)
w = torch.randn((64, 512, 3, 3)).contiguous()
outs = []
for r in (0, 3, 0x102, -1):
    p = capi.OpParams()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks = 1, 512, 14, 14, 512, 64, 14, 14, 64
    p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.reserved = 3, 3, 1, 1, 1, 1, 1, r
    buf = torch.zeros(L.pb_op_pack_weights(capi.STAGE_CONV_UMMA, C.byref(p), w.data_ptr(), None), dtype=torch.uint8)
    L.pb_op_pack_weights(capi.STAGE_CONV_UMMA, C.byref(p), w.data_ptr(), buf.data_ptr())
    wd, scratch = buf.cuda(), torch.zeros(256, dtype=torch.uint8, device="cuda")
    p.x, p.w, p.scratch, p.scratch_bytes = x.data_ptr(), wd.data_ptr(), scratch.data_ptr(), 256
    for call in ("launch", "noalloc", "time"):
        y = torch.zeros((1, 14, 14, 64), device="cuda", dtype=torch.bfloat16)
        p.y = y.data_ptr()
        us = C.c_double()
        rc = {"launch": lambda: L.pb_op_launch(capi.STAGE_CONV_UMMA, C.byref(p), None, 0, None),
              "noalloc": lambda: L.pb_conv2d_umma_noalloc(C.byref(p), None, 0, None),
              "time": lambda: L.pb_conv_umma_time(C.byref(p), 0, 1, 0, C.byref(us))}[call]()
        assert rc == 0, (r, call, L.pb_last_error())
        torch.cuda.synchronize()
        outs.append(y)
assert float(outs[0].float().abs().max()) > 0 and all(torch.equal(o, outs[0]) for o in outs)
print("same")
"""


def _child(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, (r.returncode, r.stderr[-2000:])


def test_host_entry_points_ignore_the_reserved_field():
    _child(HOST)


@pytest.mark.gpu
def test_launching_entry_points_ignore_the_reserved_field():
    _child(DEVICE)
