"""Options of the serving path that change how a model's launches are cut or when its inputs are copied."""
import ctypes as C
import os

import numpy as np
import pytest

from oracle import graph as og
from paella_b200 import capi, packer
from tests import gpu_util as gu
from tests.test_gpu_gang import _pinned, _run_until, _server

pytestmark = pytest.mark.gpu


def _register(L, s, job):
    j, ib, ob, sb = C.c_uint32(), C.c_size_t(), C.c_size_t(), C.c_size_t()
    capi.check(L.pb_server_register_job(s, capi.plugin_path(job).encode(), C.byref(j)), "register " + job)
    L.pb_server_job_io_bytes(s, j, C.byref(ib), C.byref(ob), C.byref(sb))
    return j.value, ib.value, ob.value, sb.value


def test_persistent_kernel_launches_report_every_block(tmp_path, monkeypatch):
    """PB_CONV_PERSIST=1 with the default split policy: the persistent kernel never splits a reduction, so a stage that ends in
    a long one declares the blocks of the unsplit launch.  (A declaration with the split in it leaves the scheduler waiting for
    blocks that do not exist.)"""
    d = tmp_path / "models_persist_served"
    d.mkdir()
    packer.write_all(str(d), ["resnet18"])
    monkeypatch.delenv("PB_PRECISION", raising=False)
    monkeypatch.setenv("PB_CONV_PERSIST", "1")
    monkeypatch.setenv("PB_STAGE_GROUP", "3")             # several stages end in a 3x3 convolution of 256 or 512 channels
    L, s = _server(str(d), monkeypatch, 1)
    job, ib, ob, sb = _register(L, s, "tvm_resnet18")
    t = _pinned(sb)
    x = np.random.default_rng(3).standard_normal((3, 224, 224), dtype=np.float32)
    t.numpy()[:ib] = np.frombuffer(x.tobytes(), np.uint8)
    capi.check(L.pb_server_launch(s, job, t.data_ptr(), 1), "launch")
    done = _run_until(L, s, 1, timeout=20.0)
    assert done == {1: 0}, "the request was not answered"
    assert gu.error_flag() == 0
    off = (ib + 7) // 8 * 8
    y = np.frombuffer(t.numpy()[off: off + ob].tobytes(), np.float32)
    ref = og.run(og.Pack(packer.MODELS["resnet18"](seed=1234).to_bytes()), x)
    assert float(np.abs(y - ref).max()) <= 1e-2 * float(np.abs(ref).max())
    L.pb_server_destroy(s)
