"""A lone MNIST image runs on a cluster of four blocks, the images of a gang on one block each: the same bits, wherever the image
starts, and the declaration of either."""
import ctypes as C
import os

import numpy as np
import pytest

from oracle import graph as og
from paella_b200 import capi, packer
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


def test_lone_image_and_gang(tmp_path):
    import torch
    L = capi.load()
    g = packer.mnist_cnn(seed=5, bias_std=0.2)
    path = g.save(os.path.join(str(tmp_path), packer.pack_file_name("mnist")))
    m, inst = C.c_void_p(), C.c_void_p()
    capi.check(L.pb_model_load(path.encode(), 0, 0, C.byref(m)), "pb_model_load")
    capi.check(L.pb_instance_create_batched(m, 8, 0, C.byref(inst)), "pb_instance_create_batched")
    gen = torch.Generator(device="cuda").manual_seed(1)
    # an image of noise, one with signs, one that is nonzero in one corner only, one empty
    x = torch.randn((4, 784), generator=gen, device="cuda")
    x[0].abs_()
    x[2] = 0
    x[2, 783] = 3.0
    x[3] = 0

    def run(n, shift):
        buf = torch.full((n * 784 + 4,), float("nan"), device="cuda")
        buf[shift:shift + n * 784] = x[:n].reshape(-1)
        y = torch.full((n, 10), 7.0, device="cuda")
        ins = (C.c_void_p * n)(*[buf.data_ptr() + 4 * (shift + 784 * i) for i in range(n)])
        outs = (C.c_void_p * n)(*[y.data_ptr() + 40 * i for i in range(n)])
        capi.check(L.pb_instance_launch_group_batched(inst, 0, n, None, 0, None, ins, outs), "launch")
        gu.sync()
        return y

    def one(i, shift):
        buf = torch.full((784 + 4,), float("nan"), device="cuda")
        buf[shift:shift + 784] = x[i]
        y = torch.full((1, 10), 7.0, device="cuda")
        capi.check(L.pb_instance_launch_group(inst, 0, None, 0, None, buf.data_ptr() + 4 * shift, y.data_ptr()), "launch")
        gu.sync()
        return y[0]

    gang = run(4, 0)
    assert torch.equal(run(4, 1), gang) and torch.equal(run(2, 3), gang[:2])
    for i in range(4):
        for shift in (0, 1, 2):
            assert torch.equal(one(i, shift), gang[i])
        ref = og.run(og.Pack(g.to_bytes()), x[i].cpu().numpy().reshape(1, 28, 28))
        assert np.abs(gang[i].cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max()
    lone, four = capi.LaunchInfo(), capi.LaunchInfo()
    capi.check(L.pb_model_group_info_batched(m, 0, 1, C.byref(lone)), "info")
    capi.check(L.pb_model_group_info_batched(m, 0, 4, C.byref(four)), "info")
    assert (lone.num_blocks, lone.threads_per_block) == (1, 1024) and (four.num_blocks, four.threads_per_block) == (4, 256)
    L.pb_instance_destroy(inst)
    L.pb_model_destroy(m)
