"""An affine (batch-norm + ReLU) that the pointwise convolution behind it applies to its own input tiles: the bits of the two
launches, at channel counts around a 64-channel k-block, maps around a 128-row tile, several images, with and without ReLU,
as the prefix of a wider concatenation, and with long reductions that are split over a cluster."""
import ctypes as C
import os

import numpy as np
import pytest

from paella_b200 import capi, packer
from tests.test_gpu_models import Model

pytestmark = pytest.mark.gpu

CASES = [
    # channels normalised, of the concatenation, outputs, map, ReLU
    (8, 8, 16, (3, 3), True),              # one vector of channels, 9 rows of a tile
    (64, 64, 32, (16, 8), True),           # exactly one k-block, exactly one tile
    (72, 104, 40, (12, 11), False),        # a k-block and a vector; a prefix; 132 rows; no ReLU
    (136, 160, 128, (14, 14), True),
    (512, 544, 128, (7, 7), True),         # eight k-blocks
    (1024, 1024, 128, (7, 7), True),       # sixteen
    (2048, 2048, 24, (4, 4), True),        # thirty-two, split
]


def _launches(m):
    """Launches of the model's first stage group."""
    order, launch = (C.c_int32 * 64)(), (C.c_int32 * 64)()
    n = m.L.pb_model_group_plan(m.m, 0, order, launch, 64)
    assert sorted(order[:n]) == list(range(n))
    return launch[n - 1] + 1


def _graph(case):
    cin, total, cout, (h, w), relu = case
    g = packer.Graph("affine", (16, h, w), seed=cin + cout, precision=1, round_weights_bf16=True)
    cat = g.tensor(total, h, w)
    for off in range(0, total, 8 if total < 64 else total // 4 // 8 * 8):
        n = min(8 if total < 64 else total // 4 // 8 * 8, total - off)
        g.conv(g.input, n, 1, act=packer.ACT_NONE, name="part%d" % off, out=cat, out_c_off=off)
    a = g.affine(cat, cin=cin, act=packer.ACT_RELU if relu else packer.ACT_NONE, name="norm")
    y = g.conv(a, cout, 1, name="conv")
    y = g.conv(y, 16, 3, 1, 1, name="next")
    g.dense(g.gap(y, name="gap"), 10, name="fc")
    return g, a


@pytest.mark.parametrize("case", CASES)
def test_affine_in_the_convolution_has_the_bits_of_two_launches(tmp_path, monkeypatch, case):
    g, a = _graph(case)
    path = g.save(str(tmp_path / "affine.bin"))
    x = np.random.default_rng(case[0]).standard_normal((16,) + case[3], dtype=np.float32)
    outs, tensors, launches = {}, {}, {}
    for flag in ("0", "1"):
        monkeypatch.setenv("PB_FUSE_AFFINE", flag)
        m = Model(path, 1)
        outs[flag] = m.run_groups(x)
        tensors[flag] = m.tensor(a, g.tensors[a])           # written by the convolution's launch or computed when asked for
        np.testing.assert_array_equal(m.run(x), outs[flag])
        launches[flag] = _launches(m)
        m.close()
    np.testing.assert_array_equal(outs["0"], outs["1"])
    np.testing.assert_array_equal(tensors["0"], tensors["1"])
    assert launches["1"] == launches["0"] - 1


@pytest.mark.parametrize("case", CASES)
def test_single_stages_after_the_groups_see_the_affine(tmp_path, monkeypatch, case):
    """The affine's tensor is this request's after the stage groups ran, for a single stage launched from it: by stage, and as an
    operator with the stage's parameters for a batch."""
    import torch
    monkeypatch.setenv("PB_FUSE_AFFINE", "1")
    g, _ = _graph(case)
    m = Model(g.save(str(tmp_path / "affine.bin")), 1)
    names = [m.L.pb_model_stage_name(m.m, s).decode() for s in range(m.L.pb_model_num_stages(m.m))]
    conv = names.index("conv")
    t = next(o.out for o in g.ops if o.name == "conv")
    xs = np.random.default_rng(1).standard_normal((3, 16) + case[3], dtype=np.float32)
    m.run(xs[0])                                            # another request was there before
    m.run_groups(xs[1])
    want = m.tensor(t, g.tensors[t])
    capi.check(m.L.pb_instance_launch_stage(m.i, conv, None, 0, None), "pb_instance_launch_stage")
    np.testing.assert_array_equal(m.tensor(t, g.tensors[t]), want)

    inst, out = C.c_void_p(), np.zeros((3, 10), np.float32)
    capi.check(m.L.pb_instance_create_batched(m.m, 3, 0, C.byref(inst)), "pb_instance_create_batched")
    p, got = capi.OpParams(), {}
    for by_groups in (0, 1):
        first = np.ascontiguousarray(xs[::-1]) if by_groups else xs
        capi.check(m.L.pb_instance_run_batch_sync(inst, 3, 0, first.ctypes.data, out.ctypes.data), "run batch")
        if by_groups:
            capi.check(m.L.pb_instance_run_batch_sync(inst, 3, 1, xs.ctypes.data, out.ctypes.data), "run batch")
        capi.check(m.L.pb_instance_stage_params(inst, conv, 3, C.byref(p)), "pb_instance_stage_params")
        y = torch.zeros((3, p.P, p.Q, p.Ks), device="cuda", dtype=torch.bfloat16)
        p.y = y.data_ptr()
        capi.check(m.L.pb_op_launch(capi.STAGE_CONV_UMMA, C.byref(p), None, 0, None), "pb_op_launch")
        torch.cuda.synchronize()
        got[by_groups] = y
    assert torch.equal(got[0], got[1])
    m.L.pb_instance_destroy(inst)
    m.close()


@pytest.mark.parametrize("case", CASES)
def test_the_launch_is_declared_with_its_constants(tmp_path, monkeypatch, case):
    """An unsplit normalising convolution holds 512 bytes for each k-block beside its pipeline (and a few more barriers); the group
    moves the affine's and the convolution's bytes less the convolution's input, which is not read back."""
    g, _ = _graph(case)
    path = g.save(str(tmp_path / "affine.bin"))
    smem, blocks, moved, li = {}, {}, {}, capi.LaunchInfo()
    capi.load().pb_set_conv_split_gain_us(1e7)              # nothing splits
    try:
        for flag in ("0", "1"):
            monkeypatch.setenv("PB_FUSE_AFFINE", flag)
            m = Model(path, 1)
            names = [m.L.pb_model_stage_name(m.m, s).decode() for s in range(m.L.pb_model_num_stages(m.m))]
            capi.check(m.L.pb_model_stage_info(m.m, names.index("conv"), C.byref(li)), "stage info")
            smem[flag], blocks[flag] = li.smem_per_block, li.num_blocks
            capi.check(m.L.pb_model_group_info(m.m, 0, C.byref(li)), "group info")
            moved[flag] = li.bytes
            m.close()
    finally:
        capi.load().pb_set_conv_split_gain_us(-1.0)
    cin, _, _, (h, w), _ = case
    assert blocks["1"] == blocks["0"]
    assert 0 <= smem["1"] - smem["0"] - 512 * -(-cin // 64) <= 64
    assert moved["0"] - moved["1"] == 2 * cin * h * w


@pytest.mark.parametrize("channels", [11776, 11784, 16384])
def test_as_many_channels_as_the_constants_have_room_for(tmp_path, monkeypatch, channels):
    """The constants of an unsplit reduction lie in one block's shared memory beside its pipeline: 184 k-blocks' at most.  Wider
    affines have a launch of their own."""
    g, _ = _graph((channels, channels, 16, (2, 2), True))
    path = g.save(str(tmp_path / "affine.bin"))
    x = np.random.default_rng(5).standard_normal((16, 2, 2), dtype=np.float32)
    outs, launches = {}, {}
    capi.load().pb_set_conv_split_gain_us(1e7)              # nothing splits
    try:
        for flag in ("0", "1"):
            monkeypatch.setenv("PB_FUSE_AFFINE", flag)
            m = Model(path, 1)
            outs[flag], launches[flag] = m.run_groups(x), _launches(m)
            m.close()
    finally:
        capi.load().pb_set_conv_split_gain_us(-1.0)
    np.testing.assert_array_equal(outs["0"], outs["1"])
    assert launches["1"] == launches["0"] - (1 if channels <= 11776 else 0)


def test_densenet_gang_with_and_without_fused_affines(models_dir, monkeypatch):
    path = os.path.join(models_dir, packer.pack_file_name("densenet121"))
    xs = np.random.default_rng(2).standard_normal((3, 3, 224, 224), dtype=np.float32)
    outs = {}
    for flag in ("0", "1"):
        monkeypatch.setenv("PB_FUSE_AFFINE", flag)
        m = Model(path, 1)
        inst, y = C.c_void_p(), np.zeros((3, 1000), np.float32)
        capi.check(m.L.pb_instance_create_batched(m.m, 3, 0, C.byref(inst)), "pb_instance_create_batched")
        capi.check(m.L.pb_instance_run_batch_sync(inst, 3, 1, xs.ctypes.data, y.ctypes.data), "run batch")
        outs[flag] = y
        m.L.pb_instance_destroy(inst)
        m.close()
    np.testing.assert_array_equal(outs["0"], outs["1"])
