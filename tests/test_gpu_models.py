"""Whole models through the graph executor (C ABI) vs the oracle and the committed golden logits.
Tolerances: fp32 path 1e-5 of the largest |logit|; bf16 tensor-core path 1e-2 of the largest
|logit| against the FP32 oracle with identical argmax (the seeds' top-1 margins are 0.7% - 28%)."""
import ctypes as C
import os

import numpy as np
import pytest

from oracle import graph as og
from paella_b200 import capi, packer
from tests import gpu_util as gu
from tests.golden.make_golden import make_input

pytestmark = pytest.mark.gpu
GOLDEN = np.load(os.path.join(os.path.dirname(__file__), "golden", "golden_logits.npz"))


class Model:
    def __init__(self, path, precision):
        self.L = capi.load()
        self.m, self.i = C.c_void_p(), C.c_void_p()
        capi.check(self.L.pb_model_load(path.encode(), 0, precision, C.byref(self.m)), "pb_model_load")
        capi.check(self.L.pb_instance_create(self.m, C.byref(self.i)), "pb_instance_create")

    def run(self, x):
        x = np.ascontiguousarray(x, np.float32)
        y = np.zeros(self.L.pb_model_output_bytes(self.m) // 4, np.float32)
        capi.check(self.L.pb_instance_run_sync(self.i, x.ctypes.data, y.ctypes.data), "run")
        assert gu.error_flag() == 0
        return y

    def run_groups(self, x):
        x = np.ascontiguousarray(x, np.float32)
        y = np.zeros(self.L.pb_model_output_bytes(self.m) // 4, np.float32)
        capi.check(self.L.pb_instance_run_groups_sync(self.i, x.ctypes.data, y.ctypes.data), "run groups")
        assert gu.error_flag() == 0
        return y

    def kinds(self):
        li = capi.LaunchInfo()
        out = []
        for s in range(self.L.pb_model_num_stages(self.m)):
            self.L.pb_model_stage_info(self.m, s, C.byref(li))
            out.append(li.kind)
        return out

    def tensor(self, t, shape):
        buf = np.zeros(int(np.prod(shape)), np.float32)
        capi.check(self.L.pb_instance_read_tensor(self.i, t, buf.ctypes.data, buf.size), "read_tensor")
        return buf.reshape(shape)

    def close(self):
        self.L.pb_instance_destroy(self.i)
        self.L.pb_model_destroy(self.m)


@pytest.mark.parametrize("fused", ["1", "0"])
def test_mnist_fp32(models_dir, monkeypatch, fused):
    monkeypatch.setenv("PB_FUSE_MNIST", fused)
    g = packer.mnist_cnn(seed=1234)
    m = Model(os.path.join(models_dir, packer.pack_file_name("mnist")), 0)
    assert (capi.STAGE_MNIST_FUSED in m.kinds()) == (fused == "1")
    pack = og.Pack(g.to_bytes())
    for seed in range(5):
        x = np.random.default_rng(seed).random((1, 28, 28), dtype=np.float32)
        y, ref = m.run(x), og.run(pack, x)
        assert float(np.abs(y - ref).max()) <= 1e-5 * float(np.abs(ref).max())
        assert int(y.argmax()) == int(ref.argmax())
    y = m.run(make_input("mnist"))
    assert float(np.abs(y - GOLDEN["mnist"]).max()) <= 1e-5 * float(np.abs(GOLDEN["mnist"]).max())
    m.close()


def test_mnist_with_biases_both_paths(tmp_path, monkeypatch):
    g = packer.mnist_cnn(seed=7, bias_std=0.2)
    path = g.save(str(tmp_path / "m.bin"))
    ref = og.run(og.Pack(g.to_bytes()), make_input("mnist"))
    for fused in ("1", "0"):
        monkeypatch.setenv("PB_FUSE_MNIST", fused)
        m = Model(path, 0)
        y = m.run(make_input("mnist"))
        assert float(np.abs(y - ref).max()) <= 1e-5 * float(np.abs(ref).max())
        m.close()


def test_small_net_layer_by_layer_bf16(tmp_path):
    """Every intermediate tensor of a small bf16 network against the bf16-emulating oracle."""
    g = packer.Graph("small", (3, 40, 40), seed=21, precision=1, bias_std=0.05)
    t = g.conv(g.input, 32, 3, 2, 1, name="stem")
    r = g.conv(t, 64, 1, 1, 0, name="expand")
    d = g.conv(r, 64, 3, 1, 1, groups=64, act=packer.ACT_RELU6, name="dw")
    t2 = g.conv(d, 64, 3, 1, 1, residual=r, name="res")
    cat = g.tensor(64 + 32 + 64, 10, 10)
    g.conv(t2, 64, 3, 2, 1, out=cat, out_c_off=0, name="b0")
    g.conv(t2, 32, (1, 7), (2, 2), (0, 3), out=cat, out_c_off=64, name="b1")
    g.maxpool(t2, 3, 2, 1, out=cat, out_c_off=96, name="b2")
    a = g.avgpool(cat, 3, 1, 1, True, name="avg")
    s = g.add(a, cat, act=packer.ACT_RELU, name="add")
    p = g.gap(s, name="gap")
    dn = g.dense(p, 24, name="fc")
    g.softmax(dn, name="sm")
    path = g.save(str(tmp_path / "small.bin"))
    m = Model(path, 1)
    assert capi.STAGE_CONV_UMMA in m.kinds() and capi.STAGE_DWCONV in m.kinds()
    x = np.random.default_rng(3).standard_normal((3, 40, 40), dtype=np.float32)
    y = m.run(x)
    ref, bufs = og.run(og.Pack(g.to_bytes()), x, emulate_bf16=True, keep_all=True)
    for t_id, shape in enumerate(g.tensors):
        if t_id == g.output:
            continue
        if t_id == g.input:
            continue        # the stem is lowered to a patch matrix: the channels-last image is never materialised
        got = m.tensor(t_id, shape)
        want = og.round_bf16(bufs[t_id])
        scale = max(float(np.abs(want).max()), 1e-6)
        tol = np.abs(want) * 2.0 ** -6 + 4e-3 * scale
        assert (np.abs(got - want) <= tol).all(), f"tensor {t_id} {shape}: worst {float(np.abs(got - want).max())} scale {scale}"
    np.testing.assert_allclose(y, ref, rtol=3e-2, atol=1e-4)
    m.close()


@pytest.mark.parametrize("model", ["resnet18", "resnet34", "inception_v3", "resnet50", "googlenet", "squeezenet1_1", "densenet121"])
def test_imagenet_models_bf16_vs_fp32_oracle(models_dir, model):
    m = Model(os.path.join(models_dir, packer.pack_file_name(model)), 1)
    kinds = m.kinds()
    assert kinds.count(capi.STAGE_CONV_UMMA) >= 20 and capi.STAGE_CONV_SIMT not in kinds
    y = m.run(make_input(model))
    ref = GOLDEN[model]                       # fp32 oracle logits
    rel = float(np.abs(y - ref).max() / np.abs(ref).max())
    assert rel <= 1e-2, rel
    assert int(y.argmax()) == int(ref.argmax())
    m.close()


@pytest.mark.parametrize("model", ["resnet18", "inception_v3"])
def test_stem_as_patch_matrix_and_as_image_agree(models_dir, monkeypatch, model):
    """The 3-channel stem convolution is lowered to a pointwise convolution over a patch matrix written by
    stage 0; PB_PATCH_INPUT=0 keeps the channels-last image and the filter taps.  Same arithmetic, other
    summation order inside the tensor core: results agree to bf16 accuracy and with the fp32 oracle."""
    path = os.path.join(models_dir, packer.pack_file_name(model))
    x = make_input(model)
    outs = {}
    for flag in ("1", "0"):
        monkeypatch.setenv("PB_PATCH_INPUT", flag)
        m = Model(path, 1)
        name0 = m.L.pb_model_stage_name(m.m, 0).decode()
        assert name0 == ("input_patches" if flag == "1" else "input_layout")
        outs[flag] = m.run(x)
        m.close()
    ref = GOLDEN[model]
    scale = float(np.abs(ref).max())
    for y in outs.values():
        assert float(np.abs(y - ref).max()) <= 1e-2 * scale and int(y.argmax()) == int(ref.argmax())
    assert float(np.abs(outs["1"] - outs["0"]).max()) <= 5e-3 * scale


def test_resnet18_fp32_path(models_dir):
    """The fp32 (direct convolution) path of the same pack: 1e-4 of the largest logit (long fp32 sums
    in a different order than the oracle)."""
    m = Model(os.path.join(models_dir, packer.pack_file_name("resnet18")), 0)
    y = m.run(make_input("resnet18"))
    ref = GOLDEN["resnet18"]
    assert float(np.abs(y - ref).max()) <= 1e-4 * float(np.abs(ref).max())
    assert int(y.argmax()) == int(ref.argmax())
    m.close()


def test_mobilenet_v2(models_dir):
    """Depthwise + ReLU6 network.  bf16 storage loses more here (narrow linear bottlenecks): the bf16
    path is held to the bf16-emulating oracle, the fp32 path to the fp32 oracle."""
    ref = GOLDEN["mobilenet"]
    m = Model(os.path.join(models_dir, packer.pack_file_name("mobilenet")), 0)
    y = m.run(make_input("mobilenet"))
    assert float(np.abs(y - ref).max()) <= 1e-4 * float(np.abs(ref).max())
    m.close()
    m = Model(os.path.join(models_dir, packer.pack_file_name("mobilenet")), 1)
    assert capi.STAGE_DWCONV in m.kinds()
    y = m.run(make_input("mobilenet"))
    emu = og.run(og.Pack(packer.mobilenet_v2(seed=1234).to_bytes()), make_input("mobilenet"), emulate_bf16=True)
    assert float(np.abs(y - emu).max()) <= 1e-2 * float(np.abs(emu).max())
    assert int(y.argmax()) == int(ref.argmax())
    m.close()


@pytest.mark.parametrize("env", [{"PB_GRAPH_BRANCHES": "1"}, {"PB_FUSE_BRANCHES": "0"}, {"PB_PDL": "0"}, {"PB_GRAPH_SINGLE": "0", "PB_STAGE_GROUP": "1"}])
def test_graph_capture_options_give_the_same_bits(models_dir, monkeypatch, env):
    """The load-time switches of the stage graphs (parallel branch paths, no grouped launches, no programmatic
    dependent launch, kernel-by-kernel without graphs) change scheduling only: bit-identical logits."""
    path = os.path.join(models_dir, packer.pack_file_name("inception_v3"))
    x = make_input("inception_v3")
    m = Model(path, 1)
    want = m.run_groups(x)
    m.close()
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    m = Model(path, 1)
    np.testing.assert_array_equal(m.run_groups(x), want)
    np.testing.assert_array_equal(m.run_groups(x), want)
    m.close()


@pytest.mark.parametrize("group", ["4", "12", "24", "64"])
@pytest.mark.parametrize("model", ["inception_v3", "googlenet"])
def test_any_stage_granularity_gives_the_same_bits(models_dir, monkeypatch, model, group):
    """PB_STAGE_GROUP restarts the dependence depth at other stages, so convolutions that do not share a launch (nor a cluster
    size) by default come out equally deep: the models load, and give the bits of the default granularity, for one image and
    a gang of eight, under either tiling policy."""
    L = capi.load()
    path = os.path.join(models_dir, packer.pack_file_name(model))
    xs = np.stack([make_input(model, seed) for seed in range(5, 13)]).astype(np.float32)
    for shared in (0, 1):
        outs = []
        for env in (None, group):
            if env is None:
                monkeypatch.delenv("PB_STAGE_GROUP", raising=False)
            else:
                monkeypatch.setenv("PB_STAGE_GROUP", env)
            m, inst = C.c_void_p(), C.c_void_p()
            capi.check(L.pb_model_load(path.encode(), 0, 1, C.byref(m)), "pb_model_load")
            capi.check(L.pb_model_set_shared_gpu(m, shared), "pb_model_set_shared_gpu")
            capi.check(L.pb_instance_create_batched(m, 8, 0, C.byref(inst)), "pb_instance_create_batched")
            y = np.zeros((9, L.pb_model_output_bytes(m) // 4), np.float32)
            capi.check(L.pb_instance_run_batch_sync(inst, 1, 1, xs.ctypes.data, y.ctypes.data), "one image")
            capi.check(L.pb_instance_run_batch_sync(inst, 8, 1, xs.ctypes.data, y[1:].ctypes.data), "eight images")
            assert gu.error_flag() == 0
            outs.append(y)
            L.pb_instance_destroy(inst)
            L.pb_model_destroy(m)
        np.testing.assert_array_equal(outs[1], outs[0])


def test_arcface_embedding(models_dir):
    """ArcFace LResNet100E-IR: 100 convolutions deep, PReLU, a 512-d embedding out (no class scores, so no
    argmax).  bf16 STORAGE through 49 residual units drifts by 1.3 % of the largest component from fp32 - the
    bf16-emulating oracle shows the same 1.3 %, and per-tensor differences between the two bf16 executions
    grow smoothly from 0.1 % after the stem to 1.7 % before the fc - so the bf16 path is held to 2.5e-2 against
    the emulating oracle and, against the fp32 oracle, to the measure an embedding is used with (cosine
    similarity >= 0.999; measured 0.99989).  The fp32 path of the same pack meets 1e-4."""
    ref = GOLDEN["arcfaceresnet100"]
    m = Model(os.path.join(models_dir, packer.pack_file_name("arcfaceresnet100")), 0)
    y32 = m.run(make_input("arcfaceresnet100"))
    assert float(np.abs(y32 - ref).max()) <= 1e-4 * float(np.abs(ref).max())
    m.close()
    m = Model(os.path.join(models_dir, packer.pack_file_name("arcfaceresnet100")), 1)
    kinds = m.kinds()
    assert kinds.count(capi.STAGE_CONV_UMMA) == 103 and capi.STAGE_CONV_SIMT not in kinds and capi.STAGE_AFFINE in kinds
    x = make_input("arcfaceresnet100")
    y = m.run(x)
    emu = og.run(og.Pack(packer.arcface_r100(seed=1234).to_bytes()), x, emulate_bf16=True)
    assert float(np.abs(y - emu).max()) <= 2.5e-2 * float(np.abs(emu).max())
    cos = float(np.dot(y, ref) / (np.linalg.norm(y) * np.linalg.norm(ref)))
    assert cos >= 0.999, cos
    np.testing.assert_array_equal(m.run_groups(x), y)       # stage-group graphs give the same bits
    m.close()


def test_ultraface_detector(models_dir):
    """The 320x240 face detector: dilated convolutions in its receptive-field block, four detection heads writing
    one output block [4420 x 2 scores | 4420 x 4 boxes].  fp32 path: 1e-4 of the output range against the
    committed oracle output.  bf16 path: scores and boxes within 3e-2 absolute of the bf16-emulating oracle
    (scores lie in [0, 1], boxes are relative to the image), and the face / background decision of a prior equals
    the fp32 oracle's wherever that oracle's score is at least 0.1 away from 0.5."""
    ref = GOLDEN["ultraface320"]
    x = make_input("ultraface320")
    m = Model(os.path.join(models_dir, packer.pack_file_name("ultraface320")), 0)
    assert m.L.pb_model_output_bytes(m.m) == 4420 * 6 * 4 and m.L.pb_model_input_bytes(m.m) == 240 * 320 * 3 * 4
    assert m.kinds().count(capi.STAGE_DETECT) == 4
    y32 = m.run(x)
    assert float(np.abs(y32 - ref).max()) <= 1e-4 * float(np.abs(ref).max())
    np.testing.assert_array_equal(m.run_groups(x), y32)
    m.close()
    m = Model(os.path.join(models_dir, packer.pack_file_name("ultraface320")), 1)
    kinds = m.kinds()
    assert kinds.count(capi.STAGE_DETECT) == 4 and kinds.count(capi.STAGE_CONV_UMMA) >= 25 and kinds.count(capi.STAGE_DWCONV) == 18
    y = m.run(x)
    emu = og.run(og.Pack(packer.ultraface_rfb320(seed=1234).to_bytes()), x, emulate_bf16=True)
    assert float(np.abs(y - emu).max()) <= 3e-2, float(np.abs(y - emu).max())
    face_ref, face = ref[1:8840:2], y[1:8840:2]
    sure = np.abs(face_ref - 0.5) >= 0.1
    assert sure.sum() > 3000 and ((face[sure] > 0.5) == (face_ref[sure] > 0.5)).all()
    np.testing.assert_allclose(y[:8840:2] + y[1:8840:2], 1.0, atol=1e-6)
    np.testing.assert_array_equal(m.run_groups(x), y)
    m.close()


def test_same_input_same_output_and_instances_are_independent(models_dir):
    m = Model(os.path.join(models_dir, packer.pack_file_name("resnet18")), 1)
    i2 = C.c_void_p()
    capi.check(m.L.pb_instance_create(m.m, C.byref(i2)), "second instance")
    x1, x2 = make_input("resnet18"), np.random.default_rng(9).standard_normal((3, 224, 224), dtype=np.float32)
    y1 = m.run(x1)
    y = np.zeros(1000, np.float32)
    capi.check(m.L.pb_instance_run_sync(i2, x2.ctypes.data, y.ctypes.data), "run")
    assert not np.array_equal(y, y1)
    np.testing.assert_array_equal(m.run(x1), y1)      # deterministic, not disturbed by the other instance
    m.L.pb_instance_destroy(i2)
    m.close()


@pytest.mark.parametrize("model,precision", [("mnist", 0), ("resnet18", 1), ("inception_v3", 1)])
def test_stage_groups_replayed_as_graphs_give_the_same_bits(models_dir, model, precision):
    """Launching a model group by group (CUDA graphs, launch-slot indirection) must reproduce the
    kernel-by-kernel result bit for bit, launch after launch."""
    m = Model(os.path.join(models_dir, packer.pack_file_name(model)), precision)
    n_stages, n_groups = m.L.pb_model_num_stages(m.m), m.L.pb_model_num_groups(m.m)
    assert 1 <= n_groups <= n_stages and n_groups == -(-n_stages // 48)
    first, count, covered, n_fused = C.c_int(), C.c_int(), 0, 0
    li = capi.LaunchInfo()
    for g in range(n_groups):
        capi.check(m.L.pb_model_group_stages(m.m, g, C.byref(first), C.byref(count)), "group stages")
        assert first.value == covered
        covered += count.value
        capi.check(m.L.pb_model_group_info(m.m, g, C.byref(li)), "group info")
        order, launch = (C.c_int32 * count.value)(), (C.c_int32 * count.value)()
        assert m.L.pb_model_group_plan(m.m, g, order, launch, count.value) == count.value
        assert sorted(order) == list(range(first.value, first.value + count.value))      # a permutation of the group
        assert list(launch) == sorted(launch) and launch[0] == 0
        n_fused += len(launch) - (launch[-1] + 1)
        last_blocks, last_kinds = 0, set()              # only the last launch of a group notifies
        for s_idx, l_idx in zip(order, launch):
            if l_idx == launch[-1]:
                si = capi.LaunchInfo()
                m.L.pb_model_stage_info(m.m, s_idx, C.byref(si))
                assert len([x for x in launch if x == l_idx]) == 1 or si.kind == 2  # PB_STAGE_CONV_UMMA
                last_blocks += si.num_blocks
                last_kinds.add(si.kind)
        assert li.num_blocks == last_blocks
    assert covered == n_stages
    if model == "inception_v3":
        assert n_fused >= 40        # the branches of every Inception block share launches
    for seed in (5, 6):
        x = make_input(model, seed)
        ref = m.run(x)
        np.testing.assert_array_equal(m.run_groups(x), ref)
        np.testing.assert_array_equal(m.run_groups(x), ref)
    m.close()


@pytest.mark.parametrize("model", ["inception_v3", "googlenet"])
def test_pooling_layers_ride_along_in_the_grouped_launches(models_dir, monkeypatch, model):
    """The 3x3 pooling branch of an Inception block shares the grouped launch of the convolutions of its depth
    (never the last launch of a group, whose block count the group declares).  Same arithmetic as the pooling
    kernels: the stage graphs give the bits of the kernel-by-kernel run and of a load with PB_FUSE_POOLS=0, for one
    request and for a gang of three."""
    path = os.path.join(models_dir, packer.pack_file_name(model))
    pools = (capi.STAGE_MAXPOOL, capi.STAGE_AVGPOOL)
    outs = {}
    for flag in ("1", "0"):
        monkeypatch.setenv("PB_FUSE_POOLS", flag)
        m = Model(path, 1)
        kinds = m.kinds()
        riding = 0
        first, count = C.c_int(), C.c_int()
        for g in range(m.L.pb_model_num_groups(m.m)):
            capi.check(m.L.pb_model_group_stages(m.m, g, C.byref(first), C.byref(count)), "group stages")
            order, launch = (C.c_int32 * count.value)(), (C.c_int32 * count.value)()
            assert m.L.pb_model_group_plan(m.m, g, order, launch, count.value) == count.value
            members = {}
            for s_idx, l_idx in zip(order, launch):
                members.setdefault(l_idx, []).append(kinds[s_idx])
            for l_idx, ks in members.items():
                if len(ks) > 1:
                    assert ks[0] == capi.STAGE_CONV_UMMA and all(k == capi.STAGE_CONV_UMMA or k in pools for k in ks)
                    n_pool = sum(1 for k in ks if k in pools)
                    riding += n_pool
                    assert n_pool == 0 or l_idx != launch[-1]
        # GoogLeNet: the max pool of every Inception module; Inception-v3: the max pools of its two reduction blocks (its
        # average pools carry the bias + ReLU tail of the convolution that runs before them and keep their own launch)
        assert (riding >= (2 if model == "inception_v3" else 8)) if flag == "1" else (riding == 0)
        x = make_input(model)
        y = m.run(x)
        np.testing.assert_array_equal(m.run_groups(x), y)
        outs[flag] = y
        m.close()
    np.testing.assert_array_equal(outs["1"], outs["0"])


def test_persistent_convolution_kernel_in_the_stage_graphs(tmp_path, monkeypatch):
    """PB_CONV_PERSIST=1 when the model is loaded: every tensor-core launch of the stage graphs runs the persistent kernel
    (a CTA walks three tiles, two accumulators in tensor memory).  Same arithmetic per output element, so with the
    reduction split switched off the logits are the bits of the kernel-by-kernel run (which uses the one-tile kernel),
    for one request and for a gang; the last group declares a third of the tiles as blocks."""
    d = tmp_path / "models_persist"           # own directory and load: the choice is made when a model is loaded
    d.mkdir()
    packer.write_all(str(d), ["inception_v3"])
    path = os.path.join(str(d), packer.pack_file_name("inception_v3"))
    L = capi.load()
    L.pb_set_conv_split_gain_us(1e9)
    try:
        plain = Model(path, 1)
        x = make_input("inception_v3")
        want = plain.run(x)
        li0 = capi.LaunchInfo()
        g_mid = 1                                  # a group that ends in a tensor-core convolution
        capi.check(L.pb_model_group_info(plain.m, g_mid, C.byref(li0)), "group info")
        plain.close()
        monkeypatch.setenv("PB_CONV_PERSIST", "1")
        m, inst = C.c_void_p(), C.c_void_p()
        capi.check(L.pb_model_load(path.encode(), 0, 1, C.byref(m)), "pb_model_load")
        capi.check(L.pb_instance_create_batched(m, 3, 0, C.byref(inst)), "pb_instance_create_batched")
        li1 = capi.LaunchInfo()
        capi.check(L.pb_model_group_info(m, g_mid, C.byref(li1)), "group info")
        assert li1.num_blocks == -(-li0.num_blocks // 3)       # a third of the tiles as CTAs: that many blocks notify
        xs = np.stack([x, make_input("inception_v3", 6), make_input("inception_v3", 7)]).astype(np.float32)
        y = np.zeros((3, 1000), np.float32)
        capi.check(L.pb_instance_run_batch_sync(inst, 1, 1, xs.ctypes.data, y.ctypes.data), "one request, graphs")
        assert gu.error_flag() == 0
        np.testing.assert_array_equal(y[0], want)
        y3 = np.zeros((3, 1000), np.float32)
        capi.check(L.pb_instance_run_batch_sync(inst, 3, 1, xs.ctypes.data, y3.ctypes.data), "gang of three, graphs")
        assert gu.error_flag() == 0
        np.testing.assert_array_equal(y3[0], want)
        ref = GOLDEN["inception_v3"]
        assert float(np.abs(y3[0] - ref).max()) <= 1e-2 * float(np.abs(ref).max())
        assert not np.array_equal(y3[1], y3[0])
        L.pb_instance_destroy(inst)
        L.pb_model_destroy(m)
    finally:
        L.pb_set_conv_split_gain_us(-1.0)
