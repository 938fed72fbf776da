"""Tiles of 256 rows on a pair of blocks, at the sizes where they can go wrong: fewer rows than one block's, rows that end in the first or
the second block, one k-block, more k-blocks than stages, ragged output channels, strides, images that straddle a tile, slices
and residuals, stores through TMA and direct.

Reference: the convolution of the bf16 operands in 64 bits.  Products of bf16 values are exact in fp32; n = C*R*S of them summed
in fp32 in any order differ from the exact sum by at most n * 2^-23 * sum |products| (every addition truncating, in the worst
order); one rounding to bf16 (2^-8 relative) follows."""
import ctypes as C
import os

import numpy as np
import pytest

from oracle import graph as og
from paella_b200 import capi, packer
from tests import gpu_util as gu
from tests.test_gpu_gang import _pinned, _run_until, _server
from tests.test_gpu_models import Model
from tests.test_gpu_serving_options import _register

pytestmark = pytest.mark.gpu

CASES = [
    # C, H, W, K, R, S, stride, pad_h, pad_w, images, act, residual, slice offset, out channels
    (8, 3, 3, 8, 1, 1, 1, 0, 0, 1, 0, False, 0, 8),               # nine rows: the second block has none; one k-block
    (64, 16, 8, 32, 1, 1, 1, 0, 0, 1, 1, True, 0, 32),            # exactly the first block's rows
    (64, 43, 3, 96, 1, 1, 1, 0, 0, 1, 1, False, 0, 96),           # one row in the second block
    (64, 16, 16, 64, 3, 3, 1, 1, 1, 1, 2, True, 0, 64),           # exactly one pair
    (72, 257, 1, 40, 1, 1, 1, 0, 0, 1, 1, False, 24, 80),         # one row of a second pair; 40 of 64 columns; a slice
    (288, 35, 35, 384, 3, 3, 1, 1, 1, 2, 1, False, 0, 384),       # two tiles of 192 columns, 45 k-blocks
    (128, 17, 17, 200, 1, 7, 1, 0, 3, 3, 1, True, 0, 200),        # 224 columns, 200 of them real
    (96, 31, 29, 256, 3, 3, 2, 0, 0, 5, 1, False, 0, 256),        # stride 2, images straddle tiles
    (64, 14, 14, 512, 1, 1, 1, 0, 0, 4, 3, False, 0, 512),        # PReLU
]


def _problem(case):
    """Operator parameters on the GPU (with what they point to) and the 64-bit result with its error bound."""
    import torch
    L = capi.load()
    c, h, w, k, r, s, stride, ph, pw, n, act, residual, off, total = case
    P, Q = (h + 2 * ph - r) // stride + 1, (w + 2 * pw - s) // stride + 1
    gen = torch.Generator(device="cuda").manual_seed(c * 131 + h)
    cs = (c + 7) // 8 * 8
    x = torch.relu(torch.randn((n, h, w, cs), generator=gen, device="cuda")).to(torch.bfloat16)
    wt = (torch.randn((k, c, r, s), generator=gen, device="cuda") * (2.0 / (c * r * s)) ** 0.5).to(torch.bfloat16)
    bias = torch.randn(2 * k, generator=gen, device="cuda") * 0.1          # PReLU: the slopes follow
    res = torch.randn((n, P, Q, k), generator=gen, device="cuda").to(torch.bfloat16)
    p = capi.OpParams()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks, p.out_c_off = 1, c, h, w, cs, k, P, Q, total, off
    p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.act, p.batch, p.dil_h, p.dil_w = r, s, stride, stride, ph, pw, 1, act, n, 1, 1
    host = wt.float().cpu().contiguous()
    size = L.pb_op_pack_weights(capi.STAGE_CONV_UMMA, C.byref(p), host.data_ptr(), None)
    packed = torch.zeros(size, dtype=torch.uint8)
    L.pb_op_pack_weights(capi.STAGE_CONV_UMMA, C.byref(p), host.data_ptr(), packed.data_ptr())
    packed = packed.cuda()
    p.x, p.w, p.bias = x.data_ptr(), packed.data_ptr(), bias.data_ptr()
    if residual:
        p.residual, p.res_Cs = res.data_ptr(), k
    xd, wd = x[..., :c].permute(0, 3, 1, 2).double().cpu(), wt.double().cpu()
    conv = lambda a, b: torch.nn.functional.conv2d(a, b, padding=(ph, pw), stride=stride).permute(0, 2, 3, 1)
    want = conv(xd, wd) + bias[:k].double().cpu()
    if residual:
        want = want + res.double().cpu()
    want = torch.relu(want) if act in (1, 2) else want
    want = torch.where(want > 0, want, want * bias[k:].double().cpu()) if act == 3 else want
    want = want.clamp(max=6.0) if act == 2 else want
    bound = c * r * s * 2.0 ** -23 * conv(xd.abs(), wd.abs()) + 2.0 ** -8 * want.abs() + 1e-6
    return p, (x, packed, bias, res), want, bound


def _launch(p):
    """The output of one launch, every channel of the destination."""
    import torch
    L = capi.load()
    y = torch.full((p.batch, p.P, p.Q, p.Ks), 7.0, device="cuda", dtype=torch.bfloat16)
    p.y = y.data_ptr()
    capi.check(L.pb_op_launch(capi.STAGE_CONV_UMMA, C.byref(p), None, 0, None), "pb_op_launch")
    torch.cuda.synchronize()
    assert gu.error_flag() == 0
    return y


def _geometry(p):
    li = capi.LaunchInfo()
    capi.check(capi.load().pb_op_info(capi.STAGE_CONV_UMMA, C.byref(p), C.byref(li)), "pb_op_info")
    return li.num_blocks, li.smem_per_block


@pytest.mark.parametrize("case", CASES)
def test_pairs_of_blocks(case, monkeypatch):
    """Both ways within the bound, and with the same bits: neither splits its reduction (no scratch memory is given)."""
    import torch
    p, keep, want, bound = _problem(case)
    k, off = case[3], case[12]
    got, geometry = {}, {}
    for mode in ("0", "1"):
        monkeypatch.setenv("PB_CONV_PAIR", mode)
        geometry[mode] = _geometry(p)
        got[mode] = _launch(p)
        y = got[mode][..., off:off + k].double().cpu()
        assert bool(((y - want).abs() <= bound).all()), float(((y - want).abs() / bound).max())
        untouched = torch.ones(p.Ks, dtype=torch.bool)
        untouched[off:off + k] = False
        assert bool((got[mode][..., untouched.cuda()] == 7.0).all())
    row_tiles, col_tiles = -(-p.batch * p.P * p.Q // 128), -(-k // 256)
    assert geometry["1"] != geometry["0"] and geometry["1"][0] == (row_tiles + 1) // 2 * 2 * col_tiles
    assert torch.equal(got["0"], got["1"])


def test_pairs_by_the_default_rule(monkeypatch):
    """50 pairs of 224 columns, 36 k-blocks: taken without the switch."""
    import torch
    p, keep, want, bound = _problem((256, 40, 40, 224, 3, 3, 1, 1, 1, 8, 1, True, 0, 224))
    got, geometry = {}, {}
    for mode in ("0", "1", ""):
        monkeypatch.setenv("PB_CONV_PAIR", mode)
        geometry[mode], got[mode] = _geometry(p), _launch(p)
    assert geometry[""] == geometry["1"] != geometry["0"]
    assert torch.equal(got[""], got["0"])
    assert bool(((got[""].double().cpu() - want).abs() <= bound).all())


def test_pairs_report_every_block_beside_other_requests(tmp_path, monkeypatch):
    """PB_CONV_PAIR=1 on a server, three launches a stage: stages end in a pair launch, behind a programmatic predecessor, which
    reports the blocks it was declared with while other requests' convolutions run on other streams."""
    d = tmp_path / "models_pairs_served"
    d.mkdir()
    packer.write_all(str(d), ["resnet18"])
    monkeypatch.delenv("PB_PRECISION", raising=False)
    monkeypatch.setenv("PB_CONV_PAIR", "1")
    monkeypatch.setenv("PB_STAGE_GROUP", "3")
    L, s = _server(str(d), monkeypatch, 1)
    job, ib, ob, sb = _register(L, s, "tvm_resnet18")
    n = 6
    t, xs = _pinned(sb * n), np.random.default_rng(3).standard_normal((n, 3, 224, 224), dtype=np.float32)
    for i in range(n):
        t.numpy()[i * sb:i * sb + ib] = np.frombuffer(xs[i].tobytes(), np.uint8)
        capi.check(L.pb_server_launch(s, job, t.data_ptr() + i * sb, i), "launch")
    done = _run_until(L, s, n, timeout=20.0)
    assert done == {i: 0 for i in range(n)}, "a request was not answered"
    assert gu.error_flag() == 0
    pack, off = og.Pack(packer.MODELS["resnet18"](seed=1234).to_bytes()), (ib + 7) // 8 * 8
    ys = [np.frombuffer(t.numpy()[i * sb + off:i * sb + off + ob].tobytes(), np.float32) for i in range(n)]
    for i in (0, n - 1):
        ref = og.run(pack, xs[i])
        assert float(np.abs(ys[i] - ref).max()) <= 1e-2 * float(np.abs(ref).max())
    L.pb_server_destroy(s)
    # the stages do end in pair launches: their declared geometry is not the lone blocks'
    path, li, ends = os.path.join(str(d), packer.pack_file_name("resnet18")), capi.LaunchInfo(), {}
    for mode in ("0", "1"):
        monkeypatch.setenv("PB_CONV_PAIR", mode)
        m = Model(path, 1)
        capi.check(L.pb_model_group_info(m.m, 1, C.byref(li)), "group info")
        ends[mode] = li.num_blocks
        m.close()
    assert ends["1"] != ends["0"] and ends["1"] % 2 == 0


def test_the_plan_of_a_model_does_not_change_its_bits(tmp_path, monkeypatch):
    """A convolution that runs on pairs of blocks in the default plan (and whose reduction lone blocks would split), with a pooling
    layer in its launch, and in launches of other groupings: the same bits."""
    g = packer.Graph("pairs", (16, 40, 40), seed=3, precision=1, round_weights_bf16=True)
    x = g.conv(g.input, 1024, 1, name="wide")
    cat = g.tensor(192 + 1024, 40, 40)
    g.conv(x, 192, 3, 1, 1, name="big", out=cat, out_c_off=0)
    g.maxpool(x, 3, 1, 1, out=cat, out_c_off=192, name="pool")
    g.dense(g.gap(g.conv(cat, 32, 1, name="next"), name="gap"), 10, name="fc")
    path = g.save(str(tmp_path / "pairs.bin"))
    xs = np.random.default_rng(4).standard_normal((8, 16, 40, 40), dtype=np.float32)
    switches = ["PB_CONV_PAIR", "PB_FUSE_POOLS", "PB_STAGE_GROUP", "PB_FUSE_BRANCHES"]
    outs, smem, split, li = {}, {}, {}, capi.LaunchInfo()
    for name, value in [(None, None), ("PB_CONV_PAIR", "0"), ("PB_FUSE_POOLS", "1"), ("PB_STAGE_GROUP", "2"), ("PB_FUSE_BRANCHES", "0")]:
        for sw in switches:
            monkeypatch.delenv(sw, raising=False)
        if name:
            monkeypatch.setenv(name, value)
        m = Model(path, 1)
        names = [m.L.pb_model_stage_name(m.m, s).decode() for s in range(m.L.pb_model_num_stages(m.m))]
        capi.check(m.L.pb_model_stage_info_batched(m.m, names.index("big"), 8, C.byref(li)), "stage info")
        smem[name], split[name] = li.smem_per_block, li.num_blocks > 100
        inst, y = C.c_void_p(), np.zeros((8, 10), np.float32)
        capi.check(m.L.pb_instance_create_batched(m.m, 8, 0, C.byref(inst)), "pb_instance_create_batched")
        capi.check(m.L.pb_instance_run_batch_sync(inst, 8, 1, xs.ctypes.data, y.ctypes.data), "run batch")
        outs[name] = y
        m.L.pb_instance_destroy(inst)
        m.close()
    assert split["PB_CONV_PAIR"] and not split[None]       # 100 row tiles: lone blocks split them, pairs do not
    assert smem[None] == smem["PB_STAGE_GROUP"] == smem["PB_FUSE_BRANCHES"] != smem["PB_FUSE_POOLS"]
    for name in ("PB_FUSE_POOLS", "PB_STAGE_GROUP", "PB_FUSE_BRANCHES"):
        np.testing.assert_array_equal(outs[name], outs[None], err_msg=name)
