"""Split reductions of the tensor-core convolution: the parts that the ranks of a cluster send each other, beside the pipeline and in its
buffers, at two, four and eight ranks and parts of 8 to 64 columns, launch after launch; the order in which they are added.

Reference: the convolution of the bf16 operands in 64 bits.  n products of bf16 values, exact in fp32, summed in fp32 in any order differ
from the exact sum by at most n * 2^-23 * sum|products| (every addition truncating); the result is rounded to bf16 once."""
import ctypes as C

import pytest

from paella_b200 import capi
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

CASES = [
    # N, C, H, K, R, columns of a tile, ranks, are the parts beside the pipeline
    (1, 256, 7, 16, 1, 16, 2, True),             # the narrowest part
    (1, 64, 14, 16, 3, 32, 4, True),
    (2, 128, 28, 256, 3, 64, 2, True),
    (8, 256, 17, 256, 3, 96, 2, True),
    (8, 256, 17, 384, 3, 128, 2, False),         # the widest part
    (2, 256, 28, 512, 3, 112, 2, False),
    (1, 64, 7, 16, 3, 32, 4, True),              # 49 rows
    (1, 256, 28, 384, 3, 96, 4, False),          # parts of 24 columns
    (1, 256, 28, 512, 3, 128, 4, False),
    (8, 256, 14, 256, 3, 128, 4, False),         # tiles straddle images
    (1, 256, 7, 64, 3, 64, 8, True),
    (1, 128, 17, 512, 3, 64, 4, True),
    (1, 512, 17, 512, 3, 128, 8, False),         # eight ranks that send into each other's buffers
    (8, 256, 17, 160, 5, 64, 4, False),          # 25 k-blocks a rank: a stage more instead of a place beside the pipeline
    (1, 520, 8, 72, 3, 64, 8, True),             # channels and columns past whole boxes and tiles
]


def _check_route(li, n, c, h, k, r, columns, ranks, beside):
    """The tile, the ranks and the place of the parts that the case is about: by the launch's blocks and shared memory (stages of 128 rows and
    `columns` of 64 values of k in 109 KB, with the other ranks' parts or under them)."""
    assert li.num_blocks == -(-n * h * h // 128) * -(-k // columns) * ranks
    stage, parts, k_blocks = 16384 + columns * 128, (columns - columns // ranks) * 512, -(-r * r * -(-c // 64) // ranks)
    stages = (111616 - (parts if beside else 0)) // stage
    room = (111616 - parts) // stage
    assert beside == (room >= max(2, min(3, k_blocks)) and (k_blocks <= 20 or room >= min(8, k_blocks, 111616 // stage)))
    pipe = max(2, min(8, k_blocks, stages)) * stage
    assert 1024 <= li.smem_per_block - (pipe + parts if beside else max(pipe, parts)) < 4096          # (alignment; barriers and biases)


def _params(case, act=1):
    n, c, h, k, r = case[:5]
    p = capi.OpParams()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks = 1, c, h, h, c, k, h, h, k
    p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.act, p.batch = r, r, 1, 1, r // 2, r // 2, 1, act, n
    return p


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("case", CASES)
def test_parts(case, residual):
    import torch
    L = capi.load()
    n, c, h, k, r = case[:5]
    gen = torch.Generator(device="cuda").manual_seed(c + k)
    rnd = lambda *s: torch.randn(s, generator=gen, device="cuda")
    x, res, b = rnd(n, h, h, c).relu().to(torch.bfloat16), rnd(n, h, h, k).to(torch.bfloat16), rnd(k) * 0.1
    w = (rnd(k, c, r, r) * (2.0 / (c * r * r)) ** 0.5).to(torch.bfloat16)
    p = _params(case)
    wd, scratch = gu.pack_weights(capi.STAGE_CONV_UMMA, p, w.float().cpu().numpy()), torch.zeros(4096, dtype=torch.uint8, device="cuda")
    ys = torch.full((6, n, h, h, k), 7.0, dtype=torch.bfloat16, device="cuda")
    p.x, p.w, p.bias, p.scratch, p.scratch_bytes = x.data_ptr(), wd.data_ptr(), b.data_ptr(), scratch.data_ptr(), 4096
    if residual:
        p.residual, p.res_Cs = res.data_ptr(), k
    p.y = ys.data_ptr()
    li = capi.LaunchInfo()
    capi.check(L.pb_op_info(capi.STAGE_CONV_UMMA, C.byref(p), C.byref(li)), "pb_op_info")
    assert li.scratch_bytes > 0                       # it does split
    _check_route(li, *case)
    for y in ys:                                      # back to back: a block's memory is the next one's
        p.y = y.data_ptr()
        capi.check(L.pb_op_launch(capi.STAGE_CONV_UMMA, C.byref(p), None, 0, None), "pb_op_launch")
    gu.sync()
    assert gu.error_flag() == 0
    for y in ys[1:]:
        assert torch.equal(y, ys[0])
    conv = lambda a, b2: torch.nn.functional.conv2d(a.permute(0, 3, 1, 2).double(), b2.double(), None, 1, r // 2).permute(0, 2, 3, 1)
    ref, mass = conv(x, w) + b.double(), conv(x.abs(), w.abs())
    if residual:
        ref = ref + res.double()
    ref = ref.relu()
    assert ((ys[0].double() - ref).abs() <= (c * r * r + 4) * 2.0 ** -23 * (mass + ref) + 2.0 ** -8 * ref).all()


@pytest.mark.parametrize("case", CASES)
def test_the_order_of_the_parts(case):
    """One product a rank, of sizes that tell the order of their sum in fp32: a column's own rank first, then the others in rank order."""
    import numpy as np
    import torch
    n, c, h, k, r, columns, ranks, _ = case
    L, p = capi.load(), _params(case, act=0)
    cpt, nkb = -(-c // 64), r * r * -(-c // 64)
    vals = np.array([2.0 ** 24, 1, -2.0 ** 24, 3, 2.0 ** 25, 5, -2.0 ** 25, 7], np.float32)[:ranks]
    w = np.zeros((k, c, r, r), np.float32)
    for z in range(ranks):
        kb = nkb * z // ranks                      # the rank's first block of 64 values of k
        w[:, kb % cpt * 64, kb // cpt // r, kb // cpt % r] = vals[z]
    x, scratch = torch.ones((n, h, h, c), dtype=torch.bfloat16, device="cuda"), torch.zeros(4096, dtype=torch.uint8, device="cuda")
    y, b, wd = torch.full((n, h, h, k), 7.0, dtype=torch.bfloat16, device="cuda"), torch.zeros(k, device="cuda"), gu.pack_weights(capi.STAGE_CONV_UMMA, p, w)
    p.x, p.w, p.bias, p.y, p.scratch, p.scratch_bytes = x.data_ptr(), wd.data_ptr(), b.data_ptr(), y.data_ptr(), scratch.data_ptr(), 4096
    capi.check(L.pb_op_launch(capi.STAGE_CONV_UMMA, C.byref(p), None, 0, None), "pb_op_launch")
    gu.sync()
    assert gu.error_flag() == 0
    want = []
    for col in range(k):
        own = col % columns // (columns // ranks)
        total = vals[own]
        for z in range(ranks):
            if z != own:
                total = np.float32(total + vals[z])
        want.append(total)
    e = r // 2                                     # (the border's windows reach outside)
    assert (y[:, e:h - e, e:h - e] == torch.tensor(np.array(want), device="cuda").to(torch.bfloat16)).all()


def test_ranks_without_k_blocks(tmp_path):
    """A 1x1 layer of one k-block in a grouped launch whose 3x3 layer splits: most ranks have nothing to send."""
    import numpy as np
    from oracle import graph as og
    from paella_b200 import packer
    L = capi.load()
    g = packer.Graph("idle", (64, 7, 7), seed=4, precision=1, round_weights_bf16=True)
    t = g.conv(g.input, 64, 1, name="first")
    cat = g.tensor(16 + 64, 7, 7)
    g.conv(t, 16, 1, name="short", out=cat, out_c_off=0)
    g.conv(t, 64, 3, 1, 1, name="long", out=cat, out_c_off=16)
    t = g.gap(cat, name="gap")
    g.dense(t, 10, name="fc")
    model, inst = C.c_void_p(), C.c_void_p()
    capi.check(L.pb_model_load(g.save(str(tmp_path / "idle.bin")).encode(), 0, 1, C.byref(model)), "pb_model_load")
    n = L.pb_model_num_stages(model)
    names = [L.pb_model_stage_name(model, i) for i in range(n)]
    order, launch = (C.c_int32 * n)(), (C.c_int32 * n)()
    assert L.pb_model_group_plan(model, 0, order, launch, n) == n
    of = {names[order[i]]: launch[i] for i in range(n)}
    assert of[b"short"] == of[b"long"]
    li = capi.LaunchInfo()
    capi.check(L.pb_model_stage_info(model, names.index(b"short"), C.byref(li)), "pb_model_stage_info")
    assert li.num_blocks >= 2                      # one row tile and one column tile: the ranks
    capi.check(L.pb_instance_create(model, C.byref(inst)), "pb_instance_create")
    for seed in range(3):
        x, y = np.random.default_rng(seed).standard_normal((64, 7, 7), dtype=np.float32), np.zeros(10, np.float32)
        capi.check(L.pb_instance_run_groups_sync(inst, x.ctypes.data, y.ctypes.data), "pb_instance_run_groups_sync")
        assert gu.error_flag() == 0
        ref = og.run(og.Pack(g.to_bytes()), x, emulate_bf16=True)
        assert np.abs(y - ref).max() <= 1e-2 * np.abs(ref).max()          # (the oracle rounds where the device does; sums in another order)
    L.pb_instance_destroy(inst)
    L.pb_model_destroy(model)
