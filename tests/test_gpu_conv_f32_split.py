"""Dense fp32 convolutions on the tensor cores (operands split into three bf16 parts) at the sizes where they can go wrong, against
torch in 64 bits.

Bound: an output is sum(x w) over n = C*R*S products.  The parts reproduce the operands exactly; the one product of parts that is left out is at
most 2^-34 of each product.  A step of 64 products is four additions of 16 exact products each to an fp32 accumulator, every one of which
may truncate (2^-23 of a partial sum, itself at most sum|x w| of the step), and one rounding to nearest adds it to the sums of the steps
before it: together at most (8 + n / 64) * 2^-23 * sum|x w|.  Bias, residual and result add one rounding each."""
import ctypes as C
import os

import pytest

from paella_b200 import capi
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

CASES = [
    # N, C, H, W, K, R, S, stride, pad_h, pad_w, dilation    (tiles of 128 rows x 64 or 32 columns, steps of two boxes of 32 channels)
    (1, 24, 8, 16, 40, 1, 1, 1, 0, 0, 1),          # the fewest channels: one box, cut; exactly one row tile
    (1, 24, 3, 43, 8, 3, 3, 1, 1, 1, 1),           # 129 rows; 8 of 32 columns; nine boxes: the last step has one
    (1, 31, 1, 127, 33, 1, 3, 1, 0, 1, 1),         # 127 rows, 33 columns of 64, rows of weights padded to 36
    (1, 32, 9, 7, 64, 1, 1, 1, 0, 0, 1),           # exactly a box and a tile's columns
    (2, 33, 9, 7, 65, 1, 1, 1, 0, 0, 1),           # a second box of one channel, a second column tile of one column, images in one tile
    (3, 63, 11, 13, 96, 3, 3, 1, 1, 1, 1),         # tiles straddle images, odd maps
    (1, 64, 20, 20, 36, 5, 5, 2, 2, 2, 1),         # stride 2, 36 columns
    (2, 65, 15, 9, 64, 3, 3, 2, 0, 0, 1),          # three boxes a tap
    (1, 48, 19, 23, 40, 3, 3, 1, 3, 2, 2),         # dilated, unequal padding
    (1, 200, 7, 7, 48, 1, 1, 1, 0, 0, 1),          # 4 steps: two ranks
    (1, 128, 14, 14, 128, 3, 3, 1, 1, 1, 1),       # 18 steps: four ranks
    (2, 512, 7, 7, 512, 3, 3, 1, 1, 1, 1),         # 72 steps: eight ranks, 98 rows
    (1, 320, 4, 8, 64, 3, 3, 1, 1, 1, 1),          # 45 steps on 32 rows: most ranks finish rows that do not exist
    (4, 96, 56, 56, 64, 3, 3, 1, 1, 1, 1),         # the operands' ring goes round
    (16, 32, 61, 59, 64, 1, 1, 1, 0, 0, 1),        # several waves of one step each
    # four channels a pixel: a row of the filter is a chunk
    (2, 3, 41, 39, 64, 7, 7, 2, 3, 3, 1),          # seven chunks, tiles straddle images
    (1, 4, 16, 8, 33, 3, 8, 1, 1, 4, 1),           # eight taps a row
    (1, 1, 3, 43, 40, 3, 3, 1, 1, 1, 1),           # one channel, 129 rows
    (1, 2, 9, 9, 64, 1, 5, 1, 0, 2, 1),            # one chunk
    (3, 3, 30, 30, 16, 3, 3, 2, 0, 0, 1),          # 16 columns
    (1, 3, 64, 5, 64, 16, 3, 1, 8, 1, 1),          # sixteen chunks: eight steps, two ranks or more
]


def _prepare(case, act=1, residual=False, cs=None, total=None, off=0, seed=0, x=None):
    import torch
    n, c, h, w, k, r, s, stride, ph, pw, d = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    cs, total = cs or (c + 3) // 4 * 4, total or (k + 3) // 4 * 4
    P, Q = (h + 2 * ph - (r - 1) * d - 1) // stride + 1, (w + 2 * pw - (s - 1) * d - 1) // stride + 1
    p = capi.OpParams()
    p.dtype, p.C, p.H, p.W, p.Cs, p.K, p.P, p.Q, p.Ks = 0, c, h, w, cs, k, P, Q, total
    p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.dil_h, p.dil_w = r, s, stride, stride, ph, pw, d, d
    p.groups, p.act, p.batch, p.out_c_off = 1, act, n, off
    t = {"x": torch.full((n, h, w, cs), float("nan"), device="cuda"), "w": rnd(k, c, r, s) * (2.0 / (c * r * s)) ** 0.5,
         "b": rnd(2 * k) * 0.1, "res": rnd(n, P, Q, k), "y": torch.full((n, P, Q, total), 7.0, device="cuda")}
    t["x"][..., :c] = rnd(n, h, w, c) if x is None else x
    t["wd"] = gu.pack_weights(capi.STAGE_CONV_SIMT, p, t["w"].cpu().numpy())
    p.x, p.w, p.bias, p.y = t["x"].data_ptr(), t["wd"].data_ptr(), t["b"].data_ptr(), t["y"].data_ptr()
    if residual:
        t["res"] = torch.nn.functional.pad(t["res"], (0, -k % 4)).contiguous()
        p.residual, p.res_Cs = t["res"].data_ptr(), t["res"].shape[-1]
    return p, t


def _launch(p):
    capi.check(capi.load().pb_op_launch(capi.STAGE_CONV_SIMT, C.byref(p), None, 0, None), "pb_op_launch")
    gu.sync()
    assert gu.error_flag() == 0


def _reference(p, t, residual):
    """The result in 64 bits, the bound on its error, and that on a chain of fp32 multiply-adds."""
    import torch
    x, w = t["x"][..., :p.C].permute(0, 3, 1, 2).double(), t["w"].double()
    conv = lambda a, b: torch.nn.functional.conv2d(a, b, None, (p.stride_h, p.stride_w), (p.pad_h, p.pad_w), (p.dil_h, p.dil_w)).permute(0, 2, 3, 1)
    y, mass = conv(x, w), conv(x.abs(), w.abs())
    y = y + t["b"][:p.K].double()
    if residual:
        y = y + t["res"][..., :p.K].double()
    n, last = p.C * p.R * p.S, 4 * 2.0 ** -24 * (y.abs() + mass)
    bound, chain = (8 + n / 64) * 2.0 ** -23 * mass + last, n * 2.0 ** -24 * mass + last
    if p.act == 3:
        slope = t["b"][p.K:].double()
        y, bound = torch.where(y > 0, y, y * slope), bound * torch.clamp(slope.abs(), min=1.0)
    elif p.act:
        y = torch.clamp(y, min=0.0, max=6.0 if p.act == 2 else None)
    return y, bound, chain


def _kernel_threads(p):
    li = capi.LaunchInfo()
    capi.check(capi.load().pb_op_info(capi.STAGE_CONV_SIMT, C.byref(p), C.byref(li)), "pb_op_info")
    return li.threads_per_block


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("case", CASES)
def test_within_the_bound(case, residual):
    p, t = _prepare(case, act=CASES.index(case) % 4, residual=residual)
    assert _kernel_threads(p) == 832
    _launch(p)
    y, bound, _ = _reference(p, t, residual)
    assert ((t["y"][..., :p.K].double() - y).abs() <= bound).all()
    assert (t["y"][..., p.K:] == 7.0).all()


@pytest.mark.parametrize("total,off", [(72, 8), (47, 3)])
def test_slice_of_a_wider_output(total, off):
    p, t = _prepare((1, 40, 9, 11, 36, 3, 3, 1, 1, 1, 1), residual=True, total=total, off=off)
    _launch(p)
    y, bound, _ = _reference(p, t, True)
    assert ((t["y"][..., off:off + 36].double() - y).abs() <= bound).all()
    assert (t["y"][..., :off] == 7.0).all() and (t["y"][..., off + 36:] == 7.0).all()


@pytest.mark.parametrize("case", [CASES[5], CASES[9], CASES[11]])
def test_no_further_off_than_the_fp32_units(case, monkeypatch):
    errors = []
    for on in "10":
        monkeypatch.setenv("PB_F32_SPLIT", on)
        p, t = _prepare(case, act=0)
        assert _kernel_threads(p) == (832 if on == "1" else 256)
        _launch(p)
        y = _reference(p, t, False)[0]
        errors.append(((t["y"][..., :p.K].double() - y).norm() / y.norm()).item())
    assert errors[0] <= errors[1]


@pytest.mark.parametrize("case", [(1, 40, 13, 11, 72, 3, 3, 1, 1, 1, 1), (1, 512, 7, 7, 64, 1, 1, 1, 0, 0, 1)])
def test_values_that_are_not_finite(case, monkeypatch):
    """Infinities, NaN, and finite values whose rounding to bf16 or whose sum is not: as on the fp32 units."""
    import torch
    n, c, h, w = case[:4]
    x = torch.randn((n, h, w, c), generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
    x[0, 1, 2, 3], x[0, 2, 5, 0], x[0, 4, 4, 5], x[0, 5, 1, 7], x[0, 6, 6, 1] = float("inf"), -float("inf"), float("nan"), 3.4e38, -3.4e38
    outs = []
    for on in "10":
        monkeypatch.setenv("PB_F32_SPLIT", on)
        p, t = _prepare(case, act=0, x=x)
        _launch(p)
        outs.append(t["y"][..., :p.K])
    a, b = outs
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isposinf(a), torch.isposinf(b)) and torch.equal(torch.isneginf(a), torch.isneginf(b))
    ok = torch.isfinite(b)
    assert 0 < ok.sum() < ok.numel()
    assert ((a[ok] - b[ok]).double().norm() <= 1e-5 * b[ok].double().norm())


@pytest.mark.parametrize("case", CASES)
def test_second_pass(case):
    """The same, and operands that are too large for the parts, at every tile, rank count and edge: not finite where the sums in 64 bits are
    not, within the bound everywhere else."""
    import torch
    n, c, h, w = case[:4]
    x = torch.randn((n, h, w, c), generator=torch.Generator(device="cuda").manual_seed(4), device="cuda")
    for i, v in enumerate((float("inf"), -float("inf"), float("nan"), 2.0 ** 113, -3.4e37)):
        x.view(-1)[(i + 1) * x.numel() // 7] = v
    p, t = _prepare(case, act=0, residual=True, x=x)
    _launch(p)
    y, bound, _ = _reference(p, t, True)
    out, want = t["y"][..., :p.K], y.float()
    ok = torch.isfinite(want)
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isposinf(out), torch.isposinf(want)) and torch.equal(torch.isneginf(out), torch.isneginf(want))
    assert ((out.double() - y).abs()[ok] <= bound[ok]).all() and (t["y"][..., p.K:] == 7.0).all()


@pytest.mark.parametrize("case", [CASES[2], CASES[10], CASES[15]])
def test_infinite_weights_meet_the_padding(case, monkeypatch):
    """Zeros beyond the edge times infinity, as on the fp32 units."""
    import torch
    outs = []
    for on in "10":
        monkeypatch.setenv("PB_F32_SPLIT", on)
        p, t = _prepare(case, act=0)
        t["w"][1, 0, 0, 0], t["w"][5, -1, -1, -1] = float("inf"), -float("inf")
        t["wd"] = gu.pack_weights(capi.STAGE_CONV_SIMT, p, t["w"].cpu().numpy())
        p.w = t["wd"].data_ptr()
        _launch(p)
        outs.append(t["y"][..., :p.K])
    a, b = outs
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isinf(a), torch.isinf(b)) and torch.isnan(b).any()


@pytest.mark.parametrize("case", [CASES[10], CASES[13], CASES[15]])
def test_poisoned_launches_take_no_longer_than_a_few_ordinary_ones(case, monkeypatch):
    """Every pixel NaN: measured at 1.4 to 2 times the launch on the fp32 units (a serial sum per output took 20 to 50)."""
    import torch
    times = []
    for on in "10":
        monkeypatch.setenv("PB_F32_SPLIT", on)
        p, t = _prepare(case, act=0)
        t["x"].fill_(float("nan"))
        _launch(p)
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        best = 1e9
        for _ in range(5):
            e[0].record()
            for _ in range(10):
                capi.load().pb_op_launch(capi.STAGE_CONV_SIMT, C.byref(p), None, 0, None)
            e[1].record()
            gu.sync()
            best = min(best, e[0].elapsed_time(e[1]))
        times.append(best)
    assert times[0] < 4 * times[1]


@pytest.mark.parametrize("act,k", [(0, 64), (3, 37)])
@pytest.mark.parametrize("exponent", [-108, -114, -122])
def test_operands_whose_parts_bf16_cannot_hold(exponent, act, k):
    """No further off than a chain of fp32 multiply-adds, the steps of the least fp32 values included."""
    import torch
    p, t = _prepare((2, 64, 9, 9, k, 3, 3, 1, 1, 1, 1), act=act, x=torch.randn((2, 9, 9, 64), generator=torch.Generator(device="cuda").manual_seed(5), device="cuda") * 2.0 ** exponent)
    t["b"][:k] = 0.0
    _launch(p)
    y, _, chain = _reference(p, t, False)
    assert ((t["y"][..., :k].double() - y).abs() <= chain + 64 * 9 * 2.0 ** -149).all()


@pytest.mark.parametrize("case", [(2, 64, 9, 9, 64, 1, 1, 1, 0, 0, 1), (1, 512, 16, 16, 40, 1, 1, 1, 0, 0, 1), (2, 3, 32, 32, 64, 3, 3, 1, 1, 1, 1)])
def test_a_sum_of_one_product_is_rounded_once(case):
    """One channel of one pixel of the window is not zero: what is left out (2^-34) and lost in the sum of the small products (eight of
    2^-8, truncated at 2^-23 each) is within 2^-27 of the result, besides the half unit, 2^-24, of its one rounding."""
    import torch
    n, c, h, w, k = case[:5]
    gen = torch.Generator(device="cuda").manual_seed(2)
    x = torch.zeros((n, h, w, c), device="cuda")
    x[:, ::3, ::3, :] = torch.nn.functional.one_hot(torch.arange(x[:, ::3, ::3, 0].numel(), device="cuda") % c, c).view_as(x[:, ::3, ::3, :]) * 1.0
    x *= 1 + torch.rand(x.shape, generator=gen, device="cuda")
    x[x > 1.98] = 1 + 2.0 ** -8 - 2.0 ** -17         # the largest second and third parts
    p, t = _prepare(case, act=0, x=x)
    t["w"] = 1 + torch.rand(t["w"].shape, generator=gen, device="cuda")
    t["w"].view(-1)[::3] = 1 + 2.0 ** -8 - 2.0 ** -17
    t["wd"], p.bias = gu.pack_weights(capi.STAGE_CONV_SIMT, p, t["w"].cpu().numpy()), None
    p.w = t["wd"].data_ptr()
    _launch(p)
    y = _reference(p, t, False)[0] - t["b"][:k].double()
    assert ((t["y"][..., :k].double() - y).abs() <= (2.0 ** -24 + 2.0 ** -27) * y.abs()).all()


@pytest.mark.parametrize("act,k", [(0, 64), (3, 37)])
@pytest.mark.parametrize("where", ["all", "channel", "image"])
@pytest.mark.parametrize("small,large", [(-118, 30), (-126, 60), (-140, 100)])
def test_small_operands_that_meet_large_factors(small, large, where, act, k):
    """Operands whose ends bf16 cannot hold, in results of any size: all of them, one output channel, one image of a batch.  The sums
    are rounded to fp32 once a rank, to a multiple of 2^-149."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn((3, 9, 9, 64), generator=gen, device="cuda")
    p, t = _prepare((3, 64, 9, 9, k, 3, 3, 1, 1, 1, 1), act=act, x=x)
    if where == "channel":
        x, t["w"][k // 2] = x * 2.0 ** large, t["w"][k // 2] * 2.0 ** small
    else:
        x[slice(None) if where == "all" else slice(1, 2)] *= 2.0 ** small
        t["w"] *= 2.0 ** large
    t["x"][..., :64] = x
    t["wd"] = gu.pack_weights(capi.STAGE_CONV_SIMT, p, t["w"].cpu().numpy())
    p.w = t["wd"].data_ptr()
    t["b"][:k] = 0.0
    _launch(p)
    y, bound, _ = _reference(p, t, False)
    assert ((t["y"][..., :k].double() - y).abs() <= bound + 8 * 2.0 ** -149).all()


@pytest.mark.parametrize("what", ["x", "w", "size", "narrow", "few", "stem"])
def test_what_stays_on_the_fp32_units(what):
    import torch
    case = {"narrow": (1, 64, 9, 9, 32, 1, 1, 1, 0, 0, 1), "few": (1, 23, 9, 9, 64, 3, 3, 1, 1, 1, 1),
            "stem": (1, 3, 20, 20, 15, 3, 3, 2, 1, 1, 1)}.get(what, (1, 64, 9, 9, 64, 3, 3, 1, 1, 1, 1))
    p, t = _prepare(case)
    rows = p.P
    if what in ("x", "w"):
        old = t["x"] if what == "x" else t["wd"].view(torch.float32)
        t["moved"] = torch.zeros(old.numel() + 1, device="cuda")
        t["moved"][1:] = old.reshape(-1)
        setattr(p, what, t["moved"].data_ptr() + 4)
    if what == "size":
        p.P = rows = 8                       # fewer rows than padding and filter give
        t["y"] = torch.full((1, 8, p.Q, p.Ks), 7.0, device="cuda")
        p.y = t["y"].data_ptr()
    assert _kernel_threads(p) == 256
    _launch(p)
    y, _, chain = _reference(p, t, False)
    assert ((t["y"][..., :p.K].double() - y[:, :rows]).abs() <= chain[:, :rows]).all()


@pytest.mark.parametrize("what", ["x", "w"])
@pytest.mark.parametrize("case", [CASES[5], CASES[10], CASES[11], CASES[14], CASES[15]])
def test_the_declared_blocks_do_not_depend_on_where_the_tensors_are(case, what):
    """Declared before the tensors are known, launched with one off 16 bytes: as many starts and ends as declared, twice."""
    import torch
    from tests.test_gpu_ring import _drain, _unpack
    from oracle import scheduler as osch
    L, ring, nf = capi.load(), C.c_void_p(), C.c_void_p()
    capi.check(L.pb_ring_create(0, 1 << 16, C.byref(ring)), "pb_ring_create")
    capi.check(L.pb_notifier_create_array(ring, 1, C.byref(nf)), "pb_notifier_create_array")
    p, t = _prepare(case)
    x, w, p.x, p.w = p.x, p.w, None, None
    li = capi.LaunchInfo()
    capi.check(L.pb_op_info(capi.STAGE_CONV_SIMT, C.byref(p), C.byref(li)), "pb_op_info")
    assert li.threads_per_block == 832
    p.x, p.w = x, w
    old = t["x"] if what == "x" else t["wd"].view(torch.float32)
    t["moved"] = torch.zeros(old.numel() + 1, device="cuda")
    t["moved"][1:] = old.reshape(-1)
    setattr(p, what, t["moved"].data_ptr() + 4)
    want = sorted(osch.notifier_records(li.num_blocks))
    for job in (5, 6):
        capi.check(L.pb_op_launch(capi.STAGE_CONV_SIMT, C.byref(p), None, job, nf), "pb_op_launch")
        gu.sync()
        recs = [_unpack(r) for r in _drain(L, ring, 2 * len(want), timeout=2.0)]
        for kind in (0, 1):
            assert sorted(r["num"] for r in recs if r["is_start"] == kind and r["job_id"] == job) == want
    L.pb_notifier_free_array(nf)
    L.pb_ring_destroy(ring)
