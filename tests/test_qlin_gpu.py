# SPDX-License-Identifier: MIT
"""Decode linears on quantised weights (csrc/qlin_kernels.cu) at the edges of their tiles.

Oracle: the exact integer products in float64.  Tolerances: the bf16 result is rounded once (rel-L2 at
most 2^-9 / sqrt(3) per element on average, 2^-8 allowed); fp32 slabs carry the int32 -> fp32 conversions
and their sum only (2^-24 each; 2^-20 allowed).  Digits: exact down to 2^-15 of a row's largest element; what
they drop of an element is at most 2^-24 of the largest and 2^-11 of the median of a row."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = a.double(), b.double()  # rows here go up to 1e31: squares need the range of a double
    return float((a - b).norm() / b.norm().clamp_min(1e-300))


TOL, TOL32 = 2.0 ** -8, 2.0 ** -20


def _g(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _x(m, k, seed, spread=False):
    x = torch.randn(m, k, generator=_g(seed), device="cuda")
    if spread:  # outliers and small elements in one row, as activations have
        x = x * torch.exp2(torch.randint(-6, 7, (m, k), generator=_g(seed + 1), device="cuda").float())
    return x.bfloat16()


def _w8(n, k, seed):
    wq = torch.randint(-127, 128, (n, k), generator=_g(seed), device="cuda", dtype=torch.int32).to(torch.int8)
    return wq, (torch.rand(n, generator=_g(seed + 1), device="cuda") * 0.01 + 1e-3).bfloat16()


def _pack4(t):  # eight values along the last dimension -> one int32
    v = sum(t.view(*t.shape[:-1], -1, 8)[..., j].long() << (4 * j) for j in range(8))
    return ((v + 2 ** 31) % 2 ** 32 - 2 ** 31).to(torch.int32)


# tokens: edges of the 16 / 32 / 64-token tiles; n: a ragged last row tile; k: a ragged last k-block
@pytest.mark.parametrize("m", [1, 16, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("n,k", [(128, 128), (200, 1040), (1000, 3584)])
def test_int8_weights_bf16_activations(ext, m, n, k):
    wq, sc = _w8(n, k, 3)
    x = _x(m, k, 5, spread=True)
    b = torch.randn(n, generator=_g(9), device="cuda").bfloat16()
    prod = (x.double() @ wq.double().t()) * sc.double()
    assert rel_l2(ext.w8a16_linear(x, wq, sc), prod) < TOL
    assert rel_l2(ext.w8a16_linear(x, wq, sc, b), prod + b.double()) < TOL
    y = prod + b.double()
    silu = torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2]
    assert rel_l2(ext.w8a16_linear(x, wq, sc, b, True), silu) < TOL
    out = ext.w8a16_linear_split(x, wq, sc)
    if out.dim() == 3:
        assert rel_l2(out.double().sum(0), prod) < TOL32
    kb = -(-k // 128)
    for splits in {1, 2, 5, kb}:
        if splits <= kb:
            assert rel_l2(ext.w8a16_linear(x, wq, sc, b, splits=splits), prod + b.double()) < TOL
    torch.cuda.synchronize()
    assert ext.w8_error_flag(0) == 0


# int8 activations: the tile of 128 tokens and its neighbours, ragged rows and k-blocks, with and without a k-split
@pytest.mark.parametrize("m", [63, 65, 127, 128])
@pytest.mark.parametrize("n,k", [(128, 128), (200, 1040), (1000, 3584)])
def test_int8_activations_up_to_128_tokens(ext, m, n, k):
    wq, sc = _w8(n, k, 3)
    x = _x(m, k, 5)
    b = torch.randn(n, generator=_g(9), device="cuda").bfloat16()
    xq, xs = ext.w8a16_quant_act(x)
    y = (xq.double() @ wq.double().t()) * xs.double()[:, None] * sc.double() + b.double()
    silu = torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2]
    for splits in (0, 1, 3):
        assert rel_l2(ext.w8a16_linear(x, wq, sc, b, splits=splits, act_int8=True), y) < TOL
        assert rel_l2(ext.w8a16_linear(x, wq, sc, b, True, splits, act_int8=True), silu) < TOL
    torch.cuda.synchronize()
    assert ext.w8_error_flag(0) == 0


# a bias that starts off a 16-byte boundary (a slice of a longer vector), with and without a k-split, and
# where the shape picks one by itself (the last)
@pytest.mark.parametrize("off", [1, 4])
@pytest.mark.parametrize("m,n,k", [(1, 136, 1040), (64, 200, 1040), (1, 4608, 3584)])
def test_bias_at_any_element(ext, off, m, n, k):
    wq, sc = _w8(n, k, 3)
    x = _x(m, k, 5)
    b = torch.randn(n + 8, generator=_g(9), device="cuda").bfloat16()[off:off + n]
    y = (x.double() @ wq.double().t()) * sc.double() + b.double()
    silu = torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2]
    for act_int8 in (False, True):
        if act_int8:
            xq, xs = ext.w8a16_quant_act(x)
            y = (xq.double() @ wq.double().t()) * xs.double()[:, None] * sc.double() + b.double()
        for splits in (0, 1, 3):
            assert rel_l2(ext.w8a16_linear(x, wq, sc, b, splits=splits, act_int8=act_int8), y) < TOL
        if not act_int8 and n % 16 == 0:
            for splits in (0, 1, 3):
                assert rel_l2(ext.w8a16_linear(x, wq, sc, b, True, splits), silu) < TOL
    torch.cuda.synchronize()
    assert ext.w8_error_flag(0) == 0


# a k-split that the caller asks for and n that the kernel behind it cannot store as vectors
@pytest.mark.parametrize("n", [129, 200, 202])
@pytest.mark.parametrize("splits", [2, 9, 99])
def test_asked_splits_of_odd_widths(ext, n, splits):
    wq, sc = _w8(n, 1040, 3)
    x = _x(3, 1040, 5)
    y = (x.double() @ wq.double().t()) * sc.double()
    assert rel_l2(ext.w8a16_linear(x, wq, sc, None, False, splits), y) < TOL
    if n % 2 == 0:
        silu = torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2]
        assert rel_l2(ext.w8a16_linear(x, wq, sc, None, True, splits), silu) < TOL


def test_no_rows(ext):
    wq, sc = _w8(200, 1024, 3)
    gs = torch.ones(200, 8, device="cuda").bfloat16()
    x = _x(1, 1024, 5)[:0]
    assert ext.w8a16_linear(x, wq, sc).shape == (0, 200)
    assert ext.w8a16_linear(x, wq, sc, None, True).shape == (0, 100)
    assert ext.w8a16_linear(x, wq, gs, act_int8=True, group_scale=gs).shape == (0, 200)


def test_too_many_rows_are_refused(ext):
    wq, sc = _w8(200, 1024, 3)
    gs = torch.ones(200, 8, device="cuda").bfloat16()
    with pytest.raises(RuntimeError, match="1..128"):
        ext.w8a16_linear_split(_x(129, 1024, 5), wq, sc)
    with pytest.raises(RuntimeError, match="at most 64"):
        ext.w8a16_linear(_x(65, 1024, 5), wq, gs, act_int8=True, group_scale=gs)
    with pytest.raises(RuntimeError, match="at most 64"):
        ext.w8a16_linear(_x(8, 1024, 5), wq, gs, group_scale=gs)


@pytest.mark.parametrize("m", [1, 32, 64])
@pytest.mark.parametrize("n,k,group", [(200, 1024, 128), (129, 768, 256)])
@pytest.mark.parametrize("act_int8", [False, True])
def test_int8_weights_group_scales(ext, m, n, k, group, act_int8):
    from barlink_sm86_b200 import ops
    wq, _ = _w8(n, k, 3)
    gs = (torch.rand(n, k // group, generator=_g(4), device="cuda") * 0.01 + 1e-3).bfloat16()
    x = _x(m, k, 5)
    if act_int8:
        xq, xs = ext.w8a16_quant_act(x)
        w = ops.ref.w8_dequant(wq, gs).double()
        want = (xq.double() @ w.t()) * xs.double()[:, None]
        got = ext.w8a16_linear(x, wq, gs, act_int8=True, group_scale=gs)
    else:
        s = ops.prepare_w8_scales(gs, k)
        w = ops.ref.w8_dequant(wq, s.rel.float() * s.row.float()[:, None]).double()
        want = x.double() @ w.t()
        got = ext.w8a16_linear(x, wq, s.row, group_rel=s.rel)
    assert rel_l2(got, want) < TOL
    torch.cuda.synchronize()
    assert ext.w8_error_flag(0) == 0


def _forms(ext, n, k):
    """(product of rows x, the same as fp32 where the form leaves slabs, dequantised weight) of the weight forms
    whose activations become digits."""
    from barlink_sm86_b200 import ops
    wq, sc = _w8(n, k, 7)
    wq[::3, ::5] = 0
    slabs = lambda y: y.double().sum(0) if y.dim() == 3 else y.double()
    yield (lambda x: ext.w8a16_linear(x, wq, sc)), (lambda x: slabs(ext.w8a16_linear_split(x, wq, sc))), wq, wq.double() * sc.double()[:, None]
    gs = (torch.rand(n, k // 128, generator=_g(4), device="cuda") * 0.01 + 1e-3).bfloat16()
    p = ops.prepare_w8_scales(gs, k)
    yield ((lambda x: ext.w8a16_linear(x, wq, p.row, group_rel=p.rel)), None, wq,
           ops.ref.w8_dequant(wq, p.rel.float() * p.row.float()[:, None]).double())
    nib = torch.randint(0, 16, (n, k), generator=_g(11), device="cuda")
    nib[::3, ::5] = 7
    zero = torch.randint(0, 16, (k // 128, n), generator=_g(12), device="cuda")
    zero[:, ::3] = 7
    s4 = (torch.rand(k // 128, n, generator=_g(13), device="cuda") * 0.01 + 1e-3).half()
    qw, qz = _pack4(nib).t().contiguous(), _pack4(zero)
    w4 = nib - zero.t().repeat_interleave(128, 1)
    yield ((lambda x: ext.w4a16_linear(x, qw, s4, qz)), (lambda x: slabs(ext.w4a16_linear(x, qw, s4, qz, want_slabs=True))),
           w4, w4.double() * s4.double().t().repeat_interleave(128, 1))


@pytest.mark.parametrize("m", [5, 16, 33])
@pytest.mark.parametrize("n,k", [(136, 384), (200, 4224), (136, 20608)])
@pytest.mark.parametrize("ratio", [12, 15, 18, 24, 60])
def test_outliers_that_meet_zero_weights(ext, m, n, k, ratio):
    """A few elements 2^ratio above the rest, in columns where a third of the weight rows are zero: those rows'
    results have only the small elements, and every one of them may be off by 2^-11 of the median at most
    (weights of a third of the rows are zero there, the others see what fp32 leaves of the large products)."""
    for f, f32, wi, w in _forms(ext, n, k):
        x = _x(m, k, 21)
        med = x.float().abs().median(1).values.double()
        cols = torch.arange(0, k, 5, device="cuda")[:: max(1, k // 5 // 7)]
        x[1::2, cols] = (x[1::2, cols].float() * 2.0 ** ratio).bfloat16()
        want = x.double() @ w.t()
        # zero weights at the outliers: rows 0, 3, 6, ... ; one bf16 rounding of the result, then the digits
        drop = 2.0 ** -11 * med[:, None] * w.abs().sum(1)[None, :]
        assert bool((wi[::3][:, cols] == 0).all())
        y = f(x).double()
        assert bool(((y - want).abs() <= 2.0 ** -8 * want.abs() + drop)[:, ::3].all())
        assert rel_l2(y, want) < TOL
        assert rel_l2(y[:, ::3], want[:, ::3]) < TOL
        if f32 is not None:
            y = f32(x)
            assert bool(((y - want).abs() <= 2.0 ** -8 * want.abs() + drop)[:, ::3].all())
            assert rel_l2(y[:, ::3], want[:, ::3]) < TOL
    torch.cuda.synchronize()
    assert ext.w8_error_flag(0) == 0


@pytest.mark.parametrize("m", [8, 40])
def test_activation_rows_with_extreme_values(ext, m):
    """Zeros, tiny and huge rows, one outlier, rows of mostly small elements, a NaN, infinities: as a sum of
    products in float64 has them."""
    for f, _, _, w in _forms(ext, 136, 1280):
        x = _x(m, 1280, 8)
        x[0] = 0
        x[1] *= 1e-30
        x[2] *= 1e30
        x[3, 7] = 3e4
        x[4] = 255.0 / 256  # largest mantissa
        x[5, 3] = float("nan")
        x[6, 3] = float("inf")
        x[7, 900], x[7, 30] = float("inf"), -float("inf")
        if m > 8:
            x[8, 640:] = float("inf")
            x[9, 100:] *= 1e-6  # the large ones are the few
            x[10] = 0
            x[10, 17] = -torch.finfo(torch.bfloat16).max
            x[11] = 0
            x[11, 5] = -float("inf")
            x[12] = 0
            x[12, 1279] = 1e-38
            x[13] *= 1e-38  # down to the smallest bf16
            x[14, ::2] *= 1e-5  # as many large as small
        y, want = f(x).double(), x.double() @ w.t()
        y = torch.where((want.abs() > 3.37e38) & (want.abs() < 3.42e38), want, y)  # bf16 ends here: either will do
        big = y.isinf() & want.isfinite() & (want.abs() > 3.4e38)
        assert torch.equal(y.isnan(), want.isnan())
        assert torch.equal(torch.where(y.isinf(), y.sign(), 0), torch.where(want.isinf() | big, want.sign(), 0))
        assert bool((y.isinf() | (want.abs() < 3.4e38) | ~want.isfinite() | (y == want)).all())
        for r in range(m):
            ok = want[r].isfinite() & ~big[r]
            if bool(ok.any()) and float(want[r][ok].abs().max()) > 0:
                # (a smallest bf16 is 2^-133: results down there are rounded to it)
                d = (y[r][ok] - want[r][ok]).norm()
                assert float(d) < TOL * float(want[r][ok].norm()) + 2.0 ** -133 * int(ok.sum()) ** 0.5, r
        assert float(y[0].abs().max()) == 0.0
    torch.cuda.synchronize()
    assert ext.w8_error_flag(0) == 0


@pytest.mark.parametrize("m", [16, 64])
def test_rows_of_mostly_outliers(ext, m):
    """The most that the epilogue can be asked to add: every row nearly half outliers, or nothing but infinities,
    in a long reduction without a k-split.  No wait of the other warps runs out, and the values are right."""
    n, k = 136, 27648
    wq, sc = _w8(n, k, 7)
    x = _x(m, k, 21)
    x[:, : k * 9 // 20] *= 2.0 ** 20
    want = (x.double() @ wq.double().t()) * sc.double()
    assert rel_l2(ext.w8a16_linear(x, wq, sc, None, False, 1), want) < TOL
    x[:] = float("inf")
    assert bool(ext.w8a16_linear(x, wq, sc, None, False, 1).isnan().all())  # weights of both signs
    qw = torch.randint(-2 ** 31, 2 ** 31 - 1, (k // 8, n), generator=_g(11), device="cuda", dtype=torch.int64).to(torch.int32)
    s4, qz = torch.ones(k // 128, n, device="cuda").half(), torch.zeros(k // 128, n // 8, dtype=torch.int32, device="cuda")
    y = ext.w4a16_linear(x, qw, s4, qz, 128, 1)  # weights 0 .. 15: infinity times zero somewhere
    assert bool(y.isnan().all())
    torch.cuda.synchronize()
    assert ext.w8_error_flag(0) == 0


# k-chunk-major weights (the reference's pair): ragged last row tile, odd n (no k-split), one k-block
@pytest.mark.parametrize("m", [1, 9, 16])
@pytest.mark.parametrize("n,k", [(128, 128), (136, 1280), (201, 640), (1000, 3584)])
def test_chunked_int8_weights(ext, m, n, k):
    wq, _ = _w8(n, k, 3)
    wq[0], wq[1] = -128, 127  # the ends of the range
    sw = torch.rand(k // 128, n, generator=_g(4), device="cuda") * 0.01 + 1e-3
    wq_t = wq.view(n, k // 16, 16).permute(1, 0, 2).contiguous()
    xq, xs = ext.w8a16_quant_act(_x(m, k, 5, spread=True))
    part = torch.einsum("mgk,ngk->gmn", xq.double().view(m, -1, 128), wq.double().view(n, -1, 128))
    want = (part * sw.double()[:, None, :]).sum(0) * xs.double()[:, None]
    assert rel_l2(ext.w8a16_gemm(xq, xs, wq_t, sw, n, k, 4), want) < TOL
    for splits in (1, 3, k // 128, 99):  # the last two: one k-block each
        assert rel_l2(ext.w8a16_gemm(xq, xs, wq_t, sw, n, k, 1, splits=splits), want) < TOL
    off = torch.empty(m * k + 4, dtype=torch.int8, device="cuda")[4:].view(m, k)  # rows off 16-byte boundaries
    off.copy_(xq)
    assert torch.equal(ext.w8a16_gemm(off, xs, wq_t, sw, n, k, 1), ext.w8a16_gemm(xq, xs, wq_t, sw, n, k, 1))
    torch.cuda.synchronize()
    assert ext.w8_error_flag(0) == 0


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 16, 17, 64, 65, 128])
@pytest.mark.parametrize("n,k", [(128, 128), (208, 1280), (1000, 3584), (136, 17408)])
def test_int4_weights(ext, m, n, k):
    from barlink_sm86_b200 import ops
    g = _g(11)
    nib = torch.randint(0, 16, (n, k), generator=g, device="cuda")
    zero = torch.randint(0, 16, (k // 128, n), generator=g, device="cuda")
    sc = (torch.rand(k // 128, n, generator=g, device="cuda") * 0.01 + 1e-3).half()
    qw, qz = _pack4(nib).t().contiguous(), _pack4(zero)
    x = _x(m, k, 5, spread=True)
    w = (nib - zero.t().repeat_interleave(128, 1)).double() * sc.double().t().repeat_interleave(128, 1)
    want = x.double() @ w.t()
    assert rel_l2(ops.w4a16_linear(x, qw, sc, qz), want) < TOL
    out = ops.w4a16_linear_split(x, qw, sc, qz)
    if out.dim() == 3:
        assert rel_l2(out.double().sum(0), want) < TOL32
    for splits in {1, 3, k // 128, 99}:
        assert rel_l2(ext.w4a16_linear(x, qw, sc, qz, 128, splits), want) < TOL
    if n % 16 == 0:
        silu = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
        for splits in (0, 1):
            assert rel_l2(ext.w4a16_linear(x, qw, sc, qz, 128, splits, True), silu) < TOL
    torch.cuda.synchronize()
    assert ext.w8_error_flag(0) == 0


def test_other_threads_run_while_a_launch_waits(ext):
    """A launch waits when the queue of launches is full; the other Python threads go on meanwhile."""
    import threading
    import time
    n, k = 200, 1024
    wq, sc = _w8(n, k, 3)
    x, xl = _x(6, k, 5), _x(300, 4096, 6)
    wq_t, sw = wq.view(n, k // 16, 16).permute(1, 0, 2).contiguous(), torch.ones(k // 128, n, device="cuda")
    xq, xs = ext.w8a16_quant_act(x)
    w = _x(512, 4096, 7)
    assert ext.gemm_row_splits(300, 512, 4096) > 1
    qw = torch.zeros(k // 8, n, dtype=torch.int32, device="cuda")
    s4, qz = torch.ones(k // 128, n, device="cuda").half(), torch.zeros(k // 128, n // 8, dtype=torch.int32, device="cuda")
    for name, f in {"w8a16_linear": lambda: ext.w8a16_linear(x, wq, sc),
                    "w8a16_linear_split": lambda: ext.w8a16_linear_split(x, wq, sc),
                    "w8a16_gemm": lambda: ext.w8a16_gemm(xq, xs, wq_t, sw, n, k, 1),
                    "w4a16_linear": lambda: ext.w4a16_linear(x, qw, s4, qz, 128, 1),
                    "linear": lambda: ext.linear(xl, w)}.items():
        f()
        torch.cuda.synchronize()
        seen = []
        for _ in range(3):  # (a busy host may hold up any one of them)
            stop, gap = threading.Event(), [0.0]

            def tick():
                last = time.perf_counter()
                while not stop.is_set():
                    time.sleep(1e-3)
                    now = time.perf_counter()
                    gap[0], last = max(gap[0], now - last), now
            th = threading.Thread(target=tick)
            th.start()
            torch.cuda._sleep(10 ** 9)  # half a second of an occupied stream
            t0 = time.perf_counter()
            for _ in range(2000):
                f()
            waited = time.perf_counter() - t0
            stop.set()
            th.join()
            torch.cuda.synchronize()
            seen.append((gap[0], waited))
            if waited > 0.2 and gap[0] < waited / 2:  # the queue was full, and the thread ran
                break
        else:
            raise AssertionError((name, seen))


# Weights that a kernel just ahead in the stream leaves behind (received, unpacked, dequantised ones): this
# library's kernels let their successors start early, so the weights may only be read behind the wait.  The
# writer here is a product whose result, seen as bytes, is the weight; `stale` is what was there before.
@pytest.mark.parametrize("form", ["pair", "int8", "bf16", "int4"])
def test_weights_written_by_the_kernel_ahead(ext, form):
    n, k, m = 4096, 4096, 8
    # [k / 8, 2 n] bf16 = [k / 8, n] int32, or [n, k / 2] bf16 = [n, k] int8
    b, a = (_x(k // 8, 8192, 2), _x(2 * n, 8192, 1)) if form == "int4" else (_x(n, 8192, 2), _x(k // 2, 8192, 1))
    buf = torch.zeros(b.shape[0], a.shape[0], dtype=torch.bfloat16, device="cuda")
    x, one = _x(m, k, 5), torch.ones(n, device="cuda").bfloat16()
    xq, xs = ext.w8a16_quant_act(x)
    s4, qz = torch.ones(k // 128, n, device="cuda").half(), torch.zeros(k // 128, n // 8, dtype=torch.int32, device="cuda")
    sw = torch.ones(k // 128, n, device="cuda")

    def product():
        if form == "int4":
            return ext.w4a16_linear(x, buf.view(torch.int32), s4, qz)
        w = buf.view(torch.int8)
        if form == "pair":
            return ext.w8a16_gemm(xq, xs, w.view(k // 16, n, 16), sw, n, k, 1)
        return ext.w8a16_linear(x, w, one, act_int8=form == "int8")
    ext.linear(b, a, out=buf)
    torch.cuda.synchronize()
    want = product()
    for _ in range(5):
        buf.zero_()
        torch.cuda.synchronize()
        ext.linear(b, a, out=buf)
        assert torch.equal(product(), want)


@pytest.mark.parametrize("k", [8208, 16384, 18944, 32768])
def test_long_rows_shared_by_blocks(ext, k):
    """Rows whose digits a cluster of blocks writes (few tokens) and one block does (38 tokens): the same results, outliers
    at the ends of the blocks' shares included."""
    n = 160
    wq, sc = _w8(n, k, 3)
    x = _x(38, k, 5)
    for p in (0, k // 8, k // 4 - 1, k // 4, k // 2 - 1, k // 2, k - 1):
        x[3, p] = 2.0 ** 14
    want = x.double() @ (wq.double() * sc.double()[:, None]).t()
    y = {m: ext.w8a16_linear(x[:m].contiguous(), wq, sc, splits=1) for m in (1, 18, 19, 37, 38)}
    for m in y:
        assert rel_l2(y[m], want[:m]) < TOL
        assert torch.equal(y[m], y[38][:m])


@pytest.mark.parametrize("k", [8, 4096, 4104, 8192, 8200, 18944, 32768, 32776])
@pytest.mark.parametrize("m", [1, 18, 37, 300])
def test_quant_act_is_the_stated_arithmetic(ext, m, k):
    """xs = max |x| / 127 and xq = x / xs to the nearest whole number, whichever kernel a row length goes to."""
    x = _x(m, k, 7) * 3
    x[0, k - 1] = 77
    xq, xs = ext.w8a16_quant_act(x)
    amax = x.float().abs().amax(1)
    s = (amax / torch.full_like(amax, 127)).clamp_min(1e-12)  # (a division by a Python number multiplies by 1 / 127)
    assert torch.equal(xs, s)
    assert torch.equal(xq, torch.round(x.float() * (1.0 / s)[:, None]).clamp(-127, 127).to(torch.int8))


@pytest.mark.parametrize("hidden", [16, 3584, 4096, 4112, 5120, 8192])
@pytest.mark.parametrize("m", [1, 16, 17, 128])
def test_norm_that_leaves_digits(ext, m, hidden):
    """The same normed rows, residual and products, bit for bit, as the norm and a linear that makes the digits itself."""
    gamma = _x(1, hidden, 2)[0].contiguous()
    wq, sc = _w8(96, hidden, 3)
    slabs = torch.randn(3, m, hidden, generator=_g(4), device="cuda")
    if hidden > 64:
        slabs[0, m - 1, hidden - 1] = 1e9  # outweighs its row: the rest has no digits but in the outliers' scale
    for x in (slabs, slabs.sum(0).bfloat16()):
        for res in (None, _x(m, hidden, 6)):
            r0, r1 = (res.clone(), res.clone()) if res is not None else (None, None)
            n0, _ = ext.rmsnorm(x, gamma, 1e-6, r0)
            n1, _, xq, xs = ext.rmsnorm_digits(x, gamma, 1e-6, r1)
            assert torch.equal(n0, n1) and (res is None or torch.equal(r0, r1))
            assert torch.equal(ext.w8a16_linear(n0, wq, sc), ext.w8a16_linear(n1, wq, sc, xq=xq, xs=xs))
            assert torch.equal(ext.w8a16_linear_split(n0, wq, sc), ext.w8a16_linear_split(n1, wq, sc, xq=xq, xs=xs))
    with pytest.raises(RuntimeError):
        ext.w8a16_linear(n1, wq, sc, xq=xq, xs=xs[:-1])
    torch.cuda.synchronize()
    assert ext.w8_error_flag(0) == 0


@pytest.mark.parametrize("n,k", [(300, 24), (256, 1040), (5, 18944), (300, 3592)])
def test_widened_weights(ext, n, k):
    """bl_w8_dequant behind a prefill linear: weights whose rows and whole are no multiple of a block's share."""
    wq, sc = _w8(n, k, 3)
    x = torch.zeros(300, k, device="cuda").bfloat16()
    idx = torch.arange(min(300, k), device="cuda")
    x[idx, idx] = 1  # rows of the widened weight itself
    want = (wq.float() * sc.float()[:, None]).bfloat16().t()[: len(idx)]
    assert torch.equal(ext.w8a16_linear(x, wq, sc)[: len(idx)], want)


@pytest.mark.parametrize("n,k", [(5, 24), (592, 1024), (593, 1024), (4000, 4000), (4001, 4000)])
def test_widened_weights_by_size(ext, n, k):
    """One, two and four vectors a thread, on both sides of the lines between them: first and last columns."""
    wq, sc = _w8(n, k, 3)
    want = (wq.float() * sc.float()[:, None]).bfloat16().t()
    for idx in (torch.arange(min(300, k), device="cuda"), torch.arange(max(0, k - 300), k, device="cuda")):
        x = torch.zeros(300, k, device="cuda").bfloat16()
        x[torch.arange(len(idx), device="cuda"), idx] = 1
        assert torch.equal(ext.w8a16_linear(x, wq, sc)[: len(idx)], want[idx])


def test_digits_that_do_not_belong_are_refused(ext):
    """Before any launch: half of a pair, other types or sizes, another device, and products that read no digits."""
    from barlink_sm86_b200 import ops
    m, k, n = 8, 1024, 96
    wq, sc = _w8(n, k, 3)
    x, _, xq, xs = ext.rmsnorm_digits(_x(m, k, 1), _x(1, k, 2)[0].contiguous(), 1e-6, None)
    want = ext.w8a16_linear(x, wq, sc)
    assert torch.equal(ext.w8a16_linear(x, wq, sc, xq=xq, xs=xs), want)
    bad = [(xq, None), (None, xs), (xq.view(torch.uint8), xs), (xq, xs.view(torch.int32)), (xq.cpu(), xs), (xq, xs.cpu()),
           (xq[1:], xs), (torch.cat([xq[:1], xq])[1:], xs), (torch.stack([xq, xq], 1)[:, 0], xs)]
    for q, s in bad:
        for call in (ext.w8a16_linear, ext.w8a16_linear_split):
            with pytest.raises(RuntimeError, match="digits"):
                call(x, wq, sc, xq=q, xs=s)
    with pytest.raises(RuntimeError, match="digits"):
        ext.w8a16_linear(x, wq, sc, act_int8=True, xq=xq, xs=xs)
    with pytest.raises(RuntimeError, match="digits"):
        ext.w8a16_linear(_x(200, k, 1), wq, sc, xq=xq, xs=xs)
    with pytest.raises(ValueError, match="digits"):
        ops.w8a16_linear(x, wq, sc, act="int8", digits=(xq, xs))
    g32 = sc[:, None].expand(n, 32).contiguous()  # groups of 32: the weight is widened
    with pytest.raises(ValueError, match="digits"):
        ops.w8a16_linear(x, wq, g32, digits=(xq, xs))
    gs = ops.prepare_w8_scales(sc[:, None].expand(n, k // 128).contiguous(), k)
    assert torch.equal(ops.w8a16_linear(x, wq, gs, digits=(xq, xs)), ops.w8a16_linear(x, wq, gs))


@pytest.mark.parametrize("m,k", [(3, 1024), (300, 4104)])
def test_rows_between_two_vectors_are_quantised(ext, m, k):
    """Rows that start off a 16-byte boundary give what their copy gives."""
    buf = _x(1, m * k + 8, 3)[0]
    wq, sc = _w8(96, k, 3)
    for off in (1, 4):
        x = buf[off:off + m * k].view(m, k)
        (q, s), (q0, s0) = ext.w8a16_quant_act(x), ext.w8a16_quant_act(x.clone())
        assert torch.equal(q, q0) and torch.equal(s, s0)
        if k % 16 == 0:
            assert torch.equal(ext.w8a16_linear(x, wq, sc, act_int8=True), ext.w8a16_linear(x.clone(), wq, sc, act_int8=True))


def test_widened_weights_between_two_vectors(ext):
    """Prefill on int8 weights that are a view at any byte."""
    n, k = 160, 1024
    wq, sc = _w8(n, k, 3)
    x = _x(300, k, 2)
    want = ext.w8a16_linear(x, wq, sc)
    for off in (1, 4, 8):
        buf = torch.empty(n * k + 16, dtype=torch.int8, device="cuda")
        view = buf[off:off + n * k].view(n, k)
        view.copy_(wq)
        assert torch.equal(ext.w8a16_linear(x, view, sc), want)
