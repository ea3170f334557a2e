# SPDX-License-Identifier: MIT
"""Int4 weight-only linear (GPTQ-v1 tensors) against the fp32 statement: the
decode GEMV for 1..16 rows, every k-split, and the widen + GEMM path."""
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# (K, N) of the reference's int4 MLP shapes (demos/qwen_tp/int4linear.py:152) plus small odd ones
SHAPES = [(5120, 17408), (17408, 5120), (5120, 6144), (256, 64), (1024, 8 * 37)]


@pytest.mark.parametrize("k,n", SHAPES)
@pytest.mark.parametrize("m", [1, 2, 3, 8, 16])
def test_w4a16_gemv(ext, k, n, m):
    from barlink_sm86_b200 import ops
    g = torch.Generator().manual_seed(k + m)
    w = torch.randn(n, k, generator=g) * 0.02
    x = torch.randn(m, k, generator=g).bfloat16()
    qw, sc, qz = ops.ref.pack_int4(w)
    want = ops.ref.w4a16_linear(x, qw, sc, qz)
    got = ops.w4a16_linear(x.cuda(), qw.cuda(), sc.cuda(), qz.cuda()).cpu()
    assert rel_l2(got, want) < 5e-3


@pytest.mark.parametrize("splits", [1, 2, 5, 40])
def test_w4a16_gemv_splits_and_groups(ext, splits):
    from barlink_sm86_b200 import ops
    g = torch.Generator().manual_seed(splits)
    k, n, group = 2048, 512, 64
    w = torch.randn(n, k, generator=g) * 0.05
    x = torch.randn(4, k, generator=g).bfloat16()
    qw, sc, qz = ops.ref.pack_int4(w, group)
    # zero points other than 8: the kernel must read them per output
    z = torch.randint(5, 12, (k // group, n), generator=g)
    qz = sum(z.view(k // group, n // 8, 8)[..., j].long() << (4 * j) for j in range(8))
    qz = ((qz + 2 ** 31) % 2 ** 32 - 2 ** 31).to(torch.int32)
    want = ops.ref.w4a16_linear(x, qw, sc, qz, group)
    a = ext.w4a16_linear(x.cuda(), qw.cuda(), sc.cuda(), qz.cuda(), group, splits)
    b = ext.w4a16_linear(x.cuda(), qw.cuda(), sc.cuda(), qz.cuda(), group, splits)
    assert rel_l2(a.cpu(), want) < 5e-3
    assert torch.equal(a, b)  # fixed reduction order: bit-identical run to run


def test_w4a16_prefill_path_and_dequant(ext):
    from barlink_sm86_b200 import ops
    g = torch.Generator().manual_seed(9)
    k, n = 1024, 768
    w = torch.randn(n, k, generator=g) * 0.02
    qw, sc, qz = ops.ref.pack_int4(w)
    dq = ext.w4_dequant(qw.cuda(), sc.cuda(), qz.cuda(), 128).float().cpu()
    assert rel_l2(dq, ops.ref.w4_dequant(qw, sc, qz)) < 5e-3
    x = torch.randn(100, k, generator=g).bfloat16()
    got = ops.w4a16_linear(x.cuda(), qw.cuda(), sc.cuda(), qz.cuda()).cpu()
    assert rel_l2(got, ops.ref.w4a16_linear(x, qw, sc, qz)) < 1e-2


@pytest.mark.parametrize("k,n", [(128, 8), (384, 40), (256, 4104), (18944, 72), (1152, 37888)])
@pytest.mark.parametrize("m", [1, 8, 9, 16])
def test_w4a16_groups_of_128(ext, k, n, m):
    """Edges of the strips of 32 outputs, of the warps' shares of the groups and of eights of tokens."""
    from barlink_sm86_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(k + n + m)
    qw = torch.randint(-2 ** 31, 2 ** 31 - 1, (k // 8, n), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    qz = torch.randint(-2 ** 31, 2 ** 31 - 1, (k // 128, n // 8), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    sc = (torch.rand(k // 128, n, generator=g, device="cuda") * 0.01 + 1e-3).half()
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    sh = 4 * torch.arange(8, device="cuda")
    w = ((qw[:, None, :] >> sh[None, :, None]) & 15).reshape(k, n)
    z = ((qz[:, :, None] >> sh) & 15).reshape(k // 128, n)
    wd = (w - z.repeat_interleave(128, 0)).double() * sc.double().repeat_interleave(128, 0)
    want = x.double() @ wd
    # one rounding to bf16, half of a unit of 2^-7 at most, on fp32 sums of a few thousand products
    tol, tol32 = 2.0 ** -8 + 1e-5, 1e-5
    assert rel_l2(ops.w4a16_linear(x, qw, sc, qz), want) < tol
    out = ops.w4a16_linear_split(x, qw, sc, qz)
    assert rel_l2(out.double().sum(0), want) < tol32 if out.dim() == 3 else rel_l2(out, want) < tol
    assert rel_l2(ext.w4a16_linear(x, qw, sc, qz, 128, 3), want) < tol
    if n % 16 == 0:
        silu = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
        # (SiLU * up of fp32 sums; __expf and the division are good to some 1e-6)
        for splits in (0, 1):
            assert rel_l2(ext.w4a16_linear(x, qw, sc, qz, 128, splits, True), silu) < tol + 1e-5


@pytest.mark.parametrize("group,m", [(64, 1), (64, 16), (128, 3), (128, 9), (128, 40)])
def test_w4a16_words_and_scales_between_two_vectors(ext, group, m):
    """Weights that are views at an odd offset: the same as their copies (groups of 128: as another kernel's result)."""
    from barlink_sm86_b200 import ops
    k, n = 512, 264
    g = torch.Generator(device="cuda").manual_seed(m)
    buf = torch.randint(-2 ** 31, 2 ** 31 - 1, (k // 8 * n + 4,), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    qz = torch.randint(-2 ** 31, 2 ** 31 - 1, (k // group, n // 8), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    sbuf = (torch.rand(k // group * n + 4, generator=g, device="cuda") * 0.01 + 1e-3).half()
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    for off, soff in ((0, 1), (1, 0), (2, 2), (3, 3)):
        qw, sc = buf[off:off + k // 8 * n].view(k // 8, n), sbuf[soff:soff + k // group * n].view(k // group, n)
        got, want = ops.w4a16_linear(x, qw, sc, qz, group), ops.w4a16_linear(x, qw.clone(), sc.clone(), qz, group)
        # (each result rounded to bf16, and from 17 rows the widened weights too: some 2^-9.2 of the norm apiece)
        assert torch.equal(got, want) if group == 64 else rel_l2(got, want) < 2.0 ** -8
