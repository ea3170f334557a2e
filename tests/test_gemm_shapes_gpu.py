# SPDX-License-Identifier: MIT
"""Linears at the sizes where a kernel or a branch of the dispatch can go wrong: edges of tiles,
remainders, the smallest and largest of a range.  Oracle: the fp32 statement of each op on the same
bf16 tensors.  Tolerance: the result is rounded once to bf16 (relative error of one rounding at most
2^-9, rms 2^-9 / sqrt(3) = 1.1e-3) on top of fp32 sums, so rel-L2 stays below 2^-8 = 3.9e-3."""
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -8


def _bf(*shape, seed, std=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(torch.bfloat16)


@pytest.mark.parametrize("m,n,k", [(512, 256, 64), (513, 600, 136), (777, 1032, 512), (1000, 1024, 72),
                                   (2049, 512, 256), (200, 512, 256), (130, 264, 64)])
@pytest.mark.parametrize("bias", [False, True])
def test_token_major_silu_mul(ext, m, n, k, bias):
    from barlink_sm86_b200 import ops
    x, w = _bf(m, k, seed=1), _bf(n, k, seed=2, std=k ** -0.5)
    b = _bf(n, seed=3) if bias else None
    want = ops.ref.linear(x.float(), w, b, silu_mul=True)
    assert rel_l2(ops.linear(x, w, b, silu_mul=True), want) < TOL
    # an output that starts off a 16-byte boundary
    buf = torch.zeros(m * (n // 2) + 1, dtype=torch.bfloat16, device="cuda")
    out = buf[1:].view(m, n // 2)
    ops.linear(x, w, b, silu_mul=True, out=out)
    assert rel_l2(out, want) < TOL and float(buf[0]) == 0.0
    torch.cuda.synchronize()
    assert ext.gemm_error_flag(0) == 0


# the paired-CTA kernel from 129 rows on: ragged row and column tiles, k-blocks that the splits do not divide.
# Against float64; one bf16 rounding of the result (2^-9 relative), twice that for SiLU*mul: rel-L2 2^-8
@pytest.mark.parametrize("rows", [129, 256, 257, 333, 511])
@pytest.mark.parametrize("n,k", [(256, 512), (272, 4104), (3600, 2048), (512, 18944)])
def test_paired_kernel_few_rows(ext, rows, n, k):
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    x = torch.randn(rows, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.05).bfloat16()
    b = torch.randn(n, generator=g, device="cuda").bfloat16()
    want = x.double() @ w.double().t()
    rel = lambda a, c: float((a.double() - c).norm() / c.norm())
    assert rel(ext.linear(x, w), want) < 2.0 ** -8
    assert rel(ext.linear(x, w, b), want + b.double()) < 2.0 ** -8
    y = want + b.double()
    silu = torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2]
    assert rel(ext.linear(x, w, b, None, True), silu) < 2.0 ** -8
    r = torch.randn(rows, n, generator=g, device="cuda").bfloat16()
    assert rel(ext.linear(x, w, b, r), y + r.double()) < 2.0 ** -8
    torch.cuda.synchronize()
    assert ext.gemm_error_flag(0) == 0


# bias, residual or output off a 16-byte boundary (slices of longer tensors): the paired kernel, and with
# bn = 128 the single-CTA one
@pytest.mark.parametrize("which", ["bias", "residual", "out"])
@pytest.mark.parametrize("rows,n,k,bn", [(129, 256, 512, 0), (600, 264, 136, 0), (200, 256, 512, 128), (200, 264, 4096, 0)])
@pytest.mark.parametrize("off", [1, 4])
def test_token_major_off_16_bytes(ext, which, rows, n, k, bn, off):
    def cut(t, on):  # the same values, starting `off` elements into a buffer when `on`
        buf = torch.zeros(t.numel() + 8, dtype=torch.bfloat16, device="cuda")
        v = buf[off if on else 0:][:t.numel()].view(t.shape)
        return v.copy_(t)
    x, w = _bf(rows, k, seed=1), _bf(n, k, seed=2, std=k ** -0.5)
    b, r = cut(_bf(n, seed=3), which == "bias"), cut(_bf(rows, n, seed=4), which == "residual")
    out = cut(torch.zeros(rows, n), which == "out")
    want = x.double() @ w.double().t() + b.double() + r.double()
    ext.linear(x, w, b, r, False, out, bn=bn)
    assert float((out.double() - want).norm() / want.norm()) < TOL
    ext.linear(x, w, b, None, False, out, bn=bn)
    assert float((out.double() - want + r.double()).norm() / want.norm()) < TOL
    torch.cuda.synchronize()
    assert ext.gemm_error_flag(0) == 0


# k-splits with every epilogue: widths that no vector divides, one column more than a tile, the last k-block ragged
@pytest.mark.parametrize("rows", [129, 300, 520])
@pytest.mark.parametrize("n,k", [(257, 4096), (520, 4104), (1022, 8192)])
def test_k_split_epilogues(ext, rows, n, k):
    assert ext.gemm_row_splits(rows, n, k) > 1
    x, w, b, r = _bf(rows, k, seed=1), _bf(n, k, seed=2, std=k ** -0.5), _bf(n, seed=3), _bf(rows, n, seed=4)
    rel = lambda a, c: float((a.double() - c).norm() / c.norm())
    y = x.double() @ w.double().t() + b.double()
    gelu = torch.nn.functional.gelu(y, approximate="tanh")
    assert rel(ext.linear(x, w, b), y) < TOL
    assert rel(ext.linear(x, w, b, r), y + r.double()) < TOL
    assert rel(ext.linear(x, w, b, gelu=True), gelu) < TOL
    assert rel(ext.linear(x, w, b, r, gelu=True), gelu + r.double()) < TOL
    even = y[:, : n // 2 * 2]
    silu = torch.nn.functional.silu(even[:, 0::2]) * even[:, 1::2]
    assert rel(ext.linear(x, w, b, None, True), silu) < TOL
    same = r.clone()  # the residual stream updated in place
    assert rel(ext.linear(x, w, b, same, False, same), y + r.double()) < TOL
    torch.cuda.synchronize()
    assert ext.gemm_error_flag(0) == 0


@pytest.mark.parametrize("rows,n,k", [(129, 256, 512), (511, 512, 4096)])
def test_trace_stamps_below_512_rows(ext, rows, n, k):
    x, w = _bf(rows, k, seed=1), _bf(n, k, seed=2, std=k ** -0.5)
    trace = torch.zeros(8 * 296, dtype=torch.int64, device="cuda")
    assert rel_l2(ext.linear(x, w, trace=trace), x.float() @ w.float().t()) < TOL
    assert bool((trace.view(-1, 8)[0, [0, 2, 3]] > 0).all())


def test_row_splits_rule(ext):
    assert ext.gemm_row_splits(128, 3584, 18944) == 1  # the swapped form
    assert ext.gemm_row_splits(333, 3584, 18944) >= 2  # 28 tiles for 74 pairs
    assert ext.gemm_row_splits(333, 37888, 3584) == 1 and ext.gemm_row_splits(8192, 3584, 18944) == 1
    assert ext.gemm_row_splits(1000, 256, 1024) == 1  # a second kernel costs more than it saves
    assert ext.gemm_row_splits(2200, 3072, 12288) == 1 and ext.gemm_row_splits(2600, 3584, 18944) == 1  # slabs beyond L2
    # just above one lap of the pairs: 75 and 84 tiles, 80 tiles of a very long reduction
    assert min(ext.gemm_row_splits(*t) for t in [(1280, 3840, 18944), (1285, 3584, 18944), (1000, 5120, 27648)]) >= 2
    for rows, n, k in [(129, 256, 64), (129, 256, 128), (300, 512, 200), (2000, 3584, 18944)]:
        s, kb = ext.gemm_row_splits(rows, n, k), -(-k // 64)
        assert (s - 1) * -(-kb // s) < kb  # no empty split
