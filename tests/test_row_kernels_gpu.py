# SPDX-License-Identifier: MIT
"""Row kernels of prefill sizes (csrc/ops_kernels.cu: one four-warp block per row) at the edges of their
range, against the fp32 statements.  Tolerance: one bf16 rounding of the result and one of an intermediate
value, 2^-9 each relative to the element: 2^-7 of the largest, and rel-L2 2^-8."""
import pytest
import torch

from barlink_sm86_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _g(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(seed, *shape):
    return torch.randn(*shape, generator=_g(seed), device="cuda").bfloat16()


def _close(a, b):
    a, b = a.double(), b.double()
    assert float((a - b).norm() / b.norm()) < 2.0 ** -8
    assert float((a - b).abs().max() / b.abs().max()) < 2.0 ** -7


# 148 | 149: the rule's first line; 1024 / 1032 vectors and 8192 / 8200 elements: the edges of the register forms;
# 300 and 700 rows: both sides of its lines at medium widths
@pytest.mark.parametrize("rows", [148, 149, 300, 700])
@pytest.mark.parametrize("hidden", [8, 264, 1024, 1032, 2048, 2056, 4096, 4104, 8192, 8200])
def test_norms(ext, rows, hidden):
    x, r, gm = _randn(1, rows, hidden), _randn(2, rows, hidden), _randn(3, hidden)
    want, _ = ref.rmsnorm(x, gm, 1e-6, None)
    _close(ext.rmsnorm(x, gm, 1e-6, None, None)[0], want)
    r2 = r.clone()
    want, wres = ref.rmsnorm(x, gm, 1e-6, r)
    got, gres = ext.rmsnorm(x, gm, 1e-6, r2, None)
    assert torch.equal(gres, wres) and gres.data_ptr() == r2.data_ptr()
    _close(got, want)
    batch = 3
    per = -(-rows // batch)
    mod = _randn(4, batch, 2 * hidden)
    sh, sc = mod[:, :hidden], mod[:, hidden:]
    _close(ext.layernorm_modulate(x, sh, sc, per, 1e-6), ref.layernorm_modulate(
        torch.cat([x, x[: batch * per - rows]]), sh, sc, per, 1e-6)[:rows])


@pytest.mark.parametrize("rows", [148, 149, 200])
@pytest.mark.parametrize("nq,nkv,hd", [(28, 4, 128), (1, 1, 128), (8, 2, 64), (3, 1, 256), (5, 1, 16), (4, 2, 96),
                                       (16, 2, 64), (40, 10, 16)])
@pytest.mark.parametrize("cached", [False, True])
def test_rope_kv_write(ext, rows, nq, nkv, hd, cached):
    bs, blocks = 16, 16
    qkv = _randn(5, rows, (nq + 2 * nkv) * hd)
    pos = torch.randint(0, 9000, (rows,), generator=_g(6), device="cuda", dtype=torch.int32)
    slots = torch.randperm(bs * blocks, generator=_g(7), device="cuda")[:rows].to(torch.int32).contiguous()
    slots[3] = -1  # a row that is not cached
    caches = [[torch.zeros(blocks, nkv, bs, hd, device="cuda", dtype=torch.bfloat16) for _ in range(2)] for _ in range(2)]
    got = qkv.clone()
    a = caches[0] if cached else [None, None]
    ext.rope_kv_write(got, pos, slots if cached else None, *a, nq, nkv, hd, bs, 1e6, None)
    # few rows take the other kernel: the same arithmetic, so the same bits
    want = qkv.clone()
    for r in range(0, rows, 100):
        b = caches[1] if cached else [None, None]
        part = want[r:r + 100].clone()
        ext.rope_kv_write(part, pos[r:r + 100].clone(), slots[r:r + 100].clone() if cached else None, *b, nq, nkv, hd,
                          bs, 1e6, None)
        want[r:r + 100] = part
    assert torch.equal(got, want)
    for x, y in zip(caches[0], caches[1]):
        assert torch.equal(x, y)


@pytest.mark.parametrize("rows,heads,pitch,offset", [(1, 24, 24 * 384, 0), (7, 25, 25 * 256, 0), (200, 3, 3 * 384 + 2, 0),
                                                     (5, 1, 384, 1), (499, 24, 24 * 384, 0), (500, 21, 21 * 384, 0),
                                                     (500, 25, 25 * 256 + 4, 4), (500, 25, 25 * 256 + 2, 0),
                                                     (500, 25, 25 * 256, 1), (1100, 12, 12 * 384, 0)])
@pytest.mark.parametrize("axes", [1, 2])
@pytest.mark.parametrize("norm", [False, True])
def test_qknorm_rope(ext, rows, heads, pitch, offset, axes, norm):
    flat = _randn(8, rows * pitch + 8)
    x = flat[offset:offset + rows * pitch].view(rows, pitch)
    before = x.clone()
    gm = [_randn(9 + i, 128) if norm else None for i in range(2)]
    pos = torch.randint(0, 100, (rows, axes), generator=_g(11), device="cuda", dtype=torch.int32)
    want = ref.qknorm_rope(before.clone(), *gm, pos, heads, 1e-6, 1e4, axes)
    ext.qknorm_rope(x, *gm, pos, heads, 1e-6, 1e4, axes)
    _close(x[:, : 256 * heads], want[:, : 256 * heads])
    assert torch.equal(x[:, 256 * heads:], before[:, 256 * heads:])
