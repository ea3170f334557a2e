# SPDX-License-Identifier: MIT
"""Tensor-core attention around the ends of its pipeline (64-key steps, scores two steps ahead, tiles in
rings of three): one to seven steps, ragged last steps, scores that grow so that the accumulator is
rescaled while products are in flight.  Oracle: float64.  Tolerance: P and the result are rounded to bf16
(2^-9 relative each, the sums over keys average P's): rel-L2 2^-8."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _want(q, k, v, scale, causal):
    s = torch.einsum("qhd,khd->hqk", q.double(), k.double()) * scale
    if causal:
        lq, lk = s.shape[1:]
        s = s.masked_fill(torch.ones(lq, lk, dtype=torch.bool, device=s.device).triu(lk - lq + 1), float("-inf"))
    return torch.einsum("hqk,khd->qhd", s.softmax(-1), v.double())


@pytest.mark.parametrize("lk", [1, 63, 64, 65, 128, 129, 192, 193, 256, 257, 400])
@pytest.mark.parametrize("growing", [False, True])
@pytest.mark.parametrize("causal", [False, True])
def test_steps(ext, lk, growing, causal):
    g = torch.Generator(device="cuda").manual_seed(lk)
    lq, nq, nkv = (lk if causal else 300), 2, 1
    q, k, v = (torch.randn(n, h, 128, generator=g, device="cuda").bfloat16() for n, h in ((lq, nq), (lk, nkv), (lk, nkv)))
    if growing:  # later keys win by far: the running maximum rises in every step
        k = (k.float() * torch.linspace(0.2, 12.0, lk, device="cuda")[:, None, None]).bfloat16()
    cu_q, cu_k = (torch.tensor([0, n], dtype=torch.int32, device="cuda") for n in (lq, lk))
    got = ext.attn_fwd(q, k, v, cu_q, cu_k, lq, 128 ** -0.5, causal, lk)
    want = _want(q, k.expand(-1, nq, -1), v.expand(-1, nq, -1), 128 ** -0.5, causal)
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8
    assert ext.attn_error_flag(0) == 0


@pytest.mark.parametrize("l0", [1, 63, 64, 65, 130])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_values_of_the_next_sequence_do_not_leak(ext, l0, bad):
    """Keys are loaded in tiles of 64, so the last tile of a sequence holds the next one's first rows."""
    from barlink_sm86_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(l0)
    l1, nq, nkv = 40, 4, 2
    q, k, v = (torch.randn(l0 + l1, h, 128, generator=g, device="cuda").bfloat16() for h in (nq, nkv, nkv))
    v[l0:l0 + 3] = bad
    cu = torch.tensor([0, l0, l0 + l1], dtype=torch.int32, device="cuda")
    one = torch.tensor([0, l0], dtype=torch.int32, device="cuda")
    for causal in (False, True):
        both = ops.attention(q, k, v, cu, cu, max(l0, l1), 0.088, causal, max_k=max(l0, l1))
        alone = ops.attention(q[:l0].contiguous(), k[:l0].contiguous(), v[:l0].contiguous(), one, one, l0, 0.088, causal,
                              max_k=l0)
        assert torch.equal(both[:l0], alone) and bool(alone.isfinite().all())


def test_values_of_other_shapes_than_the_keys(ext):
    """Tensor maps end with the shorter of K and V, so that no box reaches beyond either; values that do not belong to
    the keys are refused before anything is launched."""
    g = torch.Generator(device="cuda").manual_seed(3)
    l, nq, nkv = 70, 4, 2
    q, k, v = (torch.randn(n, h, 128, generator=g, device="cuda").bfloat16() for n, h in ((l, nq), (200, nkv), (l, nkv)))
    cu = torch.tensor([0, l], dtype=torch.int32, device="cuda")

    def run(k, v, cu_k=cu, lk=l):
        return ext.attn_fwd(q, k, v, cu, cu_k, l, 0.088, False, lk)

    want = run(k[:l].contiguous(), v)
    more = torch.cat([v, torch.full((9, nkv, 128), float("nan"), device="cuda").bfloat16()])
    assert torch.equal(run(k, v), want) and torch.equal(run(k[:l], more), want)
    wide = torch.cat([v, v[:, :1]], 1)  # more heads than the keys have
    assert torch.equal(run(k, wide), want)
    # all rows at one address, and a single row of any stride
    assert torch.equal(run(k, v[:1].expand(l, -1, -1)), run(k, v[:1].repeat(l, 1, 1)))
    one = torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    row = torch.as_strided(v, (1, nkv, 128), (3, 128, 1))
    assert torch.equal(run(k, row, one, 1), run(k, v[:1].contiguous(), one, 1))
    for bad_k, bad_v in ((k, v[:, :1].contiguous()), (k, v[..., :64].contiguous()), (k[..., :64].contiguous(), v)):
        for lk in (l, 0):
            with pytest.raises(RuntimeError, match="head_dim"):
                run(bad_k, bad_v, lk=lk)


def test_max_q_is_a_bound(ext):
    """Any bound of the sequence lengths does, also one of more row blocks than a grid has along z."""
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(700, h, 128, generator=g, device="cuda").bfloat16() for h in (2, 1, 1))
    cu = torch.tensor([0, 130, 700], dtype=torch.int32, device="cuda")
    for causal in (False, True):
        want = ext.attn_fwd(q, k, v, cu, cu, 570, 0.088, causal, 570)
        for bound in (1024, 256 * 65535 + 1):
            assert torch.equal(ext.attn_fwd(q, k, v, cu, cu, bound, 0.088, causal, 570), want)
