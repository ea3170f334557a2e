# SPDX-License-Identifier: MIT
"""Workloads of one GPU whose speed matters to a user of this library, and how to run each of them.

Four kinds of work, all through the public entry points:

  decode    one step of the Qwen2-style decoder: every sequence of the batch gets its next token's
            logits and the greedy token against a paged KV cache (`Qwen2Model.decode_hidden`,
            `.logits`, `ops.argmax`).  A serving loop captures the step in a CUDA graph once and
            replays it, and so does `prepare` (case["graph"]); graph=False is the eager step.
            Sequences of a batch are at different lengths and their pages are scattered over the
            cache, as in continuous batching.
  prefill   the prompts of a batch through the decoder, KV cache written, logits of the last
            position (`Qwen2Model.prefill`, `.logits`).
  mmdit     one forward (denoising step) of the 12B MMDiT image model (`MMDiTModel.forward`).
  w8_layer  the four linears of one decoder layer on int8 weights, in the forms the op surface
            offers: "pair" = w8a16_quant_act + w8a16_gemm (the reference's two calls, group-128
            scales), "int8" = per-channel scales with activations quantised per token, "int8_g128" /
            "bf16_g128" = group-128 scales with int8 / bf16 activations.

A case is a dict of plain values; `prepare` makes weights, caches and inputs from the seed alone.
"""
import math
import random

import torch

from barlink_sm86_b200 import load_extension, ops
from barlink_sm86_b200.models import MMDiTConfig, MMDiTModel, Qwen2Config, Qwen2Model
from barlink_sm86_b200.models.mmdit import MMDiTWeights, grid_positions
from barlink_sm86_b200.models.qwen2 import PagedKV, RandomSource
from barlink_sm86_b200.parallel import TPComm

# Decoder shapes: the 7B and 32B shapes of the headline benchmark and of the serving demo, and the
# two-layer shape of the smoke run.
CONFIGS = {
    "7b": Qwen2Config.qwen25_7b,
    "32b": Qwen2Config.qwen25_32b,
    "small": lambda: Qwen2Config(hidden=1024, layers=2, n_heads=8, n_kv_heads=2, head_dim=128, intermediate=2816,
                                 vocab=8192, name="small"),
}
WEIGHT_BYTES = {"none": 2.0, "w8a16": 1.0, "w4a16": 1.0}  # w4a16: 0.5 for the MLP, int8 elsewhere


def listed():
    return [
        # the smallest call: an eager step of a two-layer model, where launches and host time count
        dict(name="decode_small_eager_b4", kind="decode", model="small", quant="none", batch=4, ctx=33, graph=False),
        # interactive use: one sequence
        dict(name="decode_7b_b1", kind="decode", model="7b", quant="none", batch=1, ctx=777, graph=True),
        # a few long conversations: attention over the cache is a large part of the step
        dict(name="decode_7b_b8_long", kind="decode", model="7b", quant="none", batch=8, ctx=8000, graph=True),
        # the headline: a full serving batch
        dict(name="decode_7b_b64", kind="decode", model="7b", quant="none", batch=64, ctx=1024, graph=True),
        # a short odd-sized prompt (time to first token of a chat turn)
        dict(name="prefill_7b_333", kind="prefill", model="7b", quant="none", batch=1, seq=333),
        # the largest prefill pass the engine makes: 8192 tokens
        dict(name="prefill_7b_8x1024", kind="prefill", model="7b", quant="none", batch=8, seq=1024),
        # an int8 model reads a prompt
        dict(name="prefill_7b_w8_1000", kind="prefill", model="7b", quant="w8a16", batch=1, seq=1000),
        # 1024 x 1024 image: 4096 image tokens and 512 text tokens
        dict(name="mmdit_4096", kind="mmdit", batch=1, height=64, width=64, txt=512),
        # a smaller image of odd proportions
        dict(name="mmdit_37x52", kind="mmdit", batch=1, height=37, width=52, txt=333),
        # the serving configuration of the int8 32B model
        dict(name="decode_32b_w8_b16", kind="decode", model="32b", quant="w8a16", batch=16, ctx=1200, graph=True),
        # the int4 demo model, one sequence
        dict(name="decode_7b_w4_b1", kind="decode", model="7b", quant="w4a16", batch=1, ctx=500, graph=True),
        # code written against the reference's op pair: one 32B layer, eight tokens
        dict(name="w8_layer_pair_m8", kind="w8_layer", form="pair", tokens=8, hidden=5120, inter=27648, qkv=7168),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """One more case of the ranges above."""
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "mmdit", "w8_layer"])
    if kind == "decode":
        model, quant, most, pages = rng.choice([("7b", "none", 128, 65536), ("7b", "none", 128, 65536),
                                                ("small", "none", 64, 8192), ("32b", "w8a16", 64, 32768),
                                                ("7b", "w8a16", 64, 32768), ("7b", "w4a16", 16, 16384)])
        batch = _logint(rng, 1, most)
        ctx = _logint(rng, 16, min(8192, pages // batch))
        return dict(kind="decode", model=model, quant=quant, batch=batch, ctx=ctx,
                    graph=model != "small" or rng.random() < 0.5)
    if kind == "prefill":
        quant = rng.choice(["none", "none", "w8a16"])
        total = _logint(rng, 32, 8192 if quant == "none" else 4096)
        batch = rng.choice([b for b in (1, 2, 3, 8) if b == 1 or total // b >= 32])
        return dict(kind="prefill", model="7b", quant=quant, batch=batch, seq=total // batch)
    if kind == "mmdit":
        batch = rng.choice([1, 1, 2])
        most = 64 if batch == 1 else 44
        return dict(kind="mmdit", batch=batch, height=rng.randint(16, most), width=rng.randint(16, most),
                    txt=rng.randint(64, 512))
    form = rng.choice(["pair", "int8", "int8_g128", "bf16_g128"])
    hidden, inter, qkv = rng.choice([(5120, 27648, 7168), (3584, 18944, 4608)])
    return dict(kind="w8_layer", form=form, tokens=_logint(rng, 1, 16 if form == "pair" else 64), hidden=hidden,
                inter=inter, qkv=qkv)


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
DEV = "cuda:0"


def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed((seed * 7919 + salt) % (1 << 31))


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32).to(torch.bfloat16)


class _Weights(RandomSource):
    """Random weights whose residual stream behaves like a trained decoder's: embeddings of unit size
    and output projections scaled by 0.4 / sqrt(2 * layers), so that every block adds a little to it.
    (Plain N(0, 0.02) makes the first block's output many times its input, and bf16 rounding then
    moves the logits of a 28-layer model by 5 % between one correct implementation and another.)"""

    def __init__(self, seed, layers):
        super().__init__(seed, DEV, torch.bfloat16)
        self.out_scale = 0.4 / math.sqrt(2 * layers)

    def weight(self, name, layer, shape, slot):
        w = super().weight(name, layer, shape, slot)
        if name in ("o_proj.weight", "down_proj.weight"):
            w.mul_(self.out_scale)
        elif name == "embed_tokens.weight":
            w.mul_(50.0)
        return w


def _decoder(case, seed):
    cfg = CONFIGS[case["model"]]()
    return Qwen2Model(cfg, TPComm.single(), DEV, torch.bfloat16, seed=seed, quant=case["quant"],
                      source=_Weights(seed, cfg.layers))


def _cache(model, batch, max_len, seed, filled):
    cache = PagedKV(len(model.w.layers), batch, max_len, model.nkv, model.hd, DEV, torch.bfloat16)
    g = _gen(seed, 2)
    if filled:  # keys and values of a context; N(0, 1) is what normalised activations times the weights give
        for t in cache.k + cache.v:
            t.copy_(torch.randn(t.shape, generator=g, device=DEV, dtype=torch.bfloat16))
    # pages are handed out in no particular order
    perm = torch.randperm(cache.block_tables.numel(), generator=g, device=DEV).to(torch.int32)
    cache.block_tables.copy_(perm.view_as(cache.block_tables))
    return cache


def _prepare_decode(case, seed):
    model, batch, ctx = _decoder(case, seed), case["batch"], case["ctx"]
    cache = _cache(model, batch, ctx + 16, seed, True)
    g = _gen(seed, 3)
    # context lengths spread over ctx / 2 .. ctx, the longest exactly ctx; the new token is the last of them
    lens = torch.randint(max(1, ctx // 2), ctx + 1, (batch,), generator=g, device=DEV, dtype=torch.int32)
    lens[batch - 1] = ctx
    s = dict(model=model, cache=cache, ctx_lens=lens, positions=(lens - 1).contiguous(),
             ids=torch.randint(0, model.cfg.vocab, (batch,), generator=g, device=DEV, dtype=torch.int32), graph=None)
    pos = s["positions"].long()
    blk = cache.block_tables[torch.arange(batch, device=DEV), pos // cache.block_size]
    s["slots"] = (blk * cache.block_size + pos % cache.block_size).to(torch.int32).contiguous()
    if case["graph"]:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                _decode_step(s)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            s["out"] = _decode_step(s)
    return s


def _decode_step(s):
    model = s["model"]
    hidden = model.decode_hidden(s["ids"], s["positions"], s["slots"], s["ctx_lens"], s["cache"])
    logits = model.logits(hidden)
    token, best = ops.argmax(logits)
    # `token` is left out: two bf16 logits at the top are often equal or one step apart, and then
    # which of them wins says nothing; `best` is the logit of the token
    del token
    # every layer's new key and value went into the next layer's input, so the last layer's cache
    # stands for the others (all of them would be 56 tensors and gigabytes)
    return {"logits": logits, "best": best, "k_cache": s["cache"].k[-1], "v_cache": s["cache"].v[-1]}


def _prepare_prefill(case, seed):
    model, batch, seq = _decoder(case, seed), case["batch"], case["seq"]
    cache = _cache(model, batch, seq + 16, seed, False)
    ids = torch.randint(0, model.cfg.vocab, (batch, seq), generator=_gen(seed, 3), device=DEV, dtype=torch.int32)
    return dict(model=model, cache=cache, ids=ids)


def _prepare_mmdit(case, seed):
    cfg = MMDiTConfig.flux_12b()
    model = MMDiTModel(cfg, MMDiTWeights(cfg, DEV, torch.bfloat16, seed=seed), TPComm.single())
    g, b, ni = _gen(seed, 4), case["batch"], case["height"] * case["width"]
    return dict(model=model, img=_randn(g, b, ni, cfg.in_channels), txt=_randn(g, b, case["txt"], cfg.txt_dim),
                t=torch.rand(b, generator=g, device=DEV), pos=grid_positions(case["height"], case["width"], DEV))


def _w8_shapes(case):
    h, f = case["hidden"], case["inter"]
    # (rows, k, input, SiLU * up) of QKV, o, gate/up, down
    return [(case["qkv"], h, "x", False), (h, h, "x", False), (2 * f, h, "x", True), (h, f, "f", False)]


def _prepare_w8_layer(case, seed):
    g, m, form = _gen(seed, 5), case["tokens"], case["form"]
    s = dict(form=form, x=_randn(g, m, case["hidden"]), f=_randn(g, m, case["inter"]), layers=[])
    for n, k, src, silu in _w8_shapes(case):
        w = torch.randn(n, k, generator=g, device=DEV) * 0.02
        if form == "int8":
            s["layers"].append((src, silu, ops.ref.quantize_w8(w)))
            continue
        wq, sc = ops.ref.quantize_w8_grouped(w, 128)
        if form == "pair":
            s["layers"].append((src, silu, (wq.view(n, k // 16, 16).permute(1, 0, 2).contiguous(),
                                            sc.float().t().contiguous(), n, k)))
        elif form == "int8_g128":
            s["layers"].append((src, silu, (wq, sc)))
        else:
            s["layers"].append((src, silu, (wq, ops.prepare_w8_scales(sc, k))))
    return s


def prepare(case, seed):
    return {"decode": _prepare_decode, "prefill": _prepare_prefill, "mmdit": _prepare_mmdit,
            "w8_layer": _prepare_w8_layer}[case["kind"]](case, seed) | {"kind": case["kind"]}


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "decode":
        if state["graph"] is None:
            return _decode_step(state)
        state["graph"].replay()
        return state["out"]
    if kind == "prefill":
        model, cache, ids = state["model"], state["cache"], state["ids"]
        hidden = model.prefill(ids, cache)
        last = hidden.view(ids.shape[0], ids.shape[1], -1)[:, -1].contiguous()
        return {"hidden": hidden, "logits": model.logits(last), "k_cache": cache.k[-1], "v_cache": cache.v[-1]}
    if kind == "mmdit":
        return state["model"].forward(state["img"], state["txt"], state["t"], state["pos"])
    if state["form"] == "pair":
        C, out = load_extension(), []
        for src, silu, (wq_t, sw_t, n, k) in state["layers"]:
            xq, xs = C.w8a16_quant_act(state[src])
            y = C.w8a16_gemm(xq, xs, wq_t, sw_t, n, k, 4)
            out.append(ops.silu_mul(y, interleaved=True) if silu else y)
        return out
    act = "bf16" if state["form"] == "bf16_g128" else "int8"
    return [ops.w8a16_linear(state[src], wq, sc, silu_mul=silu, act=act) for src, silu, (wq, sc) in state["layers"]]


# ---------------------------------------------------------------------------
# work and tolerance
# ---------------------------------------------------------------------------
def _decoder_params(cfg):
    """(attention, MLP) weights of one layer."""
    qkv = (cfg.n_heads + 2 * cfg.n_kv_heads) * cfg.head_dim * cfg.hidden
    return qkv + cfg.n_heads * cfg.head_dim * cfg.hidden, 3 * cfg.hidden * cfg.intermediate


def _decoder_weight_bytes(cfg, quant):
    attn, mlp = _decoder_params(cfg)
    wb = WEIGHT_BYTES[quant]
    mlp_b = 0.5 + 2.0 / 128 + 0.5 / 128 if quant == "w4a16" else wb  # nibbles, fp16 scales and zero points per 128
    return cfg.layers * (attn * wb + mlp * mlp_b) + cfg.vocab * cfg.hidden * wb


def work(case):
    kind = case["kind"]
    if kind == "decode":
        cfg, b = CONFIGS[case["model"]](), case["batch"]
        attn, mlp = _decoder_params(cfg)
        tokens = b * 0.75 * case["ctx"]  # mean length is three quarters of the longest
        kv = 2 * cfg.n_kv_heads * cfg.head_dim * 2 * cfg.layers
        return {"bytes": _decoder_weight_bytes(cfg, case["quant"]) + tokens * kv + b * (cfg.vocab + cfg.hidden) * 2,
                "flops": 2.0 * b * (cfg.layers * (attn + mlp) + cfg.vocab * cfg.hidden)
                + 4.0 * tokens * cfg.n_heads * cfg.head_dim * cfg.layers}
    if kind == "prefill":
        cfg, b, s = CONFIGS[case["model"]](), case["batch"], case["seq"]
        attn, mlp = _decoder_params(cfg)
        kv = 2 * cfg.n_kv_heads * cfg.head_dim * 2 * cfg.layers
        return {"bytes": _decoder_weight_bytes(cfg, case["quant"]) + b * s * (kv + 4 * cfg.hidden) + b * cfg.vocab * 2,
                "flops": 2.0 * b * s * cfg.layers * (attn + mlp) + 2.0 * b * cfg.vocab * cfg.hidden
                + 2.0 * b * s * (s + 1) * cfg.n_heads * cfg.head_dim * cfg.layers}
    if kind == "mmdit":
        cfg = MMDiTConfig.flux_12b()
        ni = case["height"] * case["width"]
        return {"bytes": 2.0 * cfg.params() + 2.0 * case["batch"] * (2 * ni * cfg.in_channels + case["txt"] * cfg.txt_dim),
                "flops": float(MMDiTModel.flops_per_forward(_Shape(cfg), case["batch"], ni, case["txt"]))}
    n_weights = sum(n * k for n, k, _, _ in _w8_shapes(case))
    scales = n_weights // 128 * (4 if case["form"] == "pair" else 2) if case["form"] != "int8" else 0
    io = sum(case["tokens"] * 2 * (k + (n // 2 if silu else n)) for n, k, _, silu in _w8_shapes(case))
    return {"bytes": float(n_weights + scales + io), "flops": 2.0 * case["tokens"] * n_weights}


class _Shape:
    """Just enough of a model for `MMDiTModel.flops_per_forward`."""

    def __init__(self, cfg):
        self.cfg = cfg


def tolerance(case):
    """What another correct implementation at the same precision may differ by.

    Measured against the same model in fp32 on the same weights: logits of the 28-layer decoder 1.4 %
    (rel) and 0.07 (max), of the 64-layer one 2.3 % and 0.12, of the two-layer one 0.4 %, MMDiT 1.5 % and
    0.07.  The library against itself with its sums in another order (other attention and GEMM kernels,
    other k-splits): 28-layer decoder 1.2 %, MMDiT 0.8 %.  bf16 rounds the residual stream after every
    block, so that a changed last bit early on moves the rest by that much.  The int8 layers: 0.17 %
    where the products are whole numbers (the bf16 rounding of the result), 1 % with group scales, which
    may be applied to the weights or to the sums."""
    if case["kind"] == "w8_layer":
        return {"rel": 0.007, "max": 0.035} if case["form"] in ("pair", "int8") else {"rel": 0.03, "max": 0.35}
    if case["kind"] == "decode" and case["model"] == "small":
        return {"rel": 0.016, "max": 0.08}
    return {"rel": 0.03, "max": 0.5 if case["kind"] != "mmdit" else 0.3}
