"""The work a user of this framework has it do, as cases to be timed: block masks, attention forward and backward,
and the token permutation, each through the public entry points on one GPU.

A case says the shape of a call; `prepare` makes its tensors, positions and segment ids from a seed (document lengths
and pads included), `run` is one pass.  Kinds:

  train    masks for forward and backward, forward, backward: one attention layer of a training step
  prefill  forward mask, forward: the prompt of a serving request, or a chunk of it on top of cached keys
  decode   forward mask, forward with a few new tokens per sequence against a cache of keys
  masks    the three masks of a packed batch alone
  permute  the load-balancing token permutation of context parallelism on token embeddings, positions and segment ids
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import kvax_b200 as kv

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(kind, batch, q_len, heads=0, kv_heads=0, head_dim=0, dtype="bf16", kv_len=None, fwd_block=(128, 128),
          bwd_block=(128, 128), doc_min=0, doc_max=0, pad=0.0, sequential=False, cp=1, name=None):
    c = dict(kind=kind, batch=batch, q_len=q_len, kv_len=kv_len or q_len, heads=heads, kv_heads=kv_heads, head_dim=head_dim,
             dtype=dtype, fwd_q_block=fwd_block[0], fwd_kv_block=fwd_block[1], bwd_q_block=bwd_block[0],
             bwd_kv_block=bwd_block[1], doc_min=doc_min or q_len, doc_max=doc_max or q_len, pad=pad, sequential=sequential, cp=cp)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The smallest call: the configuration the reference's tests run, fp32 with head_dim 64.  Latency and launches.
        _case("train", 1, 512, 4, 2, 64, "fp32", fwd_block=(64, 64), bwd_block=(64, 64), doc_min=64, doc_max=256, pad=32 / 512,
              name="train_tiny_fp32_512"),
        # Llama-3-8B attention layer on one packed 8k sequence.
        _case("train", 1, 8192, 32, 8, 128, doc_min=128, doc_max=4096, pad=0.025, name="train_llama8b_8k"),
        # Dense causal limit, multi-head attention: no tile to skip.
        _case("train", 4, 16384, 16, 16, 128, name="train_dense_mha_16k"),
        # Long packed sequences with padding: the configuration the benchmark is quoted on.
        _case("train", 2, 32768, 32, 8, 128, doc_min=256, doc_max=16384, pad=0.10, name="train_docmask_32k"),
        # Llama-3-70B attention layer on a 128k sequence: the largest.
        _case("train", 1, 131072, 64, 8, 128, doc_min=1024, doc_max=65536, name="train_docmask_128k"),
        # A small model's layer: head_dim 64, fp16, mask blocks of 64, a length that is no multiple of 128.
        _case("train", 8, 2112, 16, 16, 64, "fp16", fwd_block=(64, 64), bwd_block=(64, 64), doc_min=64, doc_max=1024, pad=0.05,
              name="train_ragged_fp16_d64_2k"),
        # An ordinary fine-tuning batch that relies on token indices as positions, with the reference's H100 block sizes.
        _case("train", 4, 4096, 32, 8, 128, bwd_block=(64, 128), doc_min=512, doc_max=4096, pad=0.02, sequential=True,
              name="train_sequential_4k"),
        # Prompts of odd length, packed.
        _case("prefill", 2, 5003, 32, 8, 128, doc_min=300, doc_max=4000, pad=0.01, name="prefill_ragged_5k"),
        # Chunked prefill: the next thousand tokens of two prompts on top of what is cached.
        _case("prefill", 2, 1000, 32, 8, 128, kv_len=17000, name="prefill_chunk_1k_of_17k"),
        # Decoding, sixteen sequences with up to 8k cached tokens each.
        _case("decode", 16, 1, 32, 8, 128, kv_len=8192, name="decode_8k_b16"),
        # The masks of a large packed batch.
        _case("masks", 16, 131072, doc_min=1024, doc_max=65536, pad=0.02, name="masks_16x128k"),
        # Embeddings (4096 wide) of a 64k sequence permuted for eight ranks.
        _case("permute", 1, 65536, 32, 0, 128, cp=8, doc_min=1024, doc_max=16384, name="permute_cp8_64k"),
    ]


def _log(rng: random.Random, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choices(("train", "prefill", "decode", "masks", "permute"), (6, 2, 2, 1, 1))[0]
    head_dim = rng.choice((128, 128, 128, 64, 32))
    kv_heads = rng.choice((1, 2, 4, 8, 16))
    heads = kv_heads * rng.choice((1, 2, 3, 4, 8)) if kv_heads < 16 else 16
    dtype = rng.choices(("bf16", "fp16", "fp32"), (6, 2, 1))[0]
    block = rng.choice(((128, 128), (128, 128), (64, 64), (128, 64)))
    if kind == "train":
        bwd = rng.choice(((128, 128), (64, 128), (64, 64)))
        seq = _log(rng, 256, 32768)
        unit = max(bwd)
        seq = max(unit, seq // unit * unit)                           # the backward pass wants whole blocks
        batch = max(1, min(16, _log(rng, 1, max(1, 131072 // seq))))
        doc_max = _log(rng, min(512, seq), seq)
        return _case(kind, batch, seq, heads, kv_heads, head_dim, dtype, fwd_block=block, bwd_block=bwd,
                     doc_min=max(16, doc_max // rng.choice((1, 8, 32))), doc_max=doc_max, pad=rng.choice((0.0, 0.03, 0.1)),
                     sequential=rng.random() < 0.25)
    if kind == "prefill":
        seq = _log(rng, 100, 20000)
        batch = max(1, min(8, _log(rng, 1, max(1, 65536 // seq))))
        if rng.random() < 0.4:
            return _case(kind, batch, _log(rng, 17, max(17, min(seq, 2048))), heads, kv_heads, head_dim, dtype, kv_len=seq,
                         fwd_block=block)
        doc_max = _log(rng, min(256, seq), seq)
        return _case(kind, batch, seq, heads, kv_heads, head_dim, dtype, fwd_block=block, doc_min=max(16, doc_max // 8),
                     doc_max=doc_max, pad=rng.choice((0.0, 0.02)))
    if kind == "decode":
        return _case(kind, _log(rng, 1, 64), rng.choice((1, 1, 1, 2, 4, 7)), heads, kv_heads, head_dim, dtype if dtype != "fp32" else "bf16",
                     kv_len=_log(rng, 200, 32768), fwd_block=block)
    seq = _log(rng, 1024, 131072)
    batch = _log(rng, 1, max(1, min(64, (1 << 21) // seq)))
    doc_max = _log(rng, 512, seq)
    if kind == "masks":
        bwd = rng.choice(((128, 128), (64, 128)))
        return _case(kind, batch, seq, fwd_block=block, bwd_block=bwd, doc_min=max(16, doc_max // 16), doc_max=doc_max,
                     pad=rng.choice((0.0, 0.02, 0.1)))
    cp = rng.choice((2, 4, 8))
    seq = max(2 * cp, seq // (2 * cp) * (2 * cp))
    return _case(kind, max(1, min(batch, 65536 // seq)), seq, rng.choice((8, 16, 32)), 0, 128, cp=cp, doc_min=max(16, doc_max // 16),
                 doc_max=doc_max)


def _documents(case, rng: np.random.Generator):
    """Document lengths of every batch row: log-uniform, cut at the row's end, padding after them."""
    n, rows = case["kv_len"], []
    real = n - int(round(case["pad"] * n))
    lo, hi = math.log(case["doc_min"]), math.log(max(case["doc_min"], case["doc_max"]))
    for _ in range(case["batch"]):
        lengths, used = [], 0
        while used < real:
            d = min(real - used, max(1, int(math.exp(rng.uniform(lo, hi)))))
            lengths.append(d)
            used += d
        rows.append(lengths)
    return rows


def _tokens(case, seed):
    """(query positions, query segment ids, kv positions, kv segment ids) on the host."""
    rng = np.random.default_rng(seed)
    batch, n, q_len = case["batch"], case["kv_len"], case["q_len"]
    pos = np.zeros((batch, n), np.int32)
    seg = np.full((batch, n), kv.PADDING_SEGMENT_ID, np.int32)
    if case["kind"] == "decode" or q_len != n:                  # new tokens behind a cache: one sequence per row
        used = rng.integers(max(q_len, n // 2), n + 1, batch) if case["kind"] == "decode" else np.full(batch, n)
        pos[:] = np.arange(n)
        q_pos = np.zeros((batch, q_len), np.int32)
        for b in range(batch):
            seg[b, :used[b]] = 0
            q_pos[b] = np.arange(used[b] - q_len, used[b])
        return q_pos, np.zeros((batch, q_len), np.int32), pos, seg
    for b, lengths in enumerate(_documents(case, rng)):
        at = 0
        for d, m in enumerate(lengths):
            seg[b, at:at + m] = d
            pos[b, at:at + m] = np.arange(at, at + m) if case["sequential"] else np.arange(m)
            at += m
        pos[b, at:] = np.arange(at, n) if case["sequential"] else np.arange(n - at)
    return pos, seg, pos, seg


def prepare(case, seed):
    q_pos, q_seg, kv_pos, kv_seg = _tokens(case, seed)
    same = q_pos is kv_pos
    state = {"case": case, "q_pos": torch.from_numpy(q_pos).cuda(), "q_seg": torch.from_numpy(q_seg).cuda()}
    state["kv_pos"] = state["q_pos"] if same else torch.from_numpy(kv_pos).cuda()
    state["kv_seg"] = state["q_seg"] if same else torch.from_numpy(kv_seg).cuda()
    state["fwd"] = kv.FlashAttentionParamsConfig(case["fwd_q_block"], case["fwd_kv_block"])
    state["bwd"] = kv.FlashAttentionParamsConfig(case["bwd_q_block"], case["bwd_kv_block"])
    kind, dtype = case["kind"], _DTYPES[case["dtype"]]
    axis = "context" if kind == "permute" else None
    state["specs"] = (("data", axis, None, None), ("data", None, None, None))
    state["mesh"] = kv.Mesh(("data", "context"), (1, case["cp"]), rank=0)
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)

    if kind == "permute":
        state["x"] = randn(case["batch"], case["q_len"], case["heads"] * case["head_dim"])
    elif kind != "masks":
        b, d = case["batch"], case["head_dim"]
        train = kind == "train"
        state["q"] = randn(b, case["q_len"], case["heads"], d).requires_grad_(train)
        state["k"] = randn(b, case["kv_len"], case["kv_heads"], d).requires_grad_(train)
        state["v"] = randn(b, case["kv_len"], case["kv_heads"], d).requires_grad_(train)
        if train:                                               # the loss does not look at padding
            real = (state["q_seg"] != kv.PADDING_SEGMENT_ID)[:, :, None, None]
            state["dout"] = randn(b, case["q_len"], case["heads"], d) * real
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    with kv.attention_specs(*state["specs"]), state["mesh"]:
        if kind == "permute":
            return kv.permute_tokens_context_parallelism((state["x"], state["q_pos"], state["q_seg"]))
        tokens = (state["q_pos"], state["q_seg"], state["kv_pos"], state["kv_seg"])
        train = kind in ("train", "masks")
        masks = kv.create_attention_mask(*tokens, fwd_params=state["fwd"], bwd_params=state["bwd"], calc_bwd_mask=train)
        if kind == "masks":
            return [(m.lower_bounds, m.upper_bounds, m.lower_full_bounds, m.upper_full_bounds) for m in masks]
        call = dict(scale=case["head_dim"] ** -0.5, fwd_params=state["fwd"], bwd_params=state["bwd"],
                    assume_sequential_positions=case["sequential"])
        if kind != "train":
            with torch.no_grad():
                return kv.flash_attention(state["q"], state["k"], state["v"], *tokens, masks, **call)
        qkv = (state["q"], state["k"], state["v"])
        out = kv.flash_attention(*qkv, *tokens, masks, **call)
        return (out.detach(), *torch.autograd.grad(out, qkv, state["dout"]))


def work(case):
    b, sq, skv, kind = case["batch"], case["q_len"], case["kv_len"], case["kind"]
    same = sq == skv and kind != "decode"
    index = 8 * b * (skv if same else sq + skv)                 # int32 positions and segment ids
    if kind == "permute":
        return {"bytes": 2 * (b * sq * case["heads"] * case["head_dim"] * 2 + index), "flops": 0}
    if kind == "masks":
        nq = -(-sq // case["fwd_q_block"]) + -(-sq // case["bwd_kv_block"]) + -(-skv // case["bwd_kv_block"])
        return {"bytes": index + 16 * b * nq, "flops": 0}
    size = 4 if case["dtype"] == "fp32" else 2
    q_bytes = b * sq * case["heads"] * case["head_dim"] * size
    kv_bytes = 2 * b * skv * case["kv_heads"] * case["head_dim"] * size
    if kind == "decode":
        kv_bytes = kv_bytes * 3 // 4                            # caches are half full to full
    if kind == "decode" or sq != skv:
        allowed = b * sq * ((0.75 if kind == "decode" else 1.0) * skv - sq / 2)
    else:                                                       # mean over document layouts
        allowed = float(np.mean([sum(m * (m + 1) // 2 for row in _documents(case, np.random.default_rng(s)) for m in row)
                                 for s in range(64)]))
    flops = 4.0 * case["head_dim"] * case["heads"] * allowed     # Q K^T and P V of the unmasked elements
    if kind != "train":
        return {"bytes": index + 2 * q_bytes + kv_bytes, "flops": flops}
    return {"bytes": index + 4 * q_bytes + 2 * kv_bytes, "flops": 3.5 * flops}   # q, out, dout, dq; k, v, dk, dv


def tolerance(case):
    """Whole numbers and moved bytes are exact.  Attention: P and dS are rounded to the 16-bit operand type before the second
    products and the results to the output type (8 bits of fraction in bf16, 11 in fp16; fp32 tensors are computed with fp16
    operands).  Measured against the same attention in fp64, the largest of out, dq, dk, dv: bf16 2.5e-3, fp16 3.2e-4, fp32
    5.5e-4; four times that is stated."""
    if case["kind"] in ("masks", "permute"):
        return "exact"
    return {"rel": {"bf16": 1e-2, "fp16": 1.3e-3, "fp32": 2.2e-3}[case["dtype"]]}
