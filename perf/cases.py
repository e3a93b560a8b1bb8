"""Workloads of the attention hot path, through the calls a user's program makes.

A case is a dict of plain values; ``prepare`` builds what such a program holds before the call (weights, caches, inputs,
masks), ``run`` makes the call once, ``work`` counts the bytes and floating-point operations one call cannot do without.

Kinds of case (``op``):
    token      one decoded token through a stack of attention layers over the ring cache (StepRunner), launched layer by
               layer or as one CUDA-graph replay; bf16 or float16 ring
    prompt     a prompt through the same stack, filling the ring (StepRunner)
    forward    one attention layer over whole sequences, inference (B200CausalSelfAttention.forward)
    attend     norm, RoPE and windowed attention on q, k, v that are already projected (ops.swa_prefill)
    train      one attention layer forward and backward under autograd
    kda        Kimi delta attention (kda.chunk_kda), dense or packed sequences
    kda_layer  the whole Kimi layer over a prompt, keeping its states (B200KimiLinearSelfAttention.prefill)
    kda_token  the Kimi layer's decode step (``step``, or ``step_graph``)
"""
from __future__ import annotations

import math

import torch

from daisy_b200 import (B200CausalSelfAttention, B200KimiLinearSelfAttention, BlockWindowMask, StepRunner, WindowMask,
                        doc_starts, ops)
from daisy_b200.accounting import FP32_EPS, kda_bytes_per_token_head, kda_flops_per_token_head
from daisy_b200.kda import chunk_kda

D = 128                      # head dimension of every configuration
EOS = 50256                  # token that opens the next document
MAX_POSITIONS = 131072       # the module's default RoPE table


def listed():
    return [
        # a chat turn's next token: four layers, batch 1, the float16 cache the generator allocates by default, launched
        # layer by layer from Python
        dict(name="token", op="token", layers=4, batch=1, heads=16, window=4096, cap=4096, ctx=5000, graph=False, f16=True),
        # the smallest decode step (d_model 768, short window), replayed as a CUDA graph
        dict(name="token_graph", op="token", layers=2, batch=1, heads=6, window=512, cap=512, ctx=700, graph=True, f16=False),
        # batched serving: 64 sequences, window 4096, a ring longer than the window
        dict(name="token_batch", op="token", layers=1, batch=64, heads=16, window=4096, cap=8192, ctx=9001, graph=False, f16=False),
        # a short, ragged prompt on the small model: latency and launches
        dict(name="prompt_short", op="prompt", layers=2, batch=1, tokens=131, heads=6, window=512, f16=False),
        # the headline prefill shape with its projections, several documents per row
        dict(name="forward", op="forward", batch=8, tokens=8192, heads=16, window=2048, docs=6, ve=False),
        # long-context prefill on projected q, k, v
        dict(name="attend_long", op="attend", batch=1, tokens=65536, heads=16, window=8192),
        # a small training step in a layer that receives a value embedding
        dict(name="train_small", op="train", batch=1, tokens=1024, heads=6, window=512, blocks=False, docs=3, ve=True),
        # the training form at the headline shape: block-granular window, documents
        dict(name="train", op="train", batch=8, tokens=8192, heads=16, window=2048, blocks=True, docs=6, ve=False),
        # KDA over long dense sequences
        dict(name="kda", op="kda", batch=4, tokens=16384, heads=16, seqs=0, state=False),
        # KDA over packed sequences of uneven length, continuing from carried states
        dict(name="kda_packed", op="kda", batch=1, tokens=5003, heads=16, seqs=11, state=True),
        # the Kimi layer over two prompts, states kept for decoding
        dict(name="kda_layer", op="kda_layer", batch=2, tokens=3001, heads=16, padded=False),
        # the Kimi layer's decode step, launched from Python
        dict(name="kda_token", op="kda_token", batch=1, heads=16, graph=False),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))


def draw(rng):
    op = rng.choice(["token", "prompt", "forward", "attend", "train", "kda", "kda_layer", "kda_token"])
    heads = rng.choice([6, 8, 12, 16])
    if op == "token":
        window = _log(rng, 128, 8192)
        cap = window * rng.choice([1, 1, 2])
        layers = rng.randint(1, 4)
        most = 2_100_000_000 // (layers * heads * window * 4 * D)            # no more cache traffic than 64 x 16 x 4096
        return dict(op=op, layers=layers, batch=min(_log(rng, 1, 64), max(1, most)), heads=heads, window=window, cap=cap,
                    ctx=cap + rng.randrange(cap), graph=rng.random() < 0.5, f16=rng.random() < 0.5)
    if op == "prompt":
        tokens = _log(rng, 16, 8192)
        return dict(op=op, layers=rng.randint(1, 4), batch=min(rng.randint(1, 4), max(1, 16384 // tokens)), tokens=tokens,
                    heads=heads, window=_log(rng, 128, 4096), f16=rng.random() < 0.5)
    if op == "forward":
        tokens = _log(rng, 128, 16384)
        return dict(op=op, batch=min(rng.randint(1, 8), max(1, 65536 // tokens)), tokens=tokens, heads=heads,
                    window=_log(rng, 128, 4096), docs=rng.choice([0, 0, rng.randint(2, 16)]), ve=rng.random() < 0.3)
    if op == "attend":
        tokens = _log(rng, 200, 65536)
        return dict(op=op, batch=min(rng.randint(1, 8), max(1, 65536 // tokens)), tokens=tokens, heads=heads,
                    window=_log(rng, 128, 8192))
    if op == "train":
        tokens, blocks = _log(rng, 256, 8192), rng.random() < 0.5
        if blocks:
            tokens = -(-tokens // 128) * 128
        window = _log(rng, 128, 2048)
        return dict(op=op, batch=min(rng.randint(1, 8), max(1, 65536 // tokens)), tokens=tokens, heads=heads,
                    window=-(-window // 128) * 128 if blocks else window, blocks=blocks,
                    docs=rng.choice([0, rng.randint(2, 12)]), ve=rng.random() < 0.3)
    if op == "kda":
        tokens = _log(rng, 40, 16384)
        seqs = rng.choice([0, 0, rng.randint(2, 16)])
        return dict(op=op, batch=1 if seqs else min(rng.randint(1, 4), max(1, 65536 // tokens)), tokens=tokens, heads=heads,
                    seqs=seqs, state=rng.random() < 0.5)
    if op == "kda_layer":
        tokens = _log(rng, 64, 8192)
        return dict(op=op, batch=min(rng.randint(1, 4), max(1, 16384 // tokens)), tokens=tokens, heads=heads,
                    padded=rng.random() < 0.3)
    return dict(op=op, batch=_log(rng, 1, 64), heads=heads, graph=rng.random() < 0.5)


# ---------------------------------------------------------------------------------------------- layout of rows
def _edges(n, parts, row=0):
    """0 = e_0 < e_1 < .. = n: uneven pieces at fixed places (multiples of the golden ratio), other ones in another row."""
    inner = {int(n * ((0.6180339887 * i + 0.37 * row) % 1.0)) for i in range(1, parts)}
    return [0] + sorted(e for e in inner if 0 < e < n) + [n]


def _documents(case):
    """Token ids ``[B,T]`` on the CPU with an EOS at every document's first position, or None."""
    if not case["docs"]:
        return None
    ids = torch.zeros(case["batch"], case["tokens"], dtype=torch.int64, device="cpu")
    for b in range(case["batch"]):
        ids[b, _edges(case["tokens"], case["docs"], b)[1:-1]] = EOS
    return ids


def _kept(case):
    """Tokens kept in each row of a padded batch."""
    return [max(1, int(case["tokens"] * (1.0 - 0.11 * ((3 * b) % 5)))) for b in range(case["batch"])]


def _pairs(case):
    """Visible (query, key) pairs over the batch."""
    B, T, W = case["batch"], case["tokens"], case["window"]
    q = torch.arange(T)
    first = (q - W + 1).clamp_(min=0)
    if case.get("blocks"):
        first = ((q // 128 - W // 128 + 1) * 128).clamp_(min=0)
    ids = _documents(case) if case.get("docs") else None
    if ids is None:
        return B * int((q - first + 1).sum())
    ds = doc_starts(ids, EOS).reshape(B, T).long()
    return int((q - torch.maximum(first, ds) + 1).sum())


# ---------------------------------------------------------------------------------------------- preparation
def _normal(*shape, std=1.0, dtype=torch.bfloat16):
    return torch.randn(*shape, dtype=dtype).mul_(std)


def _attention(heads, ve=False):
    dim = heads * D
    a = B200CausalSelfAttention(dim, heads, D, receives_ve=ve, layer_idx=0 if ve else None, max_seq_len=MAX_POSITIONS)
    with torch.no_grad():
        a.qkvo_w.copy_(torch.randn(4, dim, dim).mul_(dim ** -0.5))
    return a


def _mask(case):
    ids = _documents(case)
    ds = None if ids is None else doc_starts(ids.cuda(), EOS)
    if case.get("blocks"):
        return BlockWindowMask(case["window"] // 128, ds)
    return WindowMask(case["window"], ds)


def _rope_tables(T):
    freq = 10000.0 ** (-torch.arange(0, D, 2, dtype=torch.float32) / D)
    angle = torch.arange(T, dtype=torch.float32)[:, None] * freq[None, :]
    return angle.cos(), angle.sin()


def prepare(case, seed):
    torch.manual_seed(seed)
    with torch.device("cuda"):
        return _PREPARE[case["op"]](case)


def _prepare_token(case):
    L, B, H, W, cap = case["layers"], case["batch"], case["heads"], case["window"], case["cap"]
    runner = StepRunner([_attention(H) for _ in range(L)], W, cache_capacity=cap, batch=B,
                        dtype=torch.float16 if case["f16"] else torch.bfloat16)
    for c in (runner.cache.k, runner.cache.v):                    # the normalised rows of `ctx` earlier tokens
        for layer in range(L):
            c[layer].normal_()
    runner.cache.set_position(case["ctx"])
    if case["graph"]:
        runner.capture_step(B, H * D)
    return dict(run=_run_token_graph if case["graph"] else _run_token, runner=runner, x=_normal(B, 1, H * D))


def _run_token(s):
    y = s["runner"]._step(s["x"])
    return y, s["runner"].cache.k, s["runner"].cache.v


def _run_token_graph(s):
    y = s["runner"]._step_graph(s["x"])
    return y, s["runner"].cache.k, s["runner"].cache.v


def _prepare_prompt(case):
    L, B, H = case["layers"], case["batch"], case["heads"]
    runner = StepRunner([_attention(H) for _ in range(L)], case["window"], batch=B,
                        dtype=torch.float16 if case["f16"] else torch.bfloat16)
    return dict(run=_run_prompt, runner=runner, x=_normal(B, case["tokens"], H * D))


def _run_prompt(s):
    y = s["runner"]._prefill(s["x"])
    return y, s["runner"].cache.k, s["runner"].cache.v


def _prepare_forward(case):
    B, T, H = case["batch"], case["tokens"], case["heads"]
    return dict(run=_run_forward, layer=_attention(H, case["ve"]), x=_normal(B, T, H * D), mask=_mask(case),
                ve=_normal(B, T, H * D) if case["ve"] else None)


def _run_forward(s):
    with torch.inference_mode():
        return s["layer"].forward(s["x"], s["ve"], attn_mask=s["mask"])


def _prepare_attend(case):
    B, T, H = case["batch"], case["tokens"], case["heads"]
    q, k, v = (_normal(B, T, H, D) for _ in range(3))
    cos, sin = _rope_tables(T)
    return dict(run=_run_attend, q=q, k=k, v=v, cos=cos, sin=sin, window=case["window"])


def _run_attend(s):
    return ops.swa_prefill(s["q"], s["k"], s["v"], s["cos"], s["sin"], s["window"], eps=FP32_EPS)


def _prepare_train(case):
    B, T, H = case["batch"], case["tokens"], case["heads"]
    layer = _attention(H, case["ve"])
    # the upstream gradient and the value embedding both have a part that all tokens share, as they do in a network (it
    # also keeps the one-number gradient of the gate away from zero)
    shared = torch.randn(H * D).mul_(0.5)
    s = dict(run=_run_train, layer=layer, x=_normal(B, T, H * D).requires_grad_(), ve=None, mask=_mask(case), blocks=case["blocks"],
             dy=(_normal(B, T, H * D) + shared).bfloat16())
    if case["ve"]:
        common = shared @ layer.qkvo_w.detach()[3].float()
        s["ve"] = (_normal(B, T, H * D) + common).bfloat16().requires_grad_()
    s["wrt"] = [s["x"], layer.qkvo_w] + ([s["ve"], layer.g_ve] if case["ve"] else [])
    return s


def _run_train(s):
    if s["blocks"]:
        y = s["layer"].forward(s["x"], s["ve"], block_mask=s["mask"])
    else:
        y = s["layer"].forward(s["x"], s["ve"], attn_mask=s["mask"])
    return (y.detach(),) + torch.autograd.grad(y, s["wrt"], s["dy"])


def _prepare_kda(case):
    B, T, H, n = case["batch"], case["tokens"], case["heads"], case["seqs"]
    q, k, v = (_normal(B, T, H, D) for _ in range(3))
    g = torch.nn.functional.logsigmoid(torch.randn(B, T, H, D))
    beta = torch.randn(B, T, H).sigmoid_()
    cu = torch.tensor(_edges(T, n), dtype=torch.int32) if n else None       # as an unpadding helper leaves it: on the device
    rows = B if cu is None else cu.numel() - 1
    h0 = torch.randn(rows, H, D, D).mul_(0.1) if case["state"] else None
    return dict(run=_run_kda, args=dict(q=q, k=k, v=v, g=g, beta=beta, initial_state=h0, output_final_state=True,
                                        use_qk_l2norm_in_kernel=True, cu_seqlens=cu))


def _run_kda(s):
    return chunk_kda(**s["args"])


def _kimi(heads):
    return B200KimiLinearSelfAttention(heads * D, heads, MAX_POSITIONS, D)


def _prepare_kda_layer(case):
    B, T, H = case["batch"], case["tokens"], case["heads"]
    mask = None
    if case["padded"]:
        mask = torch.zeros(B, T, dtype=torch.int64)
        for b, n in enumerate(_kept(case)):
            mask[b, T - n:] = 1
    return dict(run=_run_kda_layer, layer=_kimi(H), x=_normal(B, T, H * D), mask=mask)


def _run_kda_layer(s):
    layer = s["layer"]
    with torch.inference_mode():
        layer.reset_history()
        y, _, _ = layer.prefill(s["x"], attn_mask=s["mask"])
        return (y, layer._recurrent_state) + tuple(layer._conv_state)


def _prepare_kda_token(case):
    B, H = case["batch"], case["heads"]
    layer = _kimi(H)
    with torch.inference_mode():
        layer.prefill(_normal(B, 200, H * D))
        if case["graph"]:
            layer.capture_step(B)
    return dict(run=_run_kda_token_graph if case["graph"] else _run_kda_token, layer=layer, x=_normal(B, 1, H * D))


def _run_kda_token(s):
    layer = s["layer"]
    with torch.inference_mode():
        y, _, _ = layer.step(s["x"])
    return (y, layer._recurrent_state) + tuple(layer._conv_state)


def _run_kda_token_graph(s):
    layer = s["layer"]
    y = layer.step_graph(s["x"])
    return (y, layer._recurrent_state) + tuple(layer._conv_state)


_PREPARE = dict(token=_prepare_token, prompt=_prepare_prompt, forward=_prepare_forward, attend=_prepare_attend,
                train=_prepare_train, kda=_prepare_kda, kda_layer=_prepare_kda_layer, kda_token=_prepare_kda_token)


def run(state):
    return state["run"](state)


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    op, B, H = case["op"], case["batch"], case["heads"]
    dim = H * D
    if op == "token":
        rows = min(case["cap"], case["window"] - 1)
        w, L = 4 * dim * dim, case["layers"]
        # weights and context rows read, the new k, v rows and the output written
        return dict(bytes=L * (2 * w + B * H * D * 2 * (2 * rows + 2)) + 4 * B * dim, flops=L * B * (2 * w + 4 * D * H * rows))
    if op in ("prompt", "forward", "attend", "train"):
        T = case["tokens"]
        M = B * T
        attend, project = 4 * D * H * _pairs(case), 8 * M * dim * dim
        if op == "prompt":
            kept = B * min(T, case["window"] - 1)
            return dict(bytes=case["layers"] * (8 * dim * dim + 4 * kept * dim) + 4 * M * dim,
                        flops=case["layers"] * (attend + project))
        if op == "forward":
            return dict(bytes=8 * dim * dim + 2 * M * dim * (3 if case["ve"] else 2), flops=attend + project)
        if op == "attend":
            return dict(bytes=12 * M * dim, flops=attend)
        # x, dy (ve) read, y, dx (its gradient) written, the weights read and their gradient written; a backward is two
        # products for each one of the projections and five for the two of the attention
        return dict(bytes=16 * dim * dim + 2 * M * dim * (6 if case["ve"] else 4), flops=3 * project + 3.5 * attend)
    if op == "kda":
        n = B * case["tokens"] * H
        states = (B if not case["seqs"] else len(_edges(case["tokens"], case["seqs"])) - 1) * H * D * D * 4
        return dict(bytes=n * kda_bytes_per_token_head() + states * (2 if case["state"] else 1), flops=n * kda_flops_per_token_head())
    weights = 4 * dim * dim + 2 * 2 * dim * D + dim * H + 3 * 4 * dim
    if op == "kda_layer":
        M = sum(_kept(case)) if case["padded"] else B * case["tokens"]
        return dict(bytes=2 * weights + 4 * M * dim + B * (H * D * D * 4 + 3 * 4 * dim * 2),
                    flops=2 * M * (4 * dim * dim + 2 * 2 * dim * D + dim * H) + M * H * kda_flops_per_token_head())
    return dict(bytes=2 * weights + 4 * B * dim + 2 * B * (H * D * D * 4 + 3 * 4 * dim * 2), flops=2 * B * (weights + 4 * H * D * D))


def tolerance(case):
    if case["op"] == "kda":
        # fp16 operands with fp32 accumulation (4e-4 of the fp32 recurrence) under a bf16 output (1.7e-3)
        return {"rel": 4e-3}
    # bf16 results of bf16 operands with fp32 accumulation, once more through each further layer of a stack
    return {"rel": 1e-2 * math.sqrt(case.get("layers", 1))}
