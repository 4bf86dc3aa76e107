"""The work that a user of landmark_attention_b200 has it do, as cases that can be timed and compared.

Kinds of case (field "kind") and where the work comes from:
  fused    fused_landmark_attention: attention of a whole sequence or of a chunk behind a key history, forward alone
           (prompt processing) or forward + backward (training), every data type, head dim and block size it is used with.
  layer    what a layer of the lm_benchmark GPT calls in a training step: rotary_apply on q and k, then
           lm_landmark_attention with landmarks at each row's own positions, then the gradients of q, k and v.
  softmax  the grouped softmax on scores that exist in memory, forward + backward, in the two flavours.
  chunk    one layer of long-context inference, prompt processing: llama_retrieval_attention of a chunk of whole or ragged
           length against a LandmarkKVCache, one selection per (head, token) or per head.
  decode   the same layer while tokens are generated: one token, or a few, behind a cache whose last block is unfinished.
  eval     one layer of the lm_benchmark evaluation with a block cache: retrieve_for_query, lm_landmark_attention over the
           retrieved prefix and the chunk, store_in_cache.
  offload  the inference layer with the blocks in pinned host memory (OffloadedLandmarkCache.attend).
"""
import math
import types

import torch

import landmark_attention_b200 as P

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZES = {"f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # a short prompt of odd length: one small launch, so latency and host time are all there is
        dict(name="fused short prompt", kind="fused", dtype="f16", B=1, H=32, Lq=77, history=0, D=128, block=64,
             backward=False, mask=False),
        # the attention of a 7B model's training step at its training length (the benchmark's headline)
        dict(name="fused training", kind="fused", dtype="bf16", B=1, H=32, Lq=2048, history=0, D=128, block=64,
             backward=True, mask=False),
        # the longest sequence of the benchmark's sweep, training
        dict(name="fused long training", kind="fused", dtype="bf16", B=1, H=32, Lq=32768, history=0, D=128, block=64,
             backward=True, mask=False),
        # a prompt chunk of odd length behind the blocks that were retrieved for it
        dict(name="fused prompt with history", kind="fused", dtype="f16", B=1, H=32, Lq=1999, history=5 * 64, D=128,
             block=64, backward=False, mask=False),
        # training with heads of 64 features
        dict(name="fused training D64", kind="fused", dtype="bf16", B=4, H=16, Lq=1024, history=0, D=64, block=64,
             backward=True, mask=False),
        # 32-bit training on a small problem with the landmark mask handed over, as the reference's own test does
        dict(name="fused f32", kind="fused", dtype="f32", B=2, H=8, Lq=512, history=0, D=64, block=64, backward=True,
             mask=True),
        # a layer of the 12-layer GPT's training step: batch 16, 512 tokens, a landmark after every 50
        dict(name="GPT layer training", kind="layer", dtype="bf16", B=16, H=8, T=512, D=128, block=51, groups=16),
        # grouped softmax of the same layer on scores in memory
        dict(name="grouped softmax", kind="softmax", flavour="lm", dtype="f32", B=16, H=8, Lq=512, Lk=512, block=51),
        # long-context prompt processing: 250 tokens and their landmarks against a cache of 32768
        dict(name="retrieval chunk", kind="chunk", dtype="bf16", B=1, H=32, T=258, D=128, block=32, n_blocks=1024,
             top_k=4, per_head=False),
        # generating the next token behind the same cache, its last block unfinished
        dict(name="retrieval decode", kind="decode", dtype="bf16", B=1, H=32, T=1, D=128, block=32, n_blocks=1024,
             tail=17, top_k=4),
        # cached evaluation of the GPT: batch 16, chunks of 250 tokens and 5 landmarks, a ring of 40 blocks, top 4
        dict(name="GPT cached evaluation", kind="eval", dtype="bf16", B=16, H=8, D=128, block=51, chunk_blocks=5,
             capacity=40, top_k=4, method="per_token_and_head"),
        # a chunk against blocks that live in host memory
        dict(name="offloaded cache chunk", kind="offload", dtype="bf16", B=1, H=32, T=256, D=128, block=64, n_blocks=128,
             top_k=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fused", "fused", "fused", "layer", "softmax", "chunk", "decode", "eval", "offload"])
    half = rng.choice(["bf16", "f16"])
    if kind == "fused":
        dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
        block = 64 if dtype == "f32" else rng.choice([64, 64, 64, 32])
        backward = rng.random() < 0.5
        D = rng.choice([64, 128, 128])
        top = 1024 if dtype == "f32" else 1700 if block == 32 else 16384
        Lq = _log(rng, 64, top)
        if dtype == "f32" and backward:
            Lq = -(-Lq // block) * block
        history = 64 * rng.choice([0, 0, 1, 3, 5])
        H = rng.choice([8, 16, 32])
        B = _log(rng, 1, 4 if dtype == "f32" else 8) if Lq * H <= 65536 else 1
        return dict(kind=kind, dtype=dtype, B=B, H=H, Lq=Lq, history=history, D=D, block=block, backward=backward,
                    mask=rng.random() < 0.2)
    if kind == "layer":
        T = 128 * rng.randint(2, 8)
        block = rng.choice([26, 51, 51, 64])
        return dict(kind=kind, dtype=half, B=_log(rng, 2, 32), H=rng.choice([8, 12, 16]), T=T, D=128, block=block,
                    groups=min(64, T // block + 2))
    if kind == "softmax":
        Lk = _log(rng, 100, 2048)
        return dict(kind=kind, flavour=rng.choice(["lm", "llama"]), dtype=rng.choice(["f32", "bf16"]), B=_log(rng, 1, 8),
                    H=rng.choice([8, 32]), Lq=Lk, Lk=Lk, block=rng.choice([32, 51, 64]))
    if kind == "chunk":
        block, per_head = rng.choice([32, 64]), rng.random() < 0.3
        return dict(kind=kind, dtype=half, B=1, H=rng.choice([8, 32, 40]), T=_log(rng, 40, 900), D=128, block=block,
                    n_blocks=_log(rng, 24, 1500), top_k=rng.randint(1, 6), per_head=per_head)
    if kind == "decode":
        block = rng.choice([32, 64])
        tail = rng.randint(1, block - 2)
        return dict(kind=kind, dtype=half, B=rng.choice([1, 1, 2, 4]), H=rng.choice([8, 32, 40]),
                    T=rng.choice([1, 1, 1, min(3, block - tail)]), D=128, block=block, n_blocks=_log(rng, 24, 1500),
                    tail=tail, top_k=rng.randint(1, 6))
    if kind == "eval":
        return dict(kind=kind, dtype=half, B=_log(rng, 2, 16), H=rng.choice([8, 12]), D=128, block=51,
                    chunk_blocks=rng.randint(3, 7), capacity=rng.randint(10, 80), top_k=rng.randint(2, 4),
                    method=rng.choice(["per_token_and_head", "per_token_and_head", "max_over_heads", "max_over_tokens"]))
    block = rng.choice([32, 64])
    return dict(kind=kind, dtype=half, B=1, H=rng.choice([8, 32]), T=block * rng.randint(2, 512 // block), D=128,
                block=block, n_blocks=_log(rng, 24, 200), top_k=rng.randint(1, 6))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, shape, dtype, std=1.0):
    return (torch.randn(shape, generator=g, device="cuda") * std).to(dtype)


def prepare(case, seed):
    g, dtype, c = _gen(seed), DTYPES[case["dtype"]], dict(case)
    s = {"case": c}
    B, H = c["B"], c["H"]
    if c["kind"] == "fused":
        Lk = c["Lq"] + c["history"]
        s["q"] = _randn(g, (B, H, c["Lq"], c["D"]), dtype, 0.5).requires_grad_(c["backward"])
        s["k"], s["v"] = [_randn(g, (B, H, Lk, c["D"]), dtype, 0.5).requires_grad_(c["backward"]) for _ in range(2)]
        s["do"] = _randn(g, (B, H, c["Lq"], c["D"]), dtype) if c["backward"] else None
        s["is_mem"] = (torch.arange(Lk, device="cuda") % c["block"] == c["block"] - 1) if c["mask"] else None
    elif c["kind"] == "layer":
        # q, k and v are views of one projection, the gradient a view of the output projection's input gradient
        T, D = c["T"], c["D"]
        qkv = _randn(g, (B, T, 3, H, D), dtype)
        s["q"], s["k"], s["v"] = [qkv[:, :, i].transpose(1, 2).detach().requires_grad_(True) for i in range(3)]
        s["dy"] = _randn(g, (B, T, H, D), dtype).transpose(1, 2)
        s["cos"], s["sin"] = P.rotary_tables_interleaved(T, D, dtype, "cuda")
        offset = torch.randint(0, c["block"], (B, 1), generator=g, device="cuda")
        s["is_mem"] = (torch.arange(T, device="cuda").view(1, T) + offset) % c["block"] == c["block"] - 1
    elif c["kind"] == "softmax":
        Lq, Lk = c["Lq"], c["Lk"]
        x = _randn(g, (B, H, Lq, Lk), dtype)
        row = (torch.arange(Lk, device="cuda") % c["block"] == c["block"] - 1).view(1, Lk).expand(B, Lk)
        hidden = torch.ones(Lq, Lk, dtype=torch.bool, device="cuda").triu(1)
        s["hidden"], s["is_mem"], s["last"] = P.prepare_landmark_masks(row, hidden)
        fill = float("-inf") if c["flavour"] == "lm" else torch.finfo(dtype).min
        s["x"] = x.masked_fill_(s["hidden"], fill).requires_grad_(True)
        s["dp"] = _randn(g, (B, H, Lq, Lk), torch.float32)
        s["groups"] = Lk // c["block"] + 3
    elif c["kind"] in ("chunk", "decode"):
        T, D = c["T"], c["D"]
        C = c["n_blocks"] * c["block"] + c.get("tail", 0)
        s["cache"] = P.LandmarkKVCache(B, H, C + T, D, dtype, "cuda")
        s["cache"].append(_randn(g, (B, H, C, D), dtype), _randn(g, (B, H, C, D), dtype))
        s["length"] = C
        s["q"], s["k"], s["v"] = [_randn(g, (B, H, T, D), dtype) for _ in range(3)]
        s["cos"], s["sin"] = P.rotary_tables_half(C + T + 1, D, dtype, "cuda")
    elif c["kind"] == "eval":
        T, D, blk = c["chunk_blocks"] * c["block"], c["D"], c["block"]
        config = types.SimpleNamespace(batch_size=B, mem_cache_size=c["capacity"], mem_cache_freq=blk - 1, n_head=H,
                                       n_embd=H * D, cache_topk=c["top_k"], cache_selection_method=c["method"])
        s["storage"] = P.MemLMCacheStorage(config, dtype=dtype, device="cuda")
        s["is_mem"] = (torch.arange(T, device="cuda") % blk == blk - 1).view(1, T).expand(B, T).contiguous()
        for n in [c["chunk_blocks"]] * (c["capacity"] // c["chunk_blocks"] + 2):      # the ring is full and has wrapped
            k, v = [_randn(g, (B, H, n * blk, D), dtype) for _ in range(2)]
            s["storage"].store_in_cache(k, {"v": v, "is_mem": s["is_mem"]})
        s["start"] = (c["top_k"] + 1) * blk
        s["q"], s["k"], s["v"] = [_randn(g, (B, H, T, D), dtype) for _ in range(3)]
        cos, sin = P.rotary_tables_interleaved(s["start"] + T, D, dtype, "cuda")
        s["q"], s["k_rot"] = P.rotary_apply(s["q"], s["k"], cos, sin, s["start"])
        s["groups"] = c["top_k"] + c["chunk_blocks"] + 2
    else:
        T, D, blk = c["T"], c["D"], c["block"]
        C = c["n_blocks"] * blk
        s["cache"] = P.OffloadedLandmarkCache(B, H, c["n_blocks"] + T // blk, blk, D, dtype, "cuda")
        s["cache"].append(_randn(g, (B, H, C, D), dtype), _randn(g, (B, H, C, D), dtype))
        s["q"], s["k"], s["v"] = [_randn(g, (B, H, T, D), dtype) for _ in range(3)]
        s["cos"], s["sin"] = P.rotary_tables_half(C + T + 1, D, dtype, "cuda")
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "fused":
        o = P.fused_landmark_attention(s["q"], s["k"], s["v"], s["is_mem"], block_size=c["block"])
        if not c["backward"]:
            return o
        return (o, *torch.autograd.grad(o, [s["q"], s["k"], s["v"]], s["do"]))
    if c["kind"] == "layer":
        q, k = P.rotary_apply(s["q"], s["k"], s["cos"], s["sin"])
        y = P.lm_landmark_attention(q, k, s["v"], s["is_mem"], max_groups=c["groups"])
        return (y, *torch.autograd.grad(y, [s["q"], s["k"], s["v"]], s["dy"]))
    if c["kind"] == "softmax":
        if c["flavour"] == "lm":
            p, _ = P.landmark_grouped_softmax_lm(s["x"], -1, s["is_mem"], s["hidden"], s["last"], False, s["groups"])
        else:
            p = P.landmark_grouped_softmax(s["x"], -1, s["is_mem"], s["last"])
        return (p, *torch.autograd.grad(p, [s["x"]], s["dp"]))
    if c["kind"] in ("chunk", "decode"):
        s["cache"].length = s["length"]                 # the chunk is attended to and stored again behind the same cache
        out, (k, v) = P.llama_retrieval_attention(
            s["q"], s["k"], s["v"], mem_freq=c["block"] - 1, cache_top_k=c["top_k"], cache=s["cache"], cos=s["cos"],
            sin=s["sin"], aggregate="max_over_tokens" if c.get("per_head") else None)
        return out, k, v
    if c["kind"] == "eval":
        prefix, values = s["storage"].retrieve_for_query(s["q"], None, None, s["start"])
        y = P.lm_landmark_attention(s["q"], s["k_rot"], s["v"], s["is_mem"], max_groups=s["groups"], att_prefix=prefix,
                                    cache_values=values)
        s["storage"].store_in_cache(s["k"], {"v": s["v"], "is_mem": s["is_mem"]})
        return y, s["storage"].cache_mem_k, s["storage"].cache_mem_v
    cache = s["cache"]
    cache.n_blocks, cache.tail_len = c["n_blocks"], 0   # the chunk is attended to and stored again behind the same blocks
    out = cache.attend(s["q"], s["k"], s["v"], c["top_k"], s["cos"], s["sin"])
    return out, cache.lm_keys, cache.k_host, cache.v_host


def _attention_flops(c):
    # forward, causal: matmuls only.  Forward + backward is 3.5 times that
    return 2 * c["B"] * c["H"] * c["Lq"] * (c["Lq"] + 2 * c["history"]) * c["D"]


def _touched(picks, n):
    """Blocks of n that `picks` independent draws touch at least once."""
    return n * (1.0 - (1.0 - 1.0 / n) ** picks)


def work(case):
    c, e = case, SIZES[case["dtype"]]
    B, H, D = c["B"], c["H"], c.get("D", 0)
    if c["kind"] == "fused":
        nq, nk, f = B * H * c["Lq"] * D, B * H * (c["Lq"] + c["history"]) * D, _attention_flops(c)
        if not c["backward"]:
            return {"bytes": e * (2 * nq + 2 * nk), "flops": f}
        return {"bytes": e * (4 * nq + 4 * nk), "flops": 3.5 * f}      # q, k, v, dO in; o, dQ, dK, dV out
    if c["kind"] == "layer":
        n = B * H * c["T"] * D
        return {"bytes": 8 * e * n, "flops": 7 * n * c["T"]}
    if c["kind"] == "softmax":
        n = B * H * c["Lq"] * c["Lk"]                                  # x, dP in; P, dx out (gradients in x's type)
        return {"bytes": n * (e + 4 + 4 + e), "flops": 10 * n}
    if c["kind"] in ("chunk", "decode"):
        # q, k, v in, out, k and v stored; every landmark key; every block that some (head, token) selects, once
        T, rows = c["T"], c["block"]
        sel = min(c["top_k"], c["n_blocks"])
        picks = sel if c.get("per_head") else T * sel
        blocks = B * H * _touched(picks, c["n_blocks"])
        tail = c.get("tail", 0)
        byts = e * D * (B * H * (6 * T + c["n_blocks"] + 2 * tail) + 2 * rows * blocks)
        flops = 2 * B * H * T * D * (c["n_blocks"] + 2 * sel * rows + 2 * tail + T)
        return {"bytes": byts, "flops": flops}
    if c["kind"] == "eval":
        T, rows = c["chunk_blocks"] * c["block"], c["block"]
        picks = {"per_token_and_head": T, "max_over_heads": T, "max_over_tokens": 1}[c["method"]] * c["top_k"]
        blocks = B * H * _touched(picks, c["capacity"])
        # q, rotated k, k, v in, y out, k and v stored; landmark keys; every selected block of keys and values once
        byts = e * D * (B * H * (7 * T + c["capacity"]) + 2 * rows * blocks)
        flops = 2 * B * H * T * D * (c["capacity"] + 2 * c["top_k"] * rows + T)
        return {"bytes": byts, "flops": flops}
    T, rows = c["T"], c["block"]
    keys = c["top_k"] * rows
    byts = e * D * B * H * (6 * T + c["n_blocks"] + T // rows + 2 * keys)
    return {"bytes": byts, "flops": 2 * B * H * T * D * (c["n_blocks"] + 2 * keys + T)}


def tolerance(case):
    # f32: sums of some thousand products in another order.  16-bit: probabilities and their gradients are rounded to the
    # data type between the products (relative steps of 2^-9 and 2^-12) and so are the results.
    if case["kind"] == "softmax":
        return {"rel": 1e-5} if case["dtype"] == "f32" else {"rel": 3e-3}
    return {"rel": {"f32": 1e-5, "f16": 4e-3, "bf16": 1e-2}[case["dtype"]]}
