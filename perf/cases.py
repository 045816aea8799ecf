"""Workloads by which the speed of this framework is measured, and their inputs.

Each case goes through the public entry points as a user's program does: the prefill attention
functions that the model classes call (alone, and with their backward), one layer's share of a
decode step on the caches of a running batch, and the generation engine.  Sizes are those of the
benchmark configurations (``sps_b200.workloads``) and of the tests, from calls that launch
latency dominates to calls that fill the machine for milliseconds; ``draw`` gives further sizes
of the same ranges.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import sps_b200
from sps_b200.generation import random_state_dict
from sps_b200.workloads import (DECODE_CONFIGS, GENERATION_CONFIGS, PREFILL_CONFIGS, geometric_docs,
                                generation_forbidden_ids, generation_step_bytes, run_lengths)

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_WHOLE = 1 << 20        # a window this long hides nothing at the sizes used here


def _attention_case(name, kind, variant, batch, heads, tokens, head_dim, *, window=64, persistent=-1, docs=0,
                    dtype="bf16", layout="token"):
    """``tokens`` per row before doubling; ``docs``: mean document length, 0 = one document per row
    and no document ids; ``persistent`` < 0: no persistent-key window; ``layout`` "token": views of
    [B, N, H, D] buffers as the model classes pass them, "head": contiguous [B, H, N, D]."""
    return dict(name=name, kind=kind, variant=variant, batch=batch, heads=heads, tokens=tokens, head_dim=head_dim,
                window=window, persistent=persistent, docs=docs, dtype=dtype, layout=layout)


def _decode_case(name, queries, seqs, heads, head_dim, ring, len_lo, len_hi, *, per_head=False, dtype="bf16"):
    return dict(name=name, kind="decode", queries=queries, seqs=seqs, heads=heads, head_dim=head_dim, ring=ring,
                len_lo=len_lo, len_hi=len_hi, per_head=per_head, dtype=dtype)


def _engine_case(name, kind, variant, layers, heads, hidden, intermediate, vocab, batch, prompt, new_tokens, *,
                 window=64, ragged=False, dtype="bf16"):
    """``ragged``: prompts of different lengths, left padded."""
    return dict(name=name, kind=kind, variant=variant, layers=layers, heads=heads, hidden=hidden,
                intermediate=intermediate, vocab=vocab, batch=batch, prompt=prompt, new_tokens=new_tokens,
                window=window, ragged=ragged, dtype=dtype)


def listed():
    b0, h0, t0, d0, w0, m0 = PREFILL_CONFIGS["cfg0_cpu_shape"]
    b1, h1, t1, d1, w1, m1 = PREFILL_CONFIGS["cfg1_s_scale"]
    b4, h4, t4, d4, w4, _ = PREFILL_CONFIGS["cfg4_full_window"]
    s2, h2, d2, r2, lo2, hi2 = DECODE_CONFIGS["cfg2_segmented_decode"]
    g3 = GENERATION_CONFIGS["cfg3_xl_generation"]
    return [
        # a short prompt batch or one small packed batch: the call is mostly latency
        _attention_case("prefill_small", "prefill", "sps", b0, h0, t0, d0, window=w0, docs=m0, layout="head"),
        # one layer's attention of an s-scale batch of packed documents
        _attention_case("prefill_packed", "prefill", "sps", b1, h1, t1, d1, window=w1, docs=m1, layout="head"),
        # full-window attention of wide heads over long single documents: the largest attention call
        _attention_case("prefill_full_window", "prefill", "sps", b4, h4, t4, d4, window=w4, layout="head"),
        # the Standard model's causal attention: odd length, odd batch, fp16, packed documents
        _attention_case("prefill_standard_ragged", "prefill", "standard", 3, 12, 3001, 64, docs=500, dtype="fp16"),
        # small models with narrow heads (the test models' width), Reverse-SPS
        _attention_case("prefill_narrow_heads", "prefill", "reverse_sps", 4, 8, 600, 32, docs=200),
        # training: forward and backward of one s-scale layer on packed documents
        _attention_case("train_packed", "train", "sps", 4, 12, 2048, 64, docs=1000),
        # training of a wide-headed Reverse-SPS layer, ragged length, single documents
        _attention_case("train_wide_ragged", "train", "reverse_sps", 2, 16, 1333, 128),
        # the Standard model decoding for a few users: one query, one layer, latency-bound
        _decode_case("decode_few", 1, 4, 16, 128, 0, 300, 900, per_head=True),
        # one layer of an SPS decode step of a large batch: attention and the cache update
        _decode_case("decode_batch", 2, s2, h2, d2, r2, lo2, hi2),
        # a program that samples by itself: prompt prefill, then single steps that hand out logits
        _engine_case("stepwise_s_scale", "stepwise", "sps", 12, 12, 768, 2048, 50304, 4, 128, 16, ragged=True),
        # greedy generation with a small model for a few prompts: launches and host count
        _engine_case("generate_small", "generate", "reverse_sps", 12, 12, 768, 2048, 50304, 2, 100, 48),
        # greedy generation at the width of the generation benchmark
        _engine_case("generate_xl", "generate", "reverse_sps", g3["n_layer"], g3["n_head"], g3["hidden_size"],
                     g3["intermediate_size"], g3["vocab_size"], g3["batch"], g3["prompt"], g3["new_tokens"],
                     window=g3["window_size"]),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["prefill"] * 4 + ["train"] * 2 + ["decode"] * 3 + ["stepwise"] + ["generate"] * 2)
    if kind in ("prefill", "train"):
        # heads of 64 and 128 as the models have them; the others now and then, forward only
        dims = [64] * 8 + [128] * 6 + ([16, 32, 256] if kind == "prefill" else [])
        d = rng.choice(dims)
        heads = rng.choice([3, 8, 12, 16])
        tokens = _log(rng, 64, 4096) if d in (64, 128) else _log(rng, 32, 1024)
        # rows x heads x width of the largest call: 4 x 16 x 8192 x 128; half of it with backward
        most = 4 * 16 * 8192 * 128 // (2 if kind == "train" else 1)
        batch = min(_log(rng, 1, 16), max(1, most // (heads * 2 * tokens * d)))
        variant = rng.choice(["sps", "sps", "reverse_sps", "standard"])
        case = _attention_case("", kind, variant, batch, heads, tokens, d, window=rng.choice([64, 64, 64, 16, 256, tokens]),
                               persistent=rng.choice([-1, -1, -1, -1, 128]) if variant != "standard" else -1,
                               docs=rng.choice([0, _log(rng, 50, 1000)]), dtype=rng.choice(["bf16", "bf16", "bf16", "fp16"]),
                               layout=rng.choice(["token", "token", "head"]))
    elif kind == "decode":
        queries = rng.choice([1, 2, 2])
        hi = _log(rng, 64, 4096)
        case = _decode_case("", queries, _log(rng, 1, 128), rng.choice([8, 12, 16]), rng.choice([64, 64, 128]),
                            64 if queries == 2 else 0, max(1, hi // 8), hi, per_head=rng.choice([False, True]),
                            dtype=rng.choice(["bf16", "bf16", "bf16", "fp16"]))
    else:
        layers, heads, hidden, inter = rng.choice([(2, 4, 512, 1024), (12, 12, 768, 2048), (24, 16, 1024, 2816),
                                                   (24, 16, 2048, 8192)])
        if kind == "generate":
            variant = rng.choice(["reverse_sps", "reverse_sps", "standard"])
            dtype, new = "bf16", _log(rng, 8, 128)
        else:
            variant = rng.choice(["sps", "reverse_sps", "delayed_state", "standard"])
            dtype, new = rng.choice(["bf16", "bf16", "bf16", "fp32"]), rng.randint(4, 24)
        case = _engine_case("", kind, variant, layers, heads, hidden, inter, rng.choice([2048, 50304]), _log(rng, 1, 32),
                            _log(rng, 16, 512), new, window=rng.choice([16, 64]), ragged=rng.choice([False, True]),
                            dtype=dtype)
    del case["name"]
    return case


# ---------------------------------------------------------------------------------------------
# attention, forward and backward

def _rows(case):
    return case["tokens"] * (1 if case["variant"] == "standard" else 2)


def _doc_ids(case, seed):
    """[B, rows] document ids: geometric document lengths, every document's rows together."""
    ids = geometric_docs(case["batch"], case["tokens"], case["docs"], seed)      # one id per doubled row
    return ids[:, ::2] if case["variant"] == "standard" else ids


def _prepare_attention(case, seed):
    b, h, n, d = case["batch"], case["heads"], _rows(case), case["head_dim"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    train = case["kind"] == "train"

    def tensor(grad):
        shape = (b, n, h, d) if case["layout"] == "token" else (b, h, n, d)
        x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).to(_DTYPES[case["dtype"]])
        x = x.transpose(1, 2) if case["layout"] == "token" else x
        return x.requires_grad_(grad)

    state = {"case": case, "q": tensor(train), "k": tensor(train), "v": tensor(train),
             "docs": torch.from_numpy(np.ascontiguousarray(_doc_ids(case, seed))).cuda() if case["docs"] else None}
    if train:
        state["d_o"] = tensor(False)
    return state


def _attend(s):
    case, scale = s["case"], 1.0 / math.sqrt(s["case"]["head_dim"])
    if case["variant"] == "standard":
        return sps_b200.full_attention(s["q"], s["k"], s["v"], scale, documents_idx_BxT=s["docs"])
    fn = sps_b200.sps_sliding_attention if case["variant"] == "sps" else sps_b200.reverse_sps_sliding_attention
    return fn(s["q"], s["k"], s["v"], scale, case["window"], documents_idx_BxT=s["docs"],
              persistent_key_window=None if case["persistent"] < 0 else case["persistent"])


def _run_attention(s):
    o = _attend(s)
    if s["case"]["kind"] == "prefill":
        return o
    dq, dk, dv = torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["d_o"])
    return {"o": o, "dq": dq, "dk": dk, "dv": dv}


def _visible_pairs(case):
    """Visible (query row, key row) pairs of one head, summed over the batch."""
    w = case["window"]
    p = case["persistent"] if case["persistent"] >= 0 else _WHOLE
    rows = _doc_ids(case, 0) if case["docs"] else np.zeros((case["batch"], _rows(case)), dtype=np.int64)
    total = 0
    for row in rows:
        for length in run_lengths(row):
            if case["variant"] == "standard":
                total += int(length) * (int(length) + 1) // 2
                continue
            t = np.arange(int(length) // 2, dtype=np.int64)
            w_in, w_ex = np.minimum(t, w) + 1, np.minimum(t, w)      # with and without the query's own token
            p_in, p_ex = np.minimum(t, p) + 1, np.minimum(t, p)
            # SPS: even keys persistent, odd ones windowed; Reverse-SPS the other way round.  The first
            # row of a token does not see its second row.
            per_token = 2 * p_in + w_ex + w_in if case["variant"] == "sps" else 2 * w_in + p_ex + p_in
            total += int(per_token.sum())
    return total


def _work_attention(case):
    size = case["batch"] * case["heads"] * _rows(case) * case["head_dim"]
    ids = case["batch"] * _rows(case) * 8 if case["docs"] else 0
    contraction = 2.0 * case["head_dim"] * case["heads"] * _visible_pairs(case)
    if case["kind"] == "prefill":
        return {"bytes": 4 * size * 2 + ids, "flops": 2 * contraction}
    # forward reads q, k, v and writes o; backward reads dO as well and writes three gradients
    return {"bytes": 8 * size * 2 + ids, "flops": 7 * contraction}


# ---------------------------------------------------------------------------------------------
# one layer of a decode step

def _prepare_decode(case, seed):
    s, h, d, ring, hi = case["seqs"], case["heads"], case["head_dim"], case["ring"], case["len_hi"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = _DTYPES[case["dtype"]]

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda", dtype=dt)

    # caches as a generation batch holds them: room for the step's token, live lengths on the device.
    # Per-head lengths of a sequence are equal, as every head retains every token.
    lens = np.random.default_rng(seed).integers(case["len_lo"], hi + 1, size=s).astype(np.int64)
    heads = np.repeat(lens[:, None], h, axis=1) if case["per_head"] or case["queries"] == 2 else lens[:, None]
    # counters: retained length of every head, ring length, ring position (the ring has wrapped)
    counters = torch.from_numpy(np.concatenate([heads.ravel(), np.full(s, ring), lens % max(ring, 1)])).cuda()
    n = heads.size
    state = {"case": case, "saved": counters.clone(), "counters": counters,
             "len": counters[:n].view(s, -1) if heads.shape[1] > 1 else counters[:n],
             "ring_len": counters[n:n + s], "ring_pos": counters[n + s:],
             "k": rnd(s, h, hi + 1, d), "v": rnd(s, h, hi + 1, d),
             "cur_k": rnd(s, h, d), "cur_v": rnd(s, h, d)}
    if case["queries"] == 1:
        state["q"] = rnd(s, h, d)
    else:
        state.update(q=rnd(s, 2, h, d), pred_k=rnd(s, h, d), pred_v=rnd(s, h, d), ring_k=rnd(s, h, ring, d),
                     ring_v=rnd(s, h, ring, d), active=torch.ones(s, dtype=torch.bool, device="cuda"))
    return state


def _run_decode(s):
    dt = _DTYPES[s["case"]["dtype"]]
    retained = sps_b200.KVSegment(s["k"], s["v"], s["len"])
    if s["case"]["queries"] == 1:
        return sps_b200.masked_kv_attention(s["q"], [retained], extra_kv=[(s["cur_k"], s["cur_v"])], attn_dtype=dt)
    s["counters"].copy_(s["saved"])          # the step starts from the same lengths each time
    ring = sps_b200.KVSegment(s["ring_k"], s["ring_v"], s["ring_len"])
    y = sps_b200.segmented_q2_attention(
        s["q"], [ring, retained], current_normal_k_BxHxD=s["cur_k"], current_normal_v_BxHxD=s["cur_v"],
        current_predict_k_BxHxD=s["pred_k"], current_predict_v_BxHxD=s["pred_v"], attn_dtype=dt)
    # the step's rows enter the caches; the ring's rows change, so outputs of a repeated pass differ
    # from the first one's only through the row that the pass before has put there
    sps_b200.fused_sps_kv_update(
        nw_k=s["ring_k"], nw_v=s["ring_v"], nw_len=s["ring_len"], nw_pos=s["ring_pos"], br_k=s["k"], br_v=s["v"],
        br_len=s["len"], k_window_BxHxD=s["pred_k"], v_window_BxHxD=s["pred_v"], k_retained_BxHxD=s["cur_k"],
        v_retained_BxHxD=s["cur_v"], active_mask_B=s["active"], window_tokens=s["case"]["ring"])
    return {"y": y, "ring_k": s["ring_k"], "ring_v": s["ring_v"], "k": s["k"], "v": s["v"], "counters": s["counters"]}


def _work_decode(case):
    s, h, d, nq = case["seqs"], case["heads"], case["head_dim"], case["queries"]
    rows = s * ((case["len_lo"] + case["len_hi"]) / 2.0 + case["ring"] + nq)       # K and V rows read
    row = h * d
    update = 4 * s * row * 2 if nq == 2 else 0                                     # rows written to the caches
    return {"bytes": rows * row * 2 * 2 + s * nq * row * (2 + 4) + update, "flops": 4.0 * nq * rows * row}


# ---------------------------------------------------------------------------------------------
# the generation engine

def _model(case):
    """The dict form that the helpers of ``workloads`` take: special ids at the end of the vocabulary."""
    v = case["vocab"]
    return dict(block_size=case["prompt"] + case["new_tokens"], vocab_size=v, n_layer=case["layers"],
                n_head=case["heads"], hidden_size=case["hidden"], intermediate_size=case["intermediate"],
                eos_token_id=v - 48, pad_token_id=v - 1, predict_token_id=v - 47, window_size=case["window"])


def _prepare_engine(case, seed):
    m = _model(case)
    dims = sps_b200.SPSDims(**m)
    dt = _DTYPES[case["dtype"]]
    sd = random_state_dict(dims, seed=seed, dtype=dt)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    if case["kind"] == "generate":
        # Greedy tokens are compared exactly, and an untrained head has near ties all over its
        # vocabulary.  As in a trained model the next token is a confident choice here: the residual
        # stream is led by the token's embedding, and the head maps it to one successor per token.
        wte = torch.randn((m["vocab_size"], m["hidden_size"]), generator=g, device="cuda").to(dt)
        successor = torch.randperm(m["eos_token_id"], generator=g, device="cuda")
        head = wte.clone()
        head[successor] = wte[:m["eos_token_id"]]
        sd["transformer.wte.weight"], sd["lm_head.weight"] = wte, head
        for layer in range(m["n_layer"]):
            sd[f"transformer.h.{layer}.mlp.down_proj.weight"].mul_(1.0 / math.sqrt(2 * m["n_layer"]))
    b, t = case["batch"], case["prompt"]
    prompt = torch.randint(0, m["eos_token_id"], (b, t), generator=g, device="cuda")
    if case["ragged"]:
        # lengths from half the prompt to all of it, the longest row full
        pads = np.random.default_rng(seed).integers(0, t // 2 + 1, size=b)
        pads[0] = 0
        column = torch.arange(t, device="cuda").unsqueeze(0)
        prompt = torch.where(column < torch.from_numpy(pads).cuda().unsqueeze(1), m["pad_token_id"], prompt)
    state = {"case": case, "prompt": prompt, "cache": None,
             "engine": sps_b200.SPSGenerator(sd, dims, variant=case["variant"], param_dtype=dt)}
    if case["kind"] == "generate":
        state["forbidden"] = torch.tensor(generation_forbidden_ids(m))
    else:
        state["tokens"] = torch.randint(0, m["eos_token_id"], (case["new_tokens"], b), generator=g, device="cuda")
        state["active"] = torch.ones(b, dtype=torch.bool, device="cuda")
    return state


def _run_engine(s):
    engine, new = s["engine"], s["case"]["new_tokens"]
    if s["case"]["kind"] == "generate":
        return engine.generate(s["prompt"], new, stop_on_eos=False, forbidden_token_ids=s["forbidden"])
    s["cache"], logits = engine.prefill(s["prompt"], new, state=s["cache"])
    out = [logits]
    for token in s["tokens"]:                # stands for the tokens that the program samples
        out.append(engine.decode_one_token(s["cache"], token, s["active"]))
    return out


def _work_engine(case):
    m = _model(case)
    c, i, layers, b, t = (case[k] for k in ("hidden", "intermediate", "layers", "batch", "prompt"))
    slots = 1 if case["variant"] == "standard" else 2
    real = t * (0.75 if case["ragged"] else 1.0)
    size = 2 if case["dtype"] == "bf16" else 4
    block = layers * (4 * c * c + 3 * c * i)
    params = (block + m["vocab_size"] * c) * size
    steps = case["new_tokens"] - (1 if case["kind"] == "generate" else 0)
    live = real + case["new_tokens"] / 2.0
    step_bytes = generation_step_bytes(m, b, live) + params - params * 2 // size       # parameters wider than bf16
    step_flops = b * (slots * 2.0 * block + 2.0 * m["vocab_size"] * c + layers * slots * 4.0 * live * c)
    prompt_flops = b * (slots * real * 2.0 * block + 2.0 * m["vocab_size"] * c
                        + layers * 2.0 * c * slots * slots * real * real / (slots if slots == 1 else 2))
    prompt_bytes = params + layers * b * real * c * 2 * 2
    return {"bytes": prompt_bytes + steps * step_bytes, "flops": prompt_flops + steps * step_flops}


# ---------------------------------------------------------------------------------------------

def prepare(case, seed):
    if case["kind"] in ("prefill", "train"):
        return _prepare_attention(case, seed)
    if case["kind"] == "decode":
        return _prepare_decode(case, seed)
    return _prepare_engine(case, seed)


def run(state):
    kind = state["case"]["kind"]
    if kind in ("prefill", "train"):
        return _run_attention(state)
    return _run_decode(state) if kind == "decode" else _run_engine(state)


def work(case):
    if case["kind"] in ("prefill", "train"):
        return _work_attention(case)
    return _work_decode(case) if case["kind"] == "decode" else _work_engine(case)


def tolerance(case):
    if case["kind"] == "generate":
        return "exact"                       # token ids
    if case["kind"] == "stepwise":
        # logits behind a stack of layers whose sums, normalised values and products are rounded to
        # bf16 one after another, or (fp32 parameters) whose attention operands are
        return {"rel": 2e-2}
    # operands, probabilities and results in 16 bits
    return {"rel": 1e-2}
