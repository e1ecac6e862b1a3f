"""Performance cases of the MLA path: what a serving or a training program has this framework do.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)` one more of the same ranges,
`prepare` the tensors and workspaces a program holds before the call, `run` one pass through `dscuda_b200.mla`,
`work` the bytes and operations the pass cannot do without, `tolerance` how far two correct implementations of
the same precision may differ.

Operations:

    decode         one paged decode call of a serving step (query already packed, cache already filled)
    decode_step    everything the framework does for one layer of a decode step: rotary embedding of the new token,
                   W_UK absorbed into the query, the new row appended to the cache, decode, W_UV on the result
    decode_fp8     the step of a server that stores its cache in FP8: append, dequantise the pool, decode
    prefill_step   one layer of a prefill: rotary embedding, up-projection of the latent, cache append, causal forward
    train          forward and backward of the non-absorbed causal attention, dense batch
    train_packed   the same for ragged sequences packed behind cu_seqlens
    absorbed       forward and backward of the causal attention in the latent space
    flash          causal grouped-query forward at head dimension 128

Lengths of ragged cases belong to the case (`layout` seeds them); all values come from the seed given to `prepare`.
"""
import math
import random

import torch

from dscuda_b200 import mla

SCALE = 192 ** -0.5
FORWARD_FLOPS = 2 * (192 + 128)                             # per causal (query, key) pair and head
BACKWARD_FLOPS = 2 * (192 + 128 + 128 + 192 + 192)
ABSORBED_FORWARD_FLOPS = 2 * (576 + 512)
ABSORBED_BACKWARD_FLOPS = 2 * (576 + 512 + 512 + 576 + 576)


def listed():
    return [
        # a chat server with two users: one short step, where launches and host time are all there is
        {"name": "decode_two_short", "op": "decode", "batch": 2, "heads": 16, "low": 1024, "high": 1024, "page": 64, "layout": 1, "checked": False},
        # a server with a handful of uneven conversations
        {"name": "decode_eight_ragged", "op": "decode", "batch": 8, "heads": 128, "low": 511, "high": 8192, "page": 64, "layout": 2, "checked": False},
        # a loaded server: the decode configuration of the benchmark suite
        {"name": "decode_loaded", "op": "decode", "batch": 64, "heads": 128, "low": 1024, "high": 32768, "page": 64, "layout": 3, "checked": False},
        # the whole layer step around a decode of moderate load
        {"name": "decode_step", "op": "decode_step", "batch": 32, "heads": 128, "low": 256, "high": 4096, "page": 64, "layout": 4, "checked": False},
        # the same for a server that stores its cache in FP8 and appends a block of tokens per sequence
        {"name": "decode_fp8", "op": "decode_fp8", "batch": 16, "heads": 128, "low": 1000, "high": 6000, "page": 64, "layout": 5, "tokens": 64},
        # the prefill configuration of the benchmark suite with the steps around it
        {"name": "prefill_step", "op": "prefill_step", "batch": 4, "seq": 4096, "heads": 128, "page": 64},
        # a short prompt
        {"name": "prefill_prompt", "op": "prefill_step", "batch": 1, "seq": 777, "heads": 16, "page": 64},
        # the suite's small training shape
        {"name": "train_small", "op": "train", "batch": 1, "seq": 256, "heads": 16},
        # the headline training step
        {"name": "train_long", "op": "train", "batch": 2, "seq": 8192, "heads": 128},
        # packed long-context training, one GPU's 16 heads
        {"name": "train_packed", "op": "train_packed", "sequences": 16, "low": 512, "high": 32768, "heads": 16, "layout": 4},
        # attention in the latent space, forward and backward
        {"name": "absorbed_train", "op": "absorbed", "batch": 4, "seq": 2048, "heads": 16},
        # grouped-query attention
        {"name": "flash_gqa", "op": "flash", "batch": 4, "seq": 4096, "heads": 64, "kv_heads": 8},
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    op = rng.choice(("decode", "decode", "decode_step", "decode_fp8", "prefill_step", "train", "train", "train_packed", "absorbed", "absorbed", "flash"))
    while True:
        case = {"op": op}
        if op in ("decode", "decode_step", "decode_fp8"):
            high = _log_uniform(rng, 64, 32768 if op == "decode" else 8192)
            case.update(batch=_log_uniform(rng, 1, 64), heads=rng.choice((16, 32, 64, 128, 128, rng.randint(1, 128))), low=max(1, _log_uniform(rng, max(1, high // 32), high)),
                        high=high, page=rng.choice((64, 64, 128)), layout=rng.randint(1, 1 << 20))
            if op == "decode_fp8":
                case["tokens"] = min(case["low"], _log_uniform(rng, 1, 256))
            else:
                case["checked"] = rng.random() < 0.25
        elif op == "train_packed":
            high = _log_uniform(rng, 128, 32768)
            case.update(sequences=rng.randint(2, 16), low=max(1, high // rng.choice((4, 16, 64))), high=high, heads=rng.choice((2, 8, 16, 16, 32)), layout=rng.randint(1, 1 << 20))
        elif op == "flash":
            heads, kv_heads = rng.choice(((2, 2), (8, 1), (16, 16), (32, 8), (64, 8)))
            case.update(batch=_log_uniform(rng, 1, 8), seq=_log_uniform(rng, 17, 8192), heads=heads, kv_heads=kv_heads)
        elif op == "absorbed":
            case.update(batch=rng.randint(1, 4), seq=_log_uniform(rng, 17, 4096), heads=rng.choice((4, 8, 16, 32, rng.randint(1, 32))))
        elif op == "prefill_step":
            case.update(batch=rng.randint(1, 4), seq=_log_uniform(rng, 33, 8192), heads=rng.choice((8, 16, 64, 128)), page=rng.choice((64, 64, 128)))
        else:
            case.update(batch=rng.randint(1, 4), seq=_log_uniform(rng, 33, 8192), heads=rng.choice((3, 8, 16, 32, 64, 128)))
        # nothing dearer than the dearest listed case of its kind
        w = work(case)
        if w["flops"] <= {"train": 1.98e13, "train_packed": 2.83e13, "prefill_step": 3.3e12}.get(op, 1.11e12) and w["bytes"] <= 5e9:
            return case


def _lengths(case):
    """Tokens of each sequence of a ragged case."""
    rng = random.Random(case["layout"])
    if case["op"] == "train_packed":
        return [_log_uniform(rng, case["low"], case["high"]) for _ in range(case["sequences"])]
    return [rng.randint(case["low"], case["high"]) for _ in range(case["batch"])]


def _normal(generator):
    def values(*shape, std=1.0):
        return torch.randn(*shape, device="cuda", generator=generator, dtype=torch.float32).mul_(std).bfloat16()
    return values


def _page_table(lengths, page, generator):
    """Block table cut from one random permutation of all pages, and the number of pages."""
    need = [-(-n // page) for n in lengths]
    order = torch.randperm(sum(need), generator=generator, device="cuda").to(torch.int32)
    table = torch.zeros(len(lengths), max(need), dtype=torch.int32, device="cuda")
    start = 0
    for b, n in enumerate(need):
        table[b, :n] = order[start:start + n]
        start += n
    return table, sum(need)


def _int32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    values = _normal(g)
    op, s = case["op"], {"op": case["op"]}
    if op in ("decode", "decode_step", "decode_fp8"):
        batch, heads, page, lengths = case["batch"], case["heads"], case["page"], _lengths(case)
        table, pages = _page_table(lengths, page, g)
        splits = mla.decode_splits(lengths, heads)
        s.update(table=table, lengths=_int32(lengths), splits=splits, workspace=mla.decode_workspace(batch, heads, splits), checked=case.get("checked", False))
        cache = torch.empty(pages, page, 1, 576, device="cuda", dtype=torch.bfloat16)
        if op != "decode_fp8":
            for start in range(0, pages, 4096):             # in pieces: the float32 draws of a whole pool would be large
                cache[start:start + 4096] = values(min(4096, pages - start), page, 1, 576)
        s["cache"] = cache
        if op == "decode_step":
            s.update(q_nope=values(batch, 1, heads, 128), q_pe=values(batch, 1, heads, 64), latent=values(batch, 1, 512), k_pe=values(batch, 1, 1, 64),
                     w_uk=values(heads * 128, 512, std=512 ** -0.5), w_uv=values(heads * 128, 512, std=512 ** -0.5),
                     start=_int32([n - 1 for n in lengths]))
        else:
            s["query"] = values(batch, 1, heads, 576)
        if op == "decode_fp8":
            tokens = case["tokens"]
            longest = max(lengths)
            s["fp8"] = torch.zeros(pages, page, mla.FP8_CACHE_ROW_BYTES, device="cuda", dtype=torch.uint8)
            for start in range(0, longest, 2048):           # what earlier steps appended
                count = min(2048, longest - start)
                mla.cache_append_fp8(s["fp8"], values(batch, count, 512), values(batch, count, 64), table, _int32([start] * batch),
                                     _int32([max(0, min(count, n - start)) for n in lengths]))
            s.update(latent=values(batch, tokens, 512), k_pe=values(batch, tokens, 64), start=_int32([n - tokens for n in lengths]))
    elif op == "prefill_step":
        batch, seq, heads, page = case["batch"], case["seq"], case["heads"], case["page"]
        table, pages = _page_table([seq] * batch, page, g)
        s.update(heads=heads, q_nope=values(batch, seq, heads, 128), q_pe=values(batch, seq, heads, 64), latent=values(batch, seq, 512), k_pe=values(batch, seq, 1, 64),
                 w_uk=values(heads * 128, 512, std=512 ** -0.5), w_uv=values(heads * 128, 512, std=512 ** -0.5), table=table,
                 cache=torch.zeros(pages, page, 1, 576, device="cuda", dtype=torch.bfloat16))
    elif op in ("train", "train_packed"):
        heads = case["heads"]
        if op == "train":
            lead, sequences, longest, total = (case["batch"], case["seq"]), case["batch"], case["seq"], case["batch"] * case["seq"]
            s.update(cu=None, longest=None)
        else:
            lengths = _lengths(case)
            lead, sequences, longest, total = (sum(lengths),), len(lengths), max(lengths), sum(lengths)
            s.update(cu=_int32([sum(lengths[:i]) for i in range(len(lengths) + 1)]), longest=longest)
        s.update(inputs=(values(*lead, heads, 128), values(*lead, heads, 64), values(*lead, heads, 128), values(*lead, 1, 64), values(*lead, heads, 128)),
                 dout=values(*lead, heads, 128, std=0.1), workspace=mla.prefill_backward_workspace(sequences, longest, total, heads))
    elif op == "absorbed":
        batch, seq, heads = case["batch"], case["seq"], case["heads"]
        s.update(inputs=(values(batch, seq, heads, 512), values(batch, seq, heads, 64), values(batch, seq, 512), values(batch, seq, 64)),
                 dout=values(batch, seq, heads, 512, std=0.1))
    else:
        batch, seq = case["batch"], case["seq"]
        s["inputs"] = (values(batch, seq, case["heads"], 128), values(batch, seq, case["kv_heads"], 128), values(batch, seq, case["kv_heads"], 128))
    return s


def run(s):
    op = s["op"]
    if op == "decode":
        return mla.mla_decode(s["query"], s["cache"], s["table"], s["lengths"], SCALE, s["splits"], s["workspace"], checked_pages=s["checked"])
    if op == "decode_step":
        batch = s["latent"].shape[0]
        mla.rope_apply(s["q_pe"], s["k_pe"], s["start"])
        query = torch.cat((mla.absorb_query(s["q_nope"], s["w_uk"]), s["q_pe"]), dim=-1)
        mla.cache_append(s["cache"], s["latent"], s["k_pe"].view(batch, 1, 64), s["table"], s["start"])
        out, lse = mla.mla_decode(query, s["cache"], s["table"], s["lengths"], SCALE, s["splits"], s["workspace"], checked_pages=s["checked"])
        return mla.unabsorb_output(out, s["w_uv"]), lse, s["cache"]
    if op == "decode_fp8":
        mla.cache_append_fp8(s["fp8"], s["latent"], s["k_pe"], s["table"], s["start"])
        mla.cache_dequantize_fp8(s["fp8"], s["cache"])
        return *mla.mla_decode(s["query"], s["cache"], s["table"], s["lengths"], SCALE, s["splits"], s["workspace"]), s["fp8"], s["cache"]
    if op == "prefill_step":
        batch, seq, _ = s["latent"].shape
        mla.rope_apply(s["q_pe"], s["k_pe"])
        k_nope, v = mla.up_project(s["latent"], s["w_uk"], s["w_uv"], s["heads"])
        mla.cache_append(s["cache"], s["latent"], s["k_pe"].view(batch, seq, 64), s["table"])
        out, lse = mla.prefill_forward(s["q_nope"], s["q_pe"], k_nope, s["k_pe"], v, SCALE)
        return out, lse, k_nope, v, s["cache"]
    if op in ("train", "train_packed"):
        out, lse = mla.prefill_forward(*s["inputs"], SCALE, s["cu"], s["longest"])
        return out, lse, *mla.prefill_backward(s["dout"], out, lse, *s["inputs"], SCALE, s["cu"], s["longest"], workspace=s["workspace"])
    if op == "absorbed":
        out, lse = mla.mla_forward(*s["inputs"], SCALE)
        return out, lse, *mla.mla_backward(s["dout"], out, lse, *s["inputs"], SCALE)
    return mla.flash_forward(*s["inputs"], 128 ** -0.5)


def _pairs(lengths):
    return sum(n * (n + 1) // 2 for n in lengths)


def work(case):
    op, heads = case["op"], case["heads"]
    if op in ("decode", "decode_step", "decode_fp8"):
        lengths, page = _lengths(case), case["page"]
        batch, tokens = len(lengths), sum(lengths)
        tables = 4 * (batch + sum(-(-n // page) for n in lengths))
        flops = ABSORBED_FORWARD_FLOPS * heads * tokens
        if op == "decode":                                  # cache rows, Q in, O and LSE out
            return {"bytes": tokens * 1152 + batch * heads * (1152 + 1024 + 4) + tables, "flops": flops}
        if op == "decode_step":                             # cache rows, both weights, the new token's tensors in (rotated ones out too), result out
            return {"bytes": tokens * 1152 + heads * 2 * 131072 + batch * heads * (256 + 256 + 256 + 4) + batch * (1024 + 256 + 1152) + tables,
                    "flops": flops + 4 * 128 * 512 * batch * heads}
        new, pool = batch * case["tokens"], sum(-(-n // page) * page for n in lengths)
        return {"bytes": new * (1152 + 656) + pool * (656 + 1152) + batch * heads * (1152 + 1024 + 4) + tables, "flops": flops}
    if op == "prefill_step":                                # activations in, weights in, K, V, O and LSE out, cache rows out, rotary tensors in and out
        rows = case["batch"] * case["seq"]
        return {"bytes": rows * heads * (256 + 2 * 128 + 3 * 256 + 4) + rows * (1024 + 256 + 1152) + heads * 2 * 131072,
                "flops": _pairs([case["seq"]]) * case["batch"] * heads * FORWARD_FLOPS + 4 * rows * heads * 128 * 512}
    if op in ("train", "train_packed"):                     # q, k, v, dO in (832 columns a head), O and the gradients out (576), rotary key and its gradient, LSE
        lengths = [case["seq"]] * case["batch"] if op == "train" else _lengths(case)
        rows = sum(lengths)
        return {"bytes": rows * heads * (2 * (576 + 576) + 4) + rows * 256, "flops": _pairs(lengths) * heads * (FORWARD_FLOPS + BACKWARD_FLOPS)}
    rows = case["batch"] * case["seq"]
    pairs = _pairs([case["seq"]]) * case["batch"] * heads
    if op == "absorbed":                                    # query, dO in, O and dquery out, LSE; latent and its gradient
        return {"bytes": rows * heads * (2 * (576 + 512 + 512 + 576) + 4) + rows * 2 * 1152, "flops": pairs * (ABSORBED_FORWARD_FLOPS + ABSORBED_BACKWARD_FLOPS)}
    return {"bytes": rows * (heads * (256 + 256 + 4) + case["kv_heads"] * 512), "flops": pairs * 4 * 128}


def tolerance(case):
    # bf16 tensors with fp32 accumulation: probabilities, their gradients and the results are rounded to eight bits.  FP8 codes and copied
    # cache rows are whole values or equal bits and fall under the same bound.
    return {"rel": 1e-2}
