"""The work a user of this framework has it do, as cases that can be timed and compared.

Every case goes through the public entry points (``flax_attention``, ``flax_attention_pallas``,
``create_block_mask``, torch autograd for the gradients) on tensors that are already on the GPU.
A case is a dict of plain values:

kind      "decode"  short query block against a long key / value cache
          "prefill" forward only
          "train"   forward and the gradients of q, k and v
          "packed"  "train" over packed documents: the BlockMask is built in the pass, from this
                    batch's document ids, as a training loop has to
          "mask"    create_block_mask alone
entry     "flax" or "pallas": which attention entry point is called
layout    "bhsd", or "bshd" (``flax_attention_pallas(bhln=False)``)
score     None, "alibi" or "checkerboard"
mask      None, "causal", "offset" (causal, the query rows at the end of the keys), "window",
          "sink"; packed cases: causal inside a document
mask_bh   whether the tables are built for every batch entry and head or broadcast
"""
import math

import numpy as np
import torch

import flaxattention_b200 as fa
from flaxattention_b200.masks import (causal_mask, generate_attention_sink, generate_causal_offset,
                                      generate_sliding_window)
from flaxattention_b200.mods import checkerboard, generate_alibi_bias

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}


def _case(kind, B, Hq, Sq, D, dtype, Skv=None, Hkv=None, score=None, mask=None, window=0, mask_bh=True,
          entry="pallas", layout="bhsd", docs=0, name=None):
    c = {"kind": kind, "B": B, "Hq": Hq, "Hkv": Hq if Hkv is None else Hkv, "Sq": Sq,
         "Skv": Sq if Skv is None else Skv, "D": D, "dtype": dtype, "score": score, "mask": mask, "window": window,
         "mask_bh": mask_bh, "entry": entry, "layout": layout, "docs": docs}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one new token against a short cache, the decoding benchmark's default length: a few
        # microseconds of GPU work per layer, so the call itself counts
        _case("decode", 8, 8, 1, 64, "f16", Skv=2048, score="alibi", mask="offset", name="decode_short_cache"),
        # the same at serving size: batch 32, 16384 cached tokens, bound by reading the cache
        _case("decode", 32, 8, 1, 64, "f16", Skv=16384, score="alibi", mask="offset", name="decode_long_cache"),
        # a block of 16 new tokens (speculative decoding, chunked prefill) on the same cache
        _case("decode", 32, 8, 16, 64, "f16", Skv=16384, score="alibi", mask="offset", name="decode_16_rows"),
        # grouped-query decoding with wide heads and a cache of no round length, no mods
        _case("decode", 16, 32, 1, 128, "bf16", Skv=8191, Hkv=8, entry="flax", name="decode_grouped_d128"),
        # the CPU-sized configuration of the reference: fp32, causal + ALiBi, forward and gradients
        _case("train", 2, 4, 256, 64, "f32", score="alibi", mask="causal", entry="flax", name="train_small_f32"),
        # the fp32 row of the reference's benchmark: forward over a checkerboard score_mod
        _case("prefill", 8, 8, 2048, 64, "f32", score="checkerboard", name="forward_f32"),
        # the headline configuration: fp16, checkerboard, no mask, forward and backward
        _case("train", 8, 8, 2048, 64, "f16", score="checkerboard", name="train_checkerboard_f16"),
        # causal + ALiBi through a BlockMask, bf16, the default entry point
        _case("train", 8, 8, 2048, 64, "bf16", score="alibi", mask="causal", entry="flax", name="train_causal_alibi_bf16"),
        # long sequences, wide heads, sliding window with attention sinks: the largest job
        _case("train", 4, 16, 8192, 128, "bf16", mask="sink", window=1024, name="train_sink_d128_bf16"),
        # prompt of no round length, grouped-query heads, token-major [B, L, H, N] tensors, inference
        _case("prefill", 2, 16, 3001, 128, "bf16", Hkv=4, mask="causal", mask_bh=False, layout="bshd",
              name="prefill_grouped_ragged"),
        # packed documents: a mask over captured ids, rebuilt for every batch
        _case("packed", 4, 8, 4096, 64, "bf16", mask_bh=False, docs=12, name="train_packed_documents"),
        # the tables of the long-sequence job
        _case("mask", 4, 16, 8192, 0, "", mask="sink", window=1024, name="build_block_mask"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """A sequence length: two in five a multiple of 128, the others whatever comes."""
    n = _log(rng, lo, hi)
    return max(lo, n // 128 * 128) if rng.random() < 0.4 and n >= 128 else n


def _heads(rng):
    hkv, g = rng.choice([1, 2, 4, 8, 16]), rng.choice([1, 1, 2, 4])
    return (hkv * g, hkv) if hkv * g <= 32 else (hkv, hkv)


def _draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "train", "train", "train", "packed", "mask"])
    hq, hkv = _heads(rng)
    entry, half = rng.choice(["flax", "pallas"]), rng.choice(["f16", "bf16"])
    if kind == "decode":
        sq = 1 if rng.random() < 0.6 else _log(rng, 2, 64)
        return _case("decode", _log(rng, 1, 32), hq, sq, rng.choice([64, 64, 128]), half, Skv=_length(rng, 1024, 32768),
                     Hkv=hkv, score=rng.choice([None, "alibi"]), mask=rng.choice([None, "offset"]),
                     mask_bh=rng.random() < 0.5, entry=entry)
    if kind == "mask":
        s = _length(rng, 1024, 8192)
        return _case("mask", rng.choice([1, 2, 4]), rng.choice([1, 8, 16]), s, 0, "",
                     mask=rng.choice(["causal", "window", "sink"]), window=_log(rng, 64, s // 2))
    if kind == "packed":
        return _case("packed", rng.choice([1, 2, 4]), hq, _length(rng, 512, 8192), rng.choice([64, 128]), half, Hkv=hkv,
                     docs=_log(rng, 2, 32), mask_bh=False, entry=entry)
    f32 = rng.random() < 0.25
    s = _length(rng, 64, 2048) if f32 else _length(rng, 128, 8192)
    mask = rng.choice([None, "causal", "causal", "window", "sink"])
    return _case(kind, rng.choice([1, 2, 4, 8]), hq, s, 64 if f32 else rng.choice([64, 64, 128]), "f32" if f32 else half,
                 Hkv=hkv, score=rng.choice([None, "alibi", "checkerboard"]), mask=mask,
                 window=_log(rng, 64, 1024) if mask in ("window", "sink") else 0, mask_bh=rng.random() < 0.5, entry=entry,
                 layout="bshd" if entry == "pallas" and rng.random() < 0.3 else "bhsd")


def _cost(case):
    """A rough time in arbitrary units: fp32 runs on the FMA pipes, 16-bit types on the tensor cores."""
    w = work(case)
    return w["bytes"] / 6e12 + w["flops"] / (4e13 if case["dtype"] == "f32" else 7e14)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        c = _draw(rng)
        if _cost(c) <= most:
            return c


def _mask_mod(case):
    if case["mask"] == "causal":
        return causal_mask
    if case["mask"] == "offset":
        return generate_causal_offset(case["Skv"] - case["Sq"])
    if case["mask"] == "window":
        return generate_sliding_window(case["window"])
    if case["mask"] == "sink":
        return generate_attention_sink(case["window"], 4)
    return None


def _score_mod(case):
    if case["score"] == "alibi":
        return generate_alibi_bias(case["Hq"])
    return checkerboard if case["score"] == "checkerboard" else None


def _document_lengths(case):
    """Lengths in proportion to 1, 2, .. n: the same work for every seed, in another order."""
    n, S = case["docs"], case["Sq"]
    edges = [S * i * (i + 1) // (n * (n + 1)) for i in range(n + 1)]
    return [b - a for a, b in zip(edges, edges[1:])]


def _visible_pairs(case):
    """(query, key) pairs of one batch entry and head that the mask leaves visible."""
    Sq, Skv = case["Sq"], case["Skv"]
    if case["kind"] == "packed":
        return sum(n * (n + 1) // 2 for n in _document_lengths(case))
    q = np.arange(Sq, dtype=np.int64)
    last = np.minimum(q + (Skv - Sq if case["mask"] == "offset" else 0), Skv - 1)
    if case["mask"] is None:
        return Sq * Skv
    if case["mask"] in ("causal", "offset"):
        return int((last + 1).sum())
    first = np.maximum(q - case["window"], 0)
    pairs = int((last - first + 1).sum())
    if case["mask"] == "sink":
        pairs += int(np.minimum(first, 5).sum())
    return pairs


def prepare(case, seed):
    state = {"case": case}
    kind = case["kind"]
    if kind == "mask":
        # inputs of another seed: the band moved by whole blocks, about the same work
        shift = 128 * (seed % 4)
        if case["mask"] == "causal":
            mod = generate_causal_offset(shift)
        else:
            mod = _mask_mod(dict(case, window=case["window"] + shift))
        state["mask_mod"] = mod
        return state
    B, Hq, Hkv, Sq, Skv, D = (case[k] for k in ("B", "Hq", "Hkv", "Sq", "Skv", "D"))
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(H, S):
        shape = (B, H, S, D) if case["layout"] == "bhsd" else (B, S, H, D)
        return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).to(DTYPES[case["dtype"]])

    q, k, v = normal(Hq, Sq), normal(Hkv, Skv), normal(Hkv, Skv)
    if kind in ("train", "packed"):
        state["dout"] = normal(Hq, Sq)
        q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    state.update(q=q, k=k, v=v, score_mod=_score_mod(case), block_mask=None)
    if kind == "packed":
        lengths = _document_lengths(case)
        order = np.random.RandomState(seed % (1 << 31)).permutation(len(lengths))
        ids = np.repeat(np.arange(len(lengths)), [lengths[i] for i in order])
        state["doc"] = torch.from_numpy(ids.astype(np.int32)).cuda()
    elif case["mask"] is not None:
        B_, H_ = (B, Hq) if case["mask_bh"] else (None, None)
        state["block_mask"] = fa.create_block_mask(_mask_mod(case), B_, H_, Sq, Skv)
    return state


def _attention(state, block_mask):
    case = state["case"]
    gqa = case["Hq"] != case["Hkv"]
    if case["entry"] == "flax":
        return fa.flax_attention(state["q"], state["k"], state["v"], score_mod=state["score_mod"], block_mask=block_mask,
                                 enable_gqa=gqa, return_lse=True)
    return fa.flax_attention_pallas(state["q"], state["k"], state["v"], score_mod=state["score_mod"],
                                    block_mask=block_mask, enable_gqa=gqa, bhln=case["layout"] == "bhsd",
                                    return_lse=True)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "mask":
        bm = fa.create_block_mask(state["mask_mod"], case["B"], case["Hq"], case["Sq"], case["Skv"])
        return [bm.kv_num_blocks, bm.kv_indices, bm.full_kv_num_blocks, bm.full_kv_indices,
                bm.q_num_blocks, bm.q_indices, bm.full_q_num_blocks, bm.full_q_indices]
    block_mask = state["block_mask"]
    if kind == "packed":
        doc = state["doc"]

        def document_causal(b, h, q_idx, kv_idx):
            return (doc[q_idx] == doc[kv_idx]) & (q_idx >= kv_idx)

        block_mask = fa.create_block_mask(document_causal, None, None, case["Sq"], case["Skv"])
    out, lse = _attention(state, block_mask)
    if kind in ("train", "packed"):
        grads = torch.autograd.grad(out, (state["q"], state["k"], state["v"]), state["dout"])
        return [out.detach(), lse.detach(), *grads]
    return [out, lse]


def work(case):
    B, Hq, Hkv, Sq, Skv, D = (case[k] for k in ("B", "Hq", "Hkv", "Sq", "Skv", "D"))
    if case["kind"] == "mask":
        n_q, n_kv = -(-Sq // 128), -(-Skv // 128)
        # the eight tables, and each row of the mask looked at once
        return {"bytes": B * Hq * 4 * (4 * n_q * n_kv + 2 * n_q + 2 * n_kv), "flops": 2 * Sq}
    es = 4 if case["dtype"] == "f32" else 2
    q_bytes, kv_bytes, lse_bytes = B * Hq * Sq * D * es, 2 * B * Hkv * Skv * D * es, B * Hq * Sq * 4
    nbytes = 2 * q_bytes + kv_bytes + lse_bytes
    products = 2
    if case["kind"] in ("train", "packed"):
        nbytes += 2 * q_bytes + kv_bytes  # dO in; dQ, dK, dV out
        products = 7
    if case["kind"] == "packed":
        nbytes += 4 * Sq
    return {"bytes": nbytes, "flops": 2 * products * B * Hq * D * _visible_pairs(case)}


def tolerance(case):
    if case["kind"] == "mask":
        return "exact"
    if case["dtype"] == "f32":
        return {"rel": 1e-5}
    # probabilities and results are rounded to the input type (2^-9 and 2^-12 relative for bf16 and
    # fp16, half a unit), and flax_attention also rounds the raw scores to it
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}
