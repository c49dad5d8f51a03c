"""Performance cases of the attention call: what a training or evaluation program has this package do, through its public
entry points, from single short sequences (host path and launch latency) to 64k-token training steps.

A case is a dict of
    batch, seqlen, nheads, nheads_k, head_dim, causal, mode      the call's shape and options
    direction   "train": forward, then the gradients of q, k and v for a given output gradient; "forward": evaluation or
                prefill under no_grad
    api         "bnhd" (dm_attn_func), "bhnd" (dm_attn_func_bhnd on head-major tensors) or "packed" (flash_attn_func on q, k, v
                that are views of one fused projection's output)
"""
import math

import torch

import delta_matching_b200 as dm


def _case(name, batch, seqlen, nheads, nheads_k, head_dim, causal, mode, direction, api="bnhd"):
    return {"name": name, "batch": batch, "seqlen": seqlen, "nheads": nheads, "nheads_k": nheads_k, "head_dim": head_dim,
            "causal": causal, "mode": mode, "direction": direction, "api": api}


def listed():
    return [
        # one short sequence and two heads, the smallest legal causal call: unit-test sized models, the tail of a curriculum
        _case("train-256-h2", 1, 256, 2, 2, 128, True, "matched", "train"),
        # scoring one short prompt on a small grouped-query model
        _case("eval-512-h8", 1, 512, 8, 2, 128, True, "matched", "forward"),
        # a fine-tuning micro-batch of short sequences, q / k / v as views of one projection (flash_attn drop-in)
        _case("train-packed-768", 4, 768, 12, 12, 128, True, "matched", "train", "packed"),
        # a bidirectional encoder layer (stale delta, the only mode without a causal mask), head-major tensors
        _case("train-encoder-1024", 3, 1024, 12, 12, 128, False, "stale", "train", "bhnd"),
        # the multi-head benchmark shape
        _case("train-2048-h16", 2, 2048, 16, 16, 128, True, "matched", "train"),
        # an odd one: multi-query heads that do not divide the machine, a length that is no power of two, stale delta
        _case("train-ragged-2816", 3, 2816, 7, 1, 128, True, "stale", "train"),
        # the grouped-query benchmark shape: one layer of an 8B-class pre-training step
        _case("train-4096-gqa", 4, 4096, 32, 8, 128, True, "matched", "train"),
        # the same layer in evaluation / prefill
        _case("eval-4096-gqa", 4, 4096, 32, 8, 128, True, "matched", "forward"),
        # head_dim 256, bidirectional, the benchmark shape
        _case("train-4096-d256", 2, 4096, 16, 4, 256, False, "stale", "train"),
        # head_dim 256, causal, few heads and an odd number of 128-key blocks
        _case("train-ragged-1920-d256", 1, 1920, 8, 2, 256, True, "matched", "train"),
        # prefill of a long prompt
        _case("eval-16384-gqa", 1, 16384, 32, 8, 128, True, "matched", "forward"),
        # long-context training: the backward is split over the heads to bound its workspace
        _case("train-65536-gqa", 1, 65536, 32, 8, 128, True, "matched", "train"),
    ]


_MOST_ELEMENTS = 1 << 28      # of q, as in the largest listed case


def draw(rng):
    while True:
        head_dim = 128 if rng.random() < 0.7 else 256
        step = 256 if head_dim == 128 else 128
        seqlen = step * max(1, round(math.exp(rng.uniform(math.log(256), math.log(32768))) / step))
        nheads_k = rng.randint(1, 16)
        nheads = nheads_k * rng.choice((1, 1, 2, 3, 4, 7, 8))
        causal = rng.random() < 0.75
        case = _case("", rng.randint(1, 8), seqlen, nheads, nheads_k, head_dim, causal,
                     "matched" if causal and rng.random() < 0.75 else "stale", "train" if rng.random() < 0.7 else "forward",
                     rng.choice(("bnhd", "bnhd", "bhnd", "packed")))
        del case["name"]
        # head_dim 256 runs at a lower rate: half the largest listed case's operations keep every draw below its time
        if nheads <= 64 and case["batch"] * seqlen * nheads * head_dim <= _MOST_ELEMENTS and work(case)["flops"] <= 6e13:
            return case


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    B, N, H, Hk, D = (case[k] for k in ("batch", "seqlen", "nheads", "nheads_k", "head_dim"))
    qkv = torch.randn(B, N, H + 2 * Hk, D, generator=gen, device="cuda", dtype=torch.bfloat16)
    # keys of a trained model carry a per-channel offset (what the K centring is for)
    qkv[:, :, H:H + Hk] += torch.randn(Hk, D, generator=gen, device="cuda", dtype=torch.bfloat16)
    q, k, v = qkv[:, :, :H], qkv[:, :, H:H + Hk], qkv[:, :, H + Hk:]
    if case["api"] == "bhnd":
        q, k, v = (t.transpose(1, 2) for t in (q, k, v))
    if case["api"] != "packed":
        q, k, v = (t.contiguous() for t in (q, k, v))
    train = case["direction"] == "train"
    q, k, v = (t.detach().requires_grad_(train) for t in (q, k, v))
    do = torch.randn(B, N, H, D, generator=gen, device="cuda", dtype=torch.bfloat16) if train else None
    return {"case": case, "q": q, "k": k, "v": v, "do": do}


def _call(case, q, k, v):
    if case["api"] == "bhnd":
        return dm.dm_attn_func_bhnd(q, k, v, causal=case["causal"], delta_mode=case["mode"])
    if case["api"] == "packed":
        return dm.flash_attn_func(q, k, v, causal=case["causal"], mode=case["mode"])
    return dm.dm_attn_func(q, k, v, causal=case["causal"], mode=case["mode"])


def run(state):
    case, q, k, v = state["case"], state["q"], state["k"], state["v"]
    if case["direction"] == "forward":
        with torch.no_grad():
            return _call(case, q, k, v)
    o = _call(case, q, k, v)
    dq, dk, dv = torch.autograd.grad(o, (q, k, v), state["do"])
    return {"o": o.detach(), "dq": dq, "dk": dk, "dv": dv}


def work(case):
    B, N, H, Hk, D = (case[k] for k in ("batch", "seqlen", "nheads", "nheads_k", "head_dim"))
    q_bytes, k_bytes = 2 * B * N * H * D, 2 * B * N * Hk * D
    matmuls = 2 if case["direction"] == "forward" else 7          # S, O; then S again with dP, dV, dK, dQ
    pairs = N * (N + 1) // 2 if case["causal"] else N * N
    bytes_ = 2 * q_bytes + 2 * k_bytes                             # q, k, v and o
    if case["direction"] == "train":
        bytes_ += 2 * q_bytes + 2 * k_bytes                        # do and dq, dk, dv
    return {"bytes": bytes_, "flops": matmuls * 2 * B * H * pairs * D}


def tolerance(case):
    # bf16 outputs of 8-bit products: an exponential or a sum rounded otherwise moves single e4m3 codes by one step (1/16 to
    # 1/8 of their value), which shows as a few 1e-3 of the result's norm
    return {"rel": 5e-3}
