"""What the attention-forward framework is timed and compared on.

Every case is one call of a public entry point (flash_attn_forward or flash_attn_varlen_forward) on inputs that live
on the GPU.  Inputs are independent standard normals, as in this repository's benchmark; the sizes are those of its
benchmark workloads and tests, and odd ones between them.
"""
import math

import torch

import tinyfa_b200

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
ESIZE = {"fp16": 2, "bf16": 2, "fp32": 4}
# Bounds of the drawn cases, below the largest listed ones: 2.4e12 operations in 16 bits, 6.9e10 in 32 bits.
MAX_FLOPS = {"fp16": 2.0e12, "bf16": 2.0e12, "fp32": 6.0e10}
MAX_BYTES = 1.0e9


def _fixed(name, dtype, causal, B, Sq, Skv, Hq, Hkv, D):
    return {"name": name, "kind": "fixed", "dtype": dtype, "causal": causal, "B": B, "Sq": Sq, "Skv": Skv, "Hq": Hq,
            "Hkv": Hkv, "D": D}


def _varlen(name, dtype, causal, nseq, lo, hi, lens_seed, Hq, Hkv, D):
    return {"name": name, "kind": "varlen", "dtype": dtype, "causal": causal, "nseq": nseq, "lo": lo, "hi": hi,
            "lens_seed": lens_seed, "Hq": Hq, "Hkv": Hkv, "D": D}


def listed():
    return [
        # the smallest call of the test lists: a known-answer check in fp32, bound by launch and latency
        _fixed("tiny_fp32", "fp32", False, 1, 128, 128, 4, 4, 64),
        # an encoder layer over a short batch, odd lengths of queries and keys (cross attention), 16 bits
        _fixed("cross_ragged_fp16", "fp16", False, 3, 333, 517, 12, 12, 96),
        # the shape the framework's throughput is quoted on, without and with the mask
        _fixed("prefill_bf16", "bf16", False, 2, 4096, 4096, 32, 32, 128),
        # training-sized batches at the head dims below and above 128
        _fixed("prefill_fp16_d64", "fp16", True, 8, 2048, 2048, 16, 16, 64),
        _fixed("prefill_fp16_d256", "fp16", True, 8, 2048, 2048, 16, 16, 256),
        # long-context prefill with grouped KV heads: the largest call
        _fixed("prefill_gqa_long", "bf16", True, 4, 8192, 8192, 32, 8, 128),
        # a packed batch of prompts of very different lengths, as a serving engine makes it
        _varlen("packed_gqa", "bf16", True, 16, 128, 8192, 0, 32, 8, 128),
        # one decode step: one sequence with a long cache, and a batch of them with an odd cache length
        _fixed("decode_b1", "bf16", False, 1, 1, 32768, 32, 8, 128),
        _fixed("decode_b8", "bf16", False, 8, 1, 20011, 32, 8, 128),
        # a block of draft tokens checked against the cache in one call: more query rows than one decode tile holds
        _fixed("draft_block", "bf16", False, 2, 8, 12289, 32, 8, 128),
        # full-precision evaluation of a model, at an ordinary size and with a mask and odd lengths
        _fixed("fp32_d128", "fp32", False, 2, 2048, 2048, 16, 16, 128),
        _fixed("fp32_causal_d64", "fp32", True, 2, 1999, 1999, 16, 4, 64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _heads(rng):
    hkv = rng.choice([1, 2, 4, 8, 16])
    return hkv * rng.choice([1, 1, 2, 4, 8] if hkv <= 4 else [1, 2, 4]), hkv


def draw(rng):
    while True:
        family = rng.choice(["prefill", "prefill", "packed", "decode", "draft", "fp32", "small"])
        D = rng.choice([32, 64, 64, 96, 128, 128, 128, 192, 256])
        dtype = rng.choice(["fp16", "bf16"])
        causal = rng.random() < 0.5
        Hq, Hkv = _heads(rng)
        if family == "packed":
            case = _varlen("", dtype, causal, _log_int(rng, 2, 24), 1 + _log_int(rng, 1, 200), _log_int(rng, 300, 6000),
                           rng.randrange(1 << 30), Hq, Hkv, D)
        elif family == "prefill":
            S = _log_int(rng, 256, 8192)
            Skv = S if rng.random() < 0.7 else _log_int(rng, 256, 8192)
            case = _fixed("", dtype, causal, _log_int(rng, 1, 8), S, Skv, Hq, Hkv, D)
        elif family == "decode":
            case = _fixed("", dtype, False, _log_int(rng, 1, 32), 1, _log_int(rng, 300, 40000), Hq, Hkv, D)
        elif family == "draft":
            case = _fixed("", dtype, False, _log_int(rng, 1, 4), _log_int(rng, 2, 64), _log_int(rng, 500, 30000), Hq, Hkv, D)
        elif family == "fp32":
            S = _log_int(rng, 100, 3000)
            Skv = S if rng.random() < 0.7 else _log_int(rng, 100, 3000)
            case = _fixed("", "fp32", causal, _log_int(rng, 1, 4), S, Skv, Hq, Hkv, D)
        else:
            S = _log_int(rng, 16, 256)
            dtype = rng.choice(["fp16", "bf16", "fp32"])
            case = _fixed("", dtype, causal, _log_int(rng, 1, 8), S, S, Hq, Hkv, D)
        del case["name"]
        w = work(case)
        if w["flops"] <= MAX_FLOPS[case["dtype"]] and w["bytes"] <= MAX_BYTES:
            return case


def _lengths(case):
    g = torch.Generator().manual_seed(int(case["lens_seed"]))
    return [int(x) for x in torch.randint(case["lo"], case["hi"] + 1, (case["nseq"],), generator=g)]


def _visible(sq, skv, causal):
    """(query, key) pairs that the mask leaves; key j is visible to query i when j <= i."""
    if not causal:
        return sq * skv
    m = min(sq, skv)
    return m * (m + 1) // 2 + max(0, sq - skv) * skv


def work(case):
    e, D, Hq, Hkv = ESIZE[case["dtype"]], case["D"], case["Hq"], case["Hkv"]
    if case["kind"] == "varlen":
        spans = [(n, n) for n in _lengths(case)]
        index = 8 * (len(spans) + 1)
    else:
        spans = [(case["Sq"], case["Skv"])] * case["B"]
        index = 0
    nbytes = index
    flops = 0
    for sq, skv in spans:
        seen = min(sq, skv) if case["causal"] else skv  # keys behind the last query's diagonal are never needed
        nbytes += e * D * (2 * sq * Hq + 2 * seen * Hkv)
        flops += 4 * D * Hq * _visible(sq, skv, case["causal"])
    return {"bytes": nbytes, "flops": flops}


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dt = DTYPES[case["dtype"]]

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=g).to(dt)

    D, Hq, Hkv = case["D"], case["Hq"], case["Hkv"]
    state = {"causal": case["causal"]}
    if case["kind"] == "varlen":
        lens = _lengths(case)
        cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
        total = sum(lens)
        state.update(Q=normal(total, Hq, D), K=normal(total, Hkv, D), V=normal(total, Hkv, D), cu=cu, longest=max(lens))
    else:
        B, Sq, Skv = case["B"], case["Sq"], case["Skv"]
        state.update(Q=normal(B, Sq, Hq, D), K=normal(B, Skv, Hkv, D), V=normal(B, Skv, Hkv, D))
    return state


def run(state):
    if "cu" in state:
        return tinyfa_b200.flash_attn_varlen_forward(state["Q"], state["K"], state["V"], state["cu"], state["cu"],
                                                     state["longest"], state["longest"], is_causal=state["causal"])
    return tinyfa_b200.flash_attn_forward(state["Q"], state["K"], state["V"], is_causal=state["causal"])


def tolerance(case):
    # 2-norm of the difference to 64-bit attention on the same inputs over that of the result, over the listed cases
    # and thirty drawn ones: bf16 1.8e-3 .. 2.35e-3, fp16 2.4e-4 .. 2.9e-4 (weights and output are rounded to 16 bits),
    # fp32 1.5e-7 .. 9.1e-7 (32-bit sums, the order of which is free).  About four times the largest.
    return {"rel": {"bf16": 1e-2, "fp16": 1.2e-3, "fp32": 3.6e-6}[case["dtype"]]}


def _attend(q, k, v, causal):
    """One sequence in 64 bits: q [sq, Hq, D], k and v [skv, Hkv, D]."""
    group = q.shape[1] // k.shape[1]
    scale = 1.0 / math.sqrt(q.shape[2])
    out = torch.empty(q.shape, dtype=torch.float64, device=q.device)
    keys = torch.arange(k.shape[0], device=q.device)
    step = max(1, (1 << 27) // max(1, k.shape[0] * group))  # query rows at a time: at most 1 GB of scores
    for h in range(k.shape[1]):
        kh, vh = k[:, h].double(), v[:, h].double()
        for i in range(0, q.shape[0], step):
            qh = q[i:i + step, h * group:(h + 1) * group].double()
            seen = min(k.shape[0], i + qh.shape[0]) if causal else k.shape[0]
            s = torch.matmul(qh.reshape(-1, q.shape[2]), kh[:seen].t()).mul_(scale).view(qh.shape[0], group, seen)
            if causal:
                rows = torch.arange(i, i + qh.shape[0], device=q.device)
                s.masked_fill_((keys[:seen][None, :] > rows[:, None])[:, None, :], float("-inf"))
            p = torch.softmax(s, dim=-1)
            out[i:i + step, h * group:(h + 1) * group] = torch.matmul(p.view(-1, seen), vh[:seen]).view(qh.shape)
    return out


def exact(case, seed):
    s = prepare(case, seed)
    if case["kind"] == "varlen":
        out = torch.empty(s["Q"].shape, dtype=torch.float64, device="cuda")
        at = 0
        for n in _lengths(case):
            part = slice(at, at + n)
            out[part] = _attend(s["Q"][part], s["K"][part], s["V"][part], case["causal"])
            at += n
        return out
    return torch.stack([_attend(s["Q"][b], s["K"][b], s["V"][b], case["causal"]) for b in range(case["B"])])
