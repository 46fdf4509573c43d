"""Tensor-core path with every query tile's keys cut into ranges, against the fp64 oracle and the uncut call (run with -m gpu).

Sizes: ranges of one block, a last range of one key, tiles with fewer blocks than a range (causal), a tile pair of which
only one half reaches a range, grouped heads, every head dim.

Bound: weights and output are rounded to 16 bits, in all 2.4e-3 (bf16) or 2.9e-4 (fp16) of the result's 2-norm, over a single row
up to four times that; the uncut call is within the same bound.  The values of the first and last key of every 128-key block are
eight times as large as the others, so that one of them lost or weighted wrongly moves its rows by about 3 / sqrt(keys): 8e-2 at 1153."""
import pytest
import torch

import tinyfa_b200 as tf
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu

SHAPES = [  # batch, seqQ, seqKV, headsQ, headsKV
    (1, 17, 257, 1, 1),
    (2, 8, 1153, 8, 2),
    (1, 129, 640, 2, 2),
    (1, 300, 1025, 3, 1),
    (2, 513, 513, 4, 4),
    (1, 700, 200, 6, 2),
]


def _run(parts, fn):
    tf.set_option("split_tc", parts)
    try:
        out = fn()
        tf.device_status()
        return out
    finally:
        tf.set_option("split_tc", -1)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [32, 64, 96, 128, 192, 256])
@pytest.mark.parametrize("shape", SHAPES)
def test_ranges(shape, D, causal):
    B, Sq, Skv, Hq, Hkv = shape
    dtype = torch.float16 if (D // 32 + Sq) % 2 else torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(Sq + D)
    Q, K, V = (torch.randn(*s, device="cuda", generator=g).to(dtype)
               for s in ((B, Sq, Hq, D), (B, Skv, Hkv, D), (B, Skv, Hkv, D)))
    V[:, sorted({*range(0, Skv, 128), *range(127, Skv, 128), Skv - 1})] *= 8
    ref = torch.from_numpy(ao.fixed(*(t.float().cpu().numpy() for t in (Q, K, V)), causal, "f64")).cuda().float()
    bound = 1.2e-3 if dtype == torch.float16 else 1e-2
    outs = {parts: _run(parts, lambda: tf.flash_attn_forward(Q, K, V, is_causal=causal)).float() for parts in (0, 2, 3, 8)}
    for parts, out in outs.items():
        for other in (ref, outs[0]):  # 2-norm of every row
            assert ((out - other).norm(dim=3) <= bound * other.norm(dim=3)).all(), parts


def test_a_nan_key_poisons_the_rows_that_see_it():
    Q, K, V = (torch.randn(*s, device="cuda").half() for s in ((1, 40, 4, 64), (1, 1000, 2, 64), (1, 1000, 2, 64)))
    K[0, 700, 0] = float("nan")
    out = _run(4, lambda: tf.flash_attn_forward(Q, K, V))
    assert torch.isnan(out[:, :, :2]).all() and torch.isfinite(out[:, :, 2:]).all()


def test_many_streams_and_repeats():
    """Calls on several streams at once use scratch of their own."""
    sets = [[torch.randn(*s, device="cuda").bfloat16() for s in ((1, 20 + i, 8, 128), (1, 4000, 2, 128), (1, 4000, 2, 128))]
            for i in range(6)]
    want = [_run(0, lambda: tf.flash_attn_forward(*s)) for s in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    torch.cuda.synchronize()
    outs = []
    for _ in range(10):
        for st, s in zip(streams, sets):
            with torch.cuda.stream(st):
                outs.append(tf.flash_attn_forward(*s))
    torch.cuda.synchronize()
    tf.device_status()
    for i, out in enumerate(outs):
        assert (out.float() - want[i % 6].float()).abs().max() <= 1.6e-2


def test_captured_calls_run_whole():
    Q, K, V = (torch.randn(*s, device="cuda").half() for s in ((1, 40, 8, 128), (1, 5000, 2, 128), (1, 5000, 2, 128)))
    want = _run(0, lambda: tf.flash_attn_forward(Q, K, V))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = tf.flash_attn_forward(Q, K, V)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
