"""fp32 on the tensor cores (three bf16 numbers per float) against the fp64 oracle and the CUDA-core kernel (run with -m gpu).

Bound: both kernels sum in fp32, so both are within a few units of 2^-24 times the number of additions of the exact
result; the tensor-core one sums 128 keys at a time and must not be further off (2-norm) than the CUDA-core one by more
than the spread between two orders of summation, for which a quarter is allowed on these short sequences."""
import numpy as np
import pytest
import torch

import tinyfa_b200 as tf
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu

SHAPES = [  # batch, seqQ, seqKV, headsQ, headsKV: tile edges, remainders, one row, one key, several blocks
    (1, 1, 1, 1, 1),
    (2, 1, 130, 4, 1),
    (1, 127, 129, 2, 1),
    (2, 128, 128, 3, 3),
    (1, 129, 255, 4, 2),
    (1, 257, 640, 6, 2),
    (2, 40, 1111, 8, 2),
    (1, 700, 300, 2, 2),
    (1, 300, 1500, 2, 1),
    (1, 1100, 1100, 2, 2),
]


def _with(option, fn):
    tf.set_option("fp32_tc", option)
    try:
        out = fn()
        torch.cuda.synchronize()
        tf.device_status()
        return out
    finally:
        tf.set_option("fp32_tc", -1)


def _inputs(B, Sq, Skv, Hq, Hkv, D, seed):
    rng = np.random.default_rng(seed)
    return [rng.normal(0, 1, s).astype(np.float32) for s in ((B, Sq, Hq, D), (B, Skv, Hkv, D), (B, Skv, Hkv, D))]


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [32, 64, 96, 128, 192, 256])
@pytest.mark.parametrize("shape", SHAPES)
def test_against_the_oracle_and_the_cuda_core_kernel(shape, D, causal):
    Q, K, V = _inputs(*shape, D, 7 + D + shape[1])
    dev = [torch.from_numpy(x).cuda() for x in (Q, K, V)]
    ref = ao.fixed(Q, K, V, causal, "f64")
    got = _with(1, lambda: tf.flash_attn_forward(*dev, is_causal=causal)).cpu().numpy()
    old = _with(0, lambda: tf.flash_attn_forward(*dev, is_causal=causal)).cpu().numpy()
    assert np.abs(got - ref).max() <= 1e-5
    assert np.linalg.norm(got - ref) <= 1.25 * np.linalg.norm(old - ref) + 1e-7 * np.linalg.norm(ref)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [32, 64, 128, 192, 256])
def test_packed_input(D, causal):
    lens_q, lens_kv = [5, 0, 200, 64, 300, 1], [40, 9, 200, 0, 511, 128]
    cu_q = np.concatenate([[0], np.cumsum(lens_q)]).astype(np.int32)
    cu_kv = np.concatenate([[0], np.cumsum(lens_kv)]).astype(np.int32)
    rng = np.random.default_rng(D)
    Q = rng.normal(0, 1, (int(cu_q[-1]), 4, D)).astype(np.float32)
    K, V = (rng.normal(0, 1, (int(cu_kv[-1]), 2, D)).astype(np.float32) for _ in range(2))
    args = [torch.from_numpy(x).cuda() for x in (Q, K, V, cu_q, cu_kv)]
    got = _with(1, lambda: tf.flash_attn_varlen_forward(*args, max(lens_q), max(lens_kv), is_causal=causal)).cpu().numpy()
    assert np.abs(got - ao.varlen(Q, K, V, cu_q, cu_kv, causal)).max() <= 1e-5


@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf"), 2.0**60, 1e-38, -2.0**-101])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_values_outside_the_exact_range_are_left_to_the_cuda_cores(which, value):
    arrays = _inputs(2, 150, 260, 4, 2, 64, 3)
    arrays[which][1, 33, 1, 5] = value
    dev = [torch.from_numpy(x).cuda() for x in arrays]
    got = _with(1, lambda: tf.flash_attn_forward(*dev))
    old = _with(0, lambda: tf.flash_attn_forward(*dev))
    assert torch.equal(got.view(torch.int32), old.view(torch.int32))


def test_magnitudes_inside_the_exact_range():
    """Magnitudes far from 1 but inside the accepted range, and zeros, go through the tensor cores without loss."""
    Q, K, V = _inputs(1, 130, 300, 2, 2, 64, 11)
    Q *= np.float32(2.0**-50)
    K *= np.float32(2.0**50)
    V *= np.float32(2.0**-60)
    V[:, ::3] = 0
    assert all(np.abs(x[x != 0]).min() > 2.0**-100 and np.abs(x).max() < 2.0**60 for x in (Q, K, V))
    dev = [torch.from_numpy(x).cuda() for x in (Q, K, V)]
    got = _with(1, lambda: tf.flash_attn_forward(*dev)).cpu().numpy().astype(np.float64)
    old = _with(0, lambda: tf.flash_attn_forward(*dev)).cpu().numpy().astype(np.float64)
    ref = ao.fixed(Q, K, V, False, "f64").astype(np.float64)
    assert np.linalg.norm(got - ref) <= 1.25 * np.linalg.norm(old - ref)


def test_captured_calls_replay():
    """Under capture the call stays on the CUDA cores; the graph replays and gives their result."""
    Q, K, V = (torch.from_numpy(x).cuda() for x in _inputs(1, 600, 600, 4, 4, 64, 5))
    want = _with(0, lambda: tf.flash_attn_forward(Q, K, V))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = tf.flash_attn_forward(Q, K, V)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


@pytest.mark.parametrize("shape,D,lens", [  # batch, seqQ, seqKV, headsQ, headsKV
    ((9, 900, 900, 32, 32), 256, None),  # pieces of batch entries, the last one smaller
    ((1, 40, 90000, 16, 8), 128, None),  # one entry: pieces of KV heads
    ((3, 0, 0, 48, 12), 192, [9000, 7000, 6000]),  # packed: pieces of KV heads
])
def test_calls_in_pieces(shape, D, lens):
    """Calls whose parts take more than the 1 GiB of workspace that is kept.  Bound: the CUDA-core kernel adds its keys one by
    one, a walk of as many roundings of 2^-24 as there are keys; the other one's error is a few such roundings."""
    B, Sq, Skv, Hq, Hkv = shape
    g = torch.Generator(device="cuda").manual_seed(D)

    def normal(*s):
        return torch.randn(*s, device="cuda", generator=g)

    if lens is None:
        Q, K, V = normal(B, Sq, Hq, D), normal(B, Skv, Hkv, D), normal(B, Skv, Hkv, D)
        call = lambda: tf.flash_attn_forward(Q, K, V)
    else:
        Q, K, V = normal(sum(lens), Hq, D), normal(sum(lens), Hkv, D), normal(sum(lens), Hkv, D)
        cu = torch.tensor([0] + lens).cumsum(0).int().cuda()
        call = lambda: tf.flash_attn_varlen_forward(Q, K, V, cu, cu, max(lens), max(lens), is_causal=True)
    assert 6 * (Q.numel() + 2 * K.numel()) > 1 << 30
    got, old = _with(1, call), _with(0, call)
    assert (got - old).abs().max() <= 1e-5
    assert (got - old).norm() <= 2.0**-24 * (max(lens or [Skv]) ** 0.5 + 8) * old.norm()
    V[(-1,) + (0,) * (V.dim() - 1)] = float("nan")  # seen by the last piece only: the whole call is the CUDA cores'
    got, old = _with(1, call), _with(0, call)
    assert torch.equal(got.view(torch.int32), old.view(torch.int32))


@pytest.mark.parametrize("shape,D,causal,cores", [  # the faster path by a factor of 1.3 at least
    ((512, 64, 64, 8, 8), 64, False, True),
    ((200, 49, 49, 12, 12), 32, False, True),
    ((2, 100, 3000, 8, 8), 128, True, True),
    ((4, 4096, 16, 8, 8), 64, False, True),
    ((64, 1, 300, 32, 32), 64, False, True),
    ((64, 256, 256, 8, 8), 64, False, False),
    ((1, 1000, 1000, 1, 1), 64, False, False),
    ((8, 1, 4096, 32, 8), 128, False, False),
    ((128, 77, 77, 12, 12), 128, False, False),
])
def test_path_by_size(shape, D, causal, cores):
    """Short sequences, few keys and few queries ahead of many masked keys stay on the CUDA cores in batches of any size."""
    B, Sq, Skv, Hq, Hkv = shape
    Q, K, V = (torch.randn(*s, device="cuda") for s in ((B, Sq, Hq, D), (B, Skv, Hkv, D), (B, Skv, Hkv, D)))
    call = lambda: tf.flash_attn_forward(Q, K, V, is_causal=causal)
    assert torch.equal(_with(-1, call), _with(0 if cores else 1, call))


@pytest.mark.parametrize("D", [64, 256])
def test_rows_of_no_sequence_do_not_matter(D):
    """Packed input with rows ahead of the first and behind the last sequence: whatever they hold, the call stays on the tensor
    cores and gives the same bits, also where a key block reaches into them."""
    cu_q = torch.tensor([7, 300, 500], dtype=torch.int32, device="cuda")
    cu_kv = torch.tensor([5, 400, 1000], dtype=torch.int32, device="cuda")
    Q, K, V = (torch.randn(*s, device="cuda") for s in ((530, 4, D), (1090, 2, D), (1090, 2, D)))
    call = lambda: tf.flash_attn_varlen_forward(Q, K, V, cu_q, cu_kv, 300, 600)
    for t, cu in ((Q, cu_q), (K, cu_kv), (V, cu_kv)):
        t[:cu[0]] = t[cu[-1]:] = 0
    want, old = _with(1, call), _with(0, call)
    assert not torch.equal(want, old)
    for t, cu in ((Q, cu_q), (K, cu_kv), (V, cu_kv)):
        t[:cu[0]] = t[cu[-1]:] = float("nan")
    assert torch.equal(_with(1, call), want)


@pytest.mark.parametrize("D", [32, 64, 96, 128, 192, 256])
@pytest.mark.parametrize("shape", [  # batch, seqQ, seqKV, headsQ, headsKV
    (1, 20, 3000, 4, 2),  # key ranges
    (2, 129, 200, 4, 4),
    (4, 260, 300, 40, 8),  # head dim 128: the 8 x 8 form behind it
])
def test_calls_left_to_the_cuda_cores_in_every_form(shape, D):
    """One NaN: the CUDA cores' result bit for bit, at every head dim, with and without key ranges, fixed length and packed."""
    B, Sq, Skv, Hq, Hkv = shape
    dev = [torch.from_numpy(x).cuda() for x in _inputs(B, Sq, Skv, Hq, Hkv, D, 9)]
    dev[2][B - 1, Skv // 2, 1, 3] = float("nan")
    call = lambda: tf.flash_attn_forward(*dev)
    got, old = _with(1, call), _with(0, call)
    assert torch.isnan(old).any() and torch.equal(got.view(torch.int32), old.view(torch.int32))
    cu = [torch.arange(B + 1, dtype=torch.int32, device="cuda") * n for n in (Sq, Skv)]
    packed = [t.flatten(0, 1) for t in dev]
    call = lambda: tf.flash_attn_varlen_forward(*packed, *cu, Sq, Skv)
    got, old = _with(1, call), _with(0, call)
    assert torch.isnan(old).any() and torch.equal(got.view(torch.int32), old.view(torch.int32))


@pytest.mark.parametrize("shape,D", [((1, 128, 128, 4, 4), 64), ((2, 200, 384, 4, 2), 128), ((1, 300, 700, 2, 2), 256)])
def test_sums_of_one_sign(shape, D):
    """An accumulator that cuts off instead of rounding has a bias, which shows where all summands have one sign: positive values,
    keys and queries with a common offset.  No further off 64 bits than the CUDA cores by more than the spread of the other tests."""
    Q, K, V = _inputs(*shape, D, 21)
    for q, k, v in ((Q, K, np.abs(V)), (Q, K, V + np.float32(10)), (Q + np.float32(1), K + np.float32(3), np.abs(V)),
                    (np.abs(Q), np.abs(K), np.abs(V)), (Q * np.float32(6), K * np.float32(6), V)):
        dev = [torch.from_numpy(x).cuda() for x in (q, k, v)]
        ref = ao.fixed(q, k, v, False, "f64")
        got = _with(1, lambda: tf.flash_attn_forward(*dev)).cpu().numpy()
        old = _with(0, lambda: tf.flash_attn_forward(*dev)).cpu().numpy()
        assert np.linalg.norm(got - ref) <= 1.25 * np.linalg.norm(old - ref)
