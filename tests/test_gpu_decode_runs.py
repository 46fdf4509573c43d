"""Even partition of the decode path: equal runs of key blocks across batch entries, against the fp64 oracle (run with -m gpu).

Sizes where it can go wrong: an entry that is one run, runs that end inside an entry and go on into the next one, last
blocks that are nearly empty, more entries than runs, one KV head and many, and the same call through the entry point that
allocates nothing.

Bound: weights and output are rounded to 16 bits, in all 2.4e-3 (bf16) or 2.9e-4 (fp16) of the result's 2-norm; over the 32
and more values of one (entry, head) up to twice that.  The values of the first and last key of every 64-key block are eight times
as large as the others, so that one of them lost or taken twice moves its rows by about 3 / sqrt(keys): 2e-2 at 20000."""
import ctypes

import pytest
import torch

import tinyfa_b200 as tf
from oracle import attention_oracle as ao
from tinyfa_b200 import _lib

pytestmark = pytest.mark.gpu

SHAPES = [  # batch, seqQ, seqKV, headsQ, headsKV
    (1, 1, 256, 1, 1),
    (3, 1, 257, 8, 8),
    (5, 2, 1000, 8, 2),
    (37, 1, 320, 32, 32),
    (1, 1, 20000, 4, 1),
    (7, 3, 4097, 10, 2),
    (300, 1, 300, 2, 1),
    (70, 1, 449, 16, 16),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 64, 96, 128, 192, 256])
@pytest.mark.parametrize("shape", SHAPES)
def test_even_partition(shape, D, dtype):
    B, Sq, Skv, Hq, Hkv = shape
    g = torch.Generator(device="cuda").manual_seed(D + Skv)
    Q, K, V = (torch.randn(*s, device="cuda", generator=g).to(dtype)
               for s in ((B, Sq, Hq, D), (B, Skv, Hkv, D), (B, Skv, Hkv, D)))
    V[:, sorted({*range(0, Skv, 64), *range(63, Skv, 64), Skv - 1})] *= 8
    def cut(how):
        tf.set_option("split_kv", how)
        out = tf.flash_attn_forward(Q, K, V)
        tf.set_option("split_kv", -1)
        return out

    got, whole, auto = cut(-2), cut(1), cut(-1)  # equal runs, whole (batch, KV head) pairs, the library's choice
    flat = torch.empty_like(Q)
    rc = _lib.load().tfa_b200_fwd_decode_noalloc(
        *(ctypes.c_void_p(t.data_ptr()) for t in (Q, K, V, flat)), 1 if dtype == torch.float16 else 2, B, Sq, Skv, Hq, Hkv,
        D, 0, 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    tf.device_status()
    assert torch.equal(auto, flat) and (torch.equal(auto, got) or torch.equal(auto, whole))
    pick = sorted({0, B // 2, B - 1})
    ref = torch.from_numpy(ao.fixed(*(t[pick].float().cpu().numpy() for t in (Q, K, V)), False, "f64")).cuda()
    bound = 6e-4 if dtype == torch.float16 else 5e-3
    for other, mine, times in ((ref.float(), got[pick].float(), 1), (whole.float(), got.float(), 2**0.5)):  # both are rounded
        assert ((mine - other).norm(dim=(1, 3)) <= times * bound * other.norm(dim=(1, 3))).all()


def test_packed_sequence_longer_than_the_stated_maximum():
    """The rows that one 16-row tile holds are computed, and no other sequence's rows are touched.  (What the further rows of
    the longer sequence hold is not defined.)"""
    g = torch.Generator(device="cuda").manual_seed(1)
    Q, K, V = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((6, 16, 64), (1400, 2, 64), (1400, 2, 64)))
    cu_q = torch.tensor([0, 1, 5, 6], dtype=torch.int32, device="cuda")
    cu_kv = torch.tensor([0, 300, 900, 1400], dtype=torch.int32, device="cuda")
    out = tf.flash_attn_varlen_forward(Q, K, V, cu_q, cu_kv, 1, 600).float()
    want = torch.cat([tf.flash_attn_forward(Q[None, a:b], K[None, c:d], V[None, c:d])[0].float()
                      for a, b, c, d in ((0, 1, 0, 300), (1, 5, 300, 900), (5, 6, 900, 1400))])
    known = [0, 1, 2, 5]  # sequence 1 has four rows of eight heads per KV head: a tile holds two of them
    assert (out - want)[known].abs().max() <= 1.6e-2


def test_nan_key_poisons_its_rows_and_no_others():
    Q, K, V = (torch.randn(*s, device="cuda").bfloat16() for s in ((4, 1, 8, 64), (4, 3000, 2, 64), (4, 3000, 2, 64)))
    K[2, 1234, 1] = float("nan")
    out = tf.flash_attn_forward(Q, K, V)
    assert torch.isnan(out[2, :, 4:]).all()
    out[2, :, 4:] = 0
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("shape", [(1, 1, 9000, 8, 2), (2, 24, 4000, 8, 2)])  # decode runs; key ranges of the tensor-core path
def test_back_to_back_calls_do_not_see_each_others_partials(shape):
    """Calls in a row on one stream get the same scratch, and a combine kernel is launched while the kernel that writes its
    partials still runs.  Inputs take turns; every result is bit for bit that of the same call made alone."""
    B, Sq, Skv, Hq, Hkv = shape
    sets = [[torch.randn(*s, device="cuda").bfloat16() for s in ((B, Sq, Hq, 128), (B, Skv, Hkv, 128), (B, Skv, Hkv, 128))]
            for _ in range(2)]
    alone = []
    for s in sets:
        torch.cuda.synchronize()
        alone.append(tf.flash_attn_forward(*s))
    torch.cuda.synchronize()
    assert not torch.equal(*alone)
    outs = [tf.flash_attn_forward(*sets[i % 2]) for i in range(40)]
    tf.device_status()
    for i, out in enumerate(outs):
        assert torch.equal(out, alone[i % 2]), i


@pytest.mark.parametrize("shape,D", [  # batch, seqQ, seqKV, headsQ, headsKV
    ((1, 1, 9000, 8, 2), 128),  # one entry in many runs
    ((40, 1, 5000, 32, 8), 64),  # more than two waves of (batch, KV head) pairs, entries across run boundaries
    ((300, 1, 300, 8, 8), 128),  # whole entries per run
    ((2, 8, 12289, 32, 8), 128),  # key ranges, combined side by side
    ((1, 512, 2048, 16, 16), 64),  # key ranges, combined one after the other
    ((2, 300, 3000, 2, 2), 256),
])
def test_rows_without_a_score_above_minus_infinity_are_zero(shape, D):
    """A mask carried in the head dim (a K column of -inf against a Q column of 1): a masked entry gives exact zeros, a masked
    half of the keys no weight, however the keys are cut."""
    B, Sq, Skv, Hq, Hkv = shape
    Q, K, V = (torch.randn(*s, device="cuda").half() for s in ((B, Sq, Hq, D), (B, Skv, Hkv, D), (B, Skv, Hkv, D)))
    Q[..., 0] = 1
    K[..., 0] = 0
    K[0, Skv // 2:, :, 0] = float("-inf")
    want = tf.flash_attn_forward(Q[:1], K[:1, :Skv // 2].contiguous(), V[:1, :Skv // 2].contiguous())
    masked = K.clone()
    masked[-1, :, :, 0] = float("-inf")
    junk = torch.full_like(Q, 7.0)
    del junk  # the allocator hands this block out again
    out = tf.flash_attn_forward(Q, masked, V)
    tf.device_status()
    assert (out[-1] == 0).all()
    if B > 1:
        assert (out[0].float() - want[0].float()).abs().max() <= 2e-3
    else:
        assert (tf.flash_attn_forward(Q, K, V).float() - want.float()).abs().max() <= 2e-3


@pytest.mark.parametrize("Hq,Hkv,most", [(16, 2, 1), (4, 4, 2), (4, 1, 3)])
def test_packed_rows_without_partials_stay_zero(Hq, Hkv, most):
    """Packed decode with key splits: rows before the first sequence, past the last one, of a sequence without keys and past a
    tile's sixteen are zero whatever the scratch held, and so are rows without a score above -inf; all others are those of a
    call on their sequence alone."""
    D, group = 64, Hq // Hkv
    cu_q = torch.tensor([3, 3 + most, 23 + most, 24 + most, 25 + most, 26 + most], dtype=torch.int32, device="cuda")
    cu_kv = torch.tensor([0, 3000, 5500, 5500, 7500, 9500], dtype=torch.int32, device="cuda")
    Q, K, V = (torch.randn(*s, device="cuda").half() for s in ((30, Hq, D), (9500, Hkv, D), (9500, Hkv, D)))
    Q[..., 0] = 1
    K[..., 0] = 0
    K[5500:7500, :, 0] = float("-inf")
    want = torch.zeros(Q.shape, device="cuda")
    rows = max(most, 16 // group)  # positions of the second, longer sequence that its tile holds
    for a, n, c, d in ((3, most, 0, 3000), (3 + most, rows, 3000, 5500), (25 + most, 1, 7500, 9500)):
        want[a:a + n] = tf.flash_attn_forward(Q[None, a:a + n], K[None, c:d], V[None, c:d])[0].float()
    for _ in range(3):
        tf.flash_attn_forward(*(torch.full(s, 50.0, device="cuda").half() for s in ((4, 1, 16, D), (4, 9000, 2, D), (4, 9000, 2, D))))
        junk = torch.full_like(Q, 7.0)
        del junk  # the allocator hands this block out again
        out = tf.flash_attn_varlen_forward(Q, K, V, cu_q, cu_kv, most, 3000).float()
        assert (out - want).abs().max() <= 2e-3
        assert (out[want.abs().amax(dim=(1, 2)) == 0] == 0).all()


@pytest.mark.parametrize("shape,D,runs", [  # the faster cut by a factor of 1.2 at least
    ((59, 2, 442, 128, 16), 32, False),
    ((172, 1, 839, 64, 4), 32, False),
    ((102, 13, 304, 8, 8), 96, False),
    ((398, 16, 519, 4, 4), 128, False),
    ((40, 1, 5000, 32, 8), 128, True),
    ((1, 1, 32768, 32, 8), 128, True),
    ((8, 1, 20011, 32, 8), 128, True),
])
def test_cut_by_cost(shape, D, runs):
    """Many short entries are not cut: the combine pass over their rows would cost more than even ends save."""
    B, Sq, Skv, Hq, Hkv = shape
    Q, K, V = (torch.randn(*s, device="cuda").bfloat16() for s in ((B, Sq, Hq, D), (B, Skv, Hkv, D), (B, Skv, Hkv, D)))
    auto = tf.flash_attn_forward(Q, K, V)
    tf.set_option("split_kv", -2 if runs else 1)
    want = tf.flash_attn_forward(Q, K, V)
    tf.set_option("split_kv", -1)
    assert torch.equal(auto, want)


@pytest.mark.parametrize("shape,D", [((5, 3, 556, 64, 32), 256), ((3, 16, 9000, 2, 2), 64), ((1, 1, 700, 8, 1), 128)])
def test_causal_calls_are_not_split_over_keys_they_do_not_see(shape, D):
    B, Sq, Skv, Hq, Hkv = shape
    Q, K, V = (torch.randn(*s, device="cuda").half() for s in ((B, Sq, Hq, D), (B, Skv, Hkv, D), (B, Skv, Hkv, D)))
    auto = tf.flash_attn_forward(Q, K, V, is_causal=True)
    tf.set_option("split_kv", 1)
    want = tf.flash_attn_forward(Q, K, V, is_causal=True)
    tf.set_option("split_kv", -1)
    assert torch.equal(auto, want)
    ref = ao.fixed(*(t.float().cpu().numpy() for t in (Q, K, V)), True, "f64")
    assert (auto.cpu().double() - torch.from_numpy(ref).double()).abs().max() <= 4e-3
