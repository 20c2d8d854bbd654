"""Float32 attention as sums of 16-bit products: the exact face from 192 keys on (qk_attention_split.cu) and the
prefill attention of a bfloat16 cache (qk_decoder.cu), against 64-bit attention over the visible keys.

Tolerance: float32 scores of magnitude s carry an error of about s 2^-23 into the weights, so 2e-6 of the
largest output (scores here stay below 16); the plain float32 kernel is held to the reference's 1e-5.  The
prefill kernel adds to a row's output on the tensor core, which truncates: six products per 32 keys, each off by up
to 2^-23 of what is there."""

import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from quantibbler_b200 import _lib  # noqa: E402
from quantibbler_b200.gpu import AttentionShape, GpuContext  # noqa: E402


@pytest.fixture(scope="module")
def ctx():
    return GpuContext.init()


def visible_attention(q, k, v, causal, skew):
    """q [H, Sq, d], k and v [KV, Sk, .]: 64 bits, every row over the keys it sees and no others."""
    H, Sq, d = q.shape
    out = np.zeros((H, Sq, v.shape[-1]))
    with np.errstate(invalid="ignore", over="ignore"):
        for h in range(H):
            kk, vv = (t[h // (H // k.shape[0])].astype(np.float64) for t in (k, v))
            for i in range(Sq):
                n = i + skew + 1 if causal else kk.shape[0]
                s = kk[:n] @ q[h, i].astype(np.float64) / math.sqrt(d)
                p = np.exp(s - s.max())
                out[h, i] = (p[:, None] * vv[:n]).sum(0) / p.sum()
    return out


def worst(got, want):
    return np.abs(got - want).max() / np.abs(want).max()


@pytest.mark.parametrize("H,KV,Sq,Sk,d,dv,causal", [
    (2, 1, 192, 192, 128, 128, True),    # the shortest that takes this path
    (1, 1, 257, 257, 64, 64, True),      # one key and one row past a tile
    (4, 2, 129, 255, 80, 80, True),      # rows that see a third of a key block more than their tile's first
    (2, 2, 1, 321, 40, 24, True),        # one row; head sizes off every multiple
    (3, 1, 127, 320, 128, 64, False),
    (2, 1, 200, 448, 65, 127, True),     # one channel past the first chunk; odd sizes
    (1, 1, 130, 193, 1, 3, False),
])
def test_exact_face_at_the_edges_of_tiles(ctx, H, KV, Sq, Sk, d, dv, causal):
    rng = np.random.default_rng(Sq * 1000 + Sk)
    q, k, v = (rng.standard_normal(s).astype(np.float32) for s in ((H, Sq, d), (KV, Sk, d), (KV, Sk, dv)))
    k += 2 * rng.standard_normal((KV, 1, d)).astype(np.float32)
    got = ctx.attention(AttentionShape(1, H, KV, Sq, Sk, d, dv), q, k, v, causal).reshape(H, Sq, dv)
    assert worst(got, visible_attention(q, k, v, causal, Sk - Sq)) < 2e-6


@pytest.mark.parametrize("qs,ks,vs", [(1e-18, 1e18, 1e-30), (1e20, 1e-20, 1e30), (1.0, 0.0, 1.0), (1e-30, 1e-30, 3.0)])
def test_exact_face_over_the_range_of_float32(ctx, qs, ks, vs):
    rng = np.random.default_rng(5)
    q, k, v = (rng.standard_normal((2, 200, 64)).astype(np.float32) * np.float32(x) for x in (qs, ks, vs))
    v[0, :, 3] *= np.float32(1e-6)     # a channel far below the others keeps its own accuracy
    got = ctx.attention(AttentionShape(1, 2, 2, 200, 200, 64, 64), q, k, v, True).reshape(2, 200, 64)
    want = visible_attention(q, k, v, True, 0)
    assert worst(got, want) < 2e-6
    assert worst(got[0, :, 3], want[0, :, 3]) < 2e-6


def test_exact_face_with_infinities_and_nan(ctx):
    """Only the rows that see such a value are touched by it."""
    rng = np.random.default_rng(6)
    q, k, v = (rng.standard_normal((2, 260, 64)).astype(np.float32) for _ in range(3))
    k[0, 150, 2], v[0, 200, 5], v[1, 130, 0], q[1, 40, 1] = np.inf, np.nan, -np.inf, np.nan
    got = ctx.attention(AttentionShape(1, 2, 2, 260, 260, 64, 64), q, k, v, True).reshape(2, 260, 64)
    want = visible_attention(q, k, v, True, 0)
    fine = np.isfinite(want)
    assert 0 < (~fine).sum() < want.size // 2
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want))
    assert np.abs(got[fine] - want[fine]).max() < 2e-6 * np.abs(want[fine]).max()


@pytest.mark.parametrize("Sk", [191, 192, 260])
@pytest.mark.parametrize("entry", [1e4, 1e6, 1e8, 1e12, 1e30])
@pytest.mark.parametrize("place", ["last key", "a key's channel where q is zero", "seen key", "last value", "seen value",
                                   "a value in every 64", "half of a query"])
def test_exact_face_with_a_large_entry_among_small_ones(ctx, place, entry, Sk):
    """A row is as exact as its own operands allow, whatever lies elsewhere in the sequence: every row is held to its
    own largest output.  (A score s is off by about s 2^-23, which weighs fully where it decides over a large value.)"""
    rng = np.random.default_rng(Sk)
    q, k, v = (rng.standard_normal((2, Sk, 64)).astype(np.float32) for _ in range(3))
    at_most = 8                  # of the scores that bear on an output
    if place == "last key":
        k[0, -1, 3] = entry
    elif place == "a key's channel where q is zero":
        q[:, :, 7], k[0, :, 7] = 0, entry
    elif place == "seen key":
        k[0, 10, 3], q[0, :, 3] = entry, -np.abs(q[0, :, 3])     # (its score is far below the others)
    elif place == "last value":
        v[0, -1, 3] = entry
    elif place == "seen value":
        v[0, 10, 3], k[0, 10], at_most = entry, -3 * q[0, 150], 30
    elif place == "a value in every 64":
        v[0, 63::64, 3] = -entry
    else:
        q[0, :, 32:] *= 1 / np.float32(entry)
        k[0, :, 32:] *= np.float32(entry)
        q[0, :, :32] *= 0.5
    got = ctx.attention(AttentionShape(1, 2, 2, Sk, Sk, 64, 64), q, k, v, True).reshape(2, Sk, 64)
    want = visible_attention(q, k, v, True, 0)
    assert (np.abs(got - want).max(-1) <= 2 * at_most * 2.0 ** -23 * np.abs(want).max(-1)).all()


def test_exact_face_of_zeros(ctx):
    """Zeros are exact: a plane, a channel, the values that the first rows see."""
    rng = np.random.default_rng(7)
    q, k, v = (rng.standard_normal((3, 256, 128)).astype(np.float32) for _ in range(3))
    v[0], k[1], v[2, :100], v[2, :, 70:] = 0, 0, 0, 0
    got = ctx.attention(AttentionShape(1, 3, 3, 256, 256, 128, 128), q, k, v, True).reshape(3, 256, 128)
    want = visible_attention(q, k, v, True, 0)
    assert not got[0].any() and not got[2, :100].any() and not got[2, :, 70:].any()
    assert np.abs(got - want).max() < 2e-6 * np.abs(want).max()


def test_exact_face_where_every_product_loses_the_same(ctx):
    """Mantissas of 1 + 2^-11 are a high term of 1 and a low one of 2^-11, whose product is not formed: 2^-22 of every
    product, with one sign.  A score s is off by s 2^-22, an output by 2^-22 and by twice the largest score error."""
    rng = np.random.default_rng(9)
    q, k, v = (rng.choice([-1.0, 1.0], (1, 256, 64)).astype(np.float32) * np.float32(1 + 2.0 ** -11) for _ in range(3))
    got = ctx.attention(AttentionShape(1, 1, 1, 256, 256, 64, 64), q, k, v, False).reshape(1, 256, 64)
    scores = np.abs(q[0].astype(np.float64) @ k[0].T / 8).max()
    assert np.abs(got - visible_attention(q, k, v, False, 0)).max() <= (1 + 2 * scores) * 2.0 ** -22 * np.abs(v).max()


@pytest.mark.parametrize("causal", [True, False])
def test_exact_face_of_2048_keys(ctx, causal):
    import torch
    gen = torch.Generator("cuda").manual_seed(11)
    q, k, v = (torch.randn(1, h, 2048, 128, device="cuda", generator=gen) for h in (8, 2, 2))
    k += 2 * torch.randn(1, 2, 1, 128, device="cuda", generator=gen)
    y = torch.full_like(q, math.nan)
    torch.cuda.synchronize()
    ctx.attention_dev(AttentionShape(1, 8, 2, 2048, 2048, 128, 128), q.data_ptr(), k.data_ptr(), v.data_ptr(), causal, y.data_ptr())
    ctx.synchronize()
    kk, vv = (t.double().repeat_interleave(4, 1) for t in (k, v))
    s = q.double() @ kk.transpose(2, 3) * 128 ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(2048, 2048, dtype=torch.bool, device="cuda").triu(1), -math.inf)
    want = torch.softmax(s, -1) @ vv
    assert float((y - want).abs().max()) < 2e-6 * float(want.abs().max())


@pytest.mark.parametrize("d,dv,Sk", [(16, 16, 255), (16, 16, 256), (17, 16, 192), (8, 3, 600), (8, 4, 600), (2, 1, 600)])
def test_exact_face_where_its_kernels_meet(ctx, d, dv, Sk):
    """Small heads, around the sizes from which the tensor-core form takes them.  (Outputs of few channels lie near zero at
    times: the error is held against the head's largest.)"""
    test_exact_face_at_the_edges_of_tiles(ctx, 4, 2, Sk - 65, Sk, d, dv, True)


def test_exact_face_without_room_for_the_terms(ctx):
    """Heads of four channels, padded to 64: the terms would take 210 GB where k and v take 13.  The call goes through all
    the same, and so does the next."""
    import torch
    B, n, d = 50000, 8192, 4
    gen = torch.Generator("cuda").manual_seed(12)
    k, v = (torch.randn(B, n, d, device="cuda", generator=gen) for _ in range(2))
    q, y = torch.randn(B, d, device="cuda", generator=gen), torch.full((B, d), math.nan, device="cuda")
    torch.cuda.synchronize()
    ctx.attention_dev(AttentionShape(B, 1, 1, 1, n, d, d), q.data_ptr(), k.data_ptr(), v.data_ptr(), False, y.data_ptr())
    ctx.synchronize()
    some = slice(None, None, 61)
    weights = torch.softmax(torch.einsum("bd,bnd->bn", q[some].double(), k[some].double()) / 2, -1)[..., None]
    want = (weights * v[some]).sum(1)
    # (8192 additions in turn, each off by half a unit of the running sum: of the weights, and of the products)
    assert bool(torch.isfinite(y).all())
    assert bool(((y[some] - want).abs() <= 2 * n * 2.0 ** -24 * (weights * v[some].abs()).sum(1)).all())
    test_exact_face_at_the_edges_of_tiles(ctx, 1, 1, 257, 257, 64, 64, True)


@pytest.mark.parametrize("H,KV,T,p0", [(4, 1, 64, 0), (4, 2, 129, 0), (6, 2, 65, 63), (3, 3, 1, 70), (8, 1, 127, 130)])
def test_prefill_attention_at_the_edges_of_tiles(ctx, H, KV, T, p0):
    import torch
    gen = torch.Generator("cuda").manual_seed(T + p0)
    draw = lambda *s: torch.randn(s, device="cuda", generator=gen)  # noqa: E731
    s_max = p0 + T + 5
    q, ck, cv = draw(T, H * 128), draw(3, KV, s_max, 128).bfloat16(), draw(3, KV, s_max, 128).bfloat16()
    ck[:, :, p0 + T:] = math.nan     # what no position has written yet is never read
    cv[:, :, p0 + T:] = math.nan
    ck[0], cv[2] = math.nan, math.nan
    out = torch.zeros(T, H * 128, device="cuda")
    torch.cuda.synchronize()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _lib.check(_lib.lib().qk_prefill_attention(ctx.handle, p(q), p(ck), p(cv), _lib.QK_BF16, 1, p0, T, H, KV, 128, s_max, p(out)))
    ctx.synchronize()
    host = lambda t: t.float().cpu().numpy()  # noqa: E731
    want = visible_attention(host(q.reshape(T, H, 128).transpose(0, 1)), host(ck[1, :, :p0 + T]), host(cv[1, :, :p0 + T]), True, p0)
    assert worst(host(out.reshape(T, H, 128).transpose(0, 1)), want) < 2e-6 + 6 * math.ceil((p0 + T) / 32) * 2.0 ** -23
