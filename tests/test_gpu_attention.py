"""GPU parity of the exact and Sage attention faces through the C ABI."""

import numpy as np
import pytest

from conftest import golden
from oracle import attention_np as anp
from quantibbler_b200.gpu import AttentionShape

pytestmark = pytest.mark.gpu

# crates/quantibbler-kernels/tests/gpu_attention_parity.rs:34-37
EXACT_RTOL, BAND = 1e-5, 1e-1
# crates/quantibbler-kernels/tests/gpu_attention_sage.rs:39-46
SAGE_RTOL, COS_MIN, REL_L1_MAX, ENVELOPE_SLACK = 1e-4, 0.999, 0.02, 1e-3


def shape_of(q, k, v):
    b, h, sq, d = q.shape
    return AttentionShape(b, h, k.shape[1], sq, k.shape[2], d, v.shape[3])


def run_exact(ctx, q, k, v, causal):
    sh = shape_of(q, k, v)
    out = ctx.attention(sh, q, k, v, causal)
    return out.reshape(sh.batch, sh.n_heads, sh.seq_q, sh.val_dim)


def run_sage(ctx, q, k, v, causal, block):
    sh = shape_of(q, k, v)
    out = ctx.attention_sage(sh, q, k, v, causal, block)
    return out.reshape(sh.batch, sh.n_heads, sh.seq_q, sh.val_dim)


def test_exact_reference_battery(gpu_ctx):
    g = golden("attention")
    cases = g.cases("tiled")
    assert len(cases) == 9
    for key in cases:
        q, k, v = g[key + "_q"], g[key + "_k"], g[key + "_v"]
        got = run_exact(gpu_ctx, q, k, v, g.meta[key]["causal"])
        inf_rel, worst = anp.parity_two_part(got, g[key + "_out"], v.shape[3], EXACT_RTOL, BAND)
        assert inf_rel <= EXACT_RTOL and worst <= EXACT_RTOL, (key, inf_rel, worst)


def test_exact_seeded_shapes(gpu_ctx):
    g = golden("attention")
    for key in g.cases("xatt"):
        q, k, v = g[key + "_q"], g[key + "_k"], g[key + "_v"]
        got = run_exact(gpu_ctx, q, k, v, g.meta[key]["causal"])
        inf_rel, worst = anp.parity_two_part(got, g[key + "_out_tiled"], v.shape[3], EXACT_RTOL,
                                             BAND)
        assert inf_rel <= EXACT_RTOL and worst <= EXACT_RTOL, (key, inf_rel, worst)
        assert np.array_equal(got, run_exact(gpu_ctx, q, k, v, g.meta[key]["causal"]))


@pytest.mark.parametrize("sq,skv", [(1, 77), (1, 4096), (5, 37), (40, 9)])
def test_exact_rectangular_causal(gpu_ctx, sq, skv):
    # decode-style shapes: bottom-right causal alignment (engine/mod.rs:1041-1067)
    rng = np.random.default_rng(sq * 1000 + skv)
    q = rng.standard_normal((2, 8, sq, 64)).astype(np.float32)
    k = rng.standard_normal((2, 2, skv, 64)).astype(np.float32)
    v = rng.standard_normal((2, 2, skv, 32)).astype(np.float32)
    got = run_exact(gpu_ctx, q, k, v, True)
    with np.errstate(invalid="ignore"):
        want = anp.attention_exact(q, k, v, causal=True)
    # rows with no admissible key are NaN in both (the reference's 0/0 contract)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert ok.any()
    assert np.abs(got[ok] - want[ok]).max() <= EXACT_RTOL * np.abs(want[ok]).max()


def test_exact_matches_scalar_decode_routine(gpu_ctx):
    import oracle
    rng = np.random.default_rng(3)
    n_heads, n_kv, d, n_pos = 8, 2, 32, 300
    q = rng.standard_normal(n_heads * d).astype(np.float32)
    keys = rng.standard_normal((n_pos, n_kv * d)).astype(np.float32)
    vals = rng.standard_normal((n_pos, n_kv * d)).astype(np.float32)
    want = oracle.gqa_attention_scalar(q, keys, vals, n_heads, n_kv, d)
    k4 = np.ascontiguousarray(keys.reshape(n_pos, n_kv, d).transpose(1, 0, 2))[None]
    v4 = np.ascontiguousarray(vals.reshape(n_pos, n_kv, d).transpose(1, 0, 2))[None]
    got = run_exact(gpu_ctx, q.reshape(1, n_heads, 1, d), k4, v4, True)
    assert np.abs(got.ravel() - want).max() <= 1e-5 * np.abs(want).max()


def test_exact_config2_shape_row_sample(gpu_ctx):
    # benchmark configuration 2 shape, full size; the oracle checks a sample of query rows
    rng = np.random.default_rng(2)
    b, h, kvh, s, d = 1, 32, 8, 8192, 128
    q = rng.standard_normal((b, h, s, d), dtype=np.float32)
    k = rng.standard_normal((b, kvh, s, d), dtype=np.float32) \
        + (2.0 * rng.standard_normal((1, kvh, 1, d))).astype(np.float32)
    v = rng.standard_normal((b, kvh, s, d), dtype=np.float32)
    got = run_exact(gpu_ctx, q, k, v, True)
    rows = np.array([0, 1, 63, 64, 1000, 4095, 4096, 8191])
    heads = [0, 5, 31]
    for hh in heads:
        kv = hh // 4
        w = anp.attention_exact(q[:, hh:hh + 1], k[:, kv:kv + 1], v[:, kv:kv + 1], causal=True,
                                rows=rows)
        gsub = got[:, hh:hh + 1][:, :, rows]
        assert np.abs(gsub - w).max() <= EXACT_RTOL * np.abs(w).max(), hh
    assert np.isfinite(got).all()


def test_validation_texts(gpu_ctx):
    z = np.zeros(64, np.float32)
    sh = AttentionShape(1, 3, 2, 4, 4, 4, 4)
    with pytest.raises(ValueError, match="n_kv_heads must divide n_heads: n_heads=3, n_kv_heads=2"):
        gpu_ctx.attention(sh, z, z, z, False)
    sh = AttentionShape(1, 2, 1, 8, 8, 4, 4)
    with pytest.raises(ValueError, match=r"key must hold 32 values for AttentionShape \{ batch: 1, "
                                         r"n_heads: 2, n_kv_heads: 1, seq_q: 8, seq_kv: 8, "
                                         r"head_dim: 4, val_dim: 4 \}, got 64"):
        gpu_ctx.attention(sh, z, z, z[:32], False)
    with pytest.raises(ValueError, match="attention requires non-empty batch and head dimensions"):
        gpu_ctx.attention(AttentionShape(0, 2, 1, 8, 8, 4, 4), z, z, z, False)
    with pytest.raises(ValueError, match="sage attention is self-attention over one cache: "
                                         "seq_q=1, seq_kv=8"):
        gpu_ctx.attention_sage(AttentionShape(1, 2, 1, 1, 8, 4, 4), z[:8], z[:32], z[:32], False, 4)
    with pytest.raises(ValueError, match="sage attention requires a positive block_size"):
        gpu_ctx.attention_sage(sh, z, z[:32], z[:32], False, 0)


def test_sage_reference_battery(gpu_ctx):
    g = golden("attention")
    cases = g.cases("sage")
    assert len(cases) == 10
    for key in cases:
        m = g.meta[key]
        q, k, v = g[key + "_q"], g[key + "_k"], g[key + "_v"]
        got = run_sage(gpu_ctx, q, k, v, m["causal"], m["block_size"])
        inf_rel, worst = anp.parity_two_part(got, g[key + "_out"], v.shape[3], SAGE_RTOL, BAND)
        assert inf_rel <= SAGE_RTOL and worst <= SAGE_RTOL, (key, inf_rel, worst)
        cos, rel_l1, _ = anp.quality_metrics(got, g[key + "_exact"])
        assert cos >= COS_MIN and rel_l1 <= REL_L1_MAX, (key, cos, rel_l1)
        ref = m["reference_metrics"]
        assert cos >= ref["cosine"] - ENVELOPE_SLACK
        assert rel_l1 <= ref["relative_l1"] + ENVELOPE_SLACK


def test_sage_seeded_shapes_against_float32_restatement(gpu_ctx):
    g = golden("attention")
    for key in g.cases("xatt"):
        m = g.meta[key]
        q, k, v = g[key + "_q"], g[key + "_k"], g[key + "_v"]
        got = run_sage(gpu_ctx, q, k, v, m["causal"], m["block_size"])
        w32 = anp.attention_sage(q, k, v, causal=m["causal"], block_size=m["block_size"],
                                 ft=np.float32)
        w64 = g[key + "_out_sage"]
        # against the float32 restatement (same arithmetic): only P codes whose exp lands
        # on a rounding tie may differ
        assert np.median(np.abs(got - w32)) <= 1e-6, key
        assert np.abs(got - w32).max() <= 2e-3 * np.abs(w32).max(), key
        # against the float64 reference: a flipped K/V/P code moves an output by ~1/127 of
        # one term, so compare in the aggregate
        cos, rel_l1, _ = anp.quality_metrics(got, w64)
        assert cos >= 0.99999 and rel_l1 <= 1e-3, (key, cos, rel_l1)
        assert np.array_equal(got, run_sage(gpu_ctx, q, k, v, m["causal"], m["block_size"]))


def test_sage_config2_shape_row_sample(gpu_ctx):
    rng = np.random.default_rng(4)
    b, h, kvh, s, d = 1, 8, 2, 2048, 128
    q = rng.standard_normal((b, h, s, d), dtype=np.float32)
    k = rng.standard_normal((b, kvh, s, d), dtype=np.float32) \
        + (2.0 * rng.standard_normal((1, kvh, 1, d))).astype(np.float32)
    v = rng.standard_normal((b, kvh, s, d), dtype=np.float32)
    got = run_sage(gpu_ctx, q, k, v, True, 64)
    rows = np.array([0, 63, 64, 777, 2047])
    for hh in (0, 7):
        kv = hh // 4
        w = anp.attention_sage(q[:, hh:hh + 1], k[:, kv:kv + 1], v[:, kv:kv + 1], causal=True,
                               block_size=64, rows=rows, ft=np.float32)
        gsub = got[:, hh:hh + 1][:, :, rows]
        assert np.abs(gsub - w).max() <= 2e-3 * np.abs(w).max(), hh
        exact = anp.attention_exact(q[:, hh:hh + 1], k[:, kv:kv + 1], v[:, kv:kv + 1],
                                    causal=True, rows=rows)
        cos, rel_l1, _ = anp.quality_metrics(gsub, exact)
        assert cos >= COS_MIN and rel_l1 <= REL_L1_MAX


def restated_codes(q, k, v, block, ft):
    """The quantisers of src/quantibbler/kernels/attention_sage.py:164-198 over whole tensors,
    in float type ``ft`` (float32 follows the device kernel's operation order:
    gpu_attention.rs:132-155 and the sequential block mean of :197-209)."""
    b, kvh, s, d = k.shape
    nb = s // block
    assert nb * block == s
    inv = ft(1.0 / np.sqrt(d)) if ft is np.float64 else ft(1.0) / np.sqrt(ft(d))
    qc, qs = anp.quantize_per_token(q.astype(ft) * inv, ft)
    kb = k.astype(ft).reshape(b, kvh, nb, block, d)
    if ft is np.float64:
        mean = kb.mean(axis=-2, keepdims=True)
    else:
        ssum = np.zeros((b, kvh, nb, 1, d), dtype=ft)
        for jj in range(block):
            ssum = (ssum + kb[:, :, :, jj:jj + 1]).astype(ft)
        mean = (ssum / ft(block)).astype(ft)
    kc, ks = anp.quantize_per_token(kb - mean, ft)
    vc, vs = anp.quantize_per_channel(v.astype(ft).reshape(b, kvh, nb, block, v.shape[3]), ft)
    return dict(q_codes=qc, q_scale=qs[..., 0], k_codes=kc.reshape(b, kvh, s, d),
                k_scale=ks.reshape(b, kvh, s), k_mean=mean[:, :, :, 0],
                v_codes=vc.reshape(b, kvh, s, v.shape[3]), v_scale=vs[:, :, :, 0])


def test_sage_at_config2_codes_and_rows(gpu_ctx):
    """benchmark configuration 2 at full size (32 query heads, 8 KV heads, 8192 tokens, head_dim 128,
    causal, key block 64).  The INT8 codes and scales the device path computes are read back
    and must equal the float32 restatement of the reference's quantisers bit for bit; against
    the float64 reference a code may differ only where a value sits within a float32 rounding
    of a tie, which is counted.  Output rows are then sampled against the quantized oracle
    and the exact one."""
    rng = np.random.default_rng(5)
    b, h, kvh, s, d, block = 1, 32, 8, 8192, 128, 64
    q = rng.standard_normal((b, h, s, d), dtype=np.float32)
    k = rng.standard_normal((b, kvh, s, d), dtype=np.float32) \
        + (2.0 * rng.standard_normal((1, kvh, 1, d))).astype(np.float32)
    v = rng.standard_normal((b, kvh, s, d), dtype=np.float32)
    sh = shape_of(q, k, v)
    got = gpu_ctx.sage_quantize(sh, q, k, v, block)
    w32 = restated_codes(q, k, v, block, np.float32)
    for name in ("q_codes", "k_codes", "v_codes", "q_scale", "k_scale", "v_scale", "k_mean"):
        assert np.array_equal(got[name], w32[name]), name   # 0 mismatches, codes and scales
    w64 = restated_codes(q, k, v, block, np.float64)
    for name in ("q_codes", "k_codes", "v_codes"):
        rate = np.mean(got[name] != w64[name])
        assert rate < 1e-3, (name, rate)
        assert np.abs(got[name].astype(np.int16) - w64[name]).max() <= 1, name
    out = run_sage(gpu_ctx, q, k, v, True, block)
    assert np.isfinite(out).all()
    rows = np.array([0, 63, 64, 1000, 4095, 8191])
    for hh in (0, 13, 31):
        kv = hh // (h // kvh)
        w = anp.attention_sage(q[:, hh:hh + 1], k[:, kv:kv + 1], v[:, kv:kv + 1], causal=True,
                               block_size=block, rows=rows, ft=np.float32)
        gsub = out[:, hh:hh + 1][:, :, rows]
        assert np.abs(gsub - w).max() <= 2e-3 * np.abs(w).max(), hh
        exact = anp.attention_exact(q[:, hh:hh + 1], k[:, kv:kv + 1], v[:, kv:kv + 1],
                                    causal=True, rows=rows)
        cos, rel_l1, _ = anp.quality_metrics(gsub, exact)
        assert cos >= COS_MIN and rel_l1 <= REL_L1_MAX, (hh, cos, rel_l1)


def test_sage_quantize_ragged_block(gpu_ctx):
    # a sequence that is not a whole number of key blocks, and the dp4a layout (head_dim 48)
    rng = np.random.default_rng(6)
    for (s, d, block) in ((100, 64, 32), (70, 48, 64)):
        q = rng.standard_normal((1, 2, s, d), dtype=np.float32)
        k = rng.standard_normal((1, 1, s, d), dtype=np.float32) + 1.5
        v = rng.standard_normal((1, 1, s, d), dtype=np.float32)
        got = gpu_ctx.sage_quantize(shape_of(q, k, v), q, k, v, block)
        _, (q_hat, k_codes, v_codes) = anp.attention_sage(q, k, v, causal=False, block_size=block,
                                                          ft=np.float32, return_codes=True)
        assert np.array_equal(got["q_codes"], q_hat)
        assert np.array_equal(got["k_codes"], np.concatenate(k_codes, axis=2))
        assert np.array_equal(got["v_codes"], np.concatenate(v_codes, axis=2))


@pytest.mark.parametrize("case", [
    # (batch, heads, kv heads, seq, head dim, block, causal)
    (1, 4, 2, 200, 128, 64, True), (2, 2, 1, 129, 64, 32, True), (1, 2, 2, 300, 128, 128, False),
    (1, 3, 1, 64, 64, 64, True), (1, 2, 1, 97, 128, 32, False)])
def test_sage_tensor_core_kernel_matches_dp4a_kernel(gpu_ctx, case):
    """The INT8 tensor-core Sage kernel and the dp4a kernel do the same arithmetic; only the
    summation order of the float32 mean shift differs, which can move a P code on a tie."""
    b, h, kvh, s, d, block, causal = case
    rng = np.random.default_rng(sum(case[:6]))
    q = rng.standard_normal((b, h, s, d), dtype=np.float32)
    k = rng.standard_normal((b, kvh, s, d), dtype=np.float32) \
        + (2.0 * rng.standard_normal((1, kvh, 1, d))).astype(np.float32)
    v = rng.standard_normal((b, kvh, s, d), dtype=np.float32)
    default = gpu_ctx.set_sage_kernel(0)
    assert default == 2
    try:
        simt = run_sage(gpu_ctx, q, k, v, causal, block)
        gpu_ctx.set_sage_kernel(1)
        tc = run_sage(gpu_ctx, q, k, v, causal, block)
        assert np.isfinite(tc).all()
        assert np.median(np.abs(tc - simt)) <= 1e-6
        assert np.abs(tc - simt).max() <= 2e-3 * np.abs(simt).max()
        w32 = anp.attention_sage(q, k, v, causal=causal, block_size=block, ft=np.float32)
        assert np.abs(tc - w32).max() <= 2e-3 * np.abs(w32).max()
        assert np.array_equal(tc, run_sage(gpu_ctx, q, k, v, causal, block))
    finally:
        gpu_ctx.set_sage_kernel(default)


@pytest.mark.parametrize("case", [
    # (batch, heads, kv heads, seq, causal): head_dim 128, key block 64, the shapes the tcgen05 kernel takes
    (1, 4, 2, 200, True), (1, 2, 1, 320, False), (2, 8, 2, 1000, True), (1, 2, 2, 64, True), (1, 1, 1, 129, False)])
def test_sage_tcgen05_kernel_matches_the_other_kernels(gpu_ctx, case):
    """Sage with both integer products on tcgen05 (kind::i8, accumulators in tensor memory)
    against the mma.sync kernel: the same scores, maxima and P codes, hence the same integer
    PV sums; only the order in which a row's P values are added into l differs.  Ragged last
    blocks, an odd number of key blocks (the second block of the last iteration is empty),
    several query tiles, GQA, causal and not."""
    b, h, kvh, s, causal = case
    d, block = 128, 64
    rng = np.random.default_rng(sum(case[:4]) + 7)
    q = rng.standard_normal((b, h, s, d), dtype=np.float32)
    k = rng.standard_normal((b, kvh, s, d), dtype=np.float32) \
        + (2.0 * rng.standard_normal((1, kvh, 1, d))).astype(np.float32)
    v = rng.standard_normal((b, kvh, s, d), dtype=np.float32)
    default = gpu_ctx.set_sage_kernel(1)
    try:
        tc = run_sage(gpu_ctx, q, k, v, causal, block)
        gpu_ctx.set_sage_kernel(2)
        um = run_sage(gpu_ctx, q, k, v, causal, block)
        gpu_ctx.synchronize()
    finally:
        gpu_ctx.set_sage_kernel(default)
    assert np.isfinite(um).all()
    assert np.abs(um - tc).max() <= 1e-5 * np.abs(tc).max()
    w32 = anp.attention_sage(q, k, v, causal=causal, block_size=block, ft=np.float32)
    assert np.abs(um - w32).max() <= 2e-3 * np.abs(w32).max()
    gpu_ctx.set_sage_kernel(2)
    try:
        assert np.array_equal(um, run_sage(gpu_ctx, q, k, v, causal, block))
    finally:
        gpu_ctx.set_sage_kernel(default)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("seq", [64, 65, 127, 128, 129, 191, 192, 193, 320, 385, 513, 1100])
def test_sage_tcgen05_kernel_at_the_edges_of_its_tiles(gpu_ctx, seq, causal):
    """Ends of query tiles, key blocks, pairs of blocks and buffer rings against the mma.sync kernel, whose integer sums
    it must reproduce (1e-5 as above: the order in which l is summed); the quantisers' codes as well.  An infinite
    value and a query row of NaN stay where they belong."""
    b, h, kvh, d, block = 2, 3, 1, 128, 64
    rng = np.random.default_rng(seq + causal)
    q = rng.standard_normal((b, h, seq, d), dtype=np.float32)
    k = rng.standard_normal((b, kvh, seq, d), dtype=np.float32) \
        + (2.0 * rng.standard_normal((1, kvh, 1, d))).astype(np.float32)
    v = rng.standard_normal((b, kvh, seq, d), dtype=np.float32)
    q[1, 2, seq // 2] = np.nan
    v[0, 0, 0, 5] = np.inf      # (a key that every row sees: a block's infinite scale reaches all rows that pass over the block)
    default = gpu_ctx.set_sage_kernel(1)
    try:
        with np.errstate(invalid="ignore"):
            tc = run_sage(gpu_ctx, q, k, v, causal, block)
            codes = gpu_ctx.sage_quantize(shape_of(q, k, v), q, k, v, block)
            gpu_ctx.set_sage_kernel(2)
            um = run_sage(gpu_ctx, q, k, v, causal, block)
            same = gpu_ctx.sage_quantize(shape_of(q, k, v), q, k, v, block)
    finally:
        gpu_ctx.set_sage_kernel(default)
    assert np.array_equal(np.isnan(um), np.isnan(tc))
    fine = np.isfinite(tc)
    assert np.array_equal(um[~fine], tc[~fine], equal_nan=True)
    assert np.abs(um[fine] - tc[fine]).max() <= 1e-5 * np.abs(tc[fine]).max()
    for name in codes:
        assert np.array_equal(codes[name], same[name], equal_nan=True), name


def test_sage_tcgen05_kernel_repeats_its_bits(gpu_ctx):
    """Many iterations of many tiles, over and over: a product issued before the one whose operand it overwrites has
    read it would show as other bits."""
    b, h, kvh, seq, d, block = 1, 16, 4, 3072, 128, 64
    rng = np.random.default_rng(77)
    q = rng.standard_normal((b, h, seq, d), dtype=np.float32) * 3
    k, v = (rng.standard_normal((b, kvh, seq, d), dtype=np.float32) for _ in range(2))
    default = gpu_ctx.set_sage_kernel(1)
    try:
        tc = run_sage(gpu_ctx, q, k, v, True, block)
        gpu_ctx.set_sage_kernel(2)
        first = run_sage(gpu_ctx, q, k, v, True, block)
        assert np.abs(first - tc).max() <= 1e-5 * np.abs(tc).max()
        for _ in range(20):
            assert np.array_equal(run_sage(gpu_ctx, q, k, v, True, block), first)
    finally:
        gpu_ctx.set_sage_kernel(default)


@pytest.mark.parametrize("which", ["q", "k", "v"])
def test_sage_inputs_need_not_lie_on_sixteen_bytes(gpu_ctx, which):
    """One input after the other on four bytes only: the bits of the aligned call (tcgen05 form)."""
    import torch
    b, h, kvh, seq, d, block = 1, 4, 2, 321, 128, 64
    rng = np.random.default_rng(5)
    host = dict(q=rng.standard_normal((b, h, seq, d), dtype=np.float32), k=rng.standard_normal((b, kvh, seq, d), dtype=np.float32),
                v=rng.standard_normal((b, kvh, seq, d), dtype=np.float32))
    shape, outs = shape_of(*host.values()), []
    default = gpu_ctx.set_sage_kernel(2)
    try:
        for shift in (0, 1):
            bufs = {}
            for name, x in host.items():
                at = shift if name == which else 0
                buf = torch.zeros(x.size + 4, device="cuda")
                buf[at:at + x.size] = torch.from_numpy(x).cuda().flatten()
                bufs[name] = buf[at:]
            out = torch.zeros(b, h, seq, d, device="cuda")
            torch.cuda.synchronize()
            gpu_ctx.attention_dev(shape, *(t.data_ptr() for t in bufs.values()), True, out.data_ptr(), block)
            gpu_ctx.synchronize()
            outs.append(out)
    finally:
        gpu_ctx.set_sage_kernel(default)
    assert bool((outs[0] != 0).any()) and torch.equal(*outs)


@pytest.mark.parametrize("dim,block", [(64, 64), (128, 32), (128, 64)])
def test_sage_scratch_is_what_the_shape_needs(dim, block):
    """A fresh context's memory after a first call: codes and scales, and records only where a kernel reads them (heads of
    128, key blocks of 64: 416 bytes a key), whichever form runs first.  (Two more megabytes twice: an allocation is rounded up
    to them, and the context's error word takes one.)"""
    import torch
    from quantibbler_b200.gpu import GpuContext
    b, h, kvh, s = 1, 2, 2, 64 * 1024
    q, k, v = (torch.zeros(b, n, s, dim, device="cuda") for n in (h, kvh, kvh))
    out, blocks = torch.zeros_like(q), s // block
    codes = kvh * s * dim + kvh * s * 4 + kvh * blocks * dim * max(block, 64) + kvh * blocks * dim * 4 + kvh * blocks * (8 * dim + 4)
    common = h * s * dim + h * s * 4 + kvh * blocks * dim * 4
    most = common + max(codes, kvh * s * 416 if (dim, block) == (128, 64) else 0) + (4 << 20)
    shape = shape_of(*(t.cpu().numpy() for t in (q, k, v)))
    ctx = GpuContext.init()
    try:
        small = torch.zeros(1, 1, 64, dim, device="cuda")
        one = shape_of(*(small.cpu().numpy() for _ in range(3)))
        for which in (2, 1):     # (the kernels are loaded)
            ctx.set_sage_kernel(which)
            ctx.attention_dev(one, small.data_ptr(), small.data_ptr(), small.data_ptr(), True, out.data_ptr(), block)
            ctx.synchronize()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        for which in (2, 1):
            ctx.set_sage_kernel(which)
            ctx.attention_dev(shape, q.data_ptr(), k.data_ptr(), v.data_ptr(), True, out.data_ptr(), block)
            ctx.synchronize()
            assert free - torch.cuda.mem_get_info()[0] <= most, which
    finally:
        ctx.close()


def test_attention_on_device_buffers(gpu_ctx):
    import torch
    rng = np.random.default_rng(11)
    b, h, kvh, s, d = 1, 4, 2, 160, 64
    q = rng.standard_normal((b, h, s, d), dtype=np.float32)
    k = rng.standard_normal((b, kvh, s, d), dtype=np.float32)
    v = rng.standard_normal((b, kvh, s, d), dtype=np.float32)
    sh = shape_of(q, k, v)
    tq, tk, tv = (torch.from_numpy(x).cuda() for x in (q, k, v))
    out = torch.zeros(b, h, s, d, device="cuda")
    torch.cuda.synchronize()
    gpu_ctx.attention_dev(sh, tq.data_ptr(), tk.data_ptr(), tv.data_ptr(), True, out.data_ptr())
    gpu_ctx.synchronize()
    assert np.array_equal(out.cpu().numpy(), run_exact(gpu_ctx, q, k, v, True))
    gpu_ctx.attention_dev(sh, tq.data_ptr(), tk.data_ptr(), tv.data_ptr(), True, out.data_ptr(),
                          block_size=32)
    gpu_ctx.synchronize()
    assert np.array_equal(out.cpu().numpy(), run_sage(gpu_ctx, q, k, v, True, 32))


@pytest.mark.parametrize("case", [
    # (batch, heads, kv heads, seq, causal)
    (1, 4, 2, 200, True), (1, 2, 1, 320, False), (2, 8, 2, 1000, True), (1, 2, 2, 64, True), (1, 1, 1, 129, False)])
def test_sage_block_scale_variant_against_its_restatement(gpu_ctx, case):
    """The benchmark specification's Sage variant (one INT8 scale per 64-token block for Q and
    K, bfloat16 P and V, the output accumulated in tensor memory and rescaled lazily): not the
    reference's arithmetic and pinned to nothing; checked against the NumPy restatement of the
    wording (exact softmax of the same quantised scores, V rounded to bfloat16), within what the
    bfloat16 rounding of P and float32 accumulation add, and against the exact attention within
    what INT8 block scales cost.  Ragged last blocks, an odd number of key blocks, several query
    tiles, GQA, causal and not; run twice for bit identity."""
    import torch
    b, h, kvh, s, causal = case
    d = 128
    rng = np.random.default_rng(sum(case[:4]) + 11)
    q = rng.standard_normal((b, h, s, d), dtype=np.float32)
    k = rng.standard_normal((b, kvh, s, d), dtype=np.float32) \
        + (2.0 * rng.standard_normal((1, kvh, 1, d))).astype(np.float32)
    v = rng.standard_normal((b, kvh, s, d), dtype=np.float32)
    sh = shape_of(q, k, v)
    tq, tk, tv = (torch.from_numpy(x).cuda() for x in (q, k, v))
    outs = []
    for _ in range(2):
        out = torch.full((b, h, s, d), float("nan"), device="cuda")
        torch.cuda.synchronize()
        gpu_ctx.attention_sage_block_dev(sh, tq.data_ptr(), tk.data_ptr(), tv.data_ptr(), causal, out.data_ptr())
        gpu_ctx.synchronize()
        outs.append(out.cpu().numpy())
    got = outs[0]
    assert np.isfinite(got).all()
    assert np.array_equal(got, outs[1])
    want = anp.attention_sage_block(q, k, v, causal=causal)
    assert np.abs(got - want).max() <= 6e-3 * np.abs(want).max()
    exact = anp.attention_exact(q, k, v, causal=causal) if hasattr(anp, "attention_exact") else None
    if exact is not None:
        assert np.abs(got - exact).max() <= 5e-2 * np.abs(exact).max()
