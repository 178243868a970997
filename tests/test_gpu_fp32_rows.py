"""fp32 path of many rows: linear layers through three bf16 terms on the tensor cores, attention over prompts in tiles, attention
of a new token with the keys spread over groups of lanes."""
import numpy as np
import pytest

import strict_b200 as sb
from strict_b200 import native as N
from strict_b200.kernel import DeviceVariable as DV
from test_gpu_models import TINY_GPT2

pytestmark = pytest.mark.gpu
L = N.lib


def _gemm(ctx, x, w, b):
    dx, dw, dy = DV.of(ctx, x), DV.of(ctx, w), DV(ctx, len(x) * len(w))
    db = DV.of(ctx, b) if b is not None else None
    N.check(L().strictb200_gemm_f32(ctx.h, len(x), len(w), x.shape[1], dx.p, dw.p, db.p if db else None, dy.p))
    y = dy.to_host().reshape(len(x), len(w))
    for v in (dx, dw, dy, db):
        if v:
            v.free()
    return y


# rows around the token tiles (32, 64, 128), channels around a block's 128, columns around the 64 of a stage, the 1024 of a block and
# two and eight blocks of a cluster; the fewest rows that come here, with a large matrix
@pytest.mark.parametrize("M,N_,K", [(17, 1, 4), (31, 127, 60), (32, 128, 64), (33, 129, 68), (64, 130, 1024), (65, 257, 1028), (128, 768, 3072),
                                    (129, 300, 772), (300, 96, 8200), (1000, 40, 14336), (5, 2800, 3072), (9, 1366, 772)])
def test_gemm_f32_many_rows(ctx, rng, M, N_, K):
    x = (rng.standard_normal((M, K)) * np.exp2(rng.integers(-6, 7, (M, K)))).astype(np.float32)
    w = (rng.standard_normal((N_, K)) * 0.02).astype(np.float32)
    b = rng.standard_normal(N_).astype(np.float32)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    size = np.abs(x).astype(np.float64) @ np.abs(w).astype(np.float64).T
    got = _gemm(ctx, x, w, None)
    # of the sum of the products' magnitudes: two cut-off instructions and two additions per 64 columns of the large product (at most
    # 2 * 2^-23 + 2^-24), one addition per 64 columns of a block's at most ceil(K / 8) or 1024 columns, seven between blocks, one unit for the rest
    per_block = max(1024, (K + 7) // 8)
    unit = 2.0 ** -24
    assert (np.abs(got - want) <= (6 + per_block / 64 + 7 + 1) * unit * size).all()
    rms = np.sqrt(np.mean((got - want) ** 2) / np.mean(want ** 2))
    assert rms < 2e-7  # plain fp32 sums of this length: 1e-7 to 1.6e-7
    assert np.allclose(_gemm(ctx, x, w, b), got + b, rtol=1e-6, atol=1e-6 * np.abs(got).max())


# the row kernel's instances: one to eight rows, one or two channels per warp, rows split over warps, rows of X that do not fit shared memory,
# two passes over a small matrix
@pytest.mark.parametrize("M,N_,K", [(9, 1, 4), (1, 9600, 300), (2, 2500, 768), (3, 4999, 1028), (4, 2400, 2048), (4, 40, 6200), (7, 500, 512), (8, 6001, 64),
                                    (8, 300, 12000), (16, 700, 1200)])
def test_gemm_f32_few_rows(ctx, rng, M, N_, K):
    x, w = rng.standard_normal((M, K)).astype(np.float32), (rng.standard_normal((N_, K)) * 0.02).astype(np.float32)
    b = rng.standard_normal(N_).astype(np.float32)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    size = np.abs(x).astype(np.float64) @ np.abs(w).astype(np.float64).T
    got = _gemm(ctx, x, w, None)
    # a lane adds its part of at most K columns four at a time, then 5 folds and 8 slices: each addition at most 2^-24 of the magnitudes
    assert (np.abs(got - want) <= (K / 32 + 4 + 5 + 8) * 2.0 ** -24 * size).all()
    assert np.sqrt(np.mean((got - want) ** 2) / np.mean(want ** 2)) < 2e-7
    assert np.allclose(_gemm(ctx, x, w, b), got + b, rtol=1e-6, atol=1e-6 * np.abs(got).max())


# operands down to the end of the fp32 range, of one side or both, next to ones that bring the products back: the terms of a value below 2^-110
# would end in bits that bf16 does not have
@pytest.mark.parametrize("ex,ew", [(-112, 60), (-118, 100), (-125, 0), (-125, 120), (120, -124), (-60, -60), (-135, 126), (-147, 126)])
def test_gemm_f32_many_rows_small_operands(ctx, rng, ex, ew):
    M, N_, K = 48, 136, 260
    x = np.ldexp(rng.uniform(1, 2, (M, K)) * rng.choice([-1, 1], (M, K)), ex).astype(np.float32)
    w = np.ldexp(rng.uniform(1, 2, (N_, K)) * rng.choice([-1, 1], (N_, K)), ew).astype(np.float32)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    size = np.abs(x).astype(np.float64) @ np.abs(w).astype(np.float64).T
    got = _gemm(ctx, x, w, None)
    # as above, and one unit at the end of the fp32 range per instruction and addition; of a value below 2^-126 the products left out are w1 x2 and
    # w2 x1, 2^-9 and 2^-17 of w times what lies below 2^-141 and 2^-133: half a unit of the value
    left_out = 2.0 ** -150 * np.abs(w).astype(np.float64).sum(1) if ex < -126 else 0
    assert (np.abs(got - want) <= (6 + 1024 / 64 + 8) * 2.0 ** -24 * size + (K / 16 + 16) * 2.0 ** -149 + left_out).all()


@pytest.mark.parametrize("M", [1, 3, 40])
def test_gemm_f32_without_early_weights(ctx, rng, M):
    x, w = rng.standard_normal((M, 772)).astype(np.float32), rng.standard_normal((300, 772)).astype(np.float32)
    want = _gemm(ctx, x, w, None)
    with ctx.option("prefetch", 0):
        assert np.array_equal(_gemm(ctx, x, w, None), want)


def test_gemm_f32_many_rows_not_finite(ctx, rng):
    """Infinities and NaN reach exactly the results they reach in a plain sum; an operand row at the end of the fp32 range is computed."""
    x, w = rng.standard_normal((40, 200)).astype(np.float32), rng.standard_normal((70, 200)).astype(np.float32)
    x[3, 5], x[7, 9], w[13, 2] = np.inf, np.nan, -np.inf
    x[11], x[11, 0] = 0.0, 3.4e38
    w[:, 0] = np.clip(w[:, 0], -0.9, 0.9)
    with np.errstate(invalid="ignore"):
        want = x.astype(np.float64) @ w.astype(np.float64).T
    got = _gemm(ctx, x, w, None).astype(np.float64)
    fine = np.isfinite(want)
    assert np.array_equal(np.isnan(want), np.isnan(got)) and np.array_equal(want[~fine & ~np.isnan(want)], got[~fine & ~np.isnan(want)])
    assert np.allclose(got[fine], want[fine], rtol=1e-5, atol=1e-4)


# head widths of the two kernels (64) and of the decode kernel alone (32, 128), one that neither takes; prompts around the 64-row tile
# a wide feed-forward: the norm in front of a product with two channels per warp
@pytest.mark.parametrize("head_dim,lens,d_ff", [(64, [1, 63, 64, 65, 130], 0), (64, [200, 3], 2560), (32, [70, 9], 0), (128, [66, 40, 5, 1, 9, 2, 3], 2560),
                                                (64, [12] * 9, 0), (48, [20, 33], 0)])
def test_gpt2_prompts_and_decode(ctx, oracle, head_dim, lens, d_ff):
    cfg = dict(TINY_GPT2, d_model=2 * head_dim, head_dim=head_dim, d_ff=d_ff or 4 * head_dim, max_pos=256, vocab=300)
    B, S, seed = len(lens), max(lens), 11
    m, om = sb.Model(ctx, cfg).init_random(seed), oracle.Model(cfg, seed)
    kv, st = m.new_cache(B, S + 40), om.new_state(B, S + 40)
    toks, lens = oracle.gen_tokens(seed, 1, B * S, cfg["vocab"]).reshape(B, S), np.array(lens, np.int32)
    want = st.prefill(toks, lens)
    # the same prompts in two portions: the second one's rows see keys that are in the cache
    head = np.maximum(1, lens // 3).astype(np.int32)
    rest = lens - head
    kv.prefill(toks, head)
    if (rest > 0).all():
        tail = np.zeros_like(toks)
        for b in range(B):
            tail[b, :rest[b]] = toks[b, head[b]:lens[b]]
        _, logits = kv.prefill(tail, rest, want_logits=True)
    else:
        kv.reset()
        _, logits = kv.prefill(toks, lens, want_logits=True)
    # fp32 on both sides: logits of size 1, a few hundred roundings apart
    assert np.abs(logits - want).max() < 2e-5
    for _ in range(34):
        ids = oracle.argmax(want)
        _, logits = kv.decode_step(ids, want_logits=True)
        want = st.decode(ids)
        assert np.abs(logits - want).max() < 2e-5
    for o in (kv, m):
        o.dispose()
    st.close(), om.close()


@pytest.mark.parametrize("head_dim", [64, 48])
def test_gpt2_infinite_token_does_not_reach_earlier_rows(ctx, oracle, head_dim):
    """Rows of a prompt in front of a token with an infinite embedding, of the same 64 keys and of others, are what they are without it."""
    cfg = dict(TINY_GPT2, d_model=2 * head_dim, head_dim=head_dim, d_ff=4 * head_dim, max_pos=256, vocab=300)
    m = sb.Model(ctx, cfg).init_random(3)
    toks = oracle.gen_tokens(3, 1, 150, 299).reshape(1, 150)
    kv = m.new_cache(1, 200)
    _, clean = kv.prefill_rows(toks, [range(150)])
    embed = m.get_tensor("embed", np.float32, 300 * cfg["d_model"]).reshape(300, -1)
    embed[299, 5] = np.inf
    m.set_tensor("embed", embed)
    for at in (1, 50, 63, 64, 130):
        toks2 = toks.copy()
        toks2[0, at] = 299
        kv.reset()
        _, rows = kv.prefill_rows(toks2, [range(150)])
        assert np.array_equal(rows[:at, :299], clean[:at, :299]) and np.isnan(rows[at:, :299]).all()
    kv.dispose(), m.dispose()


@pytest.mark.parametrize("head_dim", [32, 64, 128, 48])
def test_gpt2_scores_of_minus_infinity(ctx, oracle, head_dim):
    """The first 70 keys of every sequence score -inf, more than a tile of a prompt and more than every group of a decode row sees first: they weigh
    nothing, and the others all the same. Rows with no other key are NaN."""
    d = 2 * head_dim
    cfg = dict(TINY_GPT2, n_layers=1, d_model=d, head_dim=head_dim, d_ff=4 * head_dim, max_pos=256, vocab=300)
    m, om = sb.Model(ctx, cfg).init_random(7), oracle.Model(cfg, 7)
    t = {n: np.array(om.tensor(n, np.float32)) for n in ("embed", "wpe", "layers.0.wqkv.w", "layers.0.wqkv.b")}
    embed, wpe, w, b = t["embed"].reshape(300, d), t["wpe"].reshape(256, d), t["layers.0.wqkv.w"].reshape(3 * d, d), t["layers.0.wqkv.b"]
    embed[:10], wpe[:] = 0, 0                       # ids 0..9 add nothing to the position
    wpe[:70, 0], wpe[:70, 1] = 1, -1                # a normed column 0 that is not zero for the first 70 positions only
    for p in range(70, 256):
        wpe[p, 2 + 2 * (p % 5)], wpe[p, 3 + 2 * (p % 5)] = 1, -1
    w[:2 * d], b[:2 * d] = 0, 0
    b[0:d:head_dim], w[d:2 * d:head_dim, 0] = 1e20, -1e30
    for n, v in t.items():
        m.set_tensor(n, v)
        om.tensor(n, np.float32)[:] = v
    om.retie()
    lens = np.array([71, 70, 128, 150], np.int32)
    toks = np.random.default_rng(1).integers(0, 10, (4, 150)).astype(np.int32)
    kv, st = m.new_cache(4, 200), om.new_state(4, 200)
    _, logits = kv.prefill(toks, lens, want_logits=True)
    want = st.prefill(toks, lens)
    assert np.isnan(want[1]).all() and np.isfinite(want[[0, 2, 3]]).all()
    for step in range(3):
        assert np.allclose(logits, want, rtol=0, atol=2e-5, equal_nan=True)
        ids = np.full(4, step, np.int32)
        _, logits = kv.decode_step(ids, want_logits=True)
        want = st.decode(ids)
    assert np.isfinite(want).all() and np.allclose(logits, want, rtol=0, atol=2e-5)
    for o in (kv, m):
        o.dispose()
    st.close(), om.close()
