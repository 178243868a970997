"""Decode steps of at most 16 sequences as a chain (norm in front of a product, product into the residual, key chunks merged in a cluster), the fp32
products (many rows on pairs of SMs, many channels as a stream) and fp32 attention over prompts in blocks of 16 and 32 queries."""
import ctypes as C

import numpy as np
import pytest

from strict_b200 import native as N
from strict_b200.kernel import DeviceVariable as DV
from conftest import TOL_F32, TOL_FP8, logits_close
from test_gpu_models import TINY_GPT2, TINY_QWEN, _run_pair

pytestmark = pytest.mark.gpu
L = N.lib


# one and two groups of 8 rows; widths of one to eight groups of 128 columns; products into the residual of at most 2048, 3072 and 4096 columns, ending inside
# a warp's steps; gated channels that end inside a block's 16; weights behind the dependency wait; a width beyond the chain
@pytest.mark.parametrize("B,over,prefetch", [(2, dict(d_model=1024, d_ff=1088), 1), (16, dict(d_model=640, d_ff=2112), 1), (8, dict(d_model=128, d_ff=3136), 1),
                                             (9, dict(d_model=896, d_ff=64), 0), (1, dict(d_model=1024, d_ff=4096), 1), (3, dict(d_model=1088, d_ff=1088), 1)])
def test_chained_step_vs_oracle(ctx, oracle, B, over, prefetch):
    cfg = dict(TINY_QWEN, n_layers=1, vocab=512, **over)
    with ctx.option("prefetch", prefetch):
        m, om, kv, st, _, logits, want = _run_pair(ctx, oracle, cfg, 7, B, 9, [9 - i % 4 for i in range(B)], 4, random_gains=True)
        for _ in range(2):
            ids = oracle.argmax(want)
            _, logits = kv.decode_step(ids, want_logits=True)
            want = st.decode(ids)
            ok, mx, rel = logits_close(logits, want, **TOL_FP8)
            assert ok, (mx, rel)
    for o in (kv, m):
        o.dispose()
    st.close(), om.close()


# key chunks of one (sequence, head) in one cluster: one chunk, several, sequences that leave the cluster's other blocks without keys, a
# new token that opens a chunk; with the first tiles behind the dependency wait
@pytest.mark.parametrize("lens,prefetch", [([300, 3], 1), ([64, 63, 127, 128], 1), ([190, 1, 65], 0)])
def test_chunks_merged_in_a_cluster_vs_oracle(ctx, oracle, lens, prefetch):
    cfg = dict(TINY_QWEN, n_layers=2, vocab=512, max_pos=512)
    with ctx.option("attn_prefetch", prefetch):
        m, om, kv, st, _, logits, want = _run_pair(ctx, oracle, cfg, 3, len(lens), max(lens), lens, 4, random_gains=True)
        for _ in range(3):
            ids = oracle.argmax(want)
            _, logits = kv.decode_step(ids, want_logits=True)
            want = st.decode(ids)
            ok, mx, rel = logits_close(logits, want, **TOL_FP8)
            assert ok, (mx, rel)
    for o in (kv, m):
        o.dispose()
    st.close(), om.close()


class GemmF32Args(C.Structure):
    _fields_ = [("M", C.c_int64), ("N", C.c_int64), ("K", C.c_int64), ("x", C.c_void_p), ("ldx", C.c_int64), ("w", C.c_void_p), ("ldw", C.c_int64),
                ("bias", C.c_void_p), ("y", C.c_void_p), ("ldy", C.c_int64), ("mode", C.c_int), ("act_pos", C.c_float), ("act_neg", C.c_float),
                ("col_scale", C.c_void_p), ("alpha", C.c_float), ("ln_gain", C.c_void_p), ("ln_bias", C.c_void_p), ("ln_eps", C.c_float)]


def _gemm_f32(ctx, x, w, y, **over):
    f = L()._Z10k_gemm_f32P14strictb200_ctxRK11GemmF32Args
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_void_p]
    d = {k: DV.of(ctx, v) for k, v in dict(x=x, w=w, y=y, **{k: v for k, v in over.items() if isinstance(v, np.ndarray)}).items()}
    a = GemmF32Args(M=len(x), N=len(w), K=x.shape[1], ldx=x.shape[1], ldw=w.shape[1], ldy=y.shape[1], alpha=1)
    for k, v in over.items():
        if not isinstance(v, np.ndarray):
            setattr(a, k, v)
    for k, v in d.items():
        setattr(a, k, v.p)
    N.check(f(ctx.h, C.addressof(a)))
    out = d["y"].to_host().reshape(y.shape)
    for v in d.values():
        v.free()
    return out


# 44 tiles of 256 channels x 128 tokens and more, ending inside a tile of either kind and inside a stage of 64 columns; rows of one stage, of several parts
# of four stages, and beyond the 16 stages after which the small products are taken out
@pytest.mark.parametrize("M,N_,K", [(129, 5633, 4), (1400, 901, 68), (1409, 1000, 260), (5505, 100, 1028), (300, 4097, 2052)])
def test_gemm_f32_on_pairs_vs_fp64(ctx, rng, M, N_, K):
    x = (rng.standard_normal((M, K)) * np.exp2(rng.integers(-6, 7, (M, K)))).astype(np.float32)
    w = (rng.standard_normal((N_, K)) * 0.02).astype(np.float32)
    b = rng.standard_normal(N_).astype(np.float32)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    size = np.abs(x).astype(np.float64) @ np.abs(w).astype(np.float64).T
    got = _gemm_f32(ctx, x, w, np.zeros((M, N_), np.float32))
    # of the magnitudes' sum: two cut-off instructions (2 * 2^-23) and the addition of a stage's two sums, four additions in a part, one per part, two for the
    # small products of 1024 columns, one unit for what is left out
    bound = (4 + 1 + 4 + (K + 255) // 256 + 2 * ((K + 1023) // 1024) + 1) * 2.0 ** -24
    assert (np.abs(got - want) <= bound * size).all()
    assert np.sqrt(np.mean((got - want) ** 2) / np.mean(want ** 2)) < 2e-7
    old = rng.standard_normal((M, N_)).astype(np.float32)
    unit = 2.0 ** -22 * (np.abs(got) + np.abs(old) + np.abs(b) + 1)  # a few roundings of the values involved
    assert (np.abs(_gemm_f32(ctx, x, w, old.copy(), bias=b, mode=1) - (old + (got + b))) <= unit).all()
    s = rng.uniform(0.5, 2, N_).astype(np.float32)
    assert (np.abs(_gemm_f32(ctx, x, w, old.copy(), col_scale=s, alpha=0.5, mode=4) - (old + 0.5 * s * got)) <= 2 * unit).all()
    z = (got + b).astype(np.float64)
    gelu = 0.5 * z * (1 + np.tanh(0.797884583 * (z + 0.044715 * z ** 3)))
    assert (np.abs(_gemm_f32(ctx, x, w, old.copy(), bias=b, mode=2) - gelu) <= 4 * unit).all()


# an infinity, a NaN and a sum beyond the range: the values they touch come out as plain fp32 sums give them, every other as without them
def test_gemm_f32_on_pairs_not_finite(ctx, rng):
    M, N_, K = 1400, 1000, 132
    x, w = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((N_, K)).astype(np.float32)
    clean = _gemm_f32(ctx, x, w, np.zeros((M, N_), np.float32))
    x2, w2 = x.copy(), w.copy()
    x2[5, 7], x2[1399, 131], w2[999, 3] = np.inf, np.nan, -np.inf
    x2[700, :], w2[20, :] = 1e30, 1e30
    old = np.ones((M, N_), np.float32)
    got = _gemm_f32(ctx, x2, w2, old.copy(), mode=1) - 1
    with np.errstate(all="ignore"):
        want = (x2.astype(np.float64) @ w2.astype(np.float64).T).astype(np.float32)
    rows, cols = np.ones(M, bool), np.ones(N_, bool)
    rows[[5, 700, 1399]], cols[[20, 999]] = False, False
    assert np.allclose(got[np.ix_(rows, cols)], clean[np.ix_(rows, cols)], rtol=1e-5, atol=1e-5)
    for part in (np.s_[5, :], np.s_[1399, :], np.s_[:, 999]):
        assert np.array_equal(np.isnan(got[part]), np.isnan(want[part])) and np.array_equal(np.isinf(got[part]), np.isinf(want[part]))
    assert np.isinf(got[700, 20]) and np.isfinite(got[700, cols]).all()


# operands of the ends of the fp32 range, as the kernel of fewer rows takes them
@pytest.mark.parametrize("ex,ew", [(-118, 100), (-125, 120), (120, -124), (-147, 126)])
def test_gemm_f32_on_pairs_small_operands(ctx, rng, ex, ew):
    M, N_, K = 1400, 1000, 132
    x = np.ldexp(rng.uniform(1, 2, (M, K)) * rng.choice([-1, 1], (M, K)), ex).astype(np.float32)
    w = np.ldexp(rng.uniform(1, 2, (N_, K)) * rng.choice([-1, 1], (N_, K)), ew).astype(np.float32)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    size = np.abs(x).astype(np.float64) @ np.abs(w).astype(np.float64).T
    got = _gemm_f32(ctx, x, w, np.zeros((M, N_), np.float32))
    # as above, and a unit at the end of the range per instruction and addition; of a value below 2^-126 half a unit is left out
    left_out = 2.0 ** -150 * np.abs(w).astype(np.float64).sum(1) if ex < -126 else 0
    assert (np.abs(got - want) <= 13 * 2.0 ** -24 * size + (K / 16 + 16) * 2.0 ** -149 + left_out).all()


# a recorded call keeps its kernel and replays after larger calls have moved the scratch
def test_gemm_f32_recorded_does_not_depend_on_scratch(ctx, rng):
    x, w = rng.standard_normal((1400, 64)).astype(np.float32), rng.standard_normal((1000, 64)).astype(np.float32)
    dx, dw, dy = DV.of(ctx, x), DV.of(ctx, w), DV(ctx, 1400 * 1000)
    with ctx.record():
        N.check(L().strictb200_gemm_f32(ctx.h, 1400, 1000, 64, dx.p, dw.p, None, dy.p))
    _gemm_f32(ctx, rng.standard_normal((4000, 512)).astype(np.float32), rng.standard_normal((2000, 512)).astype(np.float32), np.zeros((4000, 2000), np.float32))
    ctx.replay(ctx.last_graph)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    assert np.allclose(dy.to_host().reshape(want.shape), want, rtol=1e-5, atol=1e-5)
    ctx.free_graph(ctx.last_graph)
    for v in (dx, dw, dy):
        v.free()


# eight channels for every warp of two blocks per SM and one more, one to four rows, rows that end inside a load of a warp
@pytest.mark.parametrize("M,N_,K", [(1, 18944, 768), (2, 18945, 4), (3, 20001, 772), (4, 19000, 1024), (1, 50257, 132)])
def test_gemm_f32_stream_vs_fp64(ctx, rng, M, N_, K):
    x, w = rng.standard_normal((M, K)).astype(np.float32), (rng.standard_normal((N_, K)) * 0.02).astype(np.float32)
    b = rng.standard_normal(N_).astype(np.float32)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    size = np.abs(x).astype(np.float64) @ np.abs(w).astype(np.float64).T
    got = _gemm_f32(ctx, x, w, np.zeros((M, N_), np.float32))
    # a lane adds its part of at most K columns four at a time, then five folds: each addition at most 2^-24 of the magnitudes
    assert (np.abs(got - want) <= (K / 32 + 4 + 5) * 2.0 ** -24 * size).all()
    assert np.array_equal(_gemm_f32(ctx, x, w, np.zeros((M, N_), np.float32), bias=b), got + b)


# two heads and 7 tiles of 32 queries: 42 sequences are the last that take blocks of 16 queries, 43 the first with 32; lengths that end inside a warp's 8 rows, a block
# and a tile of keys; a step over the keys they leave
@pytest.mark.parametrize("B", [3, 42, 43])
def test_gpt2_prompts_in_blocks_vs_oracle(ctx, oracle, B):
    cfg = dict(TINY_GPT2, max_pos=256)
    lens = [200 - (i * 37) % 200 for i in range(B)]
    m, om, kv, st, _, logits, want = _run_pair(ctx, oracle, cfg, 5, B, 200, lens, 2, random_gains=True)
    ok, mx, rel = logits_close(logits, want, **TOL_F32)
    assert ok, (mx, rel)
    ids = oracle.argmax(want)
    _, logits = kv.decode_step(ids, want_logits=True)
    ok, mx, rel = logits_close(logits, st.decode(ids), **TOL_F32)
    assert ok, (mx, rel)
    for o in (kv, m):
        o.dispose()
    st.close(), om.close()


# rows of a warp each (2368 rows and more) and of a block each; the narrowest and the widest of a warp, rows that end inside a lane's loads, wider ones
@pytest.mark.parametrize("M,d", [(2368, 768), (2367, 768), (2375, 4), (2369, 772), (2370, 1024), (2368, 1028), (2400, 257)])
def test_layer_norm_of_many_rows_vs_fp64(ctx, rng, M, d):
    x = (rng.standard_normal((M, d)) + rng.uniform(-2, 2, (M, 1))).astype(np.float32)
    g, b = rng.uniform(0.5, 1.5, d).astype(np.float32), rng.standard_normal(d).astype(np.float32)
    dx, dg, db, dy = DV.of(ctx, x), DV.of(ctx, g), DV.of(ctx, b), DV(ctx, M * d)
    N.check(L().strictb200_layernorm(ctx.h, dx.p, dg.p, db.p, 1e-5, M, d, dy.p))
    got = dy.to_host().reshape(M, d)
    x64 = x.astype(np.float64)
    mean, var = x64.mean(1, keepdims=True), x64.var(1, keepdims=True)
    r = 1 / np.sqrt(var + 1e-5)
    # at most 16 additions in a row for each sum; of the mean that is 16 * 2^-24 of the magnitudes, of the variance half of it again in the root; a few roundings of the result
    unit = 2.0 ** -24
    bound = (20 * unit * (np.abs(x64).mean(1, keepdims=True) + np.abs(x64 - mean)) * r) * np.abs(g) + 4 * unit * (np.abs(b) + np.abs((x64 - mean) * r * g))
    # a mean that is off moves the deviations together: its square enters the variance
    assert (np.abs(got - ((x64 - mean) * r * g + b)) <= bound).all()
    for v in (dx, dg, db, dy):
        v.free()


# the layer norm in front of the product, which is that of the whole row where two warps share a channel's columns too (one row, 512 columns and more, at
# most 1184 channels): both sides of that line, the ends of the registers that hold a row (384, 768, 1024 columns), a narrow row, a wide matrix, several rows
@pytest.mark.parametrize("M,N_,K", [(1, 512, 512), (1, 1024, 512), (1, 700, 640), (1, 768, 768), (1, 40, 772), (1, 1184, 1024), (1, 1185, 1024), (1, 1184, 508), (1, 9, 384),
                                    (1, 9, 388), (1, 3072, 768), (1, 64, 4), (2, 768, 768), (8, 512, 1024)])
def test_gemm_f32_norm_in_front_vs_fp64(ctx, rng, M, N_, K):
    x = (rng.standard_normal((M, K)) * np.linspace(0.2, 3, K) + rng.uniform(-2, 2, (M, 1))).astype(np.float32)  # a row whose parts differ in size
    w = (rng.standard_normal((N_, K)) * 0.02).astype(np.float32)
    g, b, c = rng.uniform(0.5, 1.5, K).astype(np.float32), rng.standard_normal(K).astype(np.float32), rng.standard_normal(N_).astype(np.float32)
    got = _gemm_f32(ctx, x, w, np.zeros((M, N_), np.float32), bias=c, ln_gain=g, ln_bias=b, ln_eps=1e-5)
    x64, w64 = x.astype(np.float64), np.abs(w).astype(np.float64)
    mean = x64.mean(1, keepdims=True)
    r = 1 / np.sqrt(x64.var(1, keepdims=True) + 1e-5)
    n = (x64 - mean) * r * g + b
    # of the norm: at most 16 additions in a row for each of its sums and a few roundings of the result; of the product: a lane's part of at most K columns, four at
    # a time, 5 folds, two slices and the bias
    unit = 2.0 ** -24
    off = 20 * unit * (np.abs(x64).mean(1, keepdims=True) + np.abs(x64 - mean)) * r * np.abs(g) + 4 * unit * (np.abs(b) + np.abs((x64 - mean) * r * g))
    assert (np.abs(got - (n @ w.astype(np.float64).T + c)) <= off @ w64.T + (K / 32 + 4 + 5 + 3) * unit * (np.abs(n) @ w64.T + np.abs(c))).all()


# decode steps of one sequence of GPT-2 models whose feed-forward is narrow enough for two warps per channel
@pytest.mark.parametrize("d,ff", [(512, 1024), (768, 768), (1024, 1152)])
def test_gpt2_one_sequence_narrow_feed_forward_vs_oracle(ctx, oracle, d, ff):
    cfg = dict(TINY_GPT2, d_model=d, n_q_heads=d // 64, n_kv_heads=d // 64, d_ff=ff)
    m, om, kv, st, _, logits, want = _run_pair(ctx, oracle, cfg, 6, 1, 5, None, 4, random_gains=True)
    for _ in range(3):
        ids = oracle.argmax(want)
        _, logits = kv.decode_step(ids, want_logits=True)
        want = st.decode(ids)
        ok, mx, rel = logits_close(logits, want, **TOL_F32)
        assert ok, (mx, rel)
    for o in (kv, m):
        o.dispose()
    st.close(), om.close()


# lengths that a kernel in front changes while the attention has already asked for keys: a product of one block that takes half a millisecond, the lengths'
# increment behind it, attention behind both, all three launched at once. Longer, shorter, across chunks and tiles, no keys at first
@pytest.mark.parametrize("lens,inc", [([200, 64, 1], 1), ([300, 63, 900], 100), ([1000, 700, 129], -100), ([0, 512, 5], 1)])
def test_decode_attention_takes_a_length_that_changes(ctx, oracle, rng, lens, inc):
    B, Hq, Hkv, D, maxlen = len(lens), 8, 2, 128, 1024
    dq, dk, dv = (DV.of(ctx, oracle.f32_to_bf16(rng.standard_normal(s).astype(np.float32))) for s in ((B, Hq, D), (B, Hkv, maxlen, D), (B, Hkv, maxlen, D)))
    _with_lengths_that_change(ctx, lens, inc, B * Hq * D, lambda dl, out: N.check(
        L().strictb200_attn_decode(ctx.h, dq.p, dk.p, dv.p, dl.p, B, Hq, Hkv, D, maxlen, D ** -0.5, out.p)))
    for v in (dq, dk, dv):
        v.free()


def _with_lengths_that_change(ctx, lens, inc, n_out, attention):
    K, out = 1 << 22, []
    dx, dw, dy = DV.of(ctx, np.ones(K, np.float32)), DV.of(ctx, np.ones(K, np.float32)), DV(ctx, 1)
    add = L()._Z9k_add_i32P14strictb200_ctxPiPKiil
    add.restype, add.argtypes = C.c_int, [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_int64]
    for late in (False, True):
        dl = DV.of(ctx, np.array(lens if late else [n + inc for n in lens], np.int32))
        got = DV(ctx, n_out, np.uint16)
        ctx.synchronize()
        if late:
            N.check(L().strictb200_gemm_f32(ctx.h, 1, 1, K, dx.p, dw.p, None, dy.p))
            N.check(add(ctx.h, dl.p, None, inc, len(lens)))
        attention(dl, got)
        out.append(got.to_host())
        assert ctx.device_status() == 0
        for v in (dl, got):
            v.free()
    assert out[0].any() and np.array_equal(out[0], out[1])
    for v in (dx, dw, dy):
        v.free()


class LatentShape(C.Structure):
    _fields_ = [("H", C.c_int), ("dim", C.c_int), ("rot", C.c_int), ("vdim", C.c_int), ("rank", C.c_int), ("window", C.c_int), ("scale", C.c_float)]


# the same of latent attention: fewer and more early tiles than the ring has stages, a window that moves with the length, one block and clusters, rows of which one
# block fills an SM
@pytest.mark.parametrize("lens,inc,rank,window,nsplit", [([200, 63, 130], 1, 256, 0, 2), ([1000, 64, 500], 24, 256, 0, 4), ([900, 700, 129], -100, 256, 256, 1),
                                                         ([500, 1000, 3], 1, 512, 0, 8), ([640, 300, 0], 65, 256, 128, 2)])
def test_latent_attention_takes_a_length_that_changes(ctx, oracle, rng, lens, inc, rank, window, nsplit):
    B, H, dim, rot, vdim, maxlen = len(lens), 16, 128, 64, 128, 1088
    s = LatentShape(H, dim, rot, vdim, rank, window, (dim + rot) ** -0.5)
    chunk = ((min(window, maxlen) if window else maxlen) + nsplit * 64 - 1) // (nsplit * 64) * 64
    dq, dk, dw = (DV.of(ctx, oracle.f32_to_bf16(0.3 * rng.standard_normal(n).astype(np.float32))) for n in ((B, H, rank + rot), (B, maxlen, rank + rot), (2 * H * dim, rank)))
    scratch = DV(ctx, B * H * rank, np.uint16)
    f = L()._Z20k_latent_attn_decodeP14strictb200_ctxRK11LatentShapePK13__nv_bfloat16S6_PKiiiiiPS4_S6_S9_l
    f.restype, f.argtypes = C.c_int, [C.c_void_p] * 5 + [C.c_int] * 4 + [C.c_void_p] * 3 + [C.c_int64]
    _with_lengths_that_change(ctx, lens, inc, B * H * vdim, lambda dl, out: N.check(
        f(ctx.h, C.addressof(s), dq.p, dk.p, dl.p, B, maxlen, chunk, nsplit, scratch.p, dw.p, out.p, H * vdim)))
    for v in (dq, dk, dw, scratch):
        v.free()


# the scratch that the products on SM pairs keep is given back before an allocation through the context is refused, and had again by the next product
def test_scratch_is_given_back_before_an_allocation_fails(ctx, rng):
    import torch
    x, w = rng.standard_normal((2000, 1024)).astype(np.float32), rng.standard_normal((4096, 1024)).astype(np.float32)
    planes = 3 * 2 * (2000 + 4096) * 1024
    clean = _gemm_f32(ctx, x, w, np.zeros((2000, 4096), np.float32))
    ctx.synchronize()
    before = torch.cuda.mem_get_info()[0]
    p = C.c_void_p()
    assert L().strictb200_malloc(ctx.h, C.c_size_t(1 << 50), C.byref(p)) != 0 and not p.value
    given = torch.cuda.mem_get_info()[0]
    assert given >= before + planes
    assert np.array_equal(_gemm_f32(ctx, x, w, np.zeros((2000, 4096), np.float32)), clean)
    ctx.synchronize()
    assert torch.cuda.mem_get_info()[0] <= given - planes


# key chunks merged in a cluster for KV heads with more than 8 query heads: 9, and the 16 that are the most
@pytest.mark.parametrize("heads,B", [(18, 2), (32, 16)])
def test_many_heads_merged_in_a_cluster_vs_oracle(ctx, oracle, heads, B):
    cfg = dict(TINY_QWEN, n_layers=1, vocab=512, n_q_heads=heads, n_kv_heads=2, d_model=256, max_pos=512)
    m, om, kv, st, _, logits, want = _run_pair(ctx, oracle, cfg, 8, B, 200, [200 - 11 * i for i in range(B)], 4, random_gains=True)
    for _ in range(2):
        ids = oracle.argmax(want)
        _, logits = kv.decode_step(ids, want_logits=True)
        want = st.decode(ids)
        ok, mx, rel = logits_close(logits, want, **TOL_FP8)
        assert ok, (mx, rel)
    for o in (kv, m):
        o.dispose()
    st.close(), om.close()


# key chunks that are merged in clusters are planned so that all clusters start together: sequences x KV heads, cache, query heads per KV head
@pytest.mark.parametrize("B,Hkv,maxlen,merge_heads,chunk", [(5, 8, 2032, 2, 256), (6, 8, 2032, 2, 320), (7, 8, 2032, 2, 384), (10, 8, 2032, 2, 512), (16, 8, 2032, 2, 704), (8, 8, 1032, 2, 256),
                                                            (8, 8, 545, 2, 128), (1, 8, 54, 2, 64), (14, 2, 2032, 16, 256), (16, 2, 2032, 16, 320)])
def test_merged_chunks_are_planned_in_clusters(ctx, B, Hkv, maxlen, merge_heads, chunk):
    f = L()._Z20sb_attn_decode_chunkP14strictb200_ctxiiiibi
    f.restype, f.argtypes = C.c_int, [C.c_void_p] + [C.c_int] * 4 + [C.c_bool, C.c_int]
    assert f(ctx.h, B, Hkv, maxlen, maxlen, True, merge_heads) == chunk
