"""Linear layers of a decode step's few rows."""
import numpy as np
import pytest

from strict_b200 import native as N
from strict_b200.kernel import DeviceVariable as DV
from conftest import TOL_FP8, logits_close
from test_gpu_models import TINY_QWEN, _run_pair

pytestmark = pytest.mark.gpu
L = N.lib


# one and two groups of 8 rows; channels around a block's 32 and 64; columns around a load's 32, a unit of 64, the 1024 a block holds ahead, and
# more of them; grids beyond two blocks per SM (two tiles per block, and one with more than 8 rows); the most channels of the kernel and one beyond
@pytest.mark.parametrize("M,N_,K", [(1, 1, 8), (8, 31, 24), (9, 33, 40), (16, 64, 1024), (3, 100, 1032), (5, 40, 5000), (8, 9600, 136), (13, 9599, 1024),
                                    (8, 16384, 1024), (2, 16385, 1024), (17, 64, 64), (8, 18944, 72), (7, 18945, 72), (9, 9473, 776), (16, 9473, 72)])
def test_gemm_bf16_few_rows(ctx, oracle, rng, M, N_, K):
    x = oracle.round_bf16(rng.standard_normal((M, K)).astype(np.float32))
    w = oracle.round_bf16((rng.standard_normal((N_, K)) * 0.05).astype(np.float32))
    want = x.astype(np.float64) @ w.astype(np.float64).T
    size = np.abs(x).astype(np.float64) @ np.abs(w).astype(np.float64).T
    dx, dw, dy = DV.of(ctx, oracle.f32_to_bf16(x)), DV.of(ctx, oracle.f32_to_bf16(w)), DV(ctx, M * N_)
    N.check(L().strictb200_gemm_bf16(ctx.h, M, N_, K, dx.p, dw.p, dy.p, 1))
    got = dy.to_host().reshape(M, N_)
    # exact products; at most one cut-off (2^-23) per product instruction and per addition of the warps' sums, of the sum of the magnitudes
    assert (np.abs(got - want) <= (K / 16 + 8) * 2.0 ** -23 * size).all()
    N.check(L().strictb200_gemm_bf16(ctx.h, M, N_, K, dx.p, dw.p, dy.p, 0))
    half = dy.to_host().view(np.uint16)[:M * N_].reshape(M, N_)
    assert np.array_equal(half, oracle.f32_to_bf16(got).reshape(M, N_))
    for v in (dx, dw, dy):
        v.free()


# the same of E4M3 weights: loads of 64 columns, 1024 columns per block, sums of several blocks per output
@pytest.mark.parametrize("M,N_,K", [(1, 16, 64), (8, 48, 192), (9, 32, 1088), (16, 1024, 2048), (5, 1600, 4160), (8, 15984, 512), (13, 7600, 1024), (16, 9472, 128), (9, 9488, 128),
                                    (3, 768, 14336), (4, 1024, 3072), (16, 2080, 4096)])
def test_gemm_fp8_few_rows(ctx, oracle, rng, M, N_, K):
    import torch
    x = oracle.round_bf16((rng.standard_normal((M, K)) * np.exp2(rng.integers(-12, 3, (M, K)))).astype(np.float32))
    q, s = oracle.split_rows_device_layout(x)
    wq = rng.integers(0, 256, (N_, K)).astype(np.uint8)
    wq[(wq & 127) == 127] = 0  # no NaN
    f64 = lambda a: torch.from_numpy(a).view(torch.float8_e4m3fn).to(torch.float64).numpy()  # noqa: E731
    terms = f64(q.reshape(-1, K)).reshape(-1, 2, 8, K)
    xs = (terms[:, 0] + terms[:, 1] / 16).reshape(-1, K)[:M] * s[:, None].astype(np.float64)
    sw = rng.uniform(0.5, 2, N_).astype(np.float32)
    w = f64(wq)
    want, size = xs @ w.T * sw, np.abs(xs) @ np.abs(w).T * sw
    dq, ds, dw, dsw, dy = DV.of(ctx, q), DV.of(ctx, s), DV.of(ctx, wq), DV.of(ctx, sw), DV(ctx, M * N_)
    N.check(L().strictb200_gemm_fp8(ctx.h, M, N_, K, dq.p, ds.p, dw.p, dsw.p, dy.p, 1, 0))
    got = dy.to_host().reshape(M, N_)
    # as above, eight more additions between blocks and the two scales
    assert (np.abs(got - want) <= (K / 16 + 18) * 2.0 ** -23 * size).all()
    for v in (dq, ds, dw, dsw, dy):
        v.free()


# one and two groups of 8 sequences and one beyond them; feed-forwards that end inside a block of 16 channel pairs' run of columns, rows wider than
# the 1024 columns a block holds; with the weights' loads behind the dependency wait
@pytest.mark.parametrize("B,over,prefetch", [(1, {}, 1), (8, dict(d_ff=192), 1), (9, dict(d_ff=320), 1), (16, dict(d_model=1152, d_ff=1216), 1), (17, dict(d_ff=192), 1),
                                             (3, dict(d_ff=320), 0)])
def test_decode_of_few_rows_vs_oracle(ctx, oracle, B, over, prefetch):
    cfg = dict(TINY_QWEN, n_layers=2, vocab=512, **over)
    with ctx.option("prefetch", prefetch):
        m, om, kv, st, _, logits, want = _run_pair(ctx, oracle, cfg, 5, B, 12, [12 - i % 5 for i in range(B)], 4, random_gains=True)
        for _ in range(3):
            ok, mx, rel = logits_close(logits, want, **TOL_FP8)
            assert ok, (mx, rel)
            ids = oracle.argmax(want)
            _, logits = kv.decode_step(ids, want_logits=True)
            want = st.decode(ids)
        ok, mx, rel = logits_close(logits, want, **TOL_FP8)
        assert ok, (mx, rel)
    for o in (kv, m):
        o.dispose()
    st.close(), om.close()


# weights that the call in front has just written, again and again in the same place, through the row split and the product's early loads
@pytest.mark.parametrize("M,N_,K", [(1, 4096, 1024), (16, 1024, 4096), (100, 4096, 2048)])
def test_weights_written_just_before(ctx, oracle, rng, M, N_, K):
    x = oracle.round_bf16(rng.standard_normal((M, K)).astype(np.float32))
    sources = [(rng.standard_normal((N_, K)) * 0.05).astype(np.float32) for _ in range(2)]
    dx, dw, ds = DV.of(ctx, oracle.f32_to_bf16(x)), DV(ctx, N_ * K, np.int8), DV(ctx, N_)
    df, dy = [DV.of(ctx, w) for w in sources], [DV(ctx, M * N_, np.uint16) for _ in range(8)]
    for i, y in enumerate(dy):
        N.check(L().strictb200_quantize_weights_int8(ctx.h, df[i % 2].p, N_, K, dw.p, ds.p))
        N.check(L().strictb200_gemm_int8w(ctx.h, M, N_, K, dx.p, dw.p, ds.p, y.p))
    for j, w in enumerate(sources):
        want = oracle.gemm_int8w(x, *oracle.quantize_weights_int8(w))
        for y in dy[j::2]:
            assert np.array_equal(y.to_host().reshape(M, N_), want)
    for v in (dx, dw, ds, *df, *dy):
        v.free()
