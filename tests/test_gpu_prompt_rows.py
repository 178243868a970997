"""Kernels that only the rows of longer prompts reach: SwiGLU in the product's epilogue, the walk over output tiles, norms, rotations and
splits of whole rows."""
import numpy as np
import pytest

from strict_b200 import native as N
from strict_b200.kernel import DeviceVariable as DV
from conftest import TOL_FP8, logits_close
from test_gpu_models import TINY_QWEN, _run_pair

pytestmark = pytest.mark.gpu
L = N.lib


# feed-forwards that end inside a tile of 128 channels; more than eight token tiles of 128 and an odd rest of them; more than 32 and fewer heads; the
# norm of whole rows (more than 1024 of them, or a width that is no multiple of 128 and takes other products) with one, two, four and
# eight column groups per thread
@pytest.mark.parametrize("over,lens", [(dict(d_ff=192), [100, 77, 40]), (dict(d_ff=320, n_q_heads=36, n_kv_heads=3, head_dim=128), [90, 211]),
                                       (dict(d_model=1152, d_ff=128), [700, 520]), (dict(d_model=4160, d_ff=128), [12, 9]), (dict(d_model=2048, d_ff=256), [1100]),
                                       (dict(d_model=640, d_ff=128), [1030]), (dict(d_model=2176, d_ff=128), [600, 430])],
                         ids=["ff192", "heads42", "d1152", "d4160", "d2048", "d640", "d2176"])
def test_prompts_vs_oracle(ctx, oracle, over, lens):
    cfg = dict(TINY_QWEN, n_layers=2, vocab=512, max_pos=1200, **over)
    m, om, kv, st, _, logits, want = _run_pair(ctx, oracle, cfg, 7, len(lens), max(lens), lens, 1, random_gains=True)
    ok, mx, rel = logits_close(logits, want, **TOL_FP8)
    assert ok, (mx, rel)
    for o in (kv, m):
        o.dispose()
    st.close(), om.close()


@pytest.mark.parametrize("K", [2048, 2064, 4096, 4112, 12288, 12304, 16384])
def test_quantize_rows_widths(ctx, oracle, rng, K):
    M = 9
    x = oracle.round_bf16((rng.standard_normal((M, K)) * rng.uniform(0.01, 30, (M, 1))).astype(np.float32))
    x[2, K - 1] = 300.0  # the largest value in the last column
    dx, dq, ds = DV.of(ctx, oracle.f32_to_bf16(x)), DV(ctx, 32 * K, np.uint8), DV(ctx, M)
    dq.zero()
    N.check(L().strictb200_quantize_rows(ctx.h, dx.p, M, K, dq.p, ds.p))
    q, s = oracle.split_rows_device_layout(x)
    assert np.array_equal(ds.to_host(), s) and np.array_equal(dq.to_host().reshape(32, K), q)
    for v in (dx, dq, ds):
        v.free()


# one, two, four and eight column groups per thread, wider rows, widths that are no multiple of 8
@pytest.mark.parametrize("M,K", [(1, 2048), (9, 2056), (16, 4104), (7, 8200), (3, 16384), (5, 16392), (10, 1028), (2, 13)])
def test_quantize_rows_int8_widths(ctx, oracle, rng, M, K):
    x = oracle.round_bf16((rng.standard_normal((M, K)) * rng.uniform(0.01, 30, (M, 1))).astype(np.float32))
    x[M // 2, K - 1] = 300.0  # the largest value in the last column
    rows = 16 * ((M + 7) // 8)
    dx, dq, ds = DV.of(ctx, oracle.f32_to_bf16(x)), DV(ctx, rows * K, np.int8), DV(ctx, M)
    N.check(L().strictb200_memset(ctx.h, dq.p, 0x55, rows * K))
    N.check(L().strictb200_quantize_rows_int8(ctx.h, dx.p, M, K, dq.p, ds.p))
    hi, lo, s = oracle.quantize_rows_int8(x)
    want = np.zeros((rows // 2, 2, K), np.int8)
    want[:M, 0], want[:M, 1] = hi, lo
    assert np.array_equal(dq.to_host().reshape(rows // 16, 2, 8, K), want.reshape(rows // 16, 8, 2, K).transpose(0, 2, 1, 3))
    assert np.array_equal(ds.to_host(), s)
    for v in (dx, dq, ds):
        v.free()


# tiles of 256 channels and 128 tokens that end inside, more than eight token tiles; sums beyond 32 bits (the last)
@pytest.mark.parametrize("M,N_,K", [(129, 256, 128), (250, 272, 384), (1100, 528, 256), (140, 400, 16384)])
def test_gemm_int8_many_rows_exact(ctx, oracle, rng, M, N_, K):
    x = oracle.round_bf16(rng.standard_normal((M, K)).astype(np.float32))
    wq, sw = rng.integers(-127, 128, (N_, K)).astype(np.int8), rng.uniform(0.01, 1, N_).astype(np.float32)
    if K > 8192:
        x[1], x[2], wq[3] = 5.0, -5.0, 127
    dx, dw, ds, dy = DV.of(ctx, oracle.f32_to_bf16(x)), DV.of(ctx, wq), DV.of(ctx, sw), DV(ctx, M * N_, np.uint16)
    N.check(L().strictb200_gemm_int8w(ctx.h, M, N_, K, dx.p, dw.p, ds.p, dy.p))
    assert np.array_equal(dy.to_host().reshape(M, N_), oracle.gemm_int8w(x, wq, sw))
    for v in (dx, dw, ds, dy):
        v.free()
