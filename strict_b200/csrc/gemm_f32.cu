// fp32 linear layer of the GPT-2 path: Y[M,N] = X[M,K] . W[N,K]^T + bias. Decode (M = 1) is
// a pure HBM stream over W; one warp (or 2-8 for a long row) per output channel or two, lanes split K with 128-bit loads,
// warp-shuffle reduction. With ln_gain the rows of X are layer-normed on the way in, by every block for itself (3 KB from L2
// against a launch of its own). Up to 8 token rows share one pass over a weight row. `accumulate`: 0
// stores the result, 1 adds it to Y (residual), 2 stores GELU(result) (the MLP's first layer), 3 xIELU(result), 4 adds
// alpha * col_scale[n] * result to Y.
// Rows of X, W and Y may be wider than the product (ldx, ldw, ldy).
#include "common.cuh"

int k_gemm_f32_tc(strictb200_ctx* ctx, const GemmF32Args& g);    // gemm_f32_tc.cu
int k_gemm_f32_pair(strictb200_ctx* ctx, const GemmF32Args& g);  // gemm_f32_pair.cu

namespace {
constexpr int F32_MT = 8;
constexpr int F32_PRE = 8;   // float4 of a weight row a lane fetches before the dependency wait, at most (a slice of at most 1024 columns)
constexpr int LN_K = 1024;   // widest row the layer norm in front of the product takes
constexpr size_t X_SMEM = 96 * 1024;

// Sum over the lanes of each of the n values (n a power of two, at most 16): the halves of the values change sides as the lanes are
// folded, n - 1 + log2(32 / n) shuffles instead of 5 n. Lane l returns the sum of the value whose index is the top log2(n) bits of l.
template <int n, int o = 16>
__device__ __forceinline__ float fold_sums(float* v, int lane) {
  if constexpr (n > 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n / 2; i++) {
      const float send = up ? v[i] : v[n / 2 + i], keep = up ? v[n / 2 + i] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
    return fold_sums<n / 2, o / 2>(v, lane);
  } else if constexpr (o > 0) {
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return fold_sums<1, o / 2>(v, lane);
  } else {
    return v[0];
  }
}

// MT rows at most, NC channels per warp. The block's 8 warps are 8/ks groups of NC channels x ks slices of K: a long row is walked by
// several warps at once so that every lane has all its weight loads in flight in one round trip; the slices' sums meet in shared
// memory and are added in slice order. STAGED: the rows of X (or their layer norm, LN) are in shared memory. X is read from L2 and is
// not declared invariant: loads of invariant data may be moved in front of the dependency wait.
// PRE: float4 of a weight row that a lane holds, as many as its slice has where that is less than F32_PRE (one row of X). The weights in
// flight are registers, and the blocks of the next kernel can only request theirs beside these, so a block takes what it needs and no more:
// with F32_PRE for all, 128 registers, the blocks of a GPT-2 step's projections started when those in front had left. The norm in front (LN) is
// that of the whole row, however many warps share the weights: with it PRE holds a row of X.
constexpr int rows_regs(int MT, int NC, bool LN, int PRE) { return MT > 1 || PRE == F32_PRE ? 128 : (40 + 4 * PRE * (NC + (LN ? 1 : 0)) + 7) / 8 * 8; }
template <int MT, int NC, bool STAGED, bool LN, int PRE>
__maxnreg__(rows_regs(MT, NC, LN, PRE)) __global__ void gemm_f32_kernel(int M, int N, int K, const float* x, int64_t ldx, const float* __restrict__ w,
                                                       int64_t ldw, const float* __restrict__ bias, float* y, int64_t ldy, int accumulate, int ks,
                                                       float act_pos, float act_neg, const float* __restrict__ col_scale, float alpha,
                                                       const float* __restrict__ ln_gain, const float* __restrict__ ln_bias, float ln_eps,
                                                       int prefetch) {
  extern __shared__ __align__(16) float xs[];
  constexpr int VALS = NC * MT, STEP = 32 / VALS;
  __shared__ float part[8][VALS];
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = 8 / ks, slice = warp % ks;
  const int n0 = (blockIdx.x * groups + warp / ks) * NC;
  const int m0 = blockIdx.y * MT, mt = min(MT, M - m0);
  const int nk4 = K / 4, per = (nk4 + ks - 1) / ks;
  const int k4_lo = slice * per, k4_hi = min(nk4, k4_lo + per);
  // the weights are constants: the slice streams in while the previous kernel still runs (streaming loads: a step reads its
  // 0.5 GB of weights once each, and they should not push the kernels' code and the activations out of L2)
  if (!prefetch) pdl_wait();
  float4 wpre[NC][PRE];
#pragma unroll
  for (int c = 0; c < NC; c++)
#pragma unroll
    for (int i = 0; i < PRE; i++)
      if (n0 + c < N && k4_lo + lane + 32 * i < k4_hi) wpre[c][i] = __ldcs((const float4*)(w + (int64_t)(n0 + c) * ldw) + k4_lo + lane + 32 * i);
  const float4 *gain = (const float4*)xs + MT * nk4, *shift = gain + nk4;
  if (LN) {
    for (int i = threadIdx.x; i < nk4; i += 256) {
      ((float4*)xs)[MT * nk4 + i] = ((const float4*)ln_gain)[i];
      ((float4*)xs)[(MT + 1) * nk4 + i] = ((const float4*)ln_bias)[i];
    }
    __syncthreads();
  }
  const int oc = n0 + lane;  // lanes that will finish a channel
  const float bn = bias && lane < NC && oc < N ? bias[oc] : 0.f;
  pdl_wait();
  if (LN) {
    if (warp < mt) {  // a warp per row
      const float4* xr = (const float4*)(x + (int64_t)(m0 + warp) * ldx);
      float4 v[PRE];
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < PRE; i++)
        if (lane + 32 * i < nk4) { v[i] = __ldcg(xr + lane + 32 * i); sum += (v[i].x + v[i].y) + (v[i].z + v[i].w); }
      const float mean = __fdiv_rn(warp_sum(sum), (float)K);
      float sq = 0.f;
#pragma unroll
      for (int i = 0; i < PRE; i++)
        if (lane + 32 * i < nk4) {
          v[i].x -= mean; v[i].y -= mean; v[i].z -= mean; v[i].w -= mean;
          sq += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
        }
      const float var = __fdiv_rn(warp_sum(sq), (float)K);
      const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(var, ln_eps)));
#pragma unroll
      for (int i = 0; i < PRE; i++)
        if (lane + 32 * i < nk4) {
          const float4 gn = gain[lane + 32 * i], sh = shift[lane + 32 * i];
          ((float4*)xs)[warp * nk4 + lane + 32 * i] = make_float4(__fadd_rn(__fmul_rn(__fmul_rn(v[i].x, r), gn.x), sh.x), __fadd_rn(__fmul_rn(__fmul_rn(v[i].y, r), gn.y), sh.y),
                                                                  __fadd_rn(__fmul_rn(__fmul_rn(v[i].z, r), gn.z), sh.z), __fadd_rn(__fmul_rn(__fmul_rn(v[i].w, r), gn.w), sh.w));
        }
    }
    __syncthreads();
  } else if (STAGED) {
    for (int i = threadIdx.x; i < mt * nk4; i += 256) ((float4*)xs)[i] = __ldcg((const float4*)(x + (int64_t)(m0 + i / nk4) * ldx) + i % nk4);
    __syncthreads();
  }
  float acc[VALS];
#pragma unroll
  for (int i = 0; i < VALS; i++) acc[i] = 0.f;
  auto fma_rows = [&](int k4, const float4* wv) {
#pragma unroll
    for (int i = 0; i < MT; i++) {
      if (i < mt) {
        const float4 xv = STAGED ? ((const float4*)xs)[i * nk4 + k4] : __ldcg((const float4*)(x + (int64_t)(m0 + i) * ldx) + k4);
#pragma unroll
        for (int c = 0; c < NC; c++) acc[c * MT + i] += wv[c].x * xv.x + wv[c].y * xv.y + wv[c].z * xv.z + wv[c].w * xv.w;
      }
    }
  };
#pragma unroll
  for (int i = 0; i < PRE; i++)
    if (k4_lo + lane + 32 * i < k4_hi) {
      float4 wv[NC];
#pragma unroll
      for (int c = 0; c < NC; c++) wv[c] = n0 + c < N ? wpre[c][i] : make_float4(0.f, 0.f, 0.f, 0.f);
      fma_rows(k4_lo + lane + 32 * i, wv);
    }
#pragma unroll 2
  for (int k4 = k4_lo + lane + 32 * PRE; k4 < k4_hi; k4 += 32) {
    float4 wv[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) wv[c] = n0 + c < N ? __ldcs((const float4*)(w + (int64_t)(n0 + c) * ldw) + k4) : make_float4(0.f, 0.f, 0.f, 0.f);
    fma_rows(k4, wv);
  }
  const float sum = fold_sums<VALS>(acc, lane);
  if (lane % STEP == 0) part[warp][lane / STEP] = sum;
  __syncthreads();
  if (slice == 0 && lane < NC && oc < N) {
    for (int i = 0; i < mt; i++) {
      float v = 0.f;
      for (int s2 = 0; s2 < ks; s2++) v += part[warp + s2][lane * MT + i];
      const int64_t o = (int64_t)(m0 + i) * ldy + oc;
      v += bn;
      if (accumulate == 4) y[o] += alpha * (col_scale ? col_scale[oc] : 1.f) * v;
      else y[o] = accumulate == 1 ? y[o] + v : accumulate == 2 ? sb_gelu_tanh(v) : accumulate == 3 ? sb_xielu(v, act_pos, act_neg) : v;
    }
  }
}

template <int MT, int NC, bool STAGED, bool LN, int PRE = F32_PRE>
int launch_rows(strictb200_ctx* ctx, const GemmF32Args& g, int ks) {
  if (LN && g.K > 128 * PRE) return sb_fail(STRICTB200_ERR_INVALID_ARG, "gemm_f32: the norm in front does not hold its row");
  const int rows = 8 / ks * NC;
  dim3 grid((unsigned)((g.N + rows - 1) / rows), (unsigned)((g.M + MT - 1) / MT));
  if (grid.y > 65535) return sb_fail(STRICTB200_ERR_INVALID_ARG, "gemm_f32: M too large");
  const size_t smem = LN ? (size_t)(MT + 2) * g.K * 4 : STAGED ? (size_t)MT * g.K * 4 : 0;
  static SbDeviceOnce once;  // one per instantiation
  SB_CUDA(once.run(ctx->device, [&] { return cudaFuncSetAttribute(gemm_f32_kernel<MT, NC, STAGED, LN, PRE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)X_SMEM); }));
  SB_CUDA(sb_launch(ctx, gemm_f32_kernel<MT, NC, STAGED, LN, PRE>, grid, dim3(256), smem, (int)g.M, (int)g.N, (int)g.K, g.x, g.ldx, g.w, g.ldw, g.bias, g.y, g.ldy, g.mode, ks,
                    g.act_pos, g.act_neg, g.col_scale, g.alpha, g.ln_gain, g.ln_bias, g.ln_eps, ctx->opt.prefetch));
  ctx->launches++;
  return STRICTB200_OK;
}
template <int MT, int NC>
int launch_rows(strictb200_ctx* ctx, const GemmF32Args& g, int ks) {
  if constexpr (MT == 1) {
    const int64_t pre = ((g.ln_gain ? g.K / 4 : (g.K / 4 + ks - 1) / ks) + 31) / 32;
    if (pre <= 3) return g.ln_gain ? launch_rows<1, NC, true, true, 3>(ctx, g, ks) : launch_rows<1, NC, false, false, 3>(ctx, g, ks);
    if (pre <= 6) return g.ln_gain ? launch_rows<1, NC, true, true, 6>(ctx, g, ks) : launch_rows<1, NC, false, false, 6>(ctx, g, ks);
  }
  if (g.ln_gain) return launch_rows<MT, NC, true, true>(ctx, g, ks);
  // one row is a few loads per lane, straight from L2; several rows would be read once per channel
  if (MT > 1 && (size_t)MT * g.K * 4 <= X_SMEM) return launch_rows<MT, NC, true, false>(ctx, g, ks);
  return launch_rows<MT, NC, false, false>(ctx, g, ks);
}
template <int MT>
int launch_rows(strictb200_ctx* ctx, const GemmF32Args& g, int ks, bool two) {
  return two ? launch_rows<MT, 2>(ctx, g, ks) : launch_rows<MT, 1>(ctx, g, ks);
}
// Many channels of short rows (the LM head) for at most four rows of X: two blocks per SM that stay, a warp walks channels and requests the next one's
// weights before it adds up the current one's. Bound by HBM: 50257 channels of 768, one row, in blocks of sixteen channels that come and go 41 us of a
// GPT-2 step (3.8 TB/s), 26 us so (6 TB/s); four rows 48 -> 42. Sums as in gemm_f32_kernel.
template <int MT, int PRE>
__global__ void __launch_bounds__(256, 2) gemm_f32_stream_kernel(int M, int N, int K, const float* x, int64_t ldx, const float* __restrict__ w, int64_t ldw,
                                                                 const float* __restrict__ bias, float* y, int64_t ldy, int prefetch) {
  extern __shared__ __align__(16) float xs[];
  pdl_trigger();
  const int lane = threadIdx.x & 31, nk4 = K / 4, step = (int)gridDim.x * 8;
  int n = (int)blockIdx.x * 8 + (threadIdx.x >> 5);
  float4 next[PRE];
  auto request = [&](int c) {
#pragma unroll
    for (int i = 0; i < PRE; i++) next[i] = c < N && lane + 32 * i < nk4 ? __ldcs((const float4*)(w + (int64_t)c * ldw) + lane + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  if (!prefetch) pdl_wait();
  request(n);
  pdl_wait();
  for (int i = threadIdx.x; i < M * nk4; i += 256) ((float4*)xs)[i] = __ldcg((const float4*)(x + (int64_t)(i / nk4) * ldx) + i % nk4);
  __syncthreads();
  for (; n < N; n += step) {
    float4 wv[PRE];
#pragma unroll
    for (int i = 0; i < PRE; i++) wv[i] = next[i];
    request(n + step);
    float acc[MT];
#pragma unroll
    for (int m = 0; m < MT; m++) acc[m] = 0.f;
#pragma unroll
    for (int i = 0; i < PRE; i++)
      if (lane + 32 * i < nk4) {
#pragma unroll
        for (int m = 0; m < MT; m++)
          if (m < M) {
            const float4 v = ((const float4*)xs)[m * nk4 + lane + 32 * i];
            acc[m] += wv[i].x * v.x + wv[i].y * v.y + wv[i].z * v.z + wv[i].w * v.w;
          }
      }
    const float sum = fold_sums<MT>(acc, lane);
    const int m = lane / (32 / MT);
    if (lane % (32 / MT) == 0 && m < M) y[(int64_t)m * ldy + n] = bias ? sum + bias[n] : sum;
  }
}
template <int MT>
int launch_stream(strictb200_ctx* ctx, const GemmF32Args& g) {
  auto go = [&](auto kernel) {
    return sb_launch(ctx, kernel, dim3((unsigned)(2 * ctx->sm_count)), dim3(256), (size_t)g.M * g.K * 4, (int)g.M, (int)g.N, (int)g.K, g.x, g.ldx, g.w, g.ldw, g.bias, g.y,
                     g.ldy, ctx->opt.prefetch);
  };
  SB_CUDA(g.K <= 768 ? go(gemm_f32_stream_kernel<MT, 6>) : go(gemm_f32_stream_kernel<MT, 8>));
  ctx->launches++;
  return STRICTB200_OK;
}
}  // namespace

bool sb_gemm_f32_takes_norm(int64_t M, int64_t K) { return M <= F32_MT && K <= LN_K; }

int k_gemm_f32(strictb200_ctx* ctx, int64_t M, int64_t N, int64_t K, const float* x, const float* w, const float* bias, float* y,
               int accumulate) {
  GemmF32Args g;
  g.M = M; g.N = N; g.K = K; g.x = x; g.ldx = K; g.w = w; g.ldw = K; g.bias = bias; g.y = y; g.ldy = N; g.mode = accumulate;
  return k_gemm_f32(ctx, g);
}

int k_gemm_f32(strictb200_ctx* ctx, const GemmF32Args& g) {
  const int64_t M = g.M, N = g.N, K = g.K;
  if (K % 4 || g.ldx % 4 || g.ldw % 4) return sb_fail(STRICTB200_ERR_INVALID_ARG, "gemm_f32: K and the row strides must be multiples of 4");
  if (((uintptr_t)g.x | (uintptr_t)g.w | (uintptr_t)g.ln_gain | (uintptr_t)g.ln_bias) % 16) return sb_fail(STRICTB200_ERR_INVALID_ARG, "gemm_f32: operands must be 16-byte aligned");
  if (g.ln_gain && !sb_gemm_f32_takes_norm(M, K)) return sb_fail(STRICTB200_ERR_INVALID_ARG, "gemm_f32: rows for the layer norm in front are at most 8 of 1024");
  // One pass over the weights per eight rows (this kernel) or per 32 to 128 (the tensor cores). Measured, us, rows = 9 / 16 / 32 / 128 / 4700:
  //   N 768  K 768    7.1 / 7.1 / 13.0 /  37.8 / 1197   against   8.5 / 8.5 /  8.7 / 13.9 /  62
  //   N 3072 K 768   13.2 / 19.8 / 33.1 / 119.8 / 6240            9.3 / 9.3 /  9.5 / 14.9 / 192
  //   N 1000 K 100    4.3 / 4.4 /  6.2 /  19.8 /  676            6.2 / 7.1 /  7.2 / 13.7 /  28
  // so two passes over a small matrix stay here, and five to eight rows over a large one go there (4096 x 4096: 46.8 us against 26.4).
  // Errors against 64 bits (2-norm, normal operands, K 768 / 3072 / 14336): 9.2e-8 / 1.0e-7 / 1.6e-7 here, 7.6e-8..8.7e-8 /
  // 9.6e-8 / 1.3e-7 there.
  const bool few = M <= 4 || (M <= F32_MT && (g.ln_gain || N * K <= (8 << 20))) || (M <= 2 * F32_MT && N * K <= (1 << 20));
  if (!few) {
    const int st = k_gemm_f32_pair(ctx, g);
    return st == STRICTB200_ERR_UNSUPPORTED ? k_gemm_f32_tc(ctx, g) : st;
  }
  // at least eight channels for every warp of two blocks per SM
  if (M <= 4 && g.mode == 0 && !g.ln_gain && K <= LN_K && N >= 8 * 16 * (int64_t)ctx->sm_count) return M == 1 ? launch_stream<1>(ctx, g) : M == 2 ? launch_stream<2>(ctx, g) : launch_stream<4>(ctx, g);
  // Warps per output channel: slices of at most 1024 columns, and two for a long enough row, while all blocks are resident at once (two
  // per SM with the norm in front or several rows, else four); two channels per warp where they would not be. With the norm in front
  // 3072 channels of 768 columns took 6.6 us as 384 blocks of two waves, 3.0 us as 192.
  const int64_t cap = (M == 1 && !g.ln_gain ? 4 : 2) * (int64_t)ctx->sm_count;
  int ks = 1;
  while (ks < 8 && K > 1024 * (int64_t)ks && (N * ks * 2 + 7) / 8 <= 2 * cap) ks *= 2;
  if (ks == 1 && K >= 512 && (N * 2 + 7) / 8 <= cap) ks = 2;
  const bool two = (N * ks + 7) / 8 > cap;
  if (M == 1) return launch_rows<1>(ctx, g, ks, two);
  if (M == 2) return launch_rows<2>(ctx, g, ks, two);
  if (M <= 4) return launch_rows<4>(ctx, g, ks, two);
  return launch_rows<8>(ctx, g, ks, two);
}
