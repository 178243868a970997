// The two products of a decode step's few rows (at most 16, at most 1024 wide, E4M3 weights) that meet the residual stream, each with the row
// work around it, so that a layer is a chain of products and attention without row kernels in between:
//   norm_rows_kernel      norm of the residual rows in front of the product: Y = norm(x) . W^T
//   residual_rows_kernel  finished product added to the residual rows: x += (Y . W^T) * sw
// What bounds a step of such sizes is the number of dependent launches (each costs 1.0 to 1.5 us between one kernel's last block and the next
// one's wait, and a round trip or two to L2), not the weights, which wait in registers before the dependency wait (see gemm_rows.cu). The
// rows enter as bf16 and the weights become bf16 (both exact), so there is no row maximum, no split into E4M3 terms and no launch for them.
//
// norm_rows_kernel: every block norms all rows itself (4 KB a row from L2, a warp per row), which is less than a launch for it. Channels and
// columns of a block as in gemm_rows.cu: 32 channels, eight warps share the columns.
//
// residual_rows_kernel: the residual can only be written where a sum is whole, so a block walks all columns of 8 channels (X is the 16-row operand
// of mma.sync, the weights the 8-column one): 128 blocks for a width of 1024, eight warps share the columns, no partial results in memory.
//
// Two things decide whether this is faster than the launches it replaces. Registers: the blocks of a kernel must fit beside those of the kernel
// in front, or their weights are requested only when those have left (then every product takes 1.5 us more). And code: a launch executes every
// instruction once or twice and fetches it cold, 4 to 5 cycles each; the norm with twice the instructions took 2.3 us after the wait, now 1.0.
#include <cuda_fp16.h>

#include "common.cuh"

namespace {
constexpr int TILE = 32;     // channels of a block of norm_rows_kernel
constexpr int MAX_D = 1024;  // widest row that is normed in front of a product: eight float4 per lane of a warp
constexpr int WARPS = 8;
constexpr int COLS = 16, STEP = 4 * COLS, WORDS = 8;  // columns of a thread's load of a weight row and of a warp's; words of a load as bf16 operands
constexpr int AHEAD = MAX_D / (WARPS * STEP);         // loads per weight row that a thread of norm_rows_kernel holds

__device__ __forceinline__ void mma16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  uint32_t v;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(hi), "f"(lo));
  return v;
}
// Sixteen E4M3 values -> bf16 pairs (exact).
__device__ __forceinline__ void operands(const uint4& u, uint32_t* o) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    uint32_t h[2];
    asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, lo;\n\tcvt.rn.f16x2.e4m3x2 %1, hi;\n\t}" : "=r"(h[0]), "=r"(h[1]) : "r"(w[i]));
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const float2 f = __half22float2(*(const __half2*)&h[j]);
      o[2 * i + j] = pack2(f.x, f.y);
    }
  }
}

struct NormRowsArgs {
  const float* x;      // [M, K]
  const float* gain;   // [K]
  float eps;
  const uint8_t* w;    // [N, K]
  int M, N, K, prefetch;
  const float* sw;     // GLU: scales of the channels
  float* out;          // [M, N] sums
  bf16* out_glu;       // GLU, w = [gate | up]: [M, N / 2]
  float* ones;         // [M] = 1, the scales of rows that were not scaled (may be null)
};

// bytes between the rows of the operand in shared memory: the 16-byte reads of a fragment's four columns and eight rows in all banks
__host__ __device__ constexpr int row_bytes(int K) { return 2 * K + 16; }

// NT: groups of 8 rows of X. GLU: 16 channels of each half of w. (24 of each, 128 blocks instead of 192 for 3072, so that all are resident early, needed
// 160 registers a thread and gained nothing: 476 us a step instead of 465.)
template <int NT, bool GLU>
__global__ void __launch_bounds__(32 * WARPS, 2) norm_rows_kernel(NormRowsArgs a) {
  extern __shared__ __align__(16) uint8_t rows[];
  __shared__ float red[WARPS][8 * NT][TILE + 4];
  __shared__ __align__(16) float gain_s[MAX_D];
  SB_TRACE_BEGIN();
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * (GLU ? TILE / 2 : TILE), half = a.N / 2;
  const int steps = a.K / STEP, s0 = warp * steps / WARPS, s1 = (warp + 1) * steps / WARPS;
  const int ldx = row_bytes(a.K);
  const uint8_t* wr = a.w + (int64_t)(n0 + g) * a.K + COLS * t;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint32_t w[AHEAD][4][WORDS];
  if (!a.prefetch) pdl_wait();
  {
    uint4 raw[AHEAD][4];
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int row = GLU ? (r >> 1) * half + 8 * (r & 1) : 8 * r;  // from the thread's first
        const bool in = GLU ? n0 + g + 8 * (r & 1) < half : n0 + g + row < a.N;
        raw[i][r] = s0 + i < s1 && in ? __ldcs((const uint4*)(wr + (int64_t)row * a.K + (s0 + i) * STEP)) : zero;
      }
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int r = 0; r < 4; r++) operands(raw[i][r], w[i][r]);
  }
  for (int k = threadIdx.x; 4 * k < a.K; k += 32 * WARPS) ((float4*)gain_s)[k] = ((const float4*)a.gain)[k];
  __syncthreads();
  pdl_wait();
  SB_TRACE_WAITED();
  const int chunks = a.K >> 7;
#pragma unroll 1
  for (int m = warp; m < a.M; m += WARPS) {  // a warp per row
    const float* xr = a.x + (int64_t)m * a.K + 4 * lane;
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = i < chunks ? __ldcg((const float4*)(xr + 128 * i)) : make_float4(0.f, 0.f, 0.f, 0.f);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) ss += fmaf(v[i].x, v[i].x, v[i].y * v[i].y) + fmaf(v[i].z, v[i].z, v[i].w * v[i].w);
    const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(warp_sum(ss), (float)a.K), a.eps)));
    uint8_t* row = rows + m * ldx + 8 * lane;
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (i < chunks) {
        const float4 gk = *(const float4*)(gain_s + 128 * i + 4 * lane);
        *(uint2*)(row + 256 * i) = make_uint2(pack2(__fmul_rn(__fmul_rn(v[i].x, r), gk.x), __fmul_rn(__fmul_rn(v[i].y, r), gk.y)),
                                              pack2(__fmul_rn(__fmul_rn(v[i].z, r), gk.z), __fmul_rn(__fmul_rn(v[i].w, r), gk.w)));
      }
  }
  __syncthreads();
  SB_TRACE_MARK(0);
  float acc[2][NT][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < NT; j++) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
#pragma unroll
  for (int i = 0; i < AHEAD; i++)
#pragma unroll
    for (int j = 0; j < NT; j++) {
      const int m = g + 8 * j;
      const bool in = s0 + i < s1 && m < a.M;
#pragma unroll
      for (int e = 0; e < WORDS; e += 4) {
        const uint4 x = in ? *(const uint4*)(rows + m * ldx + 2 * ((s0 + i) * STEP + COLS * t) + 4 * e) : zero;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          mma16816(acc[h][j], w[i][2 * h][e], w[i][2 * h + 1][e], w[i][2 * h][e + 1], w[i][2 * h + 1][e + 1], x.x, x.y);
          mma16816(acc[h][j], w[i][2 * h][e + 2], w[i][2 * h + 1][e + 2], w[i][2 * h][e + 3], w[i][2 * h + 1][e + 3], x.z, x.w);
        }
      }
    }
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) red[warp][8 * j + 2 * t + (e & 1)][16 * h + g + 8 * (e >> 1)] = acc[h][j][e];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NT; j++) {
    const int m = 8 * j + warp;
    if (m >= a.M) continue;
    float v = red[0][m][lane];
#pragma unroll
    for (int i = 1; i < WARPS; i++) v += red[i][m][lane];
    if constexpr (GLU) {  // lanes 0..15 hold the gates, the others the up values of the same channels
      const int n = (lane >> 4) * half + n0 + (lane & 15);
      const bool in = n0 + (lane & 15) < half;
      v = in ? __fmul_rn(v, a.sw[n]) : 0.f;
      const float up = __shfl_down_sync(0xffffffffu, v, 16);
      if (lane < 16 && in) a.out_glu[(int64_t)m * half + n] = __float2bfloat16_rn(sb_silu_mul(v, up));
    } else if (n0 + lane < a.N) {
      a.out[(int64_t)m * a.N + n0 + lane] = v;
    }
  }
  if (a.ones && blockIdx.x == 0 && (int)threadIdx.x < a.M) a.ones[threadIdx.x] = 1.f;
  SB_TRACE_END(SB_K_GEMM, (uint32_t)a.N ^ ((uint32_t)a.K << 12));
}

struct ResidualRowsArgs {
  const bf16* x;     // [M, K]
  const uint8_t* w;  // [N, K]
  const float* sw;   // [N]
  float* res;        // [M, N], in and out
  int M, N, K, prefetch;
};

// NT: groups of 8 rows. STEPS: 64-byte steps along K per warp, all of whose weights are in registers before the dependency wait. The rows of X come
// straight into registers (through private places in shared memory by cp.async they took 4.1 us instead of 1.2).
template <int NT, int STEPS>
__global__ void __launch_bounds__(32 * WARPS, 2) residual_rows_kernel(ResidualRowsArgs a) {
  constexpr int XS = NT * STEPS <= 4 ? STEPS : NT == 1 ? (STEPS + 1) / 2 : 2;  // steps whose rows are in flight at once
  __shared__ float red[WARPS][8 * NT][9];
  SB_TRACE_BEGIN();
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * 8;
  const int steps = (a.K + STEP - 1) / STEP, s0 = warp * steps / WARPS, s1 = (warp + 1) * steps / WARPS;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const uint8_t* wr = a.w + (int64_t)(n0 + g) * a.K + COLS * t;
  uint32_t w[STEPS][WORDS];
  if (!a.prefetch) pdl_wait();
  {
    uint4 raw[STEPS];
#pragma unroll
    for (int i = 0; i < STEPS; i++) {
      const int k = (s0 + i) * STEP;
      raw[i] = s0 + i < s1 && k + COLS * t < a.K && n0 + g < a.N ? __ldcs((const uint4*)(wr + k)) : zero;
    }
#pragma unroll
    for (int i = 0; i < STEPS; i++) operands(raw[i], w[i]);
  }
  // the thread's output in the end
  const int om = threadIdx.x >> 3, on = n0 + (threadIdx.x & 7);
  const bool out = om < a.M && om < 8 * NT && on < a.N;
  const float scale = out ? a.sw[on] : 0.f;
  pdl_wait();
  SB_TRACE_WAITED();
  float old = 0.f;
  float acc[2][4];  // alternating sums
#pragma unroll
  for (int i = 0; i < 4; i++) acc[0][i] = acc[1][i] = 0.f;
  const bf16* xr = a.x + (int64_t)g * a.K + COLS * t;
#pragma unroll
  for (int i0 = 0; i0 < STEPS; i0 += XS) {
    uint4 x[XS][NT][2];
#pragma unroll
    for (int i = 0; i < XS; i++)
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int k = (s0 + i0 + i) * STEP;
          const bool in = i0 + i < STEPS && s0 + i0 + i < s1 && k + COLS * t < a.K && g + 8 * j < a.M;
          x[i][j][e] = in ? __ldcg((const uint4*)(xr + (int64_t)(8 * j) * a.K + k + 8 * e)) : zero;
        }
    if (i0 == 0 && out) old = __ldcg(a.res + (int64_t)om * a.N + on);
#pragma unroll
    for (int i = 0; i < XS; i++) {
      if (i0 + i >= STEPS) break;
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const uint4 p = x[i][0][e], q = NT > 1 ? x[i][NT - 1][e] : zero;
        const uint32_t* b = w[i0 + i] + 4 * e;
        mma16816(acc[0], p.x, q.x, p.y, q.y, b[0], b[1]);
        mma16816(acc[1], p.z, q.z, p.w, q.w, b[2], b[3]);
      }
    }
  }
  SB_TRACE_MARK(0);
#pragma unroll
  for (int e = 0; e < 2 * NT; e++) red[warp][g + 8 * (e >> 1)][2 * t + (e & 1)] = acc[0][e] + acc[1][e];
  __syncthreads();
  if (out) {
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < WARPS; j++) v += red[j][om][on - n0];
    a.res[(int64_t)om * a.N + on] = __fadd_rn(old, __fmul_rn(v, scale));
  }
  SB_TRACE_END(SB_K_GEMM, (uint32_t)a.N ^ ((uint32_t)a.K << 12));
}

template <int NT, bool GLU>
int launch_norm(strictb200_ctx* ctx, const NormRowsArgs& a) {
  const size_t smem = (size_t)8 * NT * row_bytes(MAX_D);
  static SbDeviceOnce once;  // one per instantiation
  auto kernel = norm_rows_kernel<NT, GLU>;
  SB_CUDA(once.run(ctx->device, [&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }));
  const int ch = GLU ? TILE / 2 : TILE, n = GLU ? a.N / 2 : a.N;
  SB_CUDA(sb_launch(ctx, kernel, dim3((unsigned)((n + ch - 1) / ch)), dim3(32 * WARPS), smem, a));
  ctx->launches++;
  return STRICTB200_OK;
}
template <int STEPS>
int launch_residual(strictb200_ctx* ctx, const ResidualRowsArgs& a) {
  const dim3 grid((unsigned)((a.N + 7) / 8)), block(32 * WARPS);
  SB_CUDA(a.M <= 8 ? sb_launch(ctx, residual_rows_kernel<1, STEPS>, grid, block, 0, a) : sb_launch(ctx, residual_rows_kernel<2, STEPS>, grid, block, 0, a));
  ctx->launches++;
  return STRICTB200_OK;
}
}  // namespace

SB_TRACE_TU(gemm_rows_chain)

// Decode steps of Qwen3-0.6B, us, with 8 launches per layer (row norms, merge of the key chunks) and with the 5 of the chain, sequences x keys:
//   1 x 40  646 -> 470    4 x 40  681 -> 502    8 x 40  693 -> 557    12 x 40  828 -> 675    16 x 40  861 -> 772
//   1 x 2000  844 -> 655    4 x 2000  872 -> 741    8 x 512  755 -> 658    8 x 2000  952 -> 887    16 x 512  998 -> 896
// The gain shrinks with the rows, which every block reads: 32 KB of residual for 8, 64 KB for 16. bf16 weights do not come here: they are twice the
// registers, so that the next kernel's blocks wait (8192 to 14336 channels of 1024: 7 to 12 us with the norm in front, 6.9 as two launches; 1024
// channels of 5120: 5.3 us in whole blocks against 2.3 in K splits).
// Rows of at most 1024 columns, and channels whose blocks are all resident at once.
bool sb_norm_rows_takes(int64_t M, int64_t N, int64_t K) { return M >= 1 && M <= 16 && K <= MAX_D && K % 128 == 0 && N <= 2 * SB_SMS * TILE; }
// Columns whose weights eight warps hold, and channels that are one round of blocks.
bool sb_residual_rows_takes(int64_t M, int64_t N, int64_t K) { return M >= 1 && M <= 16 && N <= 8 * SB_SMS && K % 16 == 0 && K <= 8 * WARPS * STEP; }

int k_norm_rows(strictb200_ctx* ctx, const NormRowsGemm& g) {
  if (!sb_norm_rows_takes(g.M, g.N, g.K) || (g.out_glu && g.N % 2)) return sb_fail(STRICTB200_ERR_UNSUPPORTED, "norm_rows: shape");
  const NormRowsArgs a{g.x, g.gain, g.eps, g.w, (int)g.M, (int)g.N, (int)g.K, ctx->opt.prefetch, g.sw, g.out, g.out_glu, g.ones};
  if (g.out_glu) return g.M <= 8 ? launch_norm<1, true>(ctx, a) : launch_norm<2, true>(ctx, a);
  return g.M <= 8 ? launch_norm<1, false>(ctx, a) : launch_norm<2, false>(ctx, a);
}
int k_residual_rows(strictb200_ctx* ctx, const ResidualRowsGemm& g) {
  if (!sb_residual_rows_takes(g.M, g.N, g.K)) return sb_fail(STRICTB200_ERR_UNSUPPORTED, "residual_rows: shape");
  const ResidualRowsArgs a{g.x, g.w, g.sw, g.res, (int)g.M, (int)g.N, (int)g.K, ctx->opt.prefetch};
  return g.K <= 4 * STEP * WARPS ? launch_residual<4>(ctx, a) : g.K <= 6 * STEP * WARPS ? launch_residual<6>(ctx, a) : launch_residual<8>(ctx, a);
}
