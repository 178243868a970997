// bf16 linear layers of a decode step's few rows: Y[M,N] = X[M,K] . W[N,K]^T with at most 16 rows of X.
//
// Bound by the stream over W, and in the chain of a decode step by what lies between the dependency wait and the last store. A tile of
// 128 channels per block (gemm_tmem_split.cu) leaves 8 to 64 blocks for the 1024 channels of an output product, each of which pulls its
// part of W through one SM. Here a block owns 32 channels and up to 1024 columns: its eight warps share the columns, and every weight a
// thread will multiply is in its registers before the wait (four 128-bit loads per 32 channels x 32 columns). Then one round trip for the
// rows of X, mma.sync, and the warps' sums meet in shared memory. A thread's eight consecutive columns of a row serve as the fragments
// of two products (the columns of a fragment may come in any order as long as W and X agree), so no operand passes shared memory.
// The legacy tensor path is enough: one product of 32 channels x 16 columns per 1 KB of weights.
// Where such blocks would not all be resident (two per SM hold 19 MB in registers) a block takes a second tile of 32 channels, whose weights
// wait in shared memory, each thread's own where it put them: 38 MB are on their way before the wait.
#include "common.cuh"

namespace {
constexpr int TILE = 32;     // channels per block
constexpr int WARPS = 8;
constexpr int STEP = 32;     // columns per load
constexpr int AHEAD = 4;     // steps whose weights a warp holds at a time

struct RowsArgs {
  const bf16 *x, *w;
  int64_t ldx, ldw;
  int M, N, K, splits;
  int kb_switch, splits0;       // in units of 64 columns, as in GemmBf16Args::k_switch
  int n_switch, x_row_off;      // rows of x of the channels from n_switch on (n_switch 0: all read the first rows)
  int group_n;
  int64_t group_k;
  float* part;                  // [splits][M, N], or a finished output
  float* out_f32;
  bf16* out_bf16;
  int64_t ldo;
};

__device__ __forceinline__ void mma_rows(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: groups of 8 rows of X. TWO: a second tile of channels, through shared memory (for at most AHEAD steps per warp).
template <int NT, bool TWO>
__global__ void __launch_bounds__(32 * WARPS, 2) gemm_rows_kernel(RowsArgs a) {
  constexpr int TILES = TWO ? 2 : 1, CH = TILES * TILE;
  extern __shared__ __align__(16) uint4 second[];  // [AHEAD * 4][threads]
  __shared__ float red[WARPS][8 * NT][CH + 4];     // the fragments of a warp in 32 banks
  SB_TRACE_BEGIN();
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * CH, z = blockIdx.y;
  const int units = (a.K + 63) / 64;
  int u0, u1;  // this block's columns, in units of 64
  if (a.splits0 > 0) {
    const bool first = z < a.splits0;
    const int base = first ? 0 : a.kb_switch, count = first ? a.kb_switch : units - a.kb_switch;
    const int i = first ? z : z - a.splits0, n = first ? a.splits0 : a.splits - a.splits0;
    u0 = base + (int)((int64_t)i * count / n);
    u1 = base + (int)((int64_t)(i + 1) * count / n);
  } else {
    u0 = (int)((int64_t)z * units / a.splits);
    u1 = (int)((int64_t)(z + 1) * units / a.splits);
  }
  // the warp's columns, in steps of 32
  const int steps_all = 2 * (u1 - u0), s0 = 2 * u0 + warp * steps_all / WARPS, s1 = 2 * u0 + (warp + 1) * steps_all / WARPS;
  const bf16* wr = a.w + (int64_t)(n0 + g) * a.ldw + 8 * t;
  const int64_t xk = a.group_n > 0 ? n0 / a.group_n * a.group_k : 0;
  const bf16* xr = a.x + (int64_t)((a.n_switch > 0 && n0 >= a.n_switch ? a.x_row_off : 0) + g) * a.ldx + xk + 8 * t;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint4 w[AHEAD][4], x[AHEAD][NT];
  auto load_w = [&](int s) {
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int k = (s + i) * STEP;
        w[i][r] = s + i < s1 && k + 8 * t < a.K && n0 + g + 8 * r < a.N ? __ldcs((const uint4*)(wr + (int64_t)(8 * r) * a.ldw + k)) : zero;
      }
  };
  load_w(s0);  // weights are constants
  if constexpr (TWO) {
    const uint64_t once = l2_evict_first_policy();
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int k = (s0 + i) * STEP;
        const bool in = s0 + i < s1 && k + 8 * t < a.K && n0 + TILE + g + 8 * r < a.N;
        const bf16* from = in ? wr + (int64_t)(TILE + 8 * r) * a.ldw + k : a.w;
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(second + (i * 4 + r) * 32 * WARPS + threadIdx.x);
        asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;" ::"r"(to), "l"(from), "r"(in ? 16 : 0), "l"(once) : "memory");
      }
  }
  pdl_wait();
  SB_TRACE_WAITED();
  float acc[2 * TILES][NT][4];
#pragma unroll
  for (int i = 0; i < 2 * TILES; i++)
#pragma unroll
    for (int j = 0; j < NT; j++) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
  auto multiply = [&](int tile) {
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          float* c = acc[2 * tile + h][j];
          mma_rows(c, w[i][2 * h].x, w[i][2 * h + 1].x, w[i][2 * h].y, w[i][2 * h + 1].y, x[i][j].x, x[i][j].y);
          mma_rows(c, w[i][2 * h].z, w[i][2 * h + 1].z, w[i][2 * h].w, w[i][2 * h + 1].w, x[i][j].z, x[i][j].w);
        }
  };
  for (int s = s0; s < s1; s += AHEAD) {
    if (s > s0) load_w(s);
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int j = 0; j < NT; j++) {
        const int k = (s + i) * STEP;
        x[i][j] = s + i < s1 && k + 8 * t < a.K && g + 8 * j < a.M ? __ldcg((const uint4*)(xr + (int64_t)(8 * j) * a.ldx + k)) : zero;
      }
    multiply(0);
    if constexpr (TWO) {
      asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
      for (int i = 0; i < AHEAD; i++)
#pragma unroll
        for (int r = 0; r < 4; r++) w[i][r] = second[(i * 4 + r) * 32 * WARPS + threadIdx.x];
      multiply(1);
    }
  }
#pragma unroll
  for (int h = 0; h < 2 * TILES; h++)
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) red[warp][8 * j + 2 * t + (e & 1)][16 * h + g + 8 * (e >> 1)] = acc[h][j][e];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TILES * NT; i++) {
    const int m = 8 * (i / TILES) + warp, c = i % TILES * TILE + lane, n = n0 + c;
    if (m >= a.M || n >= a.N) continue;
    float v = red[0][m][c];
#pragma unroll
    for (int j = 1; j < WARPS; j++) v += red[j][m][c];
    if (a.part) a.part[((int64_t)z * a.M + m) * a.N + n] = v;
    else if (a.out_f32) a.out_f32[m * a.ldo + n] = v;
    else a.out_bf16[m * a.ldo + n] = __float2bfloat16_rn(v);
  }
  SB_TRACE_END(SB_K_GEMM, (uint32_t)a.N ^ ((uint32_t)a.K << 12));
}

template <int NT, bool TWO>
int launch(strictb200_ctx* ctx, const RowsArgs& a) {
  constexpr size_t smem = TWO ? AHEAD * 4 * 32 * WARPS * sizeof(uint4) : 0;
  static SbDeviceOnce once;  // one per instantiation
  if (TWO) SB_CUDA(once.run(ctx->device, [&] { return cudaFuncSetAttribute(gemm_rows_kernel<NT, TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }));
  const int ch = TWO ? 2 * TILE : TILE;
  SB_CUDA(sb_launch(ctx, gemm_rows_kernel<NT, TWO>, dim3((unsigned)((a.N + ch - 1) / ch), (unsigned)a.splits), dim3(32 * WARPS), smem, a));
  ctx->launches++;
  return STRICTB200_OK;
}
}  // namespace

SB_TRACE_TU(gemm_rows)

// Linear layers of 1 / 8 / 16 rows, us, the 128-channel tiles in front (weights from HBM):
//   N 1024  K 1024   7.4 / 7.6 / 7.4  ->  5.5 / 4.0 / 4.0        N 14336 K 1024    9.1 /  9.2 /  9.3  ->  5.9 /  6.2 /  9.1
//   N 4096  K 1024   7.6 / 7.6 / 7.6  ->  4.0 / 4.1 / 4.0        N 4096  K 4096   21.3 / 21.3 / 21.3  ->  9.1 /  9.2 / 12.6
//   N 1024  K 5120  25.5 / 25.6 / 25.6 -> 8.6 / 8.7 / 11.3       N 14336 K 4096   23.2 / 23.0 / 23.1, beyond what the blocks hold ahead
// and error against 64 bits (K 1024 / 5120): 9.8e-7 / 5.6e-6 there (tcgen05 cuts off after every instruction), 1.3e-7 / 6.0e-7 here.
// A decode step of 8 sequences (28 layers of latent attention, 1024 wide): 926 -> 763 us.
bool sb_gemm_rows_takes(int64_t M, int64_t N, int64_t K) { return M <= 16 && K % 8 == 0 && N * K <= (16 << 20); }
int sb_gemm_rows_splits(strictb200_ctx* ctx, int64_t N, int64_t K) {
  const int64_t tiles = (N + TILE - 1) / TILE, units = (K + 63) / 64;
  int64_t s = (K + STEP * AHEAD * WARPS - 1) / (STEP * AHEAD * WARPS);             // every weight in registers before the wait
  s = std::max(s, std::min((int64_t)ctx->sm_count / tiles, units / 4));           // a block per SM, while a warp has a step
  return (int)std::max<int64_t>(1, std::min<int64_t>(s, 8));                       // eight results are what the consumers take
}
int k_gemm_rows_bf16(strictb200_ctx* ctx, const GemmBf16Args& b) {
  const RowsArgs a{b.x, b.w, b.ldx, b.ldw, (int)b.M, (int)b.N, (int)b.K, b.splits, (int)(b.k_switch / 64), b.k_switch ? b.splits0 : 0,
                   b.e.n_switch, b.e.x_row_off, b.group_n, b.group_k, b.part, b.e.out_f32, b.e.out_bf16, b.e.ldo};
  // longest run of columns a block gets, in units of 64
  const int64_t units = (b.K + 63) / 64, u0 = b.k_switch ? b.k_switch / 64 : 0;
  const int64_t run = b.k_switch ? std::max((u0 + b.splits0 - 1) / b.splits0, (units - u0 + b.splits - b.splits0 - 1) / (b.splits - b.splits0)) : (units + b.splits - 1) / b.splits;
  const bool two = (b.N + TILE - 1) / TILE * b.splits > 2 * (int64_t)ctx->sm_count && 2 * run <= AHEAD * WARPS;
  if (b.M <= 8) return two ? launch<1, true>(ctx, a) : launch<1, false>(ctx, a);
  return two ? launch<2, true>(ctx, a) : launch<2, false>(ctx, a);
}
