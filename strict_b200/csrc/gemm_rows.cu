// Linear layers of a decode step's few rows, bf16 or E4M3 weights: Y[M,N] = X[M,K] . W[N,K]^T with at most 16 rows of X.
//
// Bound by the stream over W, and in the chain of a decode step by what lies between the dependency wait and the last store. A tile of
// 128 channels per block (gemm_tmem_split.cu) leaves 8 to 64 blocks for the 1024 channels of an output product, each of which pulls its
// part of W through one SM. Here a block owns 32 channels and up to 1024 columns: its eight warps share the columns, and every weight a
// thread will multiply is in its registers before the wait (four 128-bit loads per 32 channels x 32 columns). Then one round trip for the
// rows of X, mma.sync, and the warps' sums meet in shared memory. A thread's eight consecutive columns of a row serve as the fragments
// of two products (the columns of a fragment may come in any order as long as W and X agree), so no operand passes shared memory.
// The legacy tensor path is enough: one product of 32 channels x 16 columns per 1 KB of weights.
// Where such blocks would not all be resident (two per SM hold 19 MB in registers) a block takes a second tile of 32 channels, whose weights
// wait in shared memory, each thread's own where it put them: 38 MB are there or on their way before the wait (bf16 only). They come by plain
// loads and stores, so that the form has no instruction that the form of one tile does not have.
// (The two halves of W = [gate | up] of a SwiGLU may share a block, 16 channels of each, which then writes bf16 silu(gate) * up.)
// E4M3: a load is 16 columns. Weights become fp16 pairs, and so does the sum of the two E4M3 terms of X, hi + lo / 16 (both without
// rounding: the sum has at most 9 significant bits down to units of 2^-13), so one product serves both terms. Rows of X that come as
// bf16 are multiplied as they are, by weights that became bf16: no row maximum, no split, no launch for them.
#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"

namespace {
constexpr int TILE = 32;     // channels per block
constexpr int WARPS = 8;
// Loads per weight row that a thread holds at a time; a load of a warp is 64 bytes of a row (a step). E4M3 weights are held as fp16.
constexpr int ahead(bool f8) { return f8 ? 2 : 4; }

struct RowsArgs {
  const void *x, *w;
  int64_t ldx, ldw;             // elements
  int M, N, K, splits;
  int prefetch;                 // load the weights before the dependency wait
  const float *sx, *sw;         // E4M3: scales of the rows of X and of the channels (finished outputs)
  int kb_switch, splits0;       // in units of 64 columns, as in GemmBf16Args::k_switch
  int n_switch, x_row_off;      // rows of x of the channels from n_switch on (n_switch 0: all read the first rows)
  int group_n;
  int64_t group_k;
  float* part;                  // [splits][M, N], or a finished output
  float* out_f32;
  bf16* out_bf16;
  int64_t ldo;
  float* ones = nullptr;        // GLU: [M]
};

template <bool F16>
__device__ __forceinline__ void mma_rows(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (F16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Four E4M3 values -> two fp16 pairs (exact).
__device__ __forceinline__ void unpack4(uint32_t v, uint32_t* h) {
  asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, lo;\n\tcvt.rn.f16x2.e4m3x2 %1, hi;\n\t}" : "=r"(h[0]), "=r"(h[1]) : "r"(v));
}
// The same values as bf16 pairs (exact).
__device__ __forceinline__ void unpack4_bf16(uint32_t v, uint32_t* h) {
  unpack4(v, h);
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const float2 f = __half22float2(*(const __half2*)&h[i]);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h[i]) : "f"(f.y), "f"(f.x));
  }
}
__device__ __forceinline__ uint32_t join_terms(uint32_t hi, uint32_t lo) {  // hi + lo / 16
  uint32_t v;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(v) : "r"(lo), "r"(0x2C002C00u), "r"(hi));
  return v;
}

enum { ROWS_BF16 = 0, ROWS_F8 = 1, ROWS_F8_BF16 = 2 };  // weights and X bf16; E4M3 and two E4M3 terms; E4M3 and bf16
// NT: groups of 8 rows of X. GLU: W = [gate | up], both of 16 channels. TWO: a second tile of channels, through shared memory (for at most AHEAD steps per warp).
template <int KIND, int NT, bool TWO, bool GLU>
__global__ void __launch_bounds__(32 * WARPS, 2) gemm_rows_kernel(RowsArgs a) {
  constexpr bool F8 = KIND != ROWS_BF16, TERMS2 = KIND == ROWS_F8;
  constexpr int TILES = TWO ? 2 : 1, CH = TILES * TILE;
  constexpr int AHEAD = ahead(F8), WORDS = F8 ? 8 : 4;  // words of a load, as operands
  constexpr int COLS = F8 ? 16 : 8, STEP = 4 * COLS;    // columns of a thread's load and of a warp's
  using T = std::conditional_t<F8, uint8_t, bf16>;
  extern __shared__ __align__(16) uint4 second[];  // [AHEAD * 4][threads]
  __shared__ float red[WARPS][8 * NT][CH + 4];     // the fragments of a warp in 32 banks
  SB_TRACE_BEGIN();
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * (GLU ? CH / 2 : CH), z = blockIdx.y, half = a.N / 2;
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
  // the warp's steps
  constexpr int PER = 64 / STEP;  // steps per unit
  const int steps_all = PER * (u1 - u0), s0 = PER * u0 + warp * steps_all / WARPS, s1 = PER * u0 + (warp + 1) * steps_all / WARPS;
  const T* wr = (const T*)a.w + (int64_t)(n0 + g) * a.ldw + COLS * t;
  const int64_t xk = a.group_n > 0 ? n0 / a.group_n * a.group_k : 0;
  using TX = std::conditional_t<TERMS2, uint8_t, bf16>;
  const TX* xr = (const TX*)a.x + (int64_t)((a.n_switch > 0 && n0 >= a.n_switch ? a.x_row_off : 0) + g) * a.ldx + xk + COLS * t;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint32_t w[AHEAD][4][WORDS], x[AHEAD][NT][WORDS];
  auto unpack = [](const uint4& u, uint32_t* o) {
    if constexpr (KIND == ROWS_F8) { unpack4(u.x, o); unpack4(u.y, o + 2); unpack4(u.z, o + 4); unpack4(u.w, o + 6); }
    else if constexpr (KIND == ROWS_F8_BF16) { unpack4_bf16(u.x, o); unpack4_bf16(u.y, o + 2); unpack4_bf16(u.z, o + 4); unpack4_bf16(u.w, o + 6); }
    else { o[0] = u.x; o[1] = u.y; o[2] = u.z; o[3] = u.w; }
  };
  auto load_w = [&](int s) {
    uint4 raw[AHEAD][4];
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int k = (s + i) * STEP;
        const int row = GLU ? (r >> 1) * half + 8 * (r & 1) : 8 * r;  // from the thread's first
        const bool in = GLU ? n0 + g + 8 * (r & 1) < half : n0 + g + row < a.N;
        raw[i][r] = s + i < s1 && k + COLS * t < a.K && in ? __ldcs((const uint4*)(wr + (int64_t)row * a.ldw + k)) : zero;
      }
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int r = 0; r < 4; r++) unpack(raw[i][r], w[i][r]);
  };
  if (!a.prefetch) pdl_wait();
  if constexpr (TWO) {  // the second tile first: its registers are free again when the first one's loads begin
    uint4 raw[AHEAD][4];
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int k = (s0 + i) * STEP;
        const bool in = s0 + i < s1 && k + COLS * t < a.K && n0 + TILE + g + 8 * r < a.N;
        raw[i][r] = in ? __ldcs((const uint4*)(wr + (int64_t)(TILE + 8 * r) * a.ldw + k)) : zero;
      }
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int r = 0; r < 4; r++) second[(i * 4 + r) * 32 * WARPS + threadIdx.x] = raw[i][r];
  }
  load_w(s0);  // weights are constants, and E4M3 ones are converted before the wait too (the conversions took longer than all that follows)
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
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int q = 0; q < WORDS; q += 2)
            mma_rows<TERMS2>(acc[2 * tile + h][j], w[i][2 * h][q], w[i][2 * h + 1][q], w[i][2 * h][q + 1], w[i][2 * h + 1][q + 1], x[i][j][q], x[i][j][q + 1]);
  };
  constexpr int TERMS = F8 ? 2 : 1;
  for (int s = s0; s < s1; s += AHEAD) {
    if (s > s0) load_w(s);
    uint4 raw[AHEAD][NT][TERMS];
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < TERMS; e++) {
          const int k = (s + i) * STEP;
          // the second load: the lo terms, eight rows further on, or (bf16 beside E4M3) the thread's other eight columns
          const TX* from = xr + (int64_t)(8 * (TERMS2 ? 2 * j + e : j)) * a.ldx + k + (TERMS2 ? 0 : 8 * e);
          raw[i][j][e] = s + i < s1 && k + COLS * t < a.K && g + 8 * j < a.M ? __ldcg((const uint4*)from) : zero;
        }
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
#pragma unroll
      for (int j = 0; j < NT; j++) {
        if constexpr (KIND == ROWS_F8_BF16) {
          const uint4 lo = raw[i][j][0], hi = raw[i][j][TERMS - 1];
          x[i][j][0] = lo.x; x[i][j][1] = lo.y; x[i][j][2] = lo.z; x[i][j][3] = lo.w;
          x[i][j][WORDS - 4] = hi.x; x[i][j][WORDS - 3] = hi.y; x[i][j][WORDS - 2] = hi.z; x[i][j][WORDS - 1] = hi.w;
          continue;
        }
        unpack(raw[i][j][0], x[i][j]);
        if constexpr (TERMS2) {
          uint32_t lo[WORDS];
          unpack(raw[i][j][1], lo);
#pragma unroll
          for (int q = 0; q < WORDS; q++) x[i][j][q] = join_terms(x[i][j][q], lo[q]);
        }
      }
    multiply(0);
    if constexpr (TWO) {
#pragma unroll
      for (int i = 0; i < AHEAD; i++)
#pragma unroll
        for (int r = 0; r < 4; r++) unpack(second[(i * 4 + r) * 32 * WARPS + threadIdx.x], w[i][r]);
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
    const int m = 8 * (i / TILES) + warp, c = i % TILES * TILE + lane, n = GLU ? (lane >> 4) * half + n0 + (lane & 15) : n0 + c;
    if constexpr (GLU) {  // lanes 0..15 hold the gates, the others the up values of the same channels
      if (m >= a.M) continue;
      const bool in = n0 + (lane & 15) < half;
      float v = red[0][m][c];
#pragma unroll
      for (int j = 1; j < WARPS; j++) v += red[j][m][c];
      v = in ? __fmul_rn(__fmul_rn(v, a.sx[m]), a.sw[n]) : 0.f;
      const float up = __shfl_down_sync(0xffffffffu, v, 16);
      if (lane < 16 && in) a.out_bf16[m * a.ldo + n] = __float2bfloat16_rn(sb_silu_mul(v, up));
      continue;
    }
    if (m >= a.M || n >= a.N) continue;
    float v = red[0][m][c];
#pragma unroll
    for (int j = 1; j < WARPS; j++) v += red[j][m][c];
    if (F8 && !a.part) v = __fmul_rn(__fmul_rn(v, a.sx[m]), a.sw[n]);
    if (a.part) a.part[((int64_t)z * a.M + m) * a.N + n] = v;
    else if (a.out_f32) a.out_f32[m * a.ldo + n] = v;
    else a.out_bf16[m * a.ldo + n] = __float2bfloat16_rn(v);
  }
  if (GLU && blockIdx.x == 0 && (int)threadIdx.x < a.M) a.ones[threadIdx.x] = 1.f;  // scales of the rows it writes
  SB_TRACE_END(SB_K_GEMM, (uint32_t)a.N ^ ((uint32_t)a.K << 12));
}

template <int KIND, int NT, bool TWO, bool GLU = false>
int launch(strictb200_ctx* ctx, const RowsArgs& a) {
  constexpr size_t smem = TWO ? ahead(KIND != ROWS_BF16) * 4 * 32 * WARPS * sizeof(uint4) : 0;
  static SbDeviceOnce once;  // one per instantiation
  auto kernel = gemm_rows_kernel<KIND, NT, TWO, GLU>;
  if (TWO) SB_CUDA(once.run(ctx->device, [&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }));
  const int ch = TWO ? 2 * TILE : GLU ? TILE / 2 : TILE, n = GLU ? a.N / 2 : a.N;
  SB_CUDA(sb_launch(ctx, kernel, dim3((unsigned)((n + ch - 1) / ch), (unsigned)a.splits), dim3(32 * WARPS), smem, a));
  ctx->launches++;
  return STRICTB200_OK;
}
template <int KIND>
int launch(strictb200_ctx* ctx, const RowsArgs& a) {
  if constexpr (KIND == ROWS_BF16) {
    // longest run of columns a block gets, in units of 64
    const int units = (a.K + 63) / 64, n0 = a.splits0, n1 = a.splits - n0;
    const int run = n0 ? std::max((a.kb_switch + n0 - 1) / n0, (units - a.kb_switch + n1 - 1) / n1) : (units + n1 - 1) / n1;
    // Two tiles per block against one, us, 8 / 16 rows: N 9600 K 1024 4.7 / 7.4 against 5.9 / 7.5, N 14336 5.8 / 9.6 against 6.7 / 8.1, N 16384 6.4 /
    // 10.5 against 7.2 / 8.9: with two groups of rows the second tile's products come on top of a longer chain.
    if (a.M <= 8 && (int64_t)((a.N + TILE - 1) / TILE) * a.splits > 2 * (int64_t)ctx->sm_count && 2 * run <= ahead(false) * WARPS) return launch<KIND, 1, true>(ctx, a);
  }
  return a.M <= 8 ? launch<KIND, 1, false>(ctx, a) : launch<KIND, 2, false>(ctx, a);
}
}  // namespace

SB_TRACE_TU(gemm_rows)

// Linear layers of 1 / 8 / 16 rows, us, the 128-channel tiles in front (weights from HBM):
//   N 1024  K 1024   7.4 / 7.6 / 7.4  ->  5.5 / 4.0 / 4.0        N 14336 K 1024    9.1 /  9.2 /  9.3  ->  5.9 /  6.2 /  9.1
//   N 4096  K 1024   7.6 / 7.6 / 7.6  ->  4.0 / 4.1 / 4.0        N 4096  K 4096   21.3 / 21.3 / 21.3  ->  9.1 /  9.2 / 12.6
//   N 1024  K 5120  25.5 / 25.6 / 25.6 -> 8.6 / 8.7 / 11.3       N 14336 K 4096   23.2 / 23.0 / 23.1, beyond what the blocks hold ahead
// and error against 64 bits (K 1024 / 5120): 9.8e-7 / 5.6e-6 there (tcgen05 cuts off after every instruction), 1.3e-7 / 6.0e-7 here.
// A decode step of 8 sequences (28 layers of latent attention, 1024 wide): 926 -> 763 us.
// Beyond 32 MB of weights the rows of X, which every block reads, and the later rounds of blocks cost more than the K splits of the large
// tiles; a finished product has no K splits there, and with few tiles it stays here (us, 8 / 16 rows here against the large tiles: 4096 x
// 14336 26.9 / 37.4 against 66.5; 1024 x 28672 40.9 / 55.7 against 130; 8192 x 8192 21.8 / 27.5 against 39.3; 8192 x 28672 71.5 / 94.0 against 131).
// Many channels of short rows run in rounds of blocks that each wait for a round trip, where the large tiles' ring goes on: up to one
// round of blocks (one_round), two with two tiles per block and at most 8 rows. us, 8 / 16 rows against the large tiles:
//   N 16384 K 256   4.1 / 5.9 against 4.6    N 18944 K 3072  18.9 against 20.1       N 9472 K 1024  4.9 / 5.4 against 7.6
//   N 32768 K 256   7.7 / 11.2 against 5.1   N 32768 K 2048  23.8 against 20.6       N 9600 K 256 5.1 (16), K 768 6.4 against 4.4, 6.5
// E4M3 weights, whose large tiles are half as long a stream and whose conversion is work here. Whole calls on bf16 rows (the row split in front
// included, weights from HBM), 1 / 16 rows, us, before and with this kernel (2 to 3 us of it the split's overlap):
//   N 4096 K 1024  10.2 / 10.4 -> 6.3 / 6.5   N 1024 K 3072  10.4 / 11.4 -> 8.3 / 8.4   N 1024 K 14336  16.5 / 16.5 -> 10.5 / 13.0
//   N 6144 K 1024  10.3 / 10.4 -> 6.3 / 6.3   N 4096 K 4096  9.6 / 10.6 on the large tiles, 9.9 / 12.6 here; N 6144 K 4096  10.4 / 11.0, 13.1 / 16.9 here
// and without the split, 8 / 16 rows against the large tiles:
//   N 16384 K 512  5.4 against 6.9    N 9600 K 256   4.4 / 5.3 against 4.7    N 12288 K 640  5.1 / 7.3 against 6.7
//   N 16384 K 256  5.0 against 4.6    N 32768 K 256  9.6 / 12.0 against 4.7   N 6144 K 1280 (two splits)  6.6 / 8.6 against 6.7
// A decode step of Qwen3-0.6B: 774 -> 711 us (batch 1).
bool sb_gemm_rows_takes(int64_t M, int64_t N, int64_t K, bool f8, bool finished) {
  if (M > 16 || K % (f8 ? 16 : 8)) return false;
  constexpr int64_t one_round = 2 * SB_SMS * TILE;  // channels whose blocks are resident at once
  const int64_t weights = N * K;
  const bool short_rounds = M <= 8 ? N <= one_round || (N <= 2 * one_round && (!f8 || K >= 512))
                                   : f8 ? N * std::min<int64_t>((K + 1023) / 1024, 8) <= one_round : N <= one_round || (N <= 2 * one_round && K >= 768);
  if (!short_rounds) return false;
  if (f8) return weights <= (8 << 20) || (N <= 1024 && weights <= (16 << 20));
  return weights <= (16 << 20) || (finished && (N <= 8192 || (M <= 8 && weights <= (64 << 20))));
}
int sb_gemm_rows_splits(strictb200_ctx* ctx, int64_t N, int64_t K, bool f8) {
  const int64_t tiles = (N + TILE - 1) / TILE, units = (K + 63) / 64, held = ahead(f8) * WARPS / (f8 ? 1 : 2);
  int64_t s = (units + held - 1) / held;                                          // every weight in registers before the wait
  s = std::max(s, std::min((int64_t)ctx->sm_count / tiles, units / (f8 ? 8 : 4)));  // a block per SM, while every warp has a step
  return (int)std::max<int64_t>(1, std::min<int64_t>(s, 8));                       // eight results are what the consumers take
}
int k_gemm_rows_bf16(strictb200_ctx* ctx, const GemmBf16Args& b) {
  return launch<ROWS_BF16>(ctx, RowsArgs{b.x, b.w, b.ldx, b.ldw, (int)b.M, (int)b.N, (int)b.K, b.splits, ctx->opt.prefetch, nullptr, nullptr, (int)(b.k_switch / 64), b.k_switch ? b.splits0 : 0,
                                     b.e.n_switch, b.e.x_row_off, b.group_n, b.group_k, b.part, b.e.out_f32, b.e.out_bf16, b.e.ldo});
}
int k_gemm_rows_fp8(strictb200_ctx* ctx, const GemmArgs& g) {
  const bool part = g.raw || g.splits > 1;
  return launch<ROWS_F8>(ctx, RowsArgs{g.xq, g.wq, g.ldx, g.ldw, (int)g.M, (int)g.N, (int)g.K, g.splits, ctx->opt.prefetch, g.sx, g.sw, 0, 0, 0, 0, 0, 0, part ? g.part : nullptr,
                                    g.out_f32 ? (float*)g.out : nullptr, g.out_f32 ? nullptr : (bf16*)g.out, g.N});
}
// W = [gate | up] [N, K]: out_bf16 [M, N / 2] = silu(gate) * up, and ones[M] = 1, the rows' scales for the next product's consumer.
int k_gemm_rows_glu(strictb200_ctx* ctx, const GemmArgs& g, float* ones) {
  const RowsArgs a{g.xq, g.wq, g.ldx, g.ldw, (int)g.M, (int)g.N, (int)g.K, 1, ctx->opt.prefetch, g.sx, g.sw, 0, 0, 0, 0, 0, 0, nullptr, nullptr, (bf16*)g.out, g.N / 2, ones};
  return g.M <= 8 ? launch<ROWS_F8, 1, false, true>(ctx, a) : launch<ROWS_F8, 2, false, true>(ctx, a);
}
// part [splits][M, N] = sums of X . W^T, X [M, K] bf16 (g.xq, row stride g.ldx elements) and E4M3 weights.
int k_gemm_rows_fp8_bf16(strictb200_ctx* ctx, const GemmArgs& g) {
  return launch<ROWS_F8_BF16>(ctx, RowsArgs{g.xq, g.wq, g.ldx, g.ldw, (int)g.M, (int)g.N, (int)g.K, g.splits, ctx->opt.prefetch, nullptr, nullptr, 0, 0, 0, 0, 0, 0, g.part,
                                            nullptr, nullptr, g.N});
}
