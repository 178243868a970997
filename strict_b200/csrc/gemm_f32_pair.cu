// fp32 linear layers of many rows on pairs of SMs: the arithmetic of gemm_f32_tc.cu (three bf16 terms per value, six products, the large one summed
// 32 columns at a time and added in registers), with the terms made once per value instead of once per tile.
//
// f32_planes_kernel writes the terms of X and W as three bf16 matrices each (4 bytes read and 6 written per value, an HBM stream). After that the
// product needs no warps that convert: a cluster of two blocks walks tiles of 256 channels x 128 tokens with tcgen05.mma.cta_group::2, and each block
// copies its 128 weight rows and 64 token rows of all three planes by TMA, 72 KB per 64 columns and 24 instructions. In gemm_f32_tc.cu the
// eight warps that split values were the bound (64 KB of fp32 in flight, each tile's split repeated by every other tile of its row and column).
//
// Roles of a block: warp 0 copies; warp 1 of the leading block issues the products of both; warps 4..11 add the sums of their block's 128 channels, half of
// the token columns each, and store finished values (persistent blocks: the stores of a tile overlap the first products of the next). The sums
// of the small products are taken out of tensor memory every 1024 columns, as far as gemm_f32_tc.cu lets one block walk.
// The bound now: a stage of 64 columns takes 2950 to 3050 cycles, 2250 of them the 24 products (128 columns of tokens per product read 8 KB of shared memory
// for 64 cycles of the pipe), the rest waits for copies and for the adding warps. Figures at k_gemm_f32_pair. Every mbarrier wait is bounded and reports through the context's error word.
#include "gemm_f32_terms.cuh"

namespace {
using namespace tc;

constexpr int CH = 128, TOK = 64;    // channels and token rows of a block; a pair's tile is 256 x 128
constexpr int BT = 2 * TOK;
constexpr int KB = 64;               // columns per stage: one 128-byte swizzle atom of bf16
constexpr int NSTAGE = 3;
constexpr int W_PLANE = CH * 128, X_PLANE = TOK * 128, STAGE = 3 * (W_PLANE + X_PLANE);
constexpr int FLUSH = 16;            // stages between two readings of the small products' sums
constexpr int PART = 4;              // stages whose sums are added up before they meet the running sum
constexpr int SUMMERS = 8, AUX = 4, THREADS = 32 * (AUX + SUMMERS);  // warps; of the first four two have work
constexpr int COLS = 4 * BT;         // two partial sums of the large product, the sums of the small ones
constexpr int HALF = BT / 2;
constexpr int RASTER = 8;            // token tiles that are walked side by side

// Values -> planes [3][rows, kp]: terms 0, 1, 2, scaled by 1, 2^8, 2^16. A thread owns eight columns of a row; columns from K to kp are zeros.
__global__ void __launch_bounds__(256) f32_planes_kernel(const float* x, int64_t ldx, int64_t M, bf16* px, const float* w, int64_t ldw, int64_t N, bf16* pw, int K, int kp) {
  pdl_trigger();
  pdl_wait();
  const int per = kp / 8;
  const int64_t nx = M * per, n = nx + N * per;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
    const bool is_w = i >= nx;
    const int64_t j = is_w ? i - nx : i, rows = is_w ? N : M, r = j / per;
    const int k = (int)(j - r * per) * 8;
    const float* from = (is_w ? w + r * ldw : x + r * ldx) + k;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (k < K) a = *(const float4*)from;
    if (k + 4 < K) b = *(const float4*)(from + 4);
    bf16* to = (is_w ? pw : px) + r * kp + k;
#pragma unroll
    for (int p = 0; p < 3; p++) {
      const uint32_t t0 = take_term(a.x, a.y), t1 = take_term(a.z, a.w), t2 = take_term(b.x, b.y), t3 = take_term(b.z, b.w);
      *(uint4*)(to + p * rows * kp) = make_uint4(t0, t1, t2, t3);
    }
  }
}

struct F32PairArgs {
  GemmF32Args g;
  int tiles_n, tiles;
  int* status;
};
// as in gemm_tmem_pair.cu: the pairs at work at a time share operands
__device__ __forceinline__ void tile_at(const F32PairArgs& a, int tile, int& tn, int& tt) {
  const int tiles_t = a.tiles / a.tiles_n, g = tile / (RASTER * a.tiles_n), r = tile - g * RASTER * a.tiles_n;
  const int h = min(RASTER, tiles_t - g * RASTER);
  tn = r / h;
  tt = g * RASTER + r - tn * h;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Copy into this block's shared memory whose bytes complete on a barrier of the leader.
__device__ __forceinline__ void tma_load_planes(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t leader_bar) {
  asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst), "l"(map), "r"(x),
               "r"(y), "r"(0), "r"(leader_bar)
               : "memory");
}
// Arrive on the barrier at this shared-memory offset in both blocks once all products so far are done.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(map_to_rank(bar, 0)) : "memory");
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(map_to_rank(bar, 1)) : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
      :
      : "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}

// Registers of the launch (384 threads x 168) to where they are needed: 128 x 40 + 256 x 224 = 62464 of 64512.
__device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 40;"); }
__device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 224;"); }

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, F32PairArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[NSTAGE], bar_empty[NSTAGE], bar_sum_full, bar_sum_empty;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const uint32_t smem = (smem_u32(smem_raw) + 1023) & ~1023u;
  const GemmF32Args& g = a.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int nkb = ((int)g.K + KB - 1) / KB;
  const int pairs = gridDim.x / 2, c = blockIdx.x / 2, my_tiles = (a.tiles - c + pairs - 1) / pairs;
  const int n_my = my_tiles * nkb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; s++) { mbar_init(smem_u32(&bar_full[s]), 1); mbar_init(smem_u32(&bar_empty[s]), 1); }
    mbar_init(smem_u32(&bar_sum_full), 1);
    mbar_init(smem_u32(&bar_sum_empty), 2 * SUMMERS);  // the leader's: a lane of every adding warp of both blocks
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_trigger();

  if (warp < AUX) reg_dec();
  if (warp == 0) {
    if (lane == 0) {
      pdl_wait();
      int tn = 0, tt = 0, kb = -1;
      for (int it = 0; it < n_my; it++) {
        const int s = it % NSTAGE;
        if (it >= NSTAGE && !mbar_wait(smem_u32(&bar_empty[s]), ((it / NSTAGE) & 1) ^ 1)) { set_status(a.status, 1); abort_flag = 1; break; }
        if (*(volatile int*)&abort_flag) break;
        if (++kb == nkb || it == 0) { kb = 0; tile_at(a, c + it / nkb * pairs, tn, tt); }
        const uint32_t full = map_to_rank(smem_u32(&bar_full[s]), 0), dst = smem + s * STAGE;
        if (rank == 0) mbar_expect_tx(smem_u32(&bar_full[s]), 2 * STAGE);  // the bytes of both blocks
        tma_load_planes(dst, &map_w, kb * KB, (2 * tn + (int)rank) * CH, full);
        tma_load_planes(dst + 3 * W_PLANE, &map_x, kb * KB, (2 * tt + (int)rank) * TOK, full);
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && lane == 0) {
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BT >> 3) << 17) | ((uint32_t)(2 * CH >> 4) << 24);
      const uint32_t big = tmem, small1 = tmem + 2 * BT, small2 = tmem + 3 * BT;
      pdl_wait();  // the bounded waits below are for progress inside this kernel
      for (int it = 0; it < n_my; it++) {
        const int s = it % NSTAGE, kb = it % nkb;
        const bool first = kb % FLUSH == 0;
        if (!mbar_wait(smem_u32(&bar_full[s]), (it / NSTAGE) & 1)) { set_status(a.status, 2); abort_flag = 1; break; }
        // the small products start new sums: the old ones must have been read
        if (first && it && !mbar_wait(smem_u32(&bar_sum_empty), (it - 1) & 1)) { set_status(a.status, 4); abort_flag = 1; break; }
        tc_fence_after();
        const uint32_t sw = smem + s * STAGE, sx = sw + 3 * W_PLANE;
        uint64_t w[3], x[3];
#pragma unroll
        for (int p = 0; p < 3; p++) { w[p] = desc_kmajor(sw + p * W_PLANE); x[p] = desc_kmajor(sx + p * X_PLANE); }
        // 20 small products and the large one in two sums of 32 columns, most of the small ones in front: the adding warps read both
        // sums together, and have until then
        auto small = [&](int j, int p) {  // 16 columns = 32 bytes inside the swizzle atom
          const uint64_t o = (uint64_t)(2 * j);
          if (p == 0) mma_pair(small1, w[0] + o, x[1] + o, idesc, first && !j ? 0u : 1u);
          else if (p == 1) mma_pair(small2, w[0] + o, x[2] + o, idesc, first && !j ? 0u : 1u);
          else if (p == 2) mma_pair(small1, w[1] + o, x[0] + o, idesc, 1u);
          else if (p == 3) mma_pair(small2, w[1] + o, x[1] + o, idesc, 1u);
          else mma_pair(small2, w[2] + o, x[0] + o, idesc, 1u);
        };
#pragma unroll
        for (int i = 0; i < 15; i++) small(i / 5, i % 5);
        if (!first && !mbar_wait(smem_u32(&bar_sum_empty), (it - 1) & 1)) { set_status(a.status, 4); abort_flag = 1; break; }
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < 2; j++) mma_pair(big, w[0] + (uint64_t)(2 * j), x[0] + (uint64_t)(2 * j), idesc, j & 1);
#pragma unroll
        for (int i = 15; i < 20; i++) small(i / 5, i % 5);
#pragma unroll
        for (int j = 2; j < 4; j++) mma_pair(big + BT, w[0] + (uint64_t)(2 * j), x[0] + (uint64_t)(2 * j), idesc, j & 1);
        commit_pair(smem_u32(&bar_empty[s]));
        commit_pair(smem_u32(&bar_sum_full));
      }
    }
    __syncwarp();
  } else if (warp >= AUX) {
    reg_inc();
    const int lg = warp & 3, half = (warp - AUX) >> 2;
    const uint32_t at = tmem + ((uint32_t)(lg * 32) << 16) + half * HALF;
    const uint32_t empty = map_to_rank(smem_u32(&bar_sum_empty), 0);
    // part: sums of up to PART stages, which are added to sum (short chains of additions, however long the row)
    float sum[HALF], part[HALF];
#pragma unroll
    for (int i = 0; i < HALF; i++) sum[i] = part[i] = 0.f;
    pdl_wait();  // the output belongs to the dependency chain
    int kb = 0, seg = 0;
    for (int it = 0; it < n_my; it++) {
      const bool last = ++kb == nkb, flush = last || kb % FLUSH == 0;
      const bool ok = mbar_wait(smem_u32(&bar_sum_full), it & 1);
      if (!__all_sync(0xffffffffu, ok)) { if (lane == 0) set_status(a.status, 3); break; }
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < HALF; q += 16) {
        uint32_t u[16], v[16];
        tc_ld16(at + q, u);
        tc_ld16(at + BT + q, v);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; i++) part[q + i] = __fadd_rn(part[q + i], __fadd_rn(__uint_as_float(u[i]), __uint_as_float(v[i])));
      }
      if (flush) {
#pragma unroll
        for (int q = 0; q < HALF; q += 16) {
          uint32_t u[16], v[16];
          tc_ld16(at + 2 * BT + q, u);
          tc_ld16(at + 3 * BT + q, v);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; i++) part[q + i] = __fmaf_rn(0x1p-8f, __fmaf_rn(0x1p-8f, __uint_as_float(v[i]), __uint_as_float(u[i])), part[q + i]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(empty) : "memory");
      if (last || kb % PART == 0) {
#pragma unroll
        for (int i = 0; i < HALF; i++) { sum[i] = __fadd_rn(sum[i], part[i]); part[i] = 0.f; }
      }
      if (!last) continue;
      int tn, tt;
      tile_at(a, c + seg * pairs, tn, tt);
      kb = 0;
      seg++;
      const int n = (2 * tn + (int)rank) * CH + lg * 32 + lane, tok0 = tt * BT + half * HALF;
      constexpr bool reads = MODE == 1 || MODE == 4;
      float* const y = g.y + (int64_t)tok0 * g.ldy + n;
      const int64_t ldy = g.ldy;
      const int toks = n < g.N ? min(HALF, (int)(g.M - tok0)) : 0;
      const float bias = g.bias && n < g.N ? g.bias[n] : 0.f, cs = MODE == 4 ? g.alpha * (g.col_scale && n < g.N ? g.col_scale[n] : 1.f) : 1.f;
      auto value = [&](float v, float old) { return finished<MODE>(g, cs, v + bias, old); };
      // The code that finishes a value is kept short and there once per sixteen tokens, which then move to the front: sixty-four
      // copies of it, of every mode and each with its checks, came cold from the instruction cache for 16 us a tile.
      uint64_t again = 0;  // tokens whose sum is not finite
      float* to = y;
#pragma unroll 1
      for (int q = 0; q < HALF; q += 16) {
        float old[16], check = 0.f;  // check: not a number once a sum is not finite
        if constexpr (reads) {
#pragma unroll
          for (int i = 0; i < 16; i++) old[i] = q + i < toks ? to[i * ldy] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 16; i++) check = fmaf(sum[i], 0.f, check);
        if (__builtin_expect(check == 0.f, 1)) {
#pragma unroll
          for (int i = 0; i < 16; i++)
            if (q + i < toks) to[i * ldy] = value(sum[i], reads ? old[i] : 0.f);
        } else {
#pragma unroll
          for (int i = 0; i < 16; i++)
            if (q + i < toks) {
              if (not_finite(sum[i])) again |= 1ull << (q + i);
              else to[i * ldy] = value(sum[i], reads ? old[i] : 0.f);
            }
        }
        to += 16 * ldy;
#pragma unroll
        for (int i = 0; i + 16 < HALF; i++) sum[i] = sum[i + 16];
      }
      while (again) {
        const int i = __ffsll((long long)again) - 1;
        again &= again - 1;
        float* p = y + i * ldy;
        *p = value(plain_dot(g.x + (int64_t)(tok0 + i) * g.ldx, g.w + (int64_t)n * g.ldw, (int)g.K), reads ? *p : 0.f);
      }
#pragma unroll
      for (int i = 0; i < HALF; i++) sum[i] = part[i] = 0.f;
    }
  }
  // nobody leaves while the other block may still signal one of its barriers or use its tensor memory
  tc_fence_before();
  __syncwarp();
  cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)COLS) : "memory");
  }
}

// [3][rows, kp] bf16, box = 64 columns x box_rows x 3 planes
int planes_map(CUtensorMap* map, const bf16* base, int64_t rows, int64_t K, int64_t kp, int box_rows) {
  EncodeFn encode;
  SB_TRY(encode_fn(&encode));
  cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, 3u};
  cuuint64_t strides[2] = {(cuuint64_t)kp * 2, (cuuint64_t)(rows * kp) * 2};
  cuuint32_t box[3] = {(cuuint32_t)KB, (cuuint32_t)box_rows, 3u};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return sb_fail(STRICTB200_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
  return STRICTB200_OK;
}

constexpr int64_t MIN_TILES = 44;                // fewer leave most pairs idle; below
constexpr size_t PLANES_MAX = (size_t)1 << 30;  // scratch a context keeps for the planes at most
constexpr int64_t ROWS_MAX = 32768;             // rows of X per pass
// Grow-only scratch of its own. Nothing that was recorded refers to it (below), so it may move. A larger one is had before the smaller one goes, and a size
// that could not be had is not asked for again until the context has freed something: neither costs the products behind it their scratch or a wait each.
bool planes_scratch(strictb200_ctx* ctx, size_t bytes) {
  if (bytes <= ctx->planes_bytes) return true;
  if (bytes >= ctx->planes_refused) return false;
  void* larger = nullptr;
  size_t want = std::min(bytes + (bytes >> 2), PLANES_MAX);
  if (cudaMalloc(&larger, want) != cudaSuccess && cudaMalloc(&larger, want = bytes) != cudaSuccess) {
    cudaGetLastError();
    ctx->planes_refused = bytes;
    return false;
  }
  if (ctx->planes) {
    cudaStreamSynchronize(ctx->stream);
    cudaFree(ctx->planes);
  }
  ctx->planes = larger;
  ctx->planes_bytes = want;
  return true;
}
template <int MODE>
int launch(strictb200_ctx* ctx, const CUtensorMap& mw, const CUtensorMap& mx, const F32PairArgs& a, int64_t pairs) {
  const size_t smem = (size_t)NSTAGE * STAGE + 1024;
  static SbDeviceOnce once;  // one per instantiation
  SB_CUDA(once.run(ctx->device, [&] { return cudaFuncSetAttribute(gemm_f32_pair_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }));
  SB_CUDA(sb_launch_cluster(ctx, gemm_f32_pair_kernel<MODE>, dim3((unsigned)(2 * pairs)), dim3(THREADS), smem, dim3(2, 1, 1), mw, mx, a));
  ctx->launches++;
  return STRICTB200_OK;
}
}  // namespace

// us, both passes, and error against 64 bits (2-norm) of normal operands, gemm_f32_tc.cu in front (rows x channels x columns):
//   4700 x 3072 x 768   183 -> 136  8.66e-8 -> 7.36e-8    4700 x 768 x 768   61 -> 51   8.65e-8 -> 7.34e-8    8192 x 4096 x 4096  2214 -> 1507  1.03e-7 -> 1.00e-7
//   4700 x 2304 x 768   148 -> 114  8.66e-8 -> 7.34e-8    4700 x 768 x 3072  211 -> 184  9.56e-8 -> 9.32e-8
// and around the rule: 48 tiles (500 x 3072 x 768) 31.5 -> 30.0, 60 tiles (2500 x 768 x 768 and x 3072) 30.9 -> 29.6 and 115 -> 97, 72 tiles (901 x 2304
// x 768) 30.8 -> 29.7, 96 tiles (901 x 3072 x 768) 59.5 -> 49.6; but 36 tiles (300 x 3072 x 768, 1500 x 768 x 768, 1500 x 768 x 3072) 22.1, 22.0 and 85.1
// there against 29.6, 29.0 and 89.6 here.
// ERR_UNSUPPORTED: the caller's other kernel takes the product (few tiles, no room for the planes, or a stream that is being recorded, whose
// calls must not depend on scratch that moves).
int k_gemm_f32_pair(strictb200_ctx* ctx, const GemmF32Args& g) {
  const int64_t tiles_n = (g.N + 2 * CH - 1) / (2 * CH), kp = (g.K + 7) / 8 * 8;
  const int64_t rows = std::min(g.M, ROWS_MAX), x_bytes = 3 * rows * kp * 2, w_bytes = 3 * g.N * kp * 2;
  if (g.M <= 128 || tiles_n * ((g.M + BT - 1) / BT) < MIN_TILES || ctx->sm_count < 2 || !ctx->opt.gemm_pair) return STRICTB200_ERR_UNSUPPORTED;
  if (g.N > (1 << 24) || g.K > (1 << 24) || (size_t)(x_bytes + w_bytes) > PLANES_MAX) return STRICTB200_ERR_UNSUPPORTED;
  cudaStreamCaptureStatus recording = cudaStreamCaptureStatusNone;
  SB_CUDA(cudaStreamIsCapturing(ctx->stream, &recording));
  if (recording != cudaStreamCaptureStatusNone || !planes_scratch(ctx, (size_t)(x_bytes + w_bytes))) return STRICTB200_ERR_UNSUPPORTED;
  bf16 *pw = (bf16*)ctx->planes, *px = pw + 3 * g.N * kp;
  CUtensorMap mw, mx;
  SB_TRY(planes_map(&mw, pw, g.N, g.K, kp, CH));
  for (int64_t m0 = 0; m0 < g.M; m0 += ROWS_MAX) {
    GemmF32Args p = g;
    p.M = std::min(g.M - m0, ROWS_MAX);
    p.x = g.x + m0 * g.ldx;
    p.y = g.y + m0 * g.ldy;
    const int64_t n = p.M + (m0 ? 0 : g.N), groups = n * (kp / 8);
    SB_CUDA(sb_launch(ctx, f32_planes_kernel, dim3((unsigned)std::min<int64_t>((groups + 255) / 256, 16 * (int64_t)ctx->sm_count)), dim3(256), 0, p.x, p.ldx, p.M, px, p.w, p.ldw,
                      m0 ? (int64_t)0 : g.N, pw, (int)g.K, (int)kp));
    ctx->launches++;
    SB_TRY(planes_map(&mx, px, p.M, g.K, kp, TOK));
    const int64_t tiles = tiles_n * ((p.M + BT - 1) / BT), pairs = std::min<int64_t>(ctx->sm_count / 2, tiles);
    const F32PairArgs a{p, (int)tiles_n, (int)tiles, ctx->d_status};
    SB_TRY(g.mode == 1 ? launch<1>(ctx, mw, mx, a, pairs) : g.mode == 2 ? launch<2>(ctx, mw, mx, a, pairs) : g.mode == 3 ? launch<3>(ctx, mw, mx, a, pairs) :
           g.mode == 4 ? launch<4>(ctx, mw, mx, a, pairs) : launch<0>(ctx, mw, mx, a, pairs));
  }
  return STRICTB200_OK;
}
