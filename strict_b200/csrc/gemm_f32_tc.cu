// fp32 linear layers of many rows on the tcgen05 tensor cores, without giving up fp32 results: Y[M,N] = X[M,K] . W[N,K]^T + bias.
//
// Every fp32 value is the exact sum of three bf16 terms, x = x0 + 2^-8 x1 + 2^-16 x2 (8 + 8 + 8 significant bits, each remainder exact).
// The factors keep the terms where bf16 has bits: without them a value below 2^-110 would lose bits of its last term, one below 2^-118 of two.
// (Below 2^-126, where fp32 itself ends in units of 2^-149, the terms no longer shrink by 2^-8, and the products left out amount to at
// most half of such a unit of the value.)
// Of the nine products of two values the six largest are computed, w0x0 + 2^-8 (w0x1 + w1x0) + 2^-16 (w0x2 + w1x1 + w2x0); the rest lies
// below 2^-24 of the product, as far down as the rounding of an fp32 product. A tensor core multiplies bf16 exactly, but it cuts its fp32
// sum off after every instruction (measured: 1e-8 of the result towards zero per 16 columns, 6e-7 after 768), so
//   - the large product w0x0 is summed over 32 columns at a time in tensor memory; two such sums are added and then added to the
//     running sum in registers, where fp32 addition rounds to nearest;
//   - the small ones stay in tensor memory for all of a block's columns, a sum for each factor: what is cut off there is 2^-8 times
//     smaller or less;
//   - no block walks more than about 1024 columns, or an eighth of K where that is more: longer rows are shared by the up to eight
//     blocks of a cluster, whose sums are added in block order through distributed shared memory (and few tiles are shared the same
//     way to fill the GPU).
// Measured error against 64 bits (2-norm, normal operands; in brackets the row kernel of gemm_f32.cu, all plain fp32 FMAs):
// see the table at k_gemm_f32 in gemm_f32.cu.
//
// One block: 128 channels x BT tokens. The bound is the tensor pipe (six products: 1/6 of the bf16 rate) next to the shared-memory
// traffic of feeding it; the splits are made once per tile by eight warps on the way from registers to shared memory, so the
// operands cross L2 as 4-byte values (split planes in memory would be 6).
//   warps 0..7    fp32 rows -> registers -> three bf16 planes in swizzled shared memory, 64 columns per stage, two stages
//   warp 8        tensor memory, tcgen05.mma: 20 small-product instructions of a stage, then 4 of the large one
//   warps 9..16   running sums: half of the token columns each, thread = channel
// A result that is not finite is computed again as a plain fp32 sum (an infinity has no bf16 remainder), so infinities, NaN and
// overflow come out as they do from the row kernel. Every mbarrier wait is bounded and reports through the context's error word.
#include "gemm_f32_terms.cuh"

namespace {
using namespace tc;

constexpr int CH = 128;   // channels per block
constexpr int KB = 64;    // columns of K per stage: one 128-byte swizzle atom of bf16
constexpr int NSTAGE = 2;
constexpr int W_PLANE = CH * 128;
constexpr int FEEDERS = 8, SUMMERS = 8;  // warps
constexpr int THREADS = 32 * (FEEDERS + 1 + SUMMERS);

struct F32TcArgs {
  GemmF32Args g;
  int ks;       // blocks of a cluster that share K
  int* status;
  int prefetch; // load the first weights before the dependency wait
};

__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster(uint32_t local, uint32_t rank) {
  uint32_t addr;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
// Eight columns of one row into the three planes at this shared-memory address.
__device__ __forceinline__ void store_terms(uint32_t addr, uint32_t plane_bytes, float4 a, float4 b) {
#pragma unroll
  for (int p = 0; p < 3; p++) {
    const uint32_t t0 = take_term(a.x, a.y), t1 = take_term(a.z, a.w), t2 = take_term(b.x, b.y), t3 = take_term(b.z, b.w);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr + p * plane_bytes), "r"(t0), "r"(t1), "r"(t2), "r"(t3) : "memory");
  }
}
__device__ __forceinline__ void finish(const GemmF32Args& g, int tok, int n, float v) {
  if (tok >= g.M || n >= g.N) return;
  float* y = g.y + (int64_t)tok * g.ldy + n;
  if (not_finite(v)) v = plain_dot(g.x + (int64_t)tok * g.ldx, g.w + (int64_t)n * g.ldw, (int)g.K);
  if (g.bias) v += g.bias[n];
  switch (g.mode) {
    case 1: *y = finished<1>(g, 1.f, v, *y); break;
    case 2: *y = finished<2>(g, 1.f, v, 0.f); break;
    case 3: *y = finished<3>(g, 1.f, v, 0.f); break;
    case 4: *y = finished<4>(g, g.alpha * (g.col_scale ? g.col_scale[n] : 1.f), v, *y); break;
    default: *y = v;
  }
}

template <int BT>
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_tc_kernel(F32TcArgs a) {
  constexpr int X_PLANE = BT * 128, STAGE = 3 * (W_PLANE + X_PLANE);
  constexpr int COLS = 4 * BT;  // two partial sums of the large product, the sums of the small ones
  constexpr int HALF = BT / 2;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[NSTAGE], bar_empty[NSTAGE], bar_sum_full, bar_sum_empty;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const uint32_t smem = (smem_u32(smem_raw) + 1023) & ~1023u;
  const GemmF32Args& g = a.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * CH, t0 = blockIdx.y * BT;
  const int nkb_all = ((int)g.K + KB - 1) / KB;
  const int kb0 = (int)((int64_t)blockIdx.z * nkb_all / a.ks), nkb = (int)((int64_t)(blockIdx.z + 1) * nkb_all / a.ks) - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; s++) { mbar_init(smem_u32(&bar_full[s]), FEEDERS); mbar_init(smem_u32(&bar_empty[s]), 1); }
    mbar_init(smem_u32(&bar_sum_full), 1);
    mbar_init(smem_u32(&bar_sum_empty), SUMMERS);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == FEEDERS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_trigger();

  if (warp < FEEDERS) {
    // thread: eight columns (chunk c) of the rows r, r + 32, ... of both tiles
    constexpr int WR = CH / 32, XR = BT / 32;
    const int c = threadIdx.x & 7, r = threadIdx.x >> 3;
    const float* wrow = g.w + (int64_t)(n0 + r) * g.ldw;
    const float* xrow = g.x + (int64_t)(t0 + r) * g.ldx;
    float4 rw[WR][2], rx[XR][2];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto load_w = [&](int kb, int i) {
      const int k = (kb0 + kb) * KB + c * 8;
#pragma unroll
      for (int h = 0; h < 2; h++)
        rw[i][h] = k + 4 * h < g.K && n0 + r + 32 * i < g.N ? __ldg((const float4*)(wrow + (int64_t)(32 * i) * g.ldw + k + 4 * h)) : zero;
    };
    auto load_x = [&](int kb, int i) {
      const int k = (kb0 + kb) * KB + c * 8;
#pragma unroll
      for (int h = 0; h < 2; h++)
        rx[i][h] = k + 4 * h < g.K && t0 + r + 32 * i < g.M ? *(const float4*)(xrow + (int64_t)(32 * i) * g.ldx + k + 4 * h) : zero;
    };
    if (!a.prefetch) pdl_wait();
#pragma unroll
    for (int i = 0; i < WR; i++) load_w(0, i);  // weights are constants
    pdl_wait();
#pragma unroll
    for (int i = 0; i < XR; i++) load_x(0, i);
    for (int kb = 0; kb < nkb; kb++) {
      const int s = kb % NSTAGE;
      if (kb >= NSTAGE && !mbar_wait(smem_u32(&bar_empty[s]), ((kb / NSTAGE) & 1) ^ 1)) { set_status(a.status, 1); abort_flag = 1; break; }
      if (*(volatile int*)&abort_flag) break;
      const bool more = kb + 1 < nkb;
      const uint32_t at = smem + (uint32_t)(s * STAGE + r * 128 + ((c ^ (r & 7)) << 4));  // (r + 32 i) & 7 == r & 7
      // a row's next columns are requested as soon as its registers are free: every load has a whole stage to arrive
#pragma unroll
      for (int i = 0; i < WR; i++) {
        store_terms(at + i * 4096, W_PLANE, rw[i][0], rw[i][1]);
        if (more) load_w(kb + 1, i);
      }
#pragma unroll
      for (int i = 0; i < XR; i++) {
        store_terms(at + 3 * W_PLANE + i * 4096, X_PLANE, rx[i][0], rx[i][1]);
        if (more) load_x(kb + 1, i);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_full[s]));
    }
  } else if (warp == FEEDERS) {
    if (lane == 0) {
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BT >> 3) << 17) | ((uint32_t)(CH >> 4) << 24);
      const uint32_t big = tmem, small1 = tmem + 2 * BT, small2 = tmem + 3 * BT;
      // The operand tiles cannot arrive before the feeders' dependency wait has returned: the same wait here keeps the bounded ones below for
      // progress inside this kernel, however long its predecessor takes.
      pdl_wait();
      for (int kb = 0; kb < nkb; kb++) {
        const int s = kb % NSTAGE;
        if (!mbar_wait(smem_u32(&bar_full[s]), (kb / NSTAGE) & 1)) { set_status(a.status, 2); abort_flag = 1; break; }
        tc_fence_after();
        const uint32_t sw = smem + s * STAGE, sx = sw + 3 * W_PLANE;
        uint64_t w[3], x[3];
#pragma unroll
        for (int p = 0; p < 3; p++) { w[p] = desc_kmajor(sw + p * W_PLANE); x[p] = desc_kmajor(sx + p * X_PLANE); }
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const uint64_t o = (uint64_t)(2 * j);  // 16 columns = 32 bytes inside the swizzle atom
          tc_mma_ss(small1, w[0] + o, x[1] + o, idesc, (kb | j) ? 1u : 0u);
          tc_mma_ss(small1, w[1] + o, x[0] + o, idesc, 1u);
          tc_mma_ss(small2, w[0] + o, x[2] + o, idesc, (kb | j) ? 1u : 0u);
          tc_mma_ss(small2, w[1] + o, x[1] + o, idesc, 1u);
          tc_mma_ss(small2, w[2] + o, x[0] + o, idesc, 1u);
        }
        if (kb && !mbar_wait(smem_u32(&bar_sum_empty), (kb - 1) & 1)) { set_status(a.status, 4); abort_flag = 1; break; }
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < 4; j++) tc_mma_ss(big + (j >> 1) * BT, w[0] + (uint64_t)(2 * j), x[0] + (uint64_t)(2 * j), idesc, j & 1);
        tc_commit(smem_u32(&bar_empty[s]));
        tc_commit(smem_u32(&bar_sum_full));
      }
    }
    __syncwarp();
  } else {
    const int lg = warp & 3, half = (warp - FEEDERS - 1) >> 2;
    const uint32_t at = tmem + ((uint32_t)(lg * 32) << 16) + half * HALF;
    float sum[HALF];
#pragma unroll
    for (int i = 0; i < HALF; i++) sum[i] = 0.f;
    pdl_wait();  // the output belongs to the dependency chain
    bool ok = true;
    for (int kb = 0; kb < nkb; kb++) {
      ok = mbar_wait(smem_u32(&bar_sum_full), kb & 1);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; if (lane == 0) set_status(a.status, 3); break; }
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < HALF; q += 8) {
        uint32_t u[8], v[8];
        tc_ld8(at + q, u);
        tc_ld8(at + BT + q, v);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; i++) sum[q + i] = __fadd_rn(sum[q + i], __fadd_rn(__uint_as_float(u[i]), __uint_as_float(v[i])));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_sum_empty));
    }
    if (ok) {
#pragma unroll
      for (int q = 0; q < HALF; q += 8) {
        uint32_t u[8], v[8];
        tc_ld8(at + 2 * BT + q, u);
        tc_ld8(at + 3 * BT + q, v);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; i++) sum[q + i] = __fmaf_rn(0x1p-8f, __fmaf_rn(0x1p-8f, __uint_as_float(v[i]), __uint_as_float(u[i])), sum[q + i]);
      }
      // the stages have been read by every product: they become [token][channel] sums of this block
      const uint32_t to = smem + (uint32_t)((half * HALF * CH + lg * 32 + lane) * 4);
#pragma unroll
      for (int i = 0; i < HALF; i++) asm volatile("st.shared.f32 [%0], %1;" ::"r"(to + i * CH * 4), "f"(sum[i]) : "memory");
    }
  }
  __syncwarp();
  if (a.ks > 1) cluster_sync();
  else __syncthreads();
  // block z of the cluster finishes its share of the token columns
  if (threadIdx.x < 512) {
    const int cols = BT / a.ks, ch = threadIdx.x & 127;
    for (int i = threadIdx.x >> 7; i < cols; i += 4) {
      const int col = (int)blockIdx.z * cols + i;
      const uint32_t from = smem + (uint32_t)((col * CH + ch) * 4);
      float v;
      if (a.ks == 1) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(from) : "memory");
      else {
        v = ld_cluster(from, 0);
        for (int z = 1; z < a.ks; z++) v = __fadd_rn(v, ld_cluster(from, (uint32_t)z));
      }
      finish(g, t0 + col, n0 + ch, v);
    }
  }
  __syncwarp();
  if (a.ks > 1) cluster_sync();  // nobody leaves while its sums may still be read
  tc_fence_before();
  __syncthreads();
  if (warp == FEEDERS) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)COLS) : "memory");
  }
}

template <int BT>
int launch(strictb200_ctx* ctx, const GemmF32Args& g) {
  const size_t smem = (size_t)NSTAGE * 3 * (W_PLANE + BT * 128) + 1024;
  static SbDeviceOnce once;  // one per instantiation
  SB_CUDA(once.run(ctx->device, [&] { return cudaFuncSetAttribute(gemm_f32_tc_kernel<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }));
  const int64_t tn = (g.N + CH - 1) / CH, tt = (g.M + BT - 1) / BT, nkb = (g.K + KB - 1) / KB;
  if (tt > 65535) return sb_fail(STRICTB200_ERR_INVALID_ARG, "gemm_f32: M too large");
  int ks = 1;
  while (ks < 8 && ks * 2 <= nkb && g.K > 1024 * (int64_t)ks) ks *= 2;                          // precision: short running sums
  while (ks < 8 && nkb >= 4 * (int64_t)ks && tn * tt * ks * 2 <= ctx->sm_count) ks *= 2;  // fill the GPU
  F32TcArgs a{g, ks, ctx->d_status, ctx->opt.prefetch};
  SB_CUDA(sb_launch_cluster(ctx, gemm_f32_tc_kernel<BT>, dim3((unsigned)tn, (unsigned)tt, (unsigned)ks), dim3(THREADS), smem, dim3(1, 1, (unsigned)ks), a));
  ctx->launches++;
  return STRICTB200_OK;
}
}  // namespace

int k_gemm_f32_tc(strictb200_ctx* ctx, const GemmF32Args& g) {
  if (g.M <= 32) return launch<32>(ctx, g);
  if (g.M <= 64) return launch<64>(ctx, g);
  return launch<128>(ctx, g);
}
