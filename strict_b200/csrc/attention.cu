// GQA attention over the bf16 KV cache (head_dim 128) and the fp32 attention of the GPT-2 path.
//
//  * prefill: flash-style causal kernel; one block = 64 query positions of one query head,
//    KV tiles of 64 keys double-buffered in shared memory by cp.async, bf16 mma.sync
//    m16n8k16 with fp32 online softmax; keys come straight from the cache, so a chunked
//    prefill (past > 0) is the same kernel.
//  * decode: split-KV. One block = one KV head of one sequence over one chunk of keys; the
//    G = Hq/Hkv query heads that share the KV head are the rows of the MMA tile, so every
//    K/V byte is read from HBM once. Each block writes (m, l, o) partials; a combine kernel
//    merges the chunks and can emit the two-term E4M3 split of the token row the next GEMM consumes.
//
// Shared-memory tiles hold rows of 128 bf16 (256 B = 16 chunks of 16 B); chunk c of row r
// lives at chunk c ^ (r & 7), which makes every ldmatrix phase conflict-free.
#include <cstdlib>
#include <mutex>

#include <cmath>

#include "common.cuh"

namespace {

constexpr int D = 128;
constexpr int KT = 64;  // keys per tile
constexpr int DEC_STAGES = 2;  // K/V tile ring of the decode kernel; 3 stages (2 blocks/SM) measured 4 % slower than 2 (3 blocks/SM)
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(uint32_t s, const void* g, bool valid) {
  int sz = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(g), "r"(sz));
}
__device__ __forceinline__ void cp_async16_hint(uint32_t s, const void* g, bool valid, uint64_t policy) {
  int sz = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;\n" ::"r"(s), "l"(g), "r"(sz), "l"(policy));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  return f32_to_bf16_bits(lo) | (f32_to_bf16_bits(hi) << 16);
}
// The softmax weights enter the P.V product as two bf16 terms, p = hi + lo (16 mantissa bits):
// a single bf16 P is off by up to 2^-9, which is enough to move the bf16-rounded attention
// output by an ulp on a few percent of its elements, and the E4M3 quantisation that follows
// turns each such ulp into a 6-12 % step. V is exact in bf16, so two MMAs recover the product.
__device__ __forceinline__ void split_bf16(float a, float b, uint32_t& hi, uint32_t& lo) {
  float ah = round_bf16(a), bh = round_bf16(b);
  hi = pack_bf16(ah, bh);
  lo = pack_bf16(a - ah, b - bh);
}
// HD = dims of a row (64 or 128): rows of HD / 8 chunks of 16 bytes, chunk c of row r at chunk c ^ (r & 7)
template <int HD = D>
__device__ __forceinline__ uint32_t tile_off(int row, int chunk) { return (uint32_t)(row * 2 * HD + ((chunk ^ (row & 7)) << 4)); }

// Copy `rows` rows of 128 bf16 (global row stride 128 elements) into a swizzled tile; rows at
// or beyond `valid_rows` are zero-filled.
__device__ __forceinline__ void load_tile(uint32_t tile, const bf16* src, int rows, int valid_rows, int nthreads) {
  for (int c = threadIdx.x; c < rows * 16; c += nthreads) {
    int r = c >> 4, cc = c & 15;
    bool v = r < valid_rows;
    cp_async16(tile + tile_off(r, cc), src + (int64_t)(v ? r : 0) * D + cc * 8, v);
  }
}

// Same for rows of HD dims, with an L2 eviction policy on the global reads (the decode kernel reads every key and
// value exactly once).
template <int HD>
__device__ __forceinline__ void load_tile_hint(uint32_t tile, const bf16* src, int rows, int valid_rows, int nthreads, uint64_t policy) {
  for (int c = threadIdx.x; c < rows * (HD / 8); c += nthreads) {
    int r = c / (HD / 8), cc = c % (HD / 8);
    bool v = r < valid_rows;
    cp_async16_hint(tile + tile_off<HD>(r, cc), src + (int64_t)(v ? r : 0) * HD + cc * 8, v, policy);
  }
}

// ------------------------------------------------------------------ prefill
// grid (ceil(S/64), Hq, B), 128 threads.
__global__ void __launch_bounds__(128) attn_prefill_kernel(const bf16* __restrict__ q, const bf16* __restrict__ kc, const bf16* __restrict__ vc,
                                                           const int32_t* __restrict__ lens, const int32_t* __restrict__ past,
                                                           const int32_t* __restrict__ qstart, int S, int Hq, int Hkv, int maxlen,
                                                           float scale_log2, bf16* __restrict__ out) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int b = blockIdx.z, h = blockIdx.y, q0 = blockIdx.x * 64;
  const int len = lens[b], pst = past ? past[b] : 0;
  const int n_new = len - pst;
  if (q0 >= n_new) return;
  const int64_t row0 = qstart ? qstart[b] : (int64_t)b * S;  // first row of this sequence in q / out
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
  const int hk = h / (Hq / Hkv);
  const uint32_t sQ = smem_u32(smem), sK = sQ + 64 * 256, sV = sK + 2 * KT * 256;
  const bf16* kbase = kc + ((int64_t)b * Hkv + hk) * maxlen * D;
  const bf16* vbase = vc + ((int64_t)b * Hkv + hk) * maxlen * D;
  // last key any row of this block may see
  const int kv_end = min(len, pst + q0 + 64);
  const int ntiles = (kv_end + KT - 1) / KT;

  // Q tile: rows q0..q0+63 of head h; global row stride Hq*D
  for (int c = threadIdx.x; c < 64 * 16; c += 128) {
    int r = c >> 4, cc = c & 15;
    bool v = q0 + r < n_new;
    cp_async16(sQ + tile_off(r, cc), q + ((row0 + (v ? q0 + r : 0)) * Hq + h) * D + cc * 8, v);
  }
  load_tile(sK, kbase, KT, min(KT, len), 128);
  load_tile(sV, vbase, KT, min(KT, len), 128);
  cp_async_commit();

  uint32_t qf[8][4];
  float o[16][4];
#pragma unroll
  for (int j = 0; j < 16; j++)
#pragma unroll
    for (int i = 0; i < 4; i++) o[j][i] = 0.f;
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  const int qpos0 = pst + q0 + warp * 16 + g;  // position of row g; row g+8 is qpos0+8
  const int mi = lane >> 3, r8 = lane & 7;

  for (int t = 0; t < ntiles; t++) {
    if (t + 1 < ntiles) {
      int k0 = (t + 1) * KT;
      load_tile(sK + ((t + 1) & 1) * KT * 256, kbase + (int64_t)k0 * D, KT, min(KT, len - k0), 128);
      load_tile(sV + ((t + 1) & 1) * KT * 256, vbase + (int64_t)k0 * D, KT, min(KT, len - k0), 128);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    if (t == 0) {
#pragma unroll
      for (int ks = 0; ks < 8; ks++) ldsm_x4(sQ + tile_off(warp * 16 + (mi & 1) * 8 + r8, 2 * ks + (mi >> 1)), qf[ks]);
    }
    const uint32_t tK = sK + (t & 1) * KT * 256, tV = sV + (t & 1) * KT * 256;
    float s[8][4];
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int i = 0; i < 4; i++) s[j][i] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 8; ks++) {
#pragma unroll
      for (int jp = 0; jp < 4; jp++) {
        uint32_t kb[4];
        ldsm_x4(tK + tile_off(jp * 16 + (mi >> 1) * 8 + r8, 2 * ks + (mi & 1)), kb);
        mma_bf16(s[2 * jp], qf[ks], kb[0], kb[1]);
        mma_bf16(s[2 * jp + 1], qf[ks], kb[2], kb[3]);
      }
    }
    // scale, mask, online softmax
    const int kbase_pos = t * KT;
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        int kpos = kbase_pos + 8 * j + 2 * tig + (i & 1);
        int qpos = qpos0 + ((i >> 1) << 3);
        float v = s[j][i] * scale_log2;
        v = (kpos > qpos || kpos >= len) ? -INFINITY : v;
        s[j][i] = v;
        mx[i >> 1] = fmaxf(mx[i >> 1], v);
      }
    float corr[2], m_use[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
      float m_new = fmaxf(m_run[r], mx[r]);
      m_use[r] = m_new == -INFINITY ? 0.f : m_new;
      corr[r] = exp2f(m_run[r] - m_use[r]);
      m_run[r] = m_new;
    }
    float ls[2] = {0.f, 0.f};
    uint32_t pf[4][4], pl[4][4];  // P = hi + lo, two bf16 terms (see split_bf16)
#pragma unroll
    for (int j = 0; j < 8; j++) {
      float p0 = exp2f(s[j][0] - m_use[0]), p1 = exp2f(s[j][1] - m_use[0]);
      float p2 = exp2f(s[j][2] - m_use[1]), p3 = exp2f(s[j][3] - m_use[1]);
      ls[0] += p0 + p1;
      ls[1] += p2 + p3;
      split_bf16(p0, p1, pf[j >> 1][(j & 1) * 2], pl[j >> 1][(j & 1) * 2]);
      split_bf16(p2, p3, pf[j >> 1][(j & 1) * 2 + 1], pl[j >> 1][(j & 1) * 2 + 1]);
    }
#pragma unroll
    for (int r = 0; r < 2; r++) l_run[r] = l_run[r] * corr[r] + ls[r];
#pragma unroll
    for (int j = 0; j < 16; j++) {
      o[j][0] *= corr[0]; o[j][1] *= corr[0];
      o[j][2] *= corr[1]; o[j][3] *= corr[1];
    }
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
#pragma unroll
      for (int jj = 0; jj < 8; jj++) {
        uint32_t vb[4];
        ldsm_x4_t(tV + tile_off(kk * 16 + (mi & 1) * 8 + r8, 2 * jj + (mi >> 1)), vb);
        mma_bf16(o[2 * jj], pf[kk], vb[0], vb[1]);
        mma_bf16(o[2 * jj + 1], pf[kk], vb[2], vb[3]);
        mma_bf16(o[2 * jj], pl[kk], vb[0], vb[1]);
        mma_bf16(o[2 * jj + 1], pl[kk], vb[2], vb[3]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 2; r++) {
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
  }
#pragma unroll
  for (int r = 0; r < 2; r++) {
    int row = q0 + warp * 16 + g + r * 8;
    if (row < n_new) {
      float inv = 1.0f / l_run[r];
      bf16* dst = out + ((row0 + row) * Hq + h) * D;
#pragma unroll
      for (int j = 0; j < 16; j++) *(uint32_t*)(dst + 8 * j + 2 * tig) = pack_bf16(o[j][2 * r] * inv, o[j][2 * r + 1] * inv);
    }
  }
}

// ------------------------------------------------------------------ decode (split-KV)
// What the decode step's RoPE kernel does for one head (rope.cu, operation for operation): sum of
// the qkv projection's split-K partials, the two scales, per-head RMS norm, rotary embedding at
// position p, rounded to bf16. One warp per head, four dimensions per lane. is_v: the value head is
// only summed, scaled and rounded.
struct RopeFuseArgs {
  const float* part;   // [splits][B][nqkv] raw accumulators of the qkv projection (null: q is read from memory)
  int splits;
  const float* sx;     // [B]
  const float* sw;     // [nqkv]
  const float* cos_t;  // [max_pos][64]
  const float* sin_t;
  const float* qgain;
  const float* kgain;
  float eps;
  int max_pos;
  bf16* kcache;        // the caches again, writable: the new token's key and value rows are appended here
  bf16* vcache;
};
// What of it does not depend on the projection: weight scales, gains, and cos and sin of the position (a constant table).
struct RopeConst {
  float4 w, g, c, s;
};
__device__ __forceinline__ RopeConst rope_const(const RopeFuseArgs& r, int64_t col0, const float* gain, int p, bool is_v, int lane) {
  RopeConst k;
  k.w = *(const float4*)(r.sw + col0 + lane * 4);
  k.g = k.c = k.s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!is_v) {
    const int i0 = (lane & 15) * 4;
    k.g = *(const float4*)(gain + lane * 4);
    k.c = *(const float4*)(r.cos_t + (int64_t)p * (D / 2) + i0);
    k.s = *(const float4*)(r.sin_t + (int64_t)p * (D / 2) + i0);
  }
  return k;
}
struct RopeParts {
  float4 v[8];
  float sx;
};
__device__ __forceinline__ RopeParts rope_parts(const RopeFuseArgs& r, int B, int b, int64_t nqkv, int64_t col0, int lane) {
  RopeParts p;
#pragma unroll
  for (int s = 0; s < 8; s++)
    if (s < r.splits) p.v[s] = *(const float4*)(r.part + ((int64_t)s * B + b) * nqkv + col0 + lane * 4);
  p.sx = r.sx[b];
  return p;
}
__device__ __forceinline__ uint2 rope_head_bf16(const RopeFuseArgs& r, const RopeConst& k, const RopeParts& p, bool is_v, int lane) {
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  const float sxr = p.sx;
#pragma unroll
  for (int s = 0; s < 8; s++)
    if (s < r.splits) { acc[0] += p.v[s].x; acc[1] += p.v[s].y; acc[2] += p.v[s].z; acc[3] += p.v[s].w; }
  float x[4] = {__fmul_rn(__fmul_rn(acc[0], sxr), k.w.x), __fmul_rn(__fmul_rn(acc[1], sxr), k.w.y), __fmul_rn(__fmul_rn(acc[2], sxr), k.w.z),
                __fmul_rn(__fmul_rn(acc[3], sxr), k.w.w)};
  float o[4];
  if (!is_v) {
    const float ss = warp_sum(x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3]);
    const float rr = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)D), r.eps)));
    const float n[4] = {__fmul_rn(__fmul_rn(x[0], rr), k.g.x), __fmul_rn(__fmul_rn(x[1], rr), k.g.y), __fmul_rn(__fmul_rn(x[2], rr), k.g.z),
                        __fmul_rn(__fmul_rn(x[3], rr), k.g.w)};
    const float cs[4] = {k.c.x, k.c.y, k.c.z, k.c.w}, sn[4] = {k.s.x, k.s.y, k.s.z, k.s.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float other = __shfl_xor_sync(0xffffffffu, n[j], 16);
      o[j] = lane < 16 ? __fsub_rn(__fmul_rn(n[j], cs[j]), __fmul_rn(other, sn[j])) : __fadd_rn(__fmul_rn(n[j], cs[j]), __fmul_rn(other, sn[j]));
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; j++) o[j] = x[j];
  }
  return make_uint2(f32_to_bf16_bits(o[0]) | (f32_to_bf16_bits(o[1]) << 16), f32_to_bf16_bits(o[2]) | (f32_to_bf16_bits(o[3]) << 16));
}

// A length that the previous step's last kernel writes: read around every cache, before and after the dependency wait.
__device__ __forceinline__ int ld_volatile_i32(const int32_t* p) {
  int v;
  asm volatile("ld.volatile.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// grid (nsplit, Hkv, B), 128 threads. Warp w owns keys [16w,16w+16) of every 64-key tile.
// HD = dims of a cache row (64 or 128).
// scratch: o_part [B][Hq][nsplit][HD] then ml_part [B][Hq][nsplit][2].
// FUSED: the queries do not come from memory; every block computes the (at most 16) query heads of
// its KV head from the qkv projection's partial results (sum, scales, QK-norm, RoPE), and the block
// whose key chunk holds the new token's position also computes that token's key and value rows,
// appends them to the cache and patches them into its own shared-memory tile (its tile load may
// have read that row before the append). One kernel less per layer of the decode step.
// MERGE: the blocks of a (sequence, KV head) are one cluster, and the merge of the key chunks happens inside it: the active blocks share the G * HD
// outputs, each pushes its part of every share to the owner's shared memory (st.async, which also counts the bytes on the owner's
// mbarrier), and the owner writes the finished bf16 values to `out`. No partial results in memory and no kernel to merge them
// (Qwen3-0.6B: 2.9 us of a layer's 22 at batch 1, 3.4 at batch 8). For consumers that take bf16 rows: a maximum over all heads of a token does not exist here.
constexpr int MERGE_MAX = 8;  // blocks of a cluster
__host__ __device__ constexpr size_t merge_bytes(int G, int HD) { return (size_t)(G * (HD / 4) + MERGE_MAX) * 16 + (size_t)MERGE_MAX * G * 8; }
template <int HD, bool FUSED, bool MERGE = false>
__global__ void __launch_bounds__(128) attn_decode_kernel(const bf16* q, const bf16* kc, const bf16* vc,
                                                          const int32_t* lens, int len_add, int B, int Hq, int Hkv, int maxlen,
                                                          int chunk, int nsplit, float scale_log2, float* __restrict__ o_part,
                                                          float* __restrict__ ml_part, RopeFuseArgs rf, int prefetch, bf16* __restrict__ out = nullptr,
                                                          int* status = nullptr) {
  static_assert(!FUSED || HD == D, "the RoPE prologue is for 128 dims");
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(16) bf16 q_s[FUSED ? 16 * HD : 8];    // the query heads of this KV head
  __shared__ __align__(16) bf16 kv_new[FUSED ? 2 * HD : 8];  // the new token's key row, then its value row
  __shared__ __align__(8) unsigned long long merge_bar;
  __shared__ int len_s;
  SB_TRACE_BEGIN();
  if (MERGE) {
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&merge_bar)));
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();  // .aligned: the whole warp at once
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  pdl_trigger();
  const int split = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
  // One reading for the whole block: the length may change at any time until the dependency wait, and what follows from it, barriers among
  // it, has to be the same for every thread.
  if (threadIdx.x == 0) len_s = ld_volatile_i32(lens + b);
  __syncthreads();
  const int G = Hq / Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
  const int k_begin = split * chunk;
  const uint32_t sK = smem_u32(smem), sV = sK + DEC_STAGES * KT * 2 * HD;
  const bf16* kbase = kc + ((int64_t)b * Hkv + hk) * maxlen * HD;
  const bf16* vbase = vc + ((int64_t)b * Hkv + hk) * maxlen * HD;
  const uint64_t kv_policy = l2_evict_first_policy();
  // Before the dependency wait: the first tiles of this block's keys and values start to stream
  // while the preceding kernels (the qkv projection's tail, RoPE) still run. Only rows that were
  // written in earlier steps are touched, never the block's last tile (it may hold the row the
  // preceding kernel appends; FUSED: whatever is read of that row is replaced by the block itself, so the last tile too), and the
  // length they are derived from is read again after the wait: if it changed, the tiles are loaded again from scratch.
  const int len_early = min(len_s + len_add, maxlen);
  int npre = 0;
  if (prefetch && k_begin < len_early) {
    const int nt = (min(len_early, k_begin + chunk) - k_begin + KT - 1) / KT;
    npre = FUSED ? min(DEC_STAGES, nt) : min(DEC_STAGES - 1, nt - 1);
    for (int t = 0; t < npre; t++) {
      const int k0 = k_begin + t * KT, valid = FUSED ? min(KT, min(len_early, k_begin + chunk) - k0) : KT;
      load_tile_hint<HD>(sK + t * KT * 2 * HD, kbase + (int64_t)k0 * HD, KT, valid, 128, kv_policy);
      load_tile_hint<HD>(sV + t * KT * 2 * HD, vbase + (int64_t)k0 * HD, KT, valid, 128, kv_policy);
      cp_async_commit();
    }
  }
  // FUSED: the warp's item of the prologue (0..G-1: the query heads; G, G+1: the new token's key and value heads), and its constants
  const int64_t nqkv = (int64_t)(Hq + 2 * Hkv) * HD;
  auto item_col = [&](int i) { return (int64_t)(i < G ? hk * G + i : Hq + (i == G + 1 ? Hkv : 0) + hk) * HD; };
  auto item_const = [&](int i, int length) {
    return rope_const(rf, item_col(i), i < G ? rf.qgain : rf.kgain, max(0, min(length - 1, rf.max_pos - 1)), i == G + 1, lane);
  };
  RopeConst rk;
  RopeParts rp;
  if (FUSED && warp < G + 2) rk = item_const(warp, len_early);
  pdl_wait();
  SB_TRACE_WAITED();
  if (FUSED && warp < G + 2) rp = rope_parts(rf, B, b, nqkv, item_col(warp), lane);  // in flight together with the length
  const int len = min(ld_volatile_i32(lens + b) + len_add, maxlen);
  if (len != len_early && npre) {  // not expected: the length belongs to the previous step
    cp_async_wait<0>();
    __syncthreads();
    npre = 0;
  }
  if (MERGE) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every block's barrier is initialised
  if (k_begin >= len) return;
  const int k_end = min(len, k_begin + chunk);
  // FUSED: position of the new token = the sequence's length before this step; its row is the last key
  const int p_new = FUSED ? len - 1 : -1;
  const bool owns_new = FUSED && p_new >= k_begin && p_new < k_end && p_new < rf.max_pos;
  const int ntiles = (k_end - k_begin + KT - 1) / KT;

  // prologue: the first DEC_STAGES-1 tiles are in flight before any is consumed (one group per tile)
  for (int t = npre; t < DEC_STAGES - 1; t++) {
    if (t < ntiles) {
      int k0 = k_begin + t * KT;
      load_tile_hint<HD>(sK + t * KT * 2 * HD, kbase + (int64_t)k0 * HD, KT, min(KT, k_end - k0), 128, kv_policy);
      load_tile_hint<HD>(sV + t * KT * 2 * HD, vbase + (int64_t)k0 * HD, KT, min(KT, k_end - k0), 128, kv_policy);
    }
    cp_async_commit();
  }

  if (FUSED) {
    for (int i = warp; i < G + (owns_new ? 2 : 0); i += 4) {
      if (i != warp || len != len_early) rk = item_const(i, len);
      if (i != warp) rp = rope_parts(rf, B, b, nqkv, item_col(i), lane);
      const bool is_v = i == G + 1;
      const uint2 w = rope_head_bf16(rf, rk, rp, is_v, lane);
      if (i < G) {
        *(uint2*)(q_s + i * HD + lane * 4) = w;
      } else {
        *(uint2*)(kv_new + (is_v ? HD : 0) + lane * 4) = w;
        bf16* cache = is_v ? rf.vcache : rf.kcache;
        *(uint2*)(cache + (((int64_t)b * Hkv + hk) * maxlen + p_new) * HD + lane * 4) = w;
      }
    }
    __syncthreads();
  }
  SB_TRACE_MARK(0);
  // Q fragments: rows = the G query heads of this KV head (zero beyond), from memory or from the prologue above
  uint32_t qf[HD / 16][4];
  {
    const bf16* q0 = FUSED ? q_s : q + ((int64_t)b * Hq + hk * G) * HD;
#pragma unroll
    for (int ks = 0; ks < HD / 16; ks++) {
      int d0 = ks * 16 + 2 * tig;
      qf[ks][0] = g < G ? *(const uint32_t*)(q0 + g * HD + d0) : 0u;
      qf[ks][1] = g + 8 < G ? *(const uint32_t*)(q0 + (g + 8) * HD + d0) : 0u;
      qf[ks][2] = g < G ? *(const uint32_t*)(q0 + g * HD + d0 + 8) : 0u;
      qf[ks][3] = g + 8 < G ? *(const uint32_t*)(q0 + (g + 8) * HD + d0 + 8) : 0u;
    }
  }
  float o[HD / 8][4];
#pragma unroll
  for (int j = 0; j < HD / 8; j++)
#pragma unroll
    for (int i = 0; i < 4; i++) o[j][i] = 0.f;
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  const int mi = lane >> 3, r8 = lane & 7;

  for (int t = 0; t < ntiles; t++) {
    {
      const int tn = t + DEC_STAGES - 1;  // refill the stage consumed in the previous iteration
      if (tn < ntiles && tn >= npre) {
        int k0 = k_begin + tn * KT;
        load_tile_hint<HD>(sK + (tn % DEC_STAGES) * KT * 2 * HD, kbase + (int64_t)k0 * HD, KT, min(KT, k_end - k0), 128, kv_policy);
        load_tile_hint<HD>(sV + (tn % DEC_STAGES) * KT * 2 * HD, vbase + (int64_t)k0 * HD, KT, min(KT, k_end - k0), 128, kv_policy);
      }
      cp_async_commit();
      cp_async_wait<DEC_STAGES - 1>();  // all but the newest DEC_STAGES-1 groups: tile t has landed
    }
    __syncthreads();
    const uint32_t tK = sK + (t % DEC_STAGES) * KT * 2 * HD, tV = sV + (t % DEC_STAGES) * KT * 2 * HD;
    if (FUSED && owns_new && p_new >= k_begin + t * KT && p_new < k_begin + (t + 1) * KT) {
      // the tile copy may have read the new token's row before it was appended: put the rows computed above in its place
      if (warp == 0) {
        const int row = p_new - (k_begin + t * KT), cc = lane & 15;
        const uint4 w = *(const uint4*)(kv_new + (lane < 16 ? 0 : HD) + cc * 8);
        *(uint4*)(smem + ((lane < 16 ? tK : tV) - sK) + tile_off<HD>(row, cc)) = w;
      }
      __syncthreads();
    }
    float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int ks = 0; ks < HD / 16; ks++) {
      uint32_t kb[4];
      ldsm_x4(tK + tile_off<HD>(warp * 16 + (mi >> 1) * 8 + r8, 2 * ks + (mi & 1)), kb);
      mma_bf16(s[0], qf[ks], kb[0], kb[1]);
      mma_bf16(s[1], qf[ks], kb[2], kb[3]);
    }
    const int kpos0 = k_begin + t * KT + warp * 16;
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        int kpos = kpos0 + 8 * j + 2 * tig + (i & 1);
        float v = kpos >= k_end ? -INFINITY : s[j][i] * scale_log2;
        s[j][i] = v;
        mx[i >> 1] = fmaxf(mx[i >> 1], v);
      }
    float corr[2], m_use[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
      float m_new = fmaxf(m_run[r], mx[r]);
      m_use[r] = m_new == -INFINITY ? 0.f : m_new;
      corr[r] = exp2f(m_run[r] - m_use[r]);
      m_run[r] = m_new;
    }
    uint32_t pf[4], pl[4];
    {
      float p[2][4];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        p[j][0] = exp2f(s[j][0] - m_use[0]); p[j][1] = exp2f(s[j][1] - m_use[0]);
        p[j][2] = exp2f(s[j][2] - m_use[1]); p[j][3] = exp2f(s[j][3] - m_use[1]);
      }
      l_run[0] = l_run[0] * corr[0] + (p[0][0] + p[0][1] + p[1][0] + p[1][1]);
      l_run[1] = l_run[1] * corr[1] + (p[0][2] + p[0][3] + p[1][2] + p[1][3]);
      split_bf16(p[0][0], p[0][1], pf[0], pl[0]); split_bf16(p[0][2], p[0][3], pf[1], pl[1]);
      split_bf16(p[1][0], p[1][1], pf[2], pl[2]); split_bf16(p[1][2], p[1][3], pf[3], pl[3]);
    }
#pragma unroll
    for (int j = 0; j < HD / 8; j++) {
      o[j][0] *= corr[0]; o[j][1] *= corr[0];
      o[j][2] *= corr[1]; o[j][3] *= corr[1];
    }
#pragma unroll
    for (int jj = 0; jj < HD / 16; jj++) {
      uint32_t vb[4];
      ldsm_x4_t(tV + tile_off<HD>(warp * 16 + (mi & 1) * 8 + r8, 2 * jj + (mi >> 1)), vb);
      mma_bf16(o[2 * jj], pf, vb[0], vb[1]);
      mma_bf16(o[2 * jj + 1], pf, vb[2], vb[3]);
      mma_bf16(o[2 * jj], pl, vb[0], vb[1]);
      mma_bf16(o[2 * jj + 1], pl, vb[2], vb[3]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 2; r++) {
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
  }
  SB_TRACE_MARK(1);
  // merge the four warps through shared memory (tiles are free after the last barrier)
  float* so = (float*)smem;                       // [4 warps][16 rows][HD]
  float* sml = so + 4 * 16 * HD;                   // [4 warps][16 rows][2]
#pragma unroll
  for (int r = 0; r < 2; r++) {
    int row = g + 8 * r;
    if (row < G) {
#pragma unroll
      for (int j = 0; j < HD / 8; j++) {
        so[(warp * 16 + row) * HD + 8 * j + 2 * tig] = o[j][2 * r];
        so[(warp * 16 + row) * HD + 8 * j + 2 * tig + 1] = o[j][2 * r + 1];
      }
      if (tig == 0) { sml[(warp * 16 + row) * 2] = m_run[r]; sml[(warp * 16 + row) * 2 + 1] = l_run[r]; }
    }
  }
  __syncthreads();
  if constexpr (MERGE) {
    const int ns = (len + chunk - 1) / chunk, e4n = G * (HD / 4), per = (e4n + ns - 1) / ns;  // float4s of all outputs and of the largest share
    const int lo = split * e4n / ns, hi = (split + 1) * e4n / ns;                              // this block's share
    float4* slots = (float4*)(smem + 2 * DEC_STAGES * KT * 2 * HD);                            // [source][per]
    float2* ml = (float2*)(slots + e4n + MERGE_MAX);                                           // [source][G]
    const uint32_t bar = smem_u32(&merge_bar);
    if (threadIdx.x == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)((ns - 1) * ((hi - lo) * 16 + G * 8))) : "memory");
    auto remote = [](uint32_t local, int rank) {
      uint32_t a;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
      return a;
    };
    for (int e = threadIdx.x; e < e4n; e += 128) {
      const int row = e / (HD / 4), d = (e % (HD / 4)) * 4;
      float M = -INFINITY;
#pragma unroll
      for (int w = 0; w < 4; w++) M = fmaxf(M, sml[(w * 16 + row) * 2]);
      float L = 0.f;
      float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < 4; w++) {
        const float mw = sml[(w * 16 + row) * 2], f = mw == -INFINITY ? 0.f : exp2f(mw - M);
        const float4 p = *(const float4*)(so + (w * 16 + row) * HD + d);
        L += sml[(w * 16 + row) * 2 + 1] * f;
        O.x += p.x * f; O.y += p.y * f; O.z += p.z * f; O.w += p.w * f;
      }
      const int owner = ((e + 1) * ns - 1) / e4n;
      float4* at = slots + split * per + (e - owner * e4n / ns);
      if (owner == split) *at = O;
      else
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(remote(smem_u32(at), owner)),
                     "r"(__float_as_uint(O.x)), "r"(__float_as_uint(O.y)), "r"(__float_as_uint(O.z)), "r"(__float_as_uint(O.w)), "r"(remote(bar, owner))
                     : "memory");
      if (d == 0) {
        ml[split * G + row] = make_float2(M, L);
        for (int r = 0; r < ns; r++)
          if (r != split)
            asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(remote(smem_u32(ml + split * G + row), r)),
                         "r"(__float_as_uint(M)), "r"(__float_as_uint(L)), "r"(remote(bar, r))
                         : "memory");
      }
    }
    __syncthreads();
    SB_TRACE_MARK(2);
    uint32_t done = 0;
    for (uint32_t spins = 0; !done && spins < (1u << 20); spins++)
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar), "r"(0u) : "memory");
    if (__builtin_expect(!__all_sync(0xffffffffu, done), 0)) {
      // What should have come did not: no output, and this block's shared memory stays until the others, which may be late, have left or given up too.
      if (lane == 0) { *(volatile int*)status = 6; __threadfence_system(); }
      __syncwarp();
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      return;
    }
    for (int e = lo + (int)threadIdx.x; e < hi; e += 128) {
      const int row = e / (HD / 4), d = (e % (HD / 4)) * 4;
      float M = -INFINITY;
      for (int s = 0; s < ns; s++) M = fmaxf(M, ml[s * G + row].x);
      float L = 0.f, O[4] = {0.f, 0.f, 0.f, 0.f};
      for (int s = 0; s < ns; s++) {
        const float2 m = ml[s * G + row];
        const float4 p = slots[s * per + e - lo];
        const float f = exp2f(m.x - M);
        L += m.y * f;
        O[0] += p.x * f; O[1] += p.y * f; O[2] += p.z * f; O[3] += p.w * f;
      }
      *(uint2*)(out + ((int64_t)b * Hq + hk * G + row) * HD + d) = make_uint2(pack_bf16(O[0] / L, O[1] / L), pack_bf16(O[2] / L, O[3] / L));
    }
    SB_TRACE_END(SB_K_ATTN, 0);
    return;
  }
  for (int e = threadIdx.x; e < G * HD; e += 128) {
    int row = e / HD, d = e - row * HD;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; w++) M = fmaxf(M, sml[(w * 16 + row) * 2]);
    float L = 0.f, O = 0.f;
#pragma unroll
    for (int w = 0; w < 4; w++) {
      float mw = sml[(w * 16 + row) * 2];
      float f = mw == -INFINITY ? 0.f : exp2f(mw - M);
      L += sml[(w * 16 + row) * 2 + 1] * f;
      O += so[(w * 16 + row) * HD + d] * f;
    }
    int64_t idx = ((int64_t)b * Hq + hk * G + row) * nsplit + split;
    o_part[idx * HD + d] = O;
    if (d == 0) { ml_part[idx * 2] = M; ml_part[idx * 2 + 1] = L; }
  }
  SB_TRACE_END(SB_K_ATTN, 0);
}

// grid B, 512 threads: merge the key chunks of every head of one token. A thread owns 8
// consecutive dims of one head (two when Hq > 32) and keeps them in registers for the optional
// two-term E4M3 split of the whole token row [Hq*128] (the o_proj input).
constexpr int CB_THREADS = 512, CB_ITEMS = 2;
__global__ void __launch_bounds__(CB_THREADS) attn_combine_kernel(const float* o_part, const float* ml_part,
                                                                  const int32_t* lens, int len_add, int Hq, int maxlen, int chunk,
                                                                  int nsplit, bf16* __restrict__ out, uint8_t* __restrict__ q_out,
                                                                  float* __restrict__ qscale) {
  __shared__ float red[32];
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.x;
  const int len = min(lens[b] + len_add, maxlen);
  const int ns = (len + chunk - 1) / chunk;
  float v[CB_ITEMS][8];
  float amax = 0.f;
#pragma unroll
  for (int it = 0; it < CB_ITEMS; it++) {
    int e8 = threadIdx.x + it * CB_THREADS;  // index of an 8-dim group of the row
    if (e8 < Hq * (D / 8)) {
      int h = e8 / (D / 8), d = (e8 - h * (D / 8)) * 8;
      int64_t base = ((int64_t)b * Hq + h) * nsplit;
      float M = -INFINITY;
      for (int s = 0; s < ns; s++) M = fmaxf(M, ml_part[(base + s) * 2]);
      float L = 0.f, O[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int s = 0; s < ns; s++) {
        float f = exp2f(ml_part[(base + s) * 2] - M);
        L += ml_part[(base + s) * 2 + 1] * f;
        const float4* op = (const float4*)(o_part + (base + s) * D + d);
        float4 o0 = op[0], o1 = op[1];
        O[0] += o0.x * f; O[1] += o0.y * f; O[2] += o0.z * f; O[3] += o0.w * f;
        O[4] += o1.x * f; O[5] += o1.y * f; O[6] += o1.z * f; O[7] += o1.w * f;
      }
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        v[it][i] = ns > 0 ? round_bf16(O[i] / L) : 0.f;
        amax = fmaxf(amax, fabsf(v[it][i]));
      }
#pragma unroll
      for (int i = 0; i < 4; i++) w[i] = pack_bf16(v[it][2 * i], v[it][2 * i + 1]);
      *(uint4*)(out + ((int64_t)b * Hq + h) * D + d) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  if (!q_out) return;
  amax = block_max(amax, red);
  int ex = sb_scale_exponent(amax);
  float inv = sb_pow2(-ex);
  if (threadIdx.x == 0) qscale[b] = sb_pow2(ex);
#pragma unroll
  for (int it = 0; it < CB_ITEMS; it++) {
    int e8 = threadIdx.x + it * CB_THREADS;
    if (e8 < Hq * (D / 8)) sb_store_split8(q_out, (int64_t)Hq * D, b, (int64_t)e8 * 8, v[it], inv);
  }
}

// The decode-step shape of the merge: one thread per 4-dim group of the token's attention row
// (blockDim.x == Hq * 32 <= 1024), at most 8 key chunks, so a thread has at most 16 small loads
// in flight. Every partial is loaded in one batch together with the sequence length (slots of
// chunks beyond the length hold stale data and are masked out of the arithmetic, which is that
// of the kernel above).
__global__ void __launch_bounds__(1024) attn_combine_decode_kernel(const float* o_part, const float* ml_part,
                                                                   const int32_t* lens, int len_add, int Hq, int maxlen, int chunk,
                                                                   int nsplit, bf16* __restrict__ out, uint8_t* __restrict__ q_out,
                                                                   float* __restrict__ qscale, int* __restrict__ status) {
  __shared__ float red[32];
  __shared__ __align__(8) ClusterExchange xch;
  SB_TRACE_BEGIN();
  if (gridDim.y > 1) cluster_exchange_init(&xch);  // the blocks of one cluster share a token (some of its heads each)
  pdl_trigger();
  pdl_wait();
  SB_TRACE_WAITED();
  const int b = blockIdx.x;
  const int e4 = blockIdx.y * blockDim.x + threadIdx.x, h = e4 >> 5, d = (e4 & 31) * 4;
  const int64_t base = ((int64_t)b * Hq + h) * nsplit;
  const int len_raw = lens[b];
  float2 ml[8];
  float4 o[8];
#pragma unroll
  for (int s = 0; s < 8; s++)
    if (s < nsplit) {
      ml[s] = *(const float2*)(ml_part + (base + s) * 2);
      o[s] = *(const float4*)(o_part + (base + s) * D + d);
    }
  const int len = min(len_raw + len_add, maxlen);
  const int ns = (len + chunk - 1) / chunk;
  float M = -INFINITY;
#pragma unroll
  for (int s = 0; s < 8; s++)
    if (s < ns) M = fmaxf(M, ml[s].x);
  float L = 0.f, O[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int s = 0; s < 8; s++)
    if (s < ns) {
      float f = exp2f(ml[s].x - M);
      L += ml[s].y * f;
      O[0] += o[s].x * f; O[1] += o[s].y * f; O[2] += o[s].z * f; O[3] += o[s].w * f;
    }
  float v[4], amax = 0.f;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    v[i] = ns > 0 ? round_bf16(O[i] / L) : 0.f;
    amax = fmaxf(amax, fabsf(v[i]));
  }
  *(uint2*)(out + ((int64_t)b * Hq + h) * D + d) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
  if (q_out) {
    amax = block_max(amax, red);
    if (gridDim.y > 1) {
      if (!cluster_exchange(&xch, amax, gridDim.y, blockIdx.y, 0) && threadIdx.x == 0) { *(volatile int*)status = 6; __threadfence_system(); }
      for (uint32_t r = 0; r < gridDim.y; r++) amax = fmaxf(amax, ((volatile float*)xch.slot[0])[r]);
    }
    const int ex = sb_scale_exponent(amax);
    if (blockIdx.y == 0 && threadIdx.x == 0) qscale[b] = sb_pow2(ex);
    sb_store_split4(q_out, (int64_t)Hq * D, b, (int64_t)e4 * 4, v, sb_pow2(-ex));
  }
  SB_TRACE_END(SB_K_COMBINE, 0);
}

}  // namespace

int k_attn_prefill_tc(strictb200_ctx* ctx, const bf16* q, const bf16* kc, const bf16* vc, const int32_t* lens, const int32_t* past,
                      const int32_t* qstart, int B, int S, int64_t q_rows, int Hq, int Hkv, int maxlen, float scale, bf16* out);  // attention_tc.cu

int k_attn_prefill(strictb200_ctx* ctx, const bf16* q, const bf16* kc, const bf16* vc, const int32_t* lens, const int32_t* past,
                   const int32_t* qstart, int B, int S, int64_t q_rows, int Hq, int Hkv, int Dh, int maxlen, float scale, bf16* out) {
  if (Dh != D) return sb_fail(STRICTB200_ERR_UNSUPPORTED, "attention: head_dim must be 128");
  // tcgen05 kernel first; the mma.sync kernel below takes what it declines
  if (ctx->opt.attn_tc != 0) {
    int st = k_attn_prefill_tc(ctx, q, kc, vc, lens, past, qstart, B, S, q_rows, Hq, Hkv, maxlen, scale, out);
    if (st != STRICTB200_ERR_UNSUPPORTED) return st;
  }
  static SbDeviceOnce once;
  size_t smem = 64 * 256 + 4 * KT * 256;
  SB_CUDA(once.run(ctx->device, [&] { return cudaFuncSetAttribute(attn_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }));
  if (Hq > 65535 || B > 65535) return sb_fail(STRICTB200_ERR_INVALID_ARG, "attention: too many heads or sequences");
  dim3 grid((S + 63) / 64, Hq, B);
  attn_prefill_kernel<<<grid, 128, smem, ctx->stream>>>(q, kc, vc, lens, past, qstart, S, Hq, Hkv, maxlen, scale * LOG2E, out);
  SB_LAUNCHED(ctx);
  return STRICTB200_OK;
}

SB_TRACE_TU(attention)

static int merge_set_up(strictb200_ctx* ctx) {
  static SbDeviceOnce once;
  SB_CUDA(once.run(ctx->device, [&] {
    const int most = (int)(2 * DEC_STAGES * KT * 256 + merge_bytes(16, D));
    const cudaError_t e = cudaFuncSetAttribute(attn_decode_kernel<D, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    return e == cudaSuccess ? cudaFuncSetAttribute(attn_decode_kernel<D, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) : e;
  }));
  return STRICTB200_OK;
}
// Clusters of `size` blocks of the merging form that run at once. A cluster needs its blocks' places in one part of the GPU, and of more than four blocks the calculator's
// number did not all start together: 48 of 48 clusters of eight, 56 of 56 of seven, 80 of 82 of five, 64 of 71 of six and 30 of 33 of eight (with 16 heads) left
// some for a second wave, 40 of 48, 48 of 71, 64 of 82 and 28 of 33 did not; 96 of 104 clusters of four neither, 128 of 142 of three hardly ever.
static int64_t merge_clusters(strictb200_ctx* ctx, bool fused, int heads, int size) {
  static std::mutex mu;
  static int known[64][2][17][MERGE_MAX + 1] = {};
  std::lock_guard<std::mutex> lock(mu);
  int& n = known[ctx->device & 63][fused][std::min(heads, 16)][std::min(size, MERGE_MAX)];
  if (!n) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)size;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)size);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = 2 * DEC_STAGES * KT * 256 + merge_bytes(heads, D);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaErrorUnknown;
    if (merge_set_up(ctx) == STRICTB200_OK)
      e = fused ? cudaOccupancyMaxActiveClusters(&n, attn_decode_kernel<D, true, true>, &cfg) : cudaOccupancyMaxActiveClusters(&n, attn_decode_kernel<D, false, true>, &cfg);
    if (e != cudaSuccess || n < 1) { cudaGetLastError(); n = 1; }
    if (size > 4) n = std::max(1, n - n / 8);
  }
  return n;
}

// Keys per block. All blocks of a launch take about the same time, so the grid runs in waves of
// (blocks resident per SM) x (SM count): the chunk is the multiple of the tile size that
// minimises waves x (tiles per chunk + per-block overhead) among the chunk sizes that leave at
// most 8 chunks for a full cache. The waves are counted for sequences of `len_plan` keys (0: a
// full cache): a cache that holds 2100 of 2432 keys in chunks of 512 runs four full chunks and a
// stub per sequence, chunks of 448 run five even ones (14 % less attention time, measured). The
// attn_blocks_per_sm option restores the plain "that many blocks per SM" rule. `fused`: the kernel with the RoPE prologue will run;
// `merge_heads`: the form that merges its chunks in a cluster, with that many query heads per KV head (0: not that one). Its waves are clusters (blocks without keys
// leave at once and are not counted). Planned by blocks, 10 sequences of 2000 keys with 8 KV heads ran 80 clusters of five in two waves: 25.3 us; 80 of four: 18.8.
static int decode_chunk(strictb200_ctx* ctx, int B, int Hkv, int maxlen, int len_plan = 0, bool fused = false, bool short_chunks = true, int merge_heads = 0) {
  const int per_sm = ctx->opt.attn_blocks_per_sm;
  const int tiles = (maxlen + KT - 1) / KT;
  const int tiles_plan = len_plan > 0 && len_plan < maxlen ? (len_plan + KT - 1) / KT : tiles;
  if (per_sm > 0) {
    int64_t c = (int64_t)maxlen * B * Hkv / ((int64_t)ctx->sm_count * per_sm);
    c = (c + KT - 1) / KT * KT;
    if (c < 256) c = 256;
    if (c > maxlen) c = (int64_t)tiles * KT;
    return (int)c;
  }
  static SbDeviceOnce once;
  static int resident_of[64] = {};  // blocks of the kernel an SM holds, per device
  const size_t smem_dec = 2 * DEC_STAGES * KT * 256;
  static int resident_fused_of[64] = {};
  once.run(ctx->device, [&] {
    cudaFuncSetAttribute(attn_decode_kernel<D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_dec);
    cudaFuncSetAttribute(attn_decode_kernel<D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_dec);
    int r = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, attn_decode_kernel<D, false>, 128, smem_dec) != cudaSuccess || r < 1) r = 1;
    resident_of[ctx->device & 63] = r;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, attn_decode_kernel<D, true>, 128, smem_dec) != cudaSuccess || r < 1) r = 1;
    resident_fused_of[ctx->device & 63] = r;
    return cudaSuccess;
  });
  const int res0 = (fused ? resident_fused_of : resident_of)[ctx->device & 63];
  const int resident = res0 > 0 ? res0 : 1;
  const int64_t slots = (int64_t)ctx->sm_count * resident, pairs = (int64_t)B * Hkv;
  auto waves_of = [&](int c) -> int64_t {
    const int chunks = (tiles_plan + c - 1) / c;
    if (!merge_heads) return (pairs * chunks + slots - 1) / slots;
    const int64_t at_once = merge_clusters(ctx, fused, merge_heads, chunks);
    return (pairs + at_once - 1) / at_once;
  };
  int best = tiles;
  double best_cost = 1e30;
  // At most 8 chunks per sequence: that is what the fast merge kernel takes. 16 chunks for the few
  // (sequence, head) pairs of TP=8 shortened the attention kernel but the general merge kernel they
  // need cost more than that (21.9 against 17.0 us per layer for the pair, measured on eight GPUs).
  // Less than four tiles (256 keys) only while all blocks are resident at once (8 sequences of 544 keys, 8 KV heads: chunks of 256 keys
  // walked four tiles one after the other on some SMs and one on others, 8.7 us; chunks of 128, 5.7 us). In several waves short chunks gain nothing and
  // multiply the partial results (`short_chunks` false: never).
  for (int c = (tiles + 7) / 8; c <= tiles; c++) {
    const int64_t waves = waves_of(c);
    if (c < 4 && c < tiles && (!short_chunks || waves > 1)) continue;
    // (counting a stub as a whole block is deliberate: weighting blocks by their length made the rule pick three long
    // chunks where five short ones measured 47 us against 66)
    const double cost = (double)waves * ((double)std::min(c, tiles_plan) + 1.5);
    if (cost < best_cost - 1e-9) { best_cost = cost; best = c; }
  }
  return best * KT;
}
static int splits_of(int maxlen, int chunk) { return (maxlen + chunk - 1) / chunk; }
int sb_attn_decode_splits(strictb200_ctx* ctx, int B, int Hkv, int maxlen) { return splits_of(maxlen, decode_chunk(ctx, B, Hkv, maxlen)); }
int sb_attn_decode_chunk(strictb200_ctx* ctx, int B, int Hkv, int maxlen, int len_plan, bool fused, int merge_heads) {
  return decode_chunk(ctx, B, Hkv, maxlen, len_plan, fused, true, merge_heads);
}
size_t sb_attn_decode_scratch(int B, int Hq, int Dh, int nsplit) { return (size_t)B * Hq * nsplit * (Dh + 2) * sizeof(float); }

// The key chunks alone, for a merge of the caller's: rows of HD = 64 or 128 dims, len_add = 1 (the new token's row is in the cache).
int k_attn_decode_chunks(strictb200_ctx* ctx, int HD, const bf16* q, const bf16* kc, const bf16* vc, const int32_t* lens, int B, int Hq, int Hkv, int maxlen,
                         float scale, int nsplit, int chunk, float* o_part, float* ml_part) {
  if ((HD != 64 && HD != 128) || Hq / Hkv > 16 || Hkv > 65535 || B > 65535) return sb_fail(STRICTB200_ERR_UNSUPPORTED, "attention: head shape the split-key kernel does not take");
  if (chunk <= 0 || chunk % KT || nsplit < 1) return sb_fail(STRICTB200_ERR_INVALID_ARG, "attention: bad key chunks");
  const size_t smem = 2 * DEC_STAGES * KT * 2 * HD;  // (for 128 dims decode_chunk has raised the kernel's limit)
  auto go = [&](auto kernel) {
    return sb_launch(ctx, kernel, dim3(nsplit, Hkv, B), dim3(128), smem, q, kc, vc, lens, 1, B, Hq, Hkv, maxlen, chunk, nsplit, scale * LOG2E, o_part, ml_part,
                     RopeFuseArgs{}, ctx->opt.attn_prefetch, (bf16*)nullptr, (int*)nullptr);
  };
  SB_CUDA(HD == 64 ? go(attn_decode_kernel<64, false>) : go(attn_decode_kernel<128, false>));
  ctx->launches++;
  return STRICTB200_OK;
}

int k_attn_decode(strictb200_ctx* ctx, const bf16* q, const bf16* kc, const bf16* vc, const int32_t* lens, int len_add, int B, int Hq, int Hkv,
                  int Dh, int maxlen, float scale, int nsplit, float* scratch, bf16* out, uint8_t* q_out, float* qscale_out, const RopeArgs* rope,
                  int chunk, bool cluster_merge) {
  if (Dh != D) return sb_fail(STRICTB200_ERR_UNSUPPORTED, "attention: head_dim must be 128");
  if (Hq / Hkv > 16) return sb_fail(STRICTB200_ERR_UNSUPPORTED, "attention: at most 16 query heads per KV head");
  if (Hq * (D / 8) > CB_THREADS * CB_ITEMS) return sb_fail(STRICTB200_ERR_UNSUPPORTED, "attention: at most 64 query heads per rank");
  if (chunk <= 0) chunk = decode_chunk(ctx, B, Hkv, maxlen);  // else the caller's plan (a multiple of the tile; it has run decode_chunk, which sets the kernel up)
  if (chunk % KT || (maxlen + chunk - 1) / chunk != nsplit) return sb_fail(STRICTB200_ERR_INVALID_ARG, "attention: split count does not match the cache size");
  size_t smem = 2 * DEC_STAGES * KT * 256;  // K and V rings; also covers the 34 KB merge area (the attribute is set by decode_chunk above)
  float* o_part = scratch;
  float* ml_part = scratch + (size_t)B * Hq * nsplit * D;
  if (Hkv > 65535 || B > 65535) return sb_fail(STRICTB200_ERR_INVALID_ARG, "attention: too many heads or sequences");
  dim3 grid(nsplit, Hkv, B);
  RopeFuseArgs rf{};
  if (rope) {
    // queries, key and value of the new token come from the qkv projection's partial results (see the kernel)
    if (!rope->part || rope->splits < 1 || rope->splits > 8 || len_add != 1 || Hq / Hkv > 16 || rope->Hq != Hq || rope->Hkv != Hkv ||
        rope->kcache != kc || rope->vcache != vc || rope->lens != lens)
      return sb_fail(STRICTB200_ERR_INVALID_ARG, "attention: the fused RoPE prologue needs split-K partials (at most 8), one new token and the same caches");
    rf = RopeFuseArgs{rope->part, rope->splits, rope->sx, rope->sw, rope->cos_t, rope->sin_t, rope->qgain, rope->kgain, rope->eps, rope->max_pos,
                      rope->kcache, rope->vcache};
  }
  if (cluster_merge) {
    if (q_out || nsplit > MERGE_MAX) return sb_fail(STRICTB200_ERR_INVALID_ARG, "attention: the merge inside a cluster writes bf16 rows of at most 8 key chunks");
    SB_TRY(merge_set_up(ctx));
    auto go = [&](auto kernel) -> int {
      SB_CUDA(sb_launch_cluster(ctx, kernel, grid, dim3(128), smem + merge_bytes(Hq / Hkv, D), dim3(nsplit, 1, 1), q, kc, vc, lens, len_add, B, Hq, Hkv, maxlen, chunk,
                                nsplit, scale * LOG2E, o_part, ml_part, rf, ctx->opt.attn_prefetch, out, ctx->d_status));
      ctx->launches++;
      return STRICTB200_OK;
    };
    return rope ? go(attn_decode_kernel<D, true, true>) : go(attn_decode_kernel<D, false, true>);
  }
  auto go = [&](auto kernel) {
    return sb_launch(ctx, kernel, grid, dim3(128), smem, q, kc, vc, lens, len_add, B, Hq, Hkv, maxlen, chunk, nsplit, scale * LOG2E, o_part, ml_part, rf,
                     ctx->opt.attn_prefetch, (bf16*)nullptr, (int*)nullptr);
  };
  SB_CUDA(rope ? go(attn_decode_kernel<D, true>) : go(attn_decode_kernel<D, false>));
  ctx->launches++;
  sb_prof_split(ctx, STRICTB200_K_ATTN_MERGE);
  // The merge stays a kernel of its own: done inside the attention kernel by the last block of every (sequence, head) and
  // of every sequence to finish (fence, counters), it cost 3 us per layer more than this launch (55.0 against 46.8 + 5.1 us).
  if (nsplit <= 8 && Hq <= 32) {
    // blocks per token (one cluster): 8 heads = 256 threads each
    const unsigned per_tok = q_out && ctx->opt.row_cluster > 1 && Hq % 8 == 0 ? (unsigned)std::min(ctx->opt.row_cluster, Hq / 8) : 1u;
    if (per_tok > 1 && Hq % per_tok == 0)
      SB_CUDA(sb_launch_cluster(ctx, attn_combine_decode_kernel, dim3(B, per_tok), dim3((unsigned)(Hq * 32 / per_tok)), 0, dim3(1, per_tok, 1), (const float*)o_part,
                                (const float*)ml_part, lens, len_add, Hq, maxlen, chunk, nsplit, out, q_out, qscale_out, ctx->d_status));
    else
      SB_CUDA(sb_launch(ctx, attn_combine_decode_kernel, dim3(B), dim3((unsigned)(Hq * 32)), 0, (const float*)o_part, (const float*)ml_part, lens, len_add, Hq,
                        maxlen, chunk, nsplit, out, q_out, qscale_out, ctx->d_status));
    ctx->launches++;
    return STRICTB200_OK;
  }
  SB_CUDA(sb_launch(ctx, attn_combine_kernel, dim3(B), dim3(CB_THREADS), 0, o_part, ml_part, lens, len_add, Hq, maxlen, chunk, nsplit, out, q_out, qscale_out));
  ctx->launches++;
  return STRICTB200_OK;
}

// ------------------------------------------------------------------ decode attention without any allocation
// Some hosts of this library must not trigger an allocation while they serve requests: a
// latency-critical decode loop cannot afford the device-wide synchronisation that cudaMalloc and
// cudaFree imply (every stream of the process stalls behind them), and a host that hands out the
// GPU's memory from its own pool at start-up leaves the driver's allocator nothing to give, so a
// late request for scratch would simply fail. For those callers the split-KV partial results live
// in a fixed array that is part of the library image: every GPU that loads the library carries
// these 4 MiB from load to exit, whether or not the entry point is ever called.
namespace {
constexpr size_t NOALLOC_SCRATCH_FLOATS = (size_t)1 << 20;  // 4 MiB of (m, l, o) partials
constexpr int NOALLOC_MAX_DEVICES = 64;
}  // namespace
static __device__ __align__(256) float g_noalloc_scratch[NOALLOC_SCRATCH_FLOATS];
namespace {
// In host code `g_noalloc_scratch` is only a handle for the symbol, never a device address; the
// address a kernel may use is asked for once per device (with that device current) and kept here.
float* g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {nullptr};
std::mutex g_noalloc_mutex;

int noalloc_scratch(strictb200_ctx* ctx, float** out) {
  if (ctx->device < 0 || ctx->device >= NOALLOC_MAX_DEVICES) return sb_fail(STRICTB200_ERR_UNSUPPORTED, "device index beyond the static scratch table");
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[ctx->device]) {
    float* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void**)&p, g_noalloc_scratch);  // the caller made ctx->device current
    if (e != cudaSuccess || !p) return sb_fail(STRICTB200_ERR_CUDA, std::string("cudaGetSymbolAddress(static scratch): ") + cudaGetErrorString(e));
    g_noalloc_ptr[ctx->device] = p;
  }
  *out = g_noalloc_ptr[ctx->device];
  return STRICTB200_OK;
}
}  // namespace

extern "C" int strictb200_attn_decode_noalloc(strictb200_ctx* ctx, const uint16_t* q, const uint16_t* kc, const uint16_t* vc,
                                              const int32_t* lens, int B, int Hq, int Hkv, int Dh, int maxlen, float scale, uint16_t* out) {
  SB_ENTER(ctx);
  if (Dh != D) return sb_fail(STRICTB200_ERR_UNSUPPORTED, "head_dim must be 128");
  SB_REQUIRE(B >= 0 && Hq > 0 && Hkv > 0 && Hq % Hkv == 0 && Hq / Hkv <= 16 && maxlen > 0, "bad shape");
  if (!B) return STRICTB200_OK;
  SB_REQUIRE(q && kc && vc && lens && out, "null pointer");
  auto floats = [&](int chunk) { return sb_attn_decode_scratch(B, Hq, Dh, splits_of(maxlen, chunk)) / sizeof(float); };
  int chunk = decode_chunk(ctx, B, Hkv, maxlen);
  if (floats(chunk) > NOALLOC_SCRATCH_FLOATS) chunk = decode_chunk(ctx, B, Hkv, maxlen, 0, false, false);  // fewer partial results
  const int nsplit = splits_of(maxlen, chunk);
  const size_t need = floats(chunk);
  if (need > NOALLOC_SCRATCH_FLOATS)
    return sb_fail(STRICTB200_ERR_INVALID_ARG, "attn_decode_noalloc: batch " + std::to_string(B) + " x " + std::to_string(Hq) + " heads x " +
                                                   std::to_string(nsplit) + " key chunks needs " + std::to_string(need * sizeof(float)) +
                                                   " bytes of partial results; the built-in scratch holds " +
                                                   std::to_string(NOALLOC_SCRATCH_FLOATS * sizeof(float)) + " (use strictb200_attn_decode)");
  float* scratch;
  SB_TRY(noalloc_scratch(ctx, &scratch));
  // Nothing in the scratch has to start at zero: each key chunk a sequence owns is written in full
  // by its block before the combine kernel reads it, and chunks beyond a sequence's length are never read.
  return k_attn_decode(ctx, (const bf16*)q, (const bf16*)kc, (const bf16*)vc, lens, 0, B, Hq, Hkv, Dh, maxlen, scale, nsplit, scratch,
                       (bf16*)out, nullptr, nullptr, nullptr, chunk);
}
