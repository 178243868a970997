// fp32 attention of the GPT-2 path: prompts in tiles, decode rows with the keys spread over half-warps, and a kernel for any head width.
// Inputs that another kernel of the chain writes are not declared const __restrict__ in these kernels: loads of invariant data may be
// moved in front of the dependency wait.
#include <type_traits>

#include "common.cuh"

namespace {
__global__ void kv_append_f32_kernel(const float* qkv, float* __restrict__ kc, float* __restrict__ vc,
                                     const int32_t* seq, const int32_t* pos, const int32_t* lens, int H,
                                     int Dh, int maxlen) {
  pdl_trigger();
  pdl_wait();
  int64_t t = blockIdx.x;
  int b = seq ? seq[t] : (int)t;
  int p = pos ? pos[t] : lens[b];
  if (p < 0 || p >= maxlen) return;
  int hd = H * Dh;
  for (int e = threadIdx.x; e < hd; e += blockDim.x) {
    int h = e / Dh, d = e - h * Dh;
    int64_t dst = (((int64_t)b * H + h) * maxlen + p) * Dh + d;
    kc[dst] = qkv[t * 3 * hd + hd + e];
    vc[dst] = qkv[t * 3 * hd + 2 * hd + e];
  }
}
// Head widths that are multiples of four, 16-byte aligned: four columns of a key and of its value per thread. 4800 tokens of 768 columns: 9.6 us,
// 19.5 with a thread per column.
__global__ void __launch_bounds__(256) kv_append_f32_vec_kernel(const float* qkv, float* __restrict__ kc, float* __restrict__ vc, const int32_t* seq, const int32_t* pos,
                                                                const int32_t* lens, uint32_t n, uint32_t hd, uint32_t Dh, int H, int maxlen) {
  // The attention behind this may start only when the product in front has left: its blocks, which all wait for the keys anyway, were dealt out over the
  // SMs that product had left free, the longest rows on top of each other. GPT-2 prompts of width 128, 3 x 500: 869 -> 790 us, 1 x 900: 1026 -> 892.
  pdl_wait();
  pdl_trigger();
  const uint32_t i = blockIdx.x * 256 + threadIdx.x, per = hd / 4;
  if (i >= n) return;
  const uint32_t t = i / per, e = (i - t * per) * 4, h = e / Dh;
  const float* row = qkv + (int64_t)t * 3 * hd + hd + e;
  const float4 k = *(const float4*)row, v = *(const float4*)(row + hd);
  const int b = seq ? seq[t] : (int)t, p = pos ? pos[t] : lens[b];
  if (p < 0 || p >= maxlen) return;
  const int64_t dst = (((int64_t)b * H + h) * maxlen + p) * Dh + (e - h * Dh);
  *(float4*)(kc + dst) = k;
  *(float4*)(vc + dst) = v;
}
// Any head width. grid (H, T), 256 threads; scores of one (token, head) live in shared memory.
__global__ void __launch_bounds__(256) attn_f32_kernel(const float* qkv, const float* kc, const float* vc,
                                                       const int32_t* seq, const int32_t* pos,
                                                       const int32_t* lens, int H, int Dh, int maxlen, float scale,
                                                       float* __restrict__ out, float* kc_new, float* vc_new) {
  // kc_new/vc_new (decode: every row is its own sequence) make this block also append its head's
  // new key and value; it then takes position p from the projection output, not from the cache.
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) float sc[];  // [maxlen rounded up to 4] scores, [Dh] query, [blockDim.x] float4 partial rows
  __shared__ float red[32];
  int h = blockIdx.x;
  int64_t t = blockIdx.y;
  int b = seq ? seq[t] : (int)t;
  int p = pos ? pos[t] : lens[b];
  if (p < 0 || p >= maxlen) return;
  int n = p + 1;
  float* qs = sc + ((maxlen + 3) & ~3);
  int hd = H * Dh;
  for (int d = threadIdx.x; d < Dh; d += blockDim.x) qs[d] = qkv[t * 3 * hd + h * Dh + d];
  __syncthreads();
  const float* kb = kc + ((int64_t)b * H + h) * maxlen * Dh;
  const float* vb = vc + ((int64_t)b * H + h) * maxlen * Dh;
  const float* k_own = qkv + t * 3 * hd + hd + h * Dh;
  const float* v_own = k_own + hd;
  const int own = kc_new ? p : -1;
  if (kc_new)
    for (int d = threadIdx.x; d < Dh; d += blockDim.x) {
      const int64_t dst = (((int64_t)b * H + h) * maxlen + p) * Dh + d;
      kc_new[dst] = k_own[d];
      vc_new[dst] = v_own[d];
    }
  float mx = -INFINITY;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    const float4* kr = (const float4*)(j == own ? k_own : kb + (int64_t)j * Dh);
    float acc = 0.f;
    for (int d4 = 0; d4 < Dh / 4; d4++) {
      float4 kv = kr[d4];
      acc += kv.x * qs[4 * d4] + kv.y * qs[4 * d4 + 1] + kv.z * qs[4 * d4 + 2] + kv.w * qs[4 * d4 + 3];
    }
    acc *= scale;
    sc[j] = acc;
    mx = fmaxf(mx, acc);
  }
  mx = block_max(mx, red);
  float l = 0.f;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    float e = expf(sc[j] - mx);
    sc[j] = e;
    l += e;
  }
  l = block_sum(l, red);
  __syncthreads();
  float inv = 1.0f / l;
  // P.V: the block's threads form groups of Dh/4 lanes; group g adds the keys g, g+G, ... with one
  // float4 of the value row per lane (a single query row would otherwise walk all keys on Dh
  // threads, one dependent step per key), then the groups' partial rows are added in group order.
  const int dl = Dh / 4, G = (int)blockDim.x / dl;
  float* part = qs + Dh;  // [blockDim.x] float4
  if (G >= 1) {
    const int g = (int)threadIdx.x / dl, c = (int)threadIdx.x % dl;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (g < G) {
#pragma unroll 8
      for (int j = g; j < n; j += G) {
        const float4 v = *(const float4*)((j == own ? v_own : vb + (int64_t)j * Dh) + 4 * c);
        const float pj = sc[j];
        acc.x += pj * v.x; acc.y += pj * v.y; acc.z += pj * v.z; acc.w += pj * v.w;
      }
    }
    *(float4*)(part + 4 * threadIdx.x) = acc;
    __syncthreads();
    for (int d = threadIdx.x; d < Dh; d += blockDim.x) {
      float o = 0.f;
      for (int gg = 0; gg < G; gg++) o += part[(gg * dl + d / 4) * 4 + (d & 3)];
      out[t * hd + h * Dh + d] = o * inv;
    }
  } else {  // head wider than four times the block: one thread per output column
    for (int d = threadIdx.x; d < Dh; d += blockDim.x) {
      float acc = 0.f;
      for (int j = 0; j < n; j++) acc += sc[j] * (j == own ? v_own[d] : vb[(int64_t)j * Dh + d]);
      out[t * hd + h * Dh + d] = acc * inv;
    }
  }
}


// ------------------------------------------------------------------ prompts, 64-dim heads
// One block: N / 4 queries of a sequence and one head, over 64 keys at a time with a running maximum; 4 x 4 results per thread and eight 128-bit
// shared-memory reads per 64 FMAs. The next keys are copied while the values are summed, the next values while the keys are. A tile's sums
// start from zero and are added to the running ones once, so that a long row is not one long chain of additions. Keys behind a row
// are left out, not weighted with zero: an infinity or NaN at a later token does not reach the rows before it. A row whose scores so far are all
// -inf has sums of zero. Bound by the issue of instructions (FMAs are 72% of them, 61% of the slots are used) and the waits for shared memory.
// Prompts of 300 to 901 tokens, batch 8: 1405 us per layer with one block per row and head, 195 us with blocks of 64 queries in the order of
// the sequences. 8 x 600: 211 us so, the busiest SM with 1.35 times the average work; 185 us with the blocks of the longest rows of all sequences
// in front, 175 us with 32 queries per block. 8 x 8 results per thread (half the shared-memory reads): 262 us, too few warps; packed FMAs: no gain.
constexpr int PT = 64, PD = 64, PS = PD + 4;  // keys per tile, head dims, row stride in shared memory
constexpr int R = 4, TX = PT / R, TY = 32 / TX, WROWS = R * TY;  // results per thread each way, a warp's threads each way, queries of a warp
constexpr int WS = PT + 16;                   // row stride of the weights: the two rows of a warp's threads in banks of their own
template <int N>
__global__ void __launch_bounds__(N, 512 / N) attn_f32_prompt_kernel(const float* qkv, const float* kc, const float* vc,
                                                                     const int32_t* qstart, const int32_t* past,
                                                                     const int32_t* after, int b0, int H, int maxlen, float scale,
                                                                     float* out) {
  constexpr int QT = N / 32 * WROWS;  // queries of the block
  extern __shared__ __align__(16) float ps[];
  float *qs = ps, *ks = qs + QT * PS, *vs = ks + PT * PS, *pr = vs + PT * PS;
  pdl_trigger();
  pdl_wait();
  const int j = blockIdx.y, h = blockIdx.x, q0 = ((int)gridDim.z - 1 - (int)blockIdx.z) * QT;  // the longest rows first
  const int p0 = past[j], n_new = after[j] - p0;
  if (q0 >= n_new) return;
  const int lane = threadIdx.x & 31, tx = lane % TX, hd = H * PD;
  const int wr = threadIdx.x / 32 * WROWS, ty = wr + lane / TX;  // the warp's first row; the thread's rows are ty + TY i
  const int64_t row0 = qstart[j] + q0;
  const float* kb = kc + ((int64_t)(b0 + j) * H + h) * maxlen * PD;
  const float* vb = vc + ((int64_t)(b0 + j) * H + h) * maxlen * PD;
  const int n_keys = p0 + min(q0 + QT, n_new);
  // rows [0, n) of a matrix of 64 columns, zeros behind `valid` rows
  auto copy = [&](float* to, const float* from, int64_t ld, int n, int valid) {
    for (int e = threadIdx.x; e < n * (PD / 4); e += N) {
      const int r = e / (PD / 4), c = e % (PD / 4) * 4;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to + r * PS + c)), "l"(from + (r < valid ? r : 0) * ld + c),
                   "r"(r < valid ? 16 : 0)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  copy(qs, qkv + row0 * 3 * hd + h * PD, 3 * hd, QT, n_new - q0);
  copy(ks, kb, PD, PT, n_keys);
  copy(vs, vb, PD, PT, n_keys);
  float o[R][R], m[R], l[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < R; c++) o[i][c] = 0.f;
  }
  for (int k0 = 0; k0 < n_keys; k0 += PT) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // the keys are there
    const bool seen = q0 + wr < n_new && k0 <= p0 + q0 + wr + WROWS - 1;  // by a row of the warp
    float s[R][R];
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
      for (int c = 0; c < R; c++) s[i][c] = 0.f;
    if (seen) {
      // scores of the keys k0 + tx + TX c
#pragma unroll 2
      for (int d = 0; d < PD; d += 4) {
        float4 a[R], b[R];
#pragma unroll
        for (int i = 0; i < R; i++) a[i] = *(const float4*)(qs + (ty + TY * i) * PS + d);
#pragma unroll
        for (int c = 0; c < R; c++) b[c] = *(const float4*)(ks + (tx + TX * c) * PS + d);
#pragma unroll
        for (int i = 0; i < R; i++)
#pragma unroll
          for (int c = 0; c < R; c++) s[i][c] = fmaf(a[i].w, b[c].w, fmaf(a[i].z, b[c].z, fmaf(a[i].y, b[c].y, fmaf(a[i].x, b[c].x, s[i][c]))));
      }
      __syncwarp();  // the warp's own rows of the weights have been read
#pragma unroll
      for (int i = 0; i < R; i++) {
        const int last = p0 + q0 + ty + TY * i - k0;  // keys up to here are visible
        float mx = m[i];
#pragma unroll
        for (int c = 0; c < R; c++) {
          s[i][c] *= scale;
          if (tx + TX * c <= last) mx = fmaxf(mx, s[i][c]);
        }
#pragma unroll
        for (int w = TX / 2; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
        const float ref = mx == -INFINITY ? 0.f : mx;
        const float alpha = expf(m[i] - ref);
        float sum = 0.f;
#pragma unroll
        for (int c = 0; c < R; c++) {
          const float e = tx + TX * c <= last ? expf(s[i][c] - ref) : 0.f;
          pr[(ty + TY * i) * WS + tx + TX * c] = e;
          sum += e;
        }
        l[i] = fmaf(l[i], alpha, sum);
        m[i] = mx;
#pragma unroll
        for (int c = 0; c < R; c++) { o[i][c] *= alpha; s[i][c] = 0.f; }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the values are there, the keys have been read
    const bool more = k0 + PT < n_keys;
    if (more) copy(ks, kb + (int64_t)(k0 + PT) * PD, PD, PT, n_keys - k0 - PT);
    if (seen) {
      // columns 4 tx + c
      auto add_values = [&](auto masked) {
#pragma unroll 2
        for (int k = 0; k < PT; k += 4) {
          float4 a[R], b[R];
#pragma unroll
          for (int i = 0; i < R; i++) a[i] = *(const float4*)(pr + (ty + TY * i) * WS + k);
#pragma unroll
          for (int c = 0; c < R; c++) b[c] = *(const float4*)(vs + (k + c) * PS + 4 * tx);
#pragma unroll
          for (int i = 0; i < R; i++) {
            const int last = decltype(masked)::value ? p0 + q0 + ty + TY * i - k0 - k : 3;
            if (last >= 0) { s[i][0] = fmaf(a[i].x, b[0].x, s[i][0]); s[i][1] = fmaf(a[i].x, b[0].y, s[i][1]); s[i][2] = fmaf(a[i].x, b[0].z, s[i][2]); s[i][3] = fmaf(a[i].x, b[0].w, s[i][3]); }
            if (last >= 1) { s[i][0] = fmaf(a[i].y, b[1].x, s[i][0]); s[i][1] = fmaf(a[i].y, b[1].y, s[i][1]); s[i][2] = fmaf(a[i].y, b[1].z, s[i][2]); s[i][3] = fmaf(a[i].y, b[1].w, s[i][3]); }
            if (last >= 2) { s[i][0] = fmaf(a[i].z, b[2].x, s[i][0]); s[i][1] = fmaf(a[i].z, b[2].y, s[i][1]); s[i][2] = fmaf(a[i].z, b[2].z, s[i][2]); s[i][3] = fmaf(a[i].z, b[2].w, s[i][3]); }
            if (last >= 3) { s[i][0] = fmaf(a[i].w, b[3].x, s[i][0]); s[i][1] = fmaf(a[i].w, b[3].y, s[i][1]); s[i][2] = fmaf(a[i].w, b[3].z, s[i][2]); s[i][3] = fmaf(a[i].w, b[3].w, s[i][3]); }
          }
        }
      };
      if (k0 + PT > p0 + q0 + wr + 1) add_values(std::true_type{});  // a key of the tile lies behind the warp's first row
      else add_values(std::false_type{});
#pragma unroll
      for (int i = 0; i < R; i++)
#pragma unroll
        for (int c = 0; c < R; c++) o[i][c] += s[i][c];
    }
    if (!more) break;
    __syncthreads();  // the values have been read
    copy(vs, vb + (int64_t)(k0 + PT) * PD, PD, PT, n_keys - k0 - PT);
  }
#pragma unroll
  for (int i = 0; i < R; i++) {
#pragma unroll
    for (int w = TX / 2; w > 0; w >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], w);
    const int r = ty + TY * i;
    if (q0 + r < n_new) {
      const float inv = 1.0f / l[i];
      *(float4*)(out + (row0 + r) * hd + h * PD + 4 * tx) = make_float4(o[i][0] * inv, o[i][1] * inv, o[i][2] * inv, o[i][3] * inv);
    }
  }
}
template <int N>
int launch_prompt(strictb200_ctx* ctx, const F32Prompts* prompts, const float* qkv, const float* kc, const float* vc, int H, int maxlen, float scale, float* out) {
  constexpr int QT = N / 32 * WROWS, smem = (QT * PS + 2 * PT * PS + QT * WS) * 4;
  static SbDeviceOnce once;
  SB_CUDA(once.run(ctx->device, [&] { return cudaFuncSetAttribute(attn_f32_prompt_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); }));
  SB_CUDA(sb_launch(ctx, attn_f32_prompt_kernel<N>, dim3((unsigned)H, (unsigned)prompts->nb, (unsigned)((prompts->max_new + QT - 1) / QT)), dim3(N),
                    (size_t)smem, qkv, kc, vc, prompts->qstart, prompts->past, prompts->after, prompts->b0, H, maxlen, scale, out));
  ctx->launches++;
  return STRICTB200_OK;
}

// ------------------------------------------------------------------ decode rows, heads of 4 LANES dims
// One block per row and head, and it appends the row's key and value to the cache. LANES lanes share a key (one 128-bit load of the
// key and one of the value per lane), each such group walks every GROUPS-th key with a running maximum and its own sum, eight keys'
// loads in flight; the groups meet in shared memory. Bound by the latency of those loads: 144 keys on average took 13.6 us of a GPT-2 step
// with a key per thread and a second pass for the values, 3.7 us with batches behind the dependency wait. The first batch (rows of earlier steps) is
// requested in front of it; the length it is derived from is read again after the wait, and the batch with it if it changed.
template <int LANES>
__global__ void __launch_bounds__(512) attn_f32_decode_kernel(const float* qkv, float* kc, float* vc, const int32_t* lens, int H,
                                                              int maxlen, float scale, float* out, int prefetch) {
  constexpr int D = 4 * LANES, GROUPS = 512 / LANES, BATCH = 8;
  __shared__ float red_m[GROUPS], red_l[GROUPS];
  __shared__ __align__(16) float red_o[GROUPS][D];
  pdl_trigger();
  const int h = blockIdx.x, b = blockIdx.y, c = threadIdx.x % LANES, grp = threadIdx.x / LANES, hd = H * D;
  float* kb = kc + ((int64_t)b * H + h) * maxlen * D + 4 * c;
  float* vb = vc + ((int64_t)b * H + h) * maxlen * D + 4 * c;
  float4 k[BATCH], v[BATCH];
  auto load = [&](int base, int len) {
#pragma unroll
    for (int i = 0; i < BATCH; i++) {
      const int j = base + grp + i * GROUPS;
      if (j < len) {
        k[i] = *(const float4*)(kb + (int64_t)j * D);
        v[i] = *(const float4*)(vb + (int64_t)j * D);
      }
    }
  };
  auto ld_len = [&] {
    int n;
    asm volatile("ld.volatile.global.s32 %0, [%1];" : "=r"(n) : "l"(lens + b) : "memory");
    return n;
  };
  const int early = prefetch ? min(ld_len(), maxlen) : -1;
  load(0, early);
  pdl_wait();
  const float* row = qkv + (int64_t)b * 3 * hd + h * D + 4 * c;
  const float4 q = *(const float4*)row, k_own = *(const float4*)(row + hd), v_own = *(const float4*)(row + 2 * hd);
  const int p = ld_len();
  if (p < 0 || p >= maxlen) return;
  if (p != early) load(0, p);
  if (grp == 0) {
    *(float4*)(kb + (int64_t)p * D) = k_own;
    *(float4*)(vb + (int64_t)p * D) = v_own;
  }
  float m = -INFINITY, l = 0.f;
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int base = 0; base <= p; base += BATCH * GROUPS) {  // the same number of rounds for every group: their lanes share warps, and shuffles
    const int j0 = base + grp;
    if (base) load(base, p);
#pragma unroll
    for (int i = 0; i < BATCH; i++)
      if (j0 + i * GROUPS >= p) { k[i] = k_own; v[i] = v_own; }
    float s[BATCH], mx = m;
#pragma unroll
    for (int i = 0; i < BATCH; i++) {
      s[i] = fmaf(k[i].w, q.w, fmaf(k[i].z, q.z, fmaf(k[i].y, q.y, k[i].x * q.x)));
#pragma unroll
      for (int w = LANES / 2; w > 0; w >>= 1) s[i] += __shfl_xor_sync(0xffffffffu, s[i], w, LANES);
      s[i] *= scale;
      if (j0 + i * GROUPS <= p) mx = fmaxf(mx, s[i]);
    }
    const float ref = mx == -INFINITY ? 0.f : mx;  // all scores of the group -inf so far: sums of zero
    const float alpha = expf(m - ref);
    m = mx;
    l *= alpha;
    o.x *= alpha; o.y *= alpha; o.z *= alpha; o.w *= alpha;
#pragma unroll
    for (int i = 0; i < BATCH; i++) {
      if (j0 + i * GROUPS <= p) {
        const float e = expf(s[i] - ref);
        l += e;
        o.x = fmaf(e, v[i].x, o.x); o.y = fmaf(e, v[i].y, o.y); o.z = fmaf(e, v[i].z, o.z); o.w = fmaf(e, v[i].w, o.w);
      }
    }
  }
  if (c == 0) { red_m[grp] = m; red_l[grp] = l; }
  *(float4*)&red_o[grp][4 * c] = o;
  __syncthreads();
  if (threadIdx.x < D) {
    const int n = min(GROUPS, p + 1);  // groups that have seen a key
    float mx = red_m[0];
    for (int g = 1; g < n; g++) mx = fmaxf(mx, red_m[g]);
    float sum = 0.f, acc = 0.f;
    for (int g = 0; g < n; g++) {
      const float e = expf(red_m[g] - mx);
      sum = fmaf(e, red_l[g], sum);
      acc = fmaf(e, red_o[g][threadIdx.x], acc);
    }
    out[(int64_t)b * hd + h * D + threadIdx.x] = acc * (1.0f / sum);
  }
}
}  // namespace

int k_attn_f32(strictb200_ctx* ctx, const float* qkv, float* kc, float* vc, const int32_t* seq, const int32_t* pos, const int32_t* lens,
               int64_t T, int H, int Dh, int maxlen, float scale, float* out, const F32Prompts* prompts) {
  if (Dh % 4) return sb_fail(STRICTB200_ERR_INVALID_ARG, "attention: head_dim must be a multiple of 4");
  const bool rows16 = (((uintptr_t)qkv | (uintptr_t)kc | (uintptr_t)vc | (uintptr_t)out) & 15) == 0;
  if (!seq && rows16 && (Dh == 32 || Dh == 64 || Dh == 128) && T <= 65535) {  // rows that are sequences of their own
    auto kernel = Dh == 32 ? attn_f32_decode_kernel<8> : Dh == 64 ? attn_f32_decode_kernel<16> : attn_f32_decode_kernel<32>;
    SB_CUDA(sb_launch(ctx, kernel, dim3((unsigned)H, (unsigned)T), dim3(512), 0, qkv, kc, vc, lens, H, maxlen, scale, out, ctx->opt.attn_prefetch));
    ctx->launches++;
    return STRICTB200_OK;
  }
  if (seq && prompts && rows16 && Dh == PD && T <= 65535 && prompts->nb <= 65535 && H <= 65535) {
    const int hd = H * Dh;
    const uint32_t n = (uint32_t)(T * (hd / 4));  // fits: qkv alone has 48 bytes per item
    SB_CUDA(sb_launch(ctx, kv_append_f32_vec_kernel, dim3((n + 255) / 256), dim3(256), 0, qkv, kc, vc, seq, pos, lens, n, (uint32_t)hd, (uint32_t)Dh, H, maxlen));
    ctx->launches++;
    // Blocks of 16 queries while those of 32 would all be resident (four per SM): 1 x 901 tokens 3.80 -> 3.60 ms for a GPT-2 prompt, 4 x 300 the same; with
    // more blocks those of 32 read the keys half as often (8 x 600: 9.05 ms against 9.41, and 9.17 with 64).
    if ((int64_t)((prompts->max_new + 31) / 32) * H * prompts->nb <= 4 * (int64_t)ctx->sm_count) return launch_prompt<64>(ctx, prompts, qkv, kc, vc, H, maxlen, scale, out);
    return launch_prompt<128>(ctx, prompts, qkv, kc, vc, H, maxlen, scale, out);
  }
  const int threads = 256;
  size_t smem = ((size_t)((maxlen + 3) & ~3) + Dh + 4 * threads) * sizeof(float);
  if (smem > 200 * 1024) return sb_fail(STRICTB200_ERR_UNSUPPORTED, "attention: fp32 path supports at most ~50k positions");
  {
    static std::mutex mu;
    static size_t attr_smem[64] = {};  // largest size this device's kernel has been opened for
    std::lock_guard<std::mutex> lock(mu);
    size_t& have = attr_smem[ctx->device & 63];
    if (have < 48 * 1024) have = 48 * 1024;
    if (smem > have) {
      SB_CUDA(cudaFuncSetAttribute(attn_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      have = smem;
    }
  }
  if (T > 65535) return sb_fail(STRICTB200_ERR_INVALID_ARG, "attention: too many rows for the fp32 path");
  // rows that are sequences of their own (decode) append inside the attention kernel; prompt rows
  // need the keys of other rows of their sequence, so those are appended by a kernel of its own first
  const bool fused_append = seq == nullptr;
  if (!fused_append) {
    SB_CUDA(sb_launch(ctx, kv_append_f32_kernel, dim3((unsigned)T), dim3(256), 0, qkv, kc, vc, seq, pos, lens, H, Dh, maxlen));
    ctx->launches++;
  }
  dim3 grid(H, (unsigned)T);
  SB_CUDA(sb_launch(ctx, attn_f32_kernel, grid, dim3(threads), smem, (const float*)qkv, (const float*)kc, (const float*)vc, seq, pos, lens, H, Dh, maxlen,
                    scale, out, fused_append ? kc : (float*)nullptr, fused_append ? vc : (float*)nullptr));
  ctx->launches++;
  return STRICTB200_OK;
}
