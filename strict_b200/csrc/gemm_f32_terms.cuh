// What the fp32 products on the tensor cores share: the three bf16 terms of a value, and how a finished sum leaves.
#pragma once
#include "tcgen05.cuh"

#ifdef __CUDACC__
namespace tc {
// Two values -> their bf16 terms, packed (the first value in the low half); u and v become 2^8 times the remainders.
__device__ __forceinline__ uint32_t take_term(float& u, float& v) {
  uint32_t t;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(t) : "f"(v), "f"(u));
  u = __fmul_rn(256.f, __fsub_rn(u, __uint_as_float(t << 16)));
  v = __fmul_rn(256.f, __fsub_rn(v, __uint_as_float(t & 0xFFFF0000u)));
  return t;
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// A sum that is not finite is computed again (an infinity has no bf16 remainder).
__device__ __forceinline__ bool not_finite(float v) { return !(fabsf(v) <= 3.402823466e38f); }
static __device__ __noinline__ float plain_dot(const float* x, const float* w, int K) {
  float s = 0.f;
  for (int k = 0; k < K; k++) s = fmaf(x[k], w[k], s);
  return s;
}
// A value of a channel (its bias added) -> what is stored; old: what is there now (modes 1 and 4), scale: the channel's (mode 4).
template <int MODE>
__device__ __forceinline__ float finished(const GemmF32Args& g, float scale, float v, float old) {
  return MODE == 4 ? old + scale * v : MODE == 1 ? old + v : MODE == 2 ? sb_gelu_tanh(v) : MODE == 3 ? sb_xielu(v, g.act_pos, g.act_neg) : v;
}
}  // namespace tc
#endif
