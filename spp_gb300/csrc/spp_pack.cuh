/* spp_pack.cuh -- headings as the neighbours of a Vicsek particle read them
 * (kernels_cells.cu, kernels_step.cu, batch.cu). */
#ifndef SPP_PACK_CUH
#define SPP_PACK_CUH
#include "spp_internal.cuh"

namespace {

/* A particle as its neighbours read it: position, and the exact fixed-point
 * parts of cos and sin (spp_fx_add: |hi| <= 32, |lo| <= 2^21), each pair packed
 * as hi << 24 | lo + 2^22. */
constexpr int PACK_BIAS = 1 << 22;
__device__ __forceinline__ float pack_parts(spp_fx a) {
  return __int_as_float((int)((uint32_t)a.hi << 24 | (uint32_t)(a.lo + PACK_BIAS)));
}
__device__ __forceinline__ spp_fx fx_parts(float v) {
  spp_fx a = {0, 0};
  spp_fx_add(&a, v);
  return a;
}
/* Sums of packed parts: the words add up modulo 2^32 and the upper bytes by
 * themselves, which leaves the sum of the lower parts exact (two additions
 * per term). */
struct PackedSum { int32_t words, hi; };
__device__ __forceinline__ void packed_add(PackedSum* a, float w) {
  const int v = __float_as_int(w);
  a->words += v;
  a->hi += v >> 24;
}
__device__ __forceinline__ spp_fx packed_value(PackedSum a, int terms) {
  return {a.hi, (int32_t)((uint32_t)a.words - ((uint32_t)a.hi << 24) - (uint32_t)terms * (uint32_t)PACK_BIAS)};
}

}  // namespace
#endif
