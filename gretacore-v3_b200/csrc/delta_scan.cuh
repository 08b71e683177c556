// What the two forms of the delta rules' scan share: arguments, padding, asynchronous copies.
#pragma once
#include "greta_common.cuh"

namespace greta {

__host__ __device__ constexpr uint32_t dim32(uint32_t d) { return (d + 31u) & ~31u; }

__device__ __forceinline__ void cp16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// What the scan reads, for either form: rows of consecutive tokens.
struct ScanArgs {
  const float *w, *k, *a, *r, *v;  // decay, key, removal rate (general) or write strength per head (gated), receptance / query, value
  uint32_t ld_w, ld_k, ld_a, ld_r, ld_v;
  uint32_t heads, per, dim, vdim;  // per: value heads that share a query / key head
  uint32_t T, pos0, slot;
  float *state;
};
// Rows of 16 bytes throughout.
inline int scan_vec(const ScanArgs &a, bool gated) {
  return a.dim % 4 == 0 && a.vdim % 4 == 0 && a.ld_w % 4 == 0 && a.ld_k % 4 == 0 && a.ld_r % 4 == 0 && a.ld_v % 4 == 0 && aligned16(a.w) &&
         aligned16(a.k) && aligned16(a.r) && aligned16(a.v) && (gated || (a.ld_a % 4 == 0 && aligned16(a.a)));
}

// Chunked form (delta_chunks.cu): bytes of scratch it takes for T tokens, 0 where it does not apply; and the scan through it.
size_t chunk_scan_bytes(uint32_t heads, uint32_t dim, uint32_t vdim, bool gated, uint32_t T);
int chunk_scan(cudaStream_t s, const ScanArgs &a, bool gated, float *o_buf, float *scratch);

}  // namespace greta
