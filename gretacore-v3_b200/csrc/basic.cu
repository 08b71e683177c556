// Format conversion and the small element-wise / reduction operators of the
// decode path (norm, residual add, SwiGLU, embedding gather, greedy arg-max).
#include <cooperative_groups.h>

#include <algorithm>

#include "greta_common.cuh"

namespace greta {
int gemm_ts_error_word(int **word);  // gemm_ts.cu
}  // namespace greta

using namespace greta;
namespace cg = cooperative_groups;
static inline cudaStream_t S(greta_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

namespace {

// One thread per GGUF block: splits {fp16 d; payload} into the two planes.
template <int FMT>
__global__ void repack_kernel(const uint8_t *__restrict__ blocks, uint8_t *__restrict__ qs,
                              uint16_t *__restrict__ d, size_t n_blocks, uint32_t nb_row) {
  constexpr int PB = payload_bytes(FMT), BB = PB + 2;
  size_t b = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n_blocks) return;
  const uint8_t *src = blocks + b * BB;   // 2-byte aligned only (18 / 34 byte stride)
  const uint16_t *s16 = reinterpret_cast<const uint16_t *>(src);
  d[(b / nb_row) * d_row_stride(nb_row) + b % nb_row] = s16[0];
  uint16_t *dst = reinterpret_cast<uint16_t *>(qs + b * PB);
#pragma unroll
  for (int i = 0; i < PB / 2; ++i) dst[i] = s16[1 + i];
}

// One thread per block of 32 weights; bit-exact (float)q * fp32(d).
template <int FMT>
__global__ void dequant_kernel(const uint8_t *__restrict__ qs, const void *__restrict__ d,
                               float *__restrict__ out, size_t n_blocks, uint32_t nb_row) {
  size_t b = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n_blocks) return;
  const size_t sb = (b / nb_row) * d_row_stride(nb_row) + b % nb_row;  // index in the padded fp16 d plane
  float *o = out + b * 32;
  if (FMT == GRETA_FMT_Q4_0) {
    float s = __half2float(reinterpret_cast<const __half *>(d)[sb]);
    const uint8_t *p = qs + b * 16;
    for (int j = 0; j < 16; ++j) {
      o[j] = __fmul_rn((float)((int)(p[j] & 0xF) - 8), s);
      o[j + 16] = __fmul_rn((float)((int)(p[j] >> 4) - 8), s);
    }
  } else if (FMT == GRETA_FMT_Q8_0) {
    float s = __half2float(reinterpret_cast<const __half *>(d)[sb]);
    const int8_t *p = reinterpret_cast<const int8_t *>(qs) + b * 32;
    for (int j = 0; j < 32; ++j) o[j] = __fmul_rn((float)p[j], s);
  } else if (FMT == GRETA_FMT_REF_INT4) {
    float s = reinterpret_cast<const float *>(d)[b];
    const uint8_t *p = qs + b * 16;
    for (int j = 0; j < 16; ++j) {
      int lo = p[j] & 0xF, hi = p[j] >> 4;
      o[2 * j] = __fmul_rn((float)(lo >= 8 ? lo - 16 : lo), s);
      o[2 * j + 1] = __fmul_rn((float)(hi >= 8 ? hi - 16 : hi), s);
    }
  } else {  // REF_INT8
    float s = reinterpret_cast<const float *>(d)[b];
    const int8_t *p = reinterpret_cast<const int8_t *>(qs) + b * 32;
    for (int j = 0; j < 32; ++j) o[j] = __fmul_rn((float)p[j], s);
  }
}

__global__ void f32_to_f16_kernel(const float *__restrict__ in, __half *__restrict__ out, size_t n) {
  size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i + 3 < n) {
    float4 v = *reinterpret_cast<const float4 *>(in + i);
    __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
    uint2 o;
    o.x = *reinterpret_cast<uint32_t *>(&a);
    o.y = *reinterpret_cast<uint32_t *>(&b);
    *reinterpret_cast<uint2 *>(out + i) = o;
  } else {
    for (; i < n; ++i) out[i] = __float2half_rn(in[i]);
  }
}
__global__ void f16_to_f32_kernel(const __half *__restrict__ in, float *__restrict__ out, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __half2float(in[i]);
}

__device__ __forceinline__ float block_sum(float v, float *sm) {
  v = warp_sum(v);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (l == 0) sm[w] = v;
  __syncthreads();
  float t = (threadIdx.x < nw) ? sm[threadIdx.x] : 0.f;
  if (w == 0) {
    t = warp_sum(t);
    if (l == 0) sm[0] = t;
  }
  __syncthreads();
  t = sm[0];
  __syncthreads();
  return t;
}

// One CTA per row: y = (x * rsqrt(mean(x^2) + eps)) * gamma.
__global__ void __launch_bounds__(256) rmsnorm_kernel(const float *__restrict__ x, const float *__restrict__ gamma,
                                                      float *__restrict__ y, uint32_t cols, float eps) {
  __shared__ float sm[32];
  const float *xr = x + (size_t)blockIdx.x * cols;
  float *yr = y + (size_t)blockIdx.x * cols;
  float ss = 0.f;
  for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) ss = fmaf(xr[c], xr[c], ss);
  ss = block_sum(ss, sm);
  float inv = rsqrtf(ss / (float)cols + eps);
  for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) yr[c] = (xr[c] * inv) * gamma[c];
}

// The same values as fp16, for the tensor-core products.  A row stays in registers (PER values per thread, all loads under way together;
// the 256-thread order of the sum is rmsnorm_kernel's, so the results are its bits): 3.8 us for 512 x 4096 in the layer against 10.8 and a
// conversion pass of 2.9 per product.  BOTH: y32 takes the fp32 values as well.
template <int PER, bool BOTH>
__global__ void __launch_bounds__(256) rmsnorm_f16_kernel(const float *x, const float *__restrict__ gamma, __half *y, float *y32, uint32_t cols, float eps) {
  __shared__ float sm[32];
  pdl_launch_dependents();
  pdl_wait();
  const float *xr = x + (size_t)blockIdx.x * cols;
  __half *yr = y + (size_t)blockIdx.x * cols;
  auto put = [&](uint32_t c, float n) {
    yr[c] = __float2half_rn(n);
    if (BOTH) y32[(size_t)blockIdx.x * cols + c] = n;
  };
  float v[PER], ss = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const uint32_t c = threadIdx.x + i * 256;
    v[i] = c < cols ? xr[c] : 0.f;
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) ss = fmaf(v[i], v[i], ss);
  for (uint32_t c = threadIdx.x + PER * 256; c < cols; c += 256) ss = fmaf(xr[c], xr[c], ss);
  ss = block_sum(ss, sm);
  const float inv = rsqrtf(ss / (float)cols + eps);
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const uint32_t c = threadIdx.x + i * 256;
    if (c < cols) put(c, (v[i] * inv) * gamma[c]);
  }
  for (uint32_t c = threadIdx.x + PER * 256; c < cols; c += 256) put(c, (xr[c] * inv) * gamma[c]);
}

__global__ void add_kernel(const float *a, const float *b, float *c, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) c[i] = a[i] + b[i];
}
__global__ void silu_kernel(const float *x, float *y, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    float v = x[i];
    y[i] = v / (1.0f + expf(-v));
  }
}
__global__ void mul_kernel(const float *a, const float *b, float *c, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) c[i] = a[i] * b[i];
}
__global__ void silu_mul_kernel(const float *g, const float *u, float *y, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    float v = g[i];
    y[i] = (v / (1.0f + expf(-v))) * u[i];
  }
}

// grid (rows, column groups of 256 * V, 65535 at most); V = 4 where the row length and the pointers allow it.  One value per thread behind two 64-bit divisions
// took 10.5 us for 512 x 4096 and 28 for 1531.
template <bool F16, int V>
__global__ void embedding_kernel(const int32_t *tokens, const void *__restrict__ table, float *out, uint32_t dim, uint32_t vocab) {
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t s = blockIdx.x;
  const int32_t t = tokens[s];
  const bool known = t >= 0 && t < (int32_t)vocab;
  for (uint32_t c = first_column<V>(); c < dim; c = next_column<V>(c, dim)) {
    const size_t src = (size_t)(known ? t : 0) * dim + c;
    float *o = out + (size_t)s * dim + c;
    if (V == 4) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (known) {
        if (F16) {
          const uint2 u = *reinterpret_cast<const uint2 *>(reinterpret_cast<const __half *>(table) + src);
          const float2 a = h2_to_f2(u.x), b = h2_to_f2(u.y);
          v = make_float4(a.x, a.y, b.x, b.y);
        } else {
          v = *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(table) + src);
        }
      }
      *reinterpret_cast<float4 *>(o) = v;
    } else {
      *o = !known ? 0.f : F16 ? __half2float(reinterpret_cast<const __half *>(table)[src]) : reinterpret_cast<const float *>(table)[src];
    }
  }
}

// First maximum (lowest index among equal values; NaN counts only in the first place, where it wins) of each row of logits: a cluster of gridDim.x CTAs of 1024 threads per row
// (per sequence of a batch).  One CTA per row is bound by the latency of its 32 dependent loads per thread, not by bandwidth: 15 us
// of a 258 us step at 32000 logits; eight CTAs take 4 loads per thread, issued together, and meet through distributed shared memory.
__global__ void __launch_bounds__(1024) argmax_kernel(const float *logits, uint32_t n,
                                                      int32_t *out, uint32_t *d_pos, int32_t *out_tokens,
                                                      uint32_t *d_count, uint32_t out_capacity, const int *code) {
  __shared__ float sv[32];
  __shared__ uint32_t si[32];
  cg::cluster_group cluster = cg::this_cluster();
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t b = blockIdx.y, rank = blockIdx.x, ctas = gridDim.x;  // sequence: its own logits row, result, position, counter and output list
  logits += (size_t)b * n;
  const bool tells = code && b == 0 && rank == 0 && threadIdx.x == 0;
  int told = 0;
  if (tells) told = __ldcg(code);  // stored at the end: nothing waits for it
  out += b;
  if (d_pos) d_pos += b;
  if (d_count) d_count += b;
  if (out_tokens) out_tokens += (size_t)b * out_capacity;
  float best = -INFINITY;
  uint32_t bi = 0xffffffffu;
  const uint32_t stride = ctas * blockDim.x;
#pragma unroll 4
  for (uint32_t i = rank * blockDim.x + threadIdx.x; i < n; i += stride) {
    float v = logits[i];
    if (v != v) v = i ? -INFINITY : INFINITY;  // as a scan from the first value on: a NaN is never greater, and nothing is greater than a NaN there
    if (v > best || bi == 0xffffffffu) {   // strided scan keeps the lowest index of this thread's maximum
      best = v;
      bi = i;
    }
  }
  auto better = [](float v, uint32_t i, float bv, uint32_t bidx) { return v > bv || (v == bv && i < bidx); };
  auto warp_best = [&] {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float ov = __shfl_xor_sync(0xffffffffu, best, o);
      uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (better(ov, oi, best, bi)) {
        best = ov;
        bi = oi;
      }
    }
  };
  warp_best();
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sv[w] = best;
    si[w] = bi;
  }
  __syncthreads();
  if (w == 0) {
    best = sv[l];
    bi = si[l];
    warp_best();
    __syncwarp();
    if (l == 0) {
      sv[0] = best;
      si[0] = bi;
    }
  }
  if (ctas > 1) cluster.sync();
  if (w == 0 && rank == 0) {
    if (ctas > 1) {
      best = -INFINITY;
      bi = 0xffffffffu;
      if ((uint32_t)l < ctas) {
        best = *cluster.map_shared_rank(&sv[0], l);
        bi = *cluster.map_shared_rank(&si[0], l);
      }
      warp_best();
    }
    if (l == 0) {
      *out = (int32_t)bi;
      if (tells) out[gridDim.y] = told;
      if (d_count) {
        uint32_t c = *d_count;
        if (out_tokens && c < out_capacity) out_tokens[c] = (int32_t)bi;
        *d_count = c + 1;
      }
      if (d_pos) *d_pos = *d_pos + 1;
    }
  }
  if (ctas > 1) cluster.sync();  // a CTA's shared memory outlives rank 0's reads
}

// Rows that one CTA covers with 4 loads per thread stay with it: a cluster's two barriers cost more than they save there.
int launch_argmax(cudaStream_t stream, const float *logits, uint32_t n, uint32_t batch, int32_t *d_out, uint32_t *d_pos, int32_t *out_tokens,
                  uint32_t *d_count, uint32_t out_capacity, const int *code = nullptr) {
  const unsigned ctas = n <= 4096 ? 1 : (n <= 8192 ? 2 : (n <= 16384 ? 4 : 8));
  GRETA_CUDA_TRY(launch_pdl_cluster(argmax_kernel, dim3(ctas, batch), dim3(1024), ctas, 0, stream, logits, n, d_out, d_pos, out_tokens, d_count,
                                    out_capacity, code));
  return launched("argmax_kernel");
}

int launch_rmsnorm_f16(cudaStream_t stream, const float *x, const float *gamma, void *y, float *y32, uint32_t rows, uint32_t cols, float eps) {
  auto go = [&](auto kernel) { return launch_pdl(kernel, dim3(rows), dim3(256), 0, stream, x, gamma, static_cast<__half *>(y), y32, cols, eps); };
  if (cols <= 256 * 8)
    GRETA_CUDA_TRY(y32 ? go(rmsnorm_f16_kernel<8, true>) : go(rmsnorm_f16_kernel<8, false>));
  else if (cols <= 256 * 16)
    GRETA_CUDA_TRY(y32 ? go(rmsnorm_f16_kernel<16, true>) : go(rmsnorm_f16_kernel<16, false>));
  else
    GRETA_CUDA_TRY(y32 ? go(rmsnorm_f16_kernel<32, true>) : go(rmsnorm_f16_kernel<32, false>));
  return launched("rmsnorm_f16_kernel");
}

inline unsigned blocks_for(size_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

extern "C" {

size_t greta_cuda_qs_bytes(int fmt, uint32_t N, uint32_t K) {
  return (size_t)N * (K / 32) * payload_bytes(fmt);
}
size_t greta_cuda_d_bytes(int fmt, uint32_t N, uint32_t K) {
  if (fmt == GRETA_FMT_F16) return 0;
  if (fmt == GRETA_FMT_REF_INT4 || fmt == GRETA_FMT_REF_INT8) return (size_t)N * (K / 32) * 4;
  return (size_t)N * d_row_stride(K / 32) * 2;
}

int greta_cuda_repack_gguf(greta_stream_t stream, int fmt, const void *blocks, void *qs, void *d, uint32_t N,
                           uint32_t K) {
  GRETA_REQUIRE(fmt == GRETA_FMT_Q4_0 || fmt == GRETA_FMT_Q8_0, "repack_gguf: format %d is not a GGUF block format", fmt);
  GRETA_REQUIRE(K % 32 == 0, "repack_gguf: K=%u is not a multiple of 32", K);
  size_t nb = (size_t)N * (K / 32);
  if (nb == 0) return GRETA_OK;
  GRETA_REQUIRE(blocks && qs && d, "repack_gguf: null pointer");
  GRETA_REQUIRE(((uintptr_t)blocks & 1) == 0 && aligned16(qs) && ((uintptr_t)d & 1) == 0, "repack_gguf: misaligned pointer");
  if (d_row_stride(K / 32) != K / 32) GRETA_CUDA_TRY(cudaMemsetAsync(d, 0, greta_cuda_d_bytes(fmt, N, K), S(stream)));  // row padding
  if (fmt == GRETA_FMT_Q4_0)
    repack_kernel<GRETA_FMT_Q4_0><<<blocks_for(nb, 256), 256, 0, S(stream)>>>((const uint8_t *)blocks, (uint8_t *)qs, (uint16_t *)d, nb, K / 32);
  else
    repack_kernel<GRETA_FMT_Q8_0><<<blocks_for(nb, 256), 256, 0, S(stream)>>>((const uint8_t *)blocks, (uint8_t *)qs, (uint16_t *)d, nb, K / 32);
  return launched("repack_kernel");
}

int greta_cuda_dequant(greta_stream_t stream, int fmt, const void *qs, const void *d, float *out, uint32_t N, uint32_t K) {
  GRETA_REQUIRE(K % 32 == 0, "dequant: K=%u is not a multiple of 32", K);
  size_t nb = (size_t)N * (K / 32);
  if (nb == 0) return GRETA_OK;
  GRETA_REQUIRE(qs && d && out, "dequant: null pointer");
  unsigned g = blocks_for(nb, 128);
  switch (fmt) {
    case GRETA_FMT_Q4_0: dequant_kernel<GRETA_FMT_Q4_0><<<g, 128, 0, S(stream)>>>((const uint8_t *)qs, d, out, nb, K / 32); break;
    case GRETA_FMT_Q8_0: dequant_kernel<GRETA_FMT_Q8_0><<<g, 128, 0, S(stream)>>>((const uint8_t *)qs, d, out, nb, K / 32); break;
    case GRETA_FMT_REF_INT4: dequant_kernel<GRETA_FMT_REF_INT4><<<g, 128, 0, S(stream)>>>((const uint8_t *)qs, d, out, nb, K / 32); break;
    case GRETA_FMT_REF_INT8: dequant_kernel<GRETA_FMT_REF_INT8><<<g, 128, 0, S(stream)>>>((const uint8_t *)qs, d, out, nb, K / 32); break;
    default: GRETA_REQUIRE(false, "dequant: unsupported format %d", fmt);
  }
  return launched("dequant_kernel");
}

int greta_cuda_f32_to_f16(greta_stream_t stream, const float *in, void *out, size_t n) {
  if (n == 0) return GRETA_OK;
  GRETA_REQUIRE(in && out, "f32_to_f16: null pointer");
  GRETA_REQUIRE(aligned16(in) && ((uintptr_t)out & 7) == 0, "f32_to_f16: misaligned pointer");
  f32_to_f16_kernel<<<blocks_for((n + 3) / 4, 256), 256, 0, S(stream)>>>(in, (__half *)out, n);
  return launched("f32_to_f16_kernel");
}
int greta_cuda_f16_to_f32(greta_stream_t stream, const void *in, float *out, size_t n) {
  if (n == 0) return GRETA_OK;
  GRETA_REQUIRE(in && out, "f16_to_f32: null pointer");
  f16_to_f32_kernel<<<blocks_for(n, 256), 256, 0, S(stream)>>>((const __half *)in, out, n);
  return launched("f16_to_f32_kernel");
}

int greta_cuda_rmsnorm(greta_stream_t stream, const float *x, const float *gamma, float *y, uint32_t rows, uint32_t cols, float eps) {
  if (rows == 0 || cols == 0) return GRETA_OK;
  GRETA_REQUIRE(x && gamma && y, "rmsnorm: null pointer");
  rmsnorm_kernel<<<rows, 256, 0, S(stream)>>>(x, gamma, y, cols, eps);
  return launched("rmsnorm_kernel");
}
int greta_cuda_rmsnorm_f16(greta_stream_t stream, const float *x, const float *gamma, void *y, uint32_t rows, uint32_t cols, float eps) {
  if (rows == 0 || cols == 0) return GRETA_OK;
  GRETA_REQUIRE(x && gamma && y, "rmsnorm_f16: null pointer");
  return launch_rmsnorm_f16(S(stream), x, gamma, y, nullptr, rows, cols, eps);
}
int greta_cuda_rmsnorm_both(greta_stream_t stream, const float *x, const float *gamma, float *y, void *y_f16, uint32_t rows, uint32_t cols, float eps) {
  if (rows == 0 || cols == 0) return GRETA_OK;
  GRETA_REQUIRE(x && gamma && y && y_f16, "rmsnorm_both: null pointer");
  return launch_rmsnorm_f16(S(stream), x, gamma, y_f16, y, rows, cols, eps);
}
int greta_cuda_add(greta_stream_t stream, const float *a, const float *b, float *c, size_t n) {
  if (n == 0) return GRETA_OK;
  GRETA_REQUIRE(a && b && c, "add: null pointer");
  add_kernel<<<blocks_for(n, 256), 256, 0, S(stream)>>>(a, b, c, n);
  return launched("add_kernel");
}
int greta_cuda_silu_mul(greta_stream_t stream, const float *g, const float *u, float *y, size_t n) {
  if (n == 0) return GRETA_OK;
  GRETA_REQUIRE(g && u && y, "silu_mul: null pointer");
  silu_mul_kernel<<<blocks_for(n, 256), 256, 0, S(stream)>>>(g, u, y, n);
  return launched("silu_mul_kernel");
}
int greta_cuda_embedding(greta_stream_t stream, const int32_t *tokens, const void *table, int table_is_f16, float *out,
                         uint32_t Sq, uint32_t dim, uint32_t vocab) {
  size_t n = (size_t)Sq * dim;
  if (n == 0) return GRETA_OK;
  GRETA_REQUIRE(tokens && table && out, "embedding: null pointer");
  const bool vec = dim % 4 == 0 && aligned16(out) && ((uintptr_t)table & (table_is_f16 ? 7u : 15u)) == 0;
  const dim3 grid(Sq, std::min<size_t>(65535, ((size_t)dim / (vec ? 4 : 1) + 255) / 256));
  auto go = [&](auto kernel) { return launch_pdl(kernel, grid, dim3(256), 0, S(stream), tokens, table, out, dim, vocab); };
  GRETA_CUDA_TRY(table_is_f16 ? (vec ? go(embedding_kernel<true, 4>) : go(embedding_kernel<true, 1>))
                              : (vec ? go(embedding_kernel<false, 4>) : go(embedding_kernel<false, 1>)));
  return launched("embedding_kernel");
}
int greta_cuda_argmax(greta_stream_t stream, const float *logits, uint32_t n, int32_t *d_out) {
  GRETA_REQUIRE(n > 0, "argmax: empty input");
  GRETA_REQUIRE(logits && d_out, "argmax: null pointer");
  return launch_argmax(S(stream), logits, n, 1, d_out, nullptr, nullptr, nullptr, 0u);
}
int greta_cuda_argmax_advance(greta_stream_t stream, const float *logits, uint32_t n, int32_t *d_next, uint32_t *d_pos,
                              int32_t *d_out_tokens, uint32_t *d_count, uint32_t out_capacity) {
  GRETA_REQUIRE(n > 0, "argmax_advance: empty input");
  GRETA_REQUIRE(logits && d_next, "argmax_advance: null pointer");
  return launch_argmax(S(stream), logits, n, 1, d_next, d_pos, d_out_tokens, d_count, out_capacity);
}
int greta_cuda_argmax_advance_batch(greta_stream_t stream, const float *logits, uint32_t n, uint32_t batch, int32_t *d_next, uint32_t *d_pos,
                                    int32_t *d_out_tokens, uint32_t *d_count, uint32_t out_capacity) {
  GRETA_REQUIRE(n > 0 && batch >= 1 && batch <= 65535, "argmax_advance_batch: n=%u, batch=%u", n, batch);
  GRETA_REQUIRE(logits && d_next, "argmax_advance_batch: null pointer");
  return launch_argmax(S(stream), logits, n, batch, d_next, d_pos, d_out_tokens, d_count, out_capacity);
}
int greta_cuda_argmax_advance_batch_status(greta_stream_t stream, const float *logits, uint32_t n, uint32_t batch, int32_t *d_next, uint32_t *d_pos,
                                           int32_t *d_out_tokens, uint32_t *d_count, uint32_t out_capacity) {
  GRETA_REQUIRE(n > 0 && batch >= 1 && batch <= 65535, "argmax_advance_batch_status: n=%u, batch=%u", n, batch);
  GRETA_REQUIRE(logits && d_next, "argmax_advance_batch_status: null pointer");
  int *code = nullptr;
  if (int rc = gemm_ts_error_word(&code)) return rc;
  return launch_argmax(S(stream), logits, n, batch, d_next, d_pos, d_out_tokens, d_count, out_capacity, code);
}
int greta_cuda_silu(greta_stream_t stream, const float *x, float *y, size_t n) {
  if (n == 0) return GRETA_OK;
  GRETA_REQUIRE(x && y, "silu: null pointer");
  silu_kernel<<<blocks_for(n, 256), 256, 0, S(stream)>>>(x, y, n);
  return launched("silu_kernel");
}
int greta_cuda_mul(greta_stream_t stream, const float *a, const float *b, float *c, size_t n) {
  if (n == 0) return GRETA_OK;
  GRETA_REQUIRE(a && b && c, "mul: null pointer");
  mul_kernel<<<blocks_for(n, 256), 256, 0, S(stream)>>>(a, b, c, n);
  return launched("mul_kernel");
}

}  // extern "C"
