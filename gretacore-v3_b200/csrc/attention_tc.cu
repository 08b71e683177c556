// Causal prefill attention on the 5th-generation tensor cores: 128 queries of one head per CTA, key tiles of 128 by TMA from the fp16 cache.
// Queries and probabilities travel as fp16 pairs (hi = half(x), lo = half(x - hi)), as in attention_mma.cu, so the products keep
// fp32 precision: S = Qhi K^T + Qlo K^T, O += Phi V + Plo V.  Scores, probabilities and outputs live in tensor memory.
//
// What bounds it: 32 MMAs of 128 x 128 x 16 per key tile, about 2400 cycles, against about 1400 for the softmax of a row per thread, which runs
// under the next tile's scores.  attention_mma.cu's mma.sync form, capped by that instruction's rate and by re-reading K and V from
// shared memory for every 16 queries, takes 256 us for 1531 queries of 32 heads of 128 over 8 KV heads (caches cold); this one 98 (0.12 of
// the measured bf16 rate by the 19 GF of the causal half, 0.35 by the MMAs issued for it: pairs, and whole tiles on the diagonal); 2048 queries
// of 64 heads of 64: 365 and 168.  Error against 64 bits, 2-norm: 1.3e-6 and 6.6e-7, 1.5e-6 and 7.7e-7; at four times the queries 2.1e-6 and 1.2e-6.
//
// Warp 0: TMA of K and V; warp 1: TMEM allocation, MMA issue; warps 2-5: queries into shared memory, softmax (one query row per thread),
// outputs.  TMEM columns: scores of even and odd tiles at 0 and 128, each overwritten by its probabilities (64 columns hi, 64 lo); outputs
// from 256 (Phi V) and from 384 (Plo V) on.  The tensor core cuts every sum off at the accumulator's last bit, so small terms come first
// (Qlo K^T) or to an accumulator of their own: half as many cuts at full size.  Waits are bounded as in gemm_ts.cu.
#include <math.h>

#include "attention_device.cuh"
#include "mma_device.cuh"
#include "tc_device.cuh"

using namespace greta;

namespace {

constexpr uint32_t AT_Q = 128, AT_KEYS = 128, AT_THREADS = 192, AT_TMEM = 512, AT_STAGES = 2;
constexpr uint32_t AT_SLAB = 128 * 128;  // bytes of 64 columns of 128 rows
constexpr float AT_LAZY = 8.f;           // a row's maximum may grow by this exponent before its sums are rescaled
constexpr float AT_LOG2E = 1.4426950408889634f;
constexpr float AT_LOWEST = -3.4028234e38f;  // a row's maximum before any score: scores of minus infinity have weight 0 whatever stands in front of them

__device__ __forceinline__ void tma_load_3d(void *smem_dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(smem_dst)),
               "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
               : "memory");
}

struct AttnTcArgs {
  CUtensorMap k, v;  // [Hkv][keys][Dh]; rows past the last key read as zeros
  const float *q;    // [S][H][Dh]
  const __half *kc, *vc;  // what `k` and `v` describe
  void *o;           // [S][H][Dh]
  uint32_t S, pos0, H, group, max_seq;
  float scale2;      // scale * log2(e)
  int *error;        // where a wait that gave up is reported
};

// A key that a row must not see has weight 0 in its products, and 0 times a value that is no finite number is none.  Takes 32 outputs of a row (position i),
// some of them no finite numbers, and sums the columns again whose values are finite up to the row and not behind it in its tiles: 2048 rows with
// one such token in the last tile take 13 ms instead of 0.1.  (Looking through the values in shared memory in front of the products took 0.2-0.5 us
// per tile on the diagonal, 1-5 % of the kernel, whichever warp did it; a look at the outputs takes 0-1 %.)
template <int DH>
__device__ __noinline__ void sum_again(const AttnTcArgs &w, const uint8_t *qs, uint32_t h, uint32_t row, uint32_t i, uint32_t tiles_end, uint32_t c, bool halved, float *y) {
  const size_t at = (size_t)(h / w.group) * w.max_seq * DH;
  const __half *k = w.kc + at, *v = w.vc + at + c;
  const uint32_t end = min(tiles_end, w.pos0 + w.S);
  uint32_t hit = 0;
  for (uint32_t e = 0; e < 32; ++e) {
    if (isfinite(y[e])) continue;
    uint32_t j = i + 1;
    while (j < end && isfinite(__half2float(v[(size_t)j * DH + e]))) ++j;
    if (j < end) hit |= 1u << e;
  }
  if (!hit) return;
  float mx = AT_LOWEST, l = 0.f, acc[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) acc[e] = 0.f;
  for (uint32_t j = 0; j <= i && hit; ++j) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (uint32_t d = 0; d < DH; d += 8) {
      const uint4 x = *reinterpret_cast<const uint4 *>(k + (size_t)j * DH + d);
      const uint8_t *qd = qs + (d / 64) * AT_SLAB + row * 128 + (((d % 64 / 8) ^ (row & 7)) << 4);
      const uint4 hi = *reinterpret_cast<const uint4 *>(qd), lo = *reinterpret_cast<const uint4 *>(qd + DH / 64 * AT_SLAB);
      const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, hw[4] = {hi.x, hi.y, hi.z, hi.w}, lw[4] = {lo.x, lo.y, lo.z, lo.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 z = h2_to_f2(xw[e]), a = h2_to_f2(hw[e]), b = h2_to_f2(lw[e]);
        s[e] = fmaf(a.x + b.x, z.x, fmaf(a.y + b.y, z.y, s[e]));
      }
    }
    const float t = ((s[0] + s[1]) + (s[2] + s[3])) * (halved ? 2.f : 1.f), nm = fmaxf(mx, t), f = ex2(mx - nm), p = ex2(t - nm);
    mx = nm;
    l = fmaf(l, f, p);
#pragma unroll
    for (int e = 0; e < 32; e += 8) {
      const uint4 b = *reinterpret_cast<const uint4 *>(v + (size_t)j * DH + e);
      const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float2 z = h2_to_f2(bw[r]);
        acc[e + 2 * r] = fmaf(acc[e + 2 * r], f, p * z.x);
        acc[e + 2 * r + 1] = fmaf(acc[e + 2 * r + 1], f, p * z.y);
      }
    }
    if (j % 64 == 0) {  // a value that the row sees is none either: left as it is
#pragma unroll
      for (int e = 0; e < 32; ++e)
        if (!isfinite(acc[e])) hit &= ~(1u << e);
    }
  }
#pragma unroll
  for (int e = 0; e < 32; ++e)
    if (hit >> e & 1) y[e] = acc[e] / l;
}

template <int DH, bool F16>
__global__ void __launch_bounds__(AT_THREADS, 1) attn_tc_prefill_kernel(const __grid_constant__ AttnTcArgs w) {
  constexpr uint32_t SD = DH / 64;  // slabs per row
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t *qs = smem, *ks = qs + 2 * SD * AT_SLAB, *vs = ks + AT_STAGES * SD * AT_SLAB;  // queries [hi, lo][slab]
  uint64_t *bars = reinterpret_cast<uint64_t *>(vs + AT_STAGES * SD * AT_SLAB);
  uint64_t *kf = bars, *ke = bars + 2, *vf = bars + 4, *ve = bars + 6, *sf = bars + 8, *pf = bars + 10, *od = bars + 12, *qf = bars + 13, *fin = bars + 14;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 15);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t h = blockIdx.x, m0 = (gridDim.y - 1 - blockIdx.y) * AT_Q;  // the longest rows of all heads first
  const uint32_t nq = min(AT_Q, w.S - m0), i0 = w.pos0 + m0, ntiles = (i0 + nq + AT_KEYS - 1) / AT_KEYS;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&kf[i], 1);
      mbar_init(&ke[i], 1);
      mbar_init(&vf[i], 1);
      mbar_init(&ve[i], 1);
      mbar_init(&sf[i], 1);
      mbar_init(&pf[i], 4);
    }
    mbar_init(od, 1);
    mbar_init(fin, 1);
    mbar_init(qf, 4);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&w.k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&w.v) : "memory");
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, AT_TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const bool leader = elect_one();
  pdl_launch_dependents();
  pdl_wait();

  // Both issuing warps run uniform loops whose lanes meet between a wait and the issue behind it (elect_one in tc_device.cuh).
  if (warp == 0) {
    const int kvh = (int)(h / w.group);
    uint32_t keys = 0, values = 0;  // copies issued
    bool ok = true;
    for (uint32_t t = 0; t < ntiles; ++t) {
      const uint32_t st = t % AT_STAGES, ph = ((t / AT_STAGES) & 1) ^ 1;
      if (ok) ok = mbar_wait(&ke[st], ph, abort_flag, 600 + st);
      __syncwarp();
      if (leader && ok) {
        mbar_arrive_expect_tx(&kf[st], SD * AT_SLAB);
        for (uint32_t c = 0; c < SD; ++c) {
          tma_load_3d(ks + (st * SD + c) * AT_SLAB, &w.k, (int)(c * 64), (int)(t * AT_KEYS), kvh, &kf[st]);
        }
        ++keys;
      }
      if (ok) ok = mbar_wait(&ve[st], ph, abort_flag, 610 + st);
      __syncwarp();
      if (leader && ok) {
        mbar_arrive_expect_tx(&vf[st], SD * AT_SLAB);
        for (uint32_t c = 0; c < SD; ++c) {
          tma_load_3d(vs + (st * SD + c) * AT_SLAB, &w.v, (int)(c * 64), (int)(t * AT_KEYS), kvh, &vf[st]);
        }
        ++values;
      }
    }
    if (leader && *abort_flag) drain_copies(kf, keys, AT_STAGES);
    if (leader && *abort_flag) drain_copies(vf, values, AT_STAGES);
  } else if (warp == 1) {
    constexpr uint32_t idesc_s = instr_desc_f16(AT_Q, AT_KEYS);
    constexpr uint32_t idesc_o = instr_desc_f16(AT_Q, DH) | (1u << 16);  // values: keys are the rows of memory (N-major operand)
    const uint32_t q_lo = smem_desc_lo(smem_u32(qs)), k_lo = smem_desc_lo(smem_u32(ks));
    const uint32_t v_lo = ((smem_u32(vs) >> 4) & 0x3FFFu) | ((AT_SLAB >> 4) << 16);  // 64-column groups are a slab apart
    bool ok = true;
    if (ok) ok = mbar_wait(qf, 0, abort_flag, 620);
    __syncwarp();
    for (uint32_t n = 0; n <= ntiles; ++n) {  // scores of tile n, then outputs of tile n - 1
      if (n < ntiles) {
        const uint32_t st = n % AT_STAGES;
        // od: the probabilities of tile n - 2 have been read, its columns are free
        if (ok) ok = mbar_wait(&kf[st], (n / AT_STAGES) & 1, abort_flag, 630 + st) && (n < 2 || mbar_wait(od, n & 1, abort_flag, 640));
        __syncwarp();
        if (leader && ok) {
          tc_fence_after();
#pragma unroll
          for (uint32_t part = 0; part < 2; ++part)
#pragma unroll
            for (uint32_t k16 = 0; k16 < DH / 16; ++k16)
              umma_f16(tmem + (n & 1) * 128, q_lo + ((1 - part) * SD + k16 / 4) * (AT_SLAB >> 4) + (k16 & 3) * 2,
                       k_lo + (st * SD + k16 / 4) * (AT_SLAB >> 4) + (k16 & 3) * 2, SMEM_DESC_HI_SW128, idesc_s, (part | k16) ? 1u : 0u);
          umma_commit(&ke[st]);
          umma_commit(&sf[n & 1]);
        }
      }
      if (n) {
        const uint32_t t = n - 1, st = t % AT_STAGES;
        if (ok) ok = mbar_wait(&vf[st], (t / AT_STAGES) & 1, abort_flag, 650 + st) && mbar_wait(&pf[t & 1], (t >> 1) & 1, abort_flag, 660 + (t & 1));
        __syncwarp();
        if (leader && ok) {
          tc_fence_after();
#pragma unroll
          for (uint32_t part = 0; part < 2; ++part)
#pragma unroll
            for (uint32_t k16 = 0; k16 < AT_KEYS / 16; ++k16)
              umma_f16_ts(tmem + 256 + part * 128, tmem + (t & 1) * 128 + part * 64 + k16 * 8, v_lo + st * SD * (AT_SLAB >> 4) + k16 * (2048 >> 4), SMEM_DESC_HI_SW128, idesc_o,
                          (t | k16) ? 1u : 0u);
          umma_commit(&ve[st]);
          umma_commit(od);
          if (t + 1 == ntiles) umma_commit(fin);
        }
      }
    }
  } else {
    const uint32_t quad = warp & 3, row = quad * 32 + lane, i = i0 + row;
    // ---- the warp's 32 queries, scaled, as pairs in the swizzled K-major layout
    constexpr uint32_t LPR = DH / 4, RPP = 32 / LPR;  // lanes per row, rows per pass
    // Half the queries, and twice their scores, where one of them is past fp16 under log2(e): the range is that of q * scale, as in attention_mma.cu.
    bool halved = false;
    for (;;) {
      const float by = halved ? 0.5f * w.scale2 : w.scale2;
      float most = 0.f;
#pragma unroll 8
      for (uint32_t r0 = 0; r0 < 32; r0 += RPP) {
        const uint32_t r = quad * 32 + r0 + lane / LPR, e = (lane % LPR) * 4;
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < nq) f = *reinterpret_cast<const float4 *>(w.q + ((size_t)(m0 + r) * w.H + h) * DH + e);
        f = make_float4(f.x * by, f.y * by, f.z * by, f.w * by);
        most = fmaxf(most, fmaxf(fmaxf(fabsf(f.x), fabsf(f.y)), fmaxf(fabsf(f.z), fabsf(f.w))));
        const uint2 hi = make_uint2(half2_bits(f.x, f.y), half2_bits(f.z, f.w));
        const float2 a = h2_to_f2(hi.x), b = h2_to_f2(hi.y);
        uint8_t *dst = qs + (e / 64) * AT_SLAB + r * 128 + ((((e % 64) / 8) ^ (r & 7)) << 4) + (e & 4) * 2;
        *reinterpret_cast<uint2 *>(dst) = hi;
        *reinterpret_cast<uint2 *>(dst + SD * AT_SLAB) = make_uint2(half2_bits(f.x - a.x, f.y - a.y), half2_bits(f.z - b.x, f.w - b.y));
      }
      if (halved || !__any_sync(0xffffffffu, most > 65504.f)) break;
      halved = true;
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(qf);
    const uint32_t lanes = tmem + (quad * 32 << 16);
    float mx = AT_LOWEST, l = 0.f;
    bool ok = true;
    for (uint32_t t = 0; t < ntiles && ok; ++t) {
      const uint32_t sb = lanes + (t & 1) * 128;
      ok = mbar_wait_warp(&sf[t & 1], (t >> 1) & 1, abort_flag, 670 + (t & 1));
      if (!ok) break;
      tc_fence_after();
      uint32_t v[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(sb + c * 32, v[c]);
      tmem_ld_wait();
      if (halved) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int j = 0; j < 32; ++j) v[c][j] = __float_as_uint(2.f * __uint_as_float(v[c][j]));
      }
      if (t * AT_KEYS + AT_KEYS - 1 > i0) {  // the diagonal runs through the tile
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (t * AT_KEYS + c * 32 + j > i) v[c][j] = 0xFF800000u;
      }
      float tm[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int j = 0; j < 32; ++j) tm[j & 3] = fmaxf(tm[j & 3], __uint_as_float(v[c][j]));
      const float nm = fmaxf(mx, fmaxf(fmaxf(tm[0], tm[1]), fmaxf(tm[2], tm[3])));
      if (t == 0) {
        mx = nm;
      } else if (__any_sync(0xffffffffu, nm > mx + AT_LAZY)) {
        const float f = nm > mx + AT_LAZY ? ex2(mx - nm) : 1.f;
        if (nm > mx + AT_LAZY) mx = nm;
        l *= f;
        ok = mbar_wait_warp(od, (t - 1) & 1, abort_flag, 680);  // every product so far is in
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (uint32_t c = 0; c < 2 * DH; c += 32) {
          const uint32_t at = lanes + 256 + (c < DH ? c : 128 + c - DH);
          uint32_t o[32];
          tmem_ld32(at, o);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
          tmem_st32(at, o);
        }
      }
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t hi[32], lo[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float p0 = ex2(__uint_as_float(v[2 * c + j / 16][(2 * j) & 31]) - mx), p1 = ex2(__uint_as_float(v[2 * c + j / 16][(2 * j + 1) & 31]) - mx);
          sum[(2 * j) & 3] += p0;
          sum[(2 * j + 1) & 3] += p1;
          hi[j] = half2_bits(p0, p1);
          const float2 b = h2_to_f2(hi[j]);
          lo[j] = half2_bits(p0 - b.x, p1 - b.y);
        }
        tmem_st32(sb + c * 32, hi);
        tmem_st32(sb + 64 + c * 32, lo);
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pf[t & 1]);
    }
    // A barrier of its own for the end: od may be two phases on by now, which a parity takes for none.
    ok = ok && mbar_wait_warp(fin, 0, abort_flag, 690);
    if (ok) {
      tc_fence_after();
      const float inv = 1.f / l;
      const size_t at = ((size_t)(m0 + row) * w.H + h) * DH;
#pragma unroll 1
      for (uint32_t c = 0; c < DH; c += 32) {
        uint32_t o[32], small[32];
        __syncwarp();
        tmem_ld32(lanes + 256 + c, o);
        tmem_ld32(lanes + 384 + c, small);
        tmem_ld_wait();
        if (row >= nq) continue;
        float z = 0.f;  // 0, or NaN
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float x = (__uint_as_float(o[j]) + __uint_as_float(small[j])) * inv;
          o[j] = __float_as_uint(x);
          z = fmaf(x, 0.f, z);
        }
        if (z != 0.f) {
          float y[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) y[j] = __uint_as_float(o[j]);
          sum_again<DH>(w, qs, h, row, i, ntiles * AT_KEYS, c, halved, y);
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(y[j]);
        }
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          float y[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) y[e] = __uint_as_float(o[j + e]);
          if (F16) {
            *reinterpret_cast<uint4 *>(static_cast<__half *>(w.o) + at + c + j) =
                make_uint4(half2_bits(y[0], y[1]), half2_bits(y[2], y[3]), half2_bits(y[4], y[5]), half2_bits(y[6], y[7]));
          } else {
            float4 *dst = reinterpret_cast<float4 *>(static_cast<float *>(w.o) + at + c + j);
            dst[0] = make_float4(y[0], y[1], y[2], y[3]);
            dst[1] = make_float4(y[4], y[5], y[6], y[7]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) atomicCAS(w.error, 0, *abort_flag);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, AT_TMEM);
  }
}

template <int DH, bool F16>
int launch_tc_prefill(cudaStream_t stream, const AttnTcArgs &w) {
  constexpr size_t smem = (size_t)(2 + 2 * AT_STAGES) * (DH / 64) * AT_SLAB + 1024 + 15 * 8 + 16;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    GRETA_CUDA_TRY(cudaFuncSetAttribute(attn_tc_prefill_kernel<DH, F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set[dev] = true;
  }
  GRETA_CUDA_TRY(launch_pdl(attn_tc_prefill_kernel<DH, F16>, dim3(w.H, (w.S + AT_Q - 1) / AT_Q), dim3(AT_THREADS), smem, stream, w));
  return launched("attn_tc_prefill_kernel");
}

}  // namespace

namespace greta {

int gemm_ts_error_word(int **word);  // gemm_ts.cu: the word that greta_cuda_gemm_segments_status reads

// S queries at positions pos0 .. against the fp16 cache, Dh 64 or 128; out fp32, or fp16 (the fp32 result rounded once).
int attn_tc_prefill(cudaStream_t stream, const AttnParams &p, uint32_t S, uint32_t pos0, uint32_t Dh, void *out, bool f16) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) {
    set_error("attn_prefill: cuTensorMapEncodeTiled is not available from this driver");
    return GRETA_ERR_NOT_IMPLEMENTED;
  }
  AttnTcArgs w{};
  const cuuint64_t dims[3] = {Dh, pos0 + S, p.Hkv}, strides[2] = {(cuuint64_t)Dh * 2, (cuuint64_t)p.max_seq * Dh * 2};
  const cuuint32_t box[3] = {64, AT_KEYS, 1}, one[3] = {1, 1, 1};
  for (int i = 0; i < 2; ++i) {
    const CUresult r = enc(i ? &w.v : &w.k, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(i ? p.vc : p.kc), dims, strides, box, one,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
      set_error("attn_prefill: cuTensorMapEncodeTiled failed with code %d", (int)r);
      return GRETA_ERR_INVALID_ARGS;
    }
  }
  if (int rc = gemm_ts_error_word(&w.error)) return rc;
  w.q = p.q;
  w.kc = static_cast<const __half *>(p.kc);
  w.vc = static_cast<const __half *>(p.vc);
  w.max_seq = p.max_seq;
  w.o = out;
  w.S = S;
  w.pos0 = pos0;
  w.H = p.H;
  w.group = p.H / p.Hkv;
  w.scale2 = p.scale * AT_LOG2E;
  if (Dh == 128) return f16 ? launch_tc_prefill<128, true>(stream, w) : launch_tc_prefill<128, false>(stream, w);
  return f16 ? launch_tc_prefill<64, true>(stream, w) : launch_tc_prefill<64, false>(stream, w);
}

}  // namespace greta
