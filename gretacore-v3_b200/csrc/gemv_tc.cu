// Batched decode products (up to 32 activation rows) on the 5th-generation tensor cores:
//   y[m][n] = epilogue(sum_k x[m][k] * W[n][k]), W in Q4_0, Q8_0 or fp16, x in fp32.
//
// gemv_batch.cu's mma.sync form is capped by that instruction's rate: 16 rows as fp16 pairs need 8 of them per 288 bytes of Q4_0 weights, which
// holds it at 0.2 of the memory bandwidth.  Here 128 weight rows are the rows of a tcgen05.mma and the activation rows its N dimension.  The
// arithmetic stays what it was: quantised weights are the exact integers of a block (its scale left out), activations fp16 pairs hi = half(x s),
// lo = half(x s - hi) with a power of two s per row; a block's sum comes out of tensor memory, takes the block's scale in fp32 and is added in fp32.
// Small terms come first in the tensor core, which cuts every sum off at its last bit.  Error against 64 bits, 2-norm of the worst row, 16 rows:
// 8192 x 8192 q4_0 1.3e-7 (mma.sync 2.2e-7), 4096 x 4096 fp16 1.5e-7 (1.6e-7).
//
// Measured in a CUDA graph with weights from HBM, both kernels of a product, us (mma.sync form behind the stroke): 16 rows q4_0 57344 x 8192 79 / 208
// (3.3 TB/s), 8192 x 8192 20.8 / 34, 4096 x 4096 11.8 / 17.1; q8_0 101 / 245 (4.9 TB/s), 26 / 39, 14.3 / 20.0; fp16 155 / 284 (6.1 TB/s), 32 / 43, 16.2 / 16.3;
// 32 rows q4_0 115 / 318, 30 / 51, 19.5 / 25.3.  What bounds q4_0: the chain load - unpack - store - multiply - read of a set of warps, of
// which four run at a time; of 91 us alone at 57344 x 8192 the products left out give 77, reading and adding the sums 79, unpacking 93.
//
// Warp roles (640 threads, one persistent CTA per SM):
//   warp 0       copies of prepared activations (an image of shared memory, made once per product by prep_image_kernel), 256 K of all rows at a time;
//   warp 1       TMEM allocation, the rows' factors;
//   warp 2       TMA of raw weights, 128 rows x 128 bytes and their scales; starts before the kernel's predecessor has finished;
//   warps 4-19   four sets of four warps: set s has half s / 2 of the step's 256 K of row tile s % 2.  It unpacks its weights into tensor memory (fp16
//                weights are multiplied out of shared memory as they came), its first warp issues the products, all scale and add the sums.
// Two row tiles share an activation buffer: with one the activations from L2 are as many bytes as the weights from HBM.
//
// Work is cut into steps of 256 K x 256 rows, and every CTA takes a run of them (row tiles one after the other, K inside; plan_shares).  A row tile that
// several CTAs share is summed through the workspace: each stores its part and takes a ticket; who comes last adds the parts in CTA order
// (the result does not depend on who that was) and finishes the rows.  Nobody waits for another CTA.
// Every wait is bounded, as in gemm_ts.cu; one that gave up is reported in the same word.
#include "gemv_device.cuh"
#include "gemv_tc.cuh"
#include "tc_device.cuh"

using namespace greta;

namespace {

constexpr uint32_t BT_STEP = 256, BT_STEP_BLOCKS = BT_STEP / 32;
constexpr uint32_t BT_RAW_PAYLOAD = 128 * 128, BT_RAW_BYTES = BT_RAW_PAYLOAD + 128 * 16;
constexpr uint32_t BT_SET_WARP0 = 4, BT_SETS = 4, BT_WORKERS = BT_SETS * 128, BT_THREADS = 32 * BT_SET_WARP0 + BT_WORKERS;
constexpr uint32_t BT_TMEM = 512, BT_D_COL = 256;  // columns: 64 of weights per set, then 64 of block sums per set
constexpr size_t BT_SMEM_MAX = 232448;

template <int FMT, int TN>
struct BtPlan {
  static constexpr bool Q4 = FMT == GRETA_FMT_Q4_0, F16 = FMT == GRETA_FMT_F16;
  static constexpr uint32_t UNITS = Q4 ? 2 : (F16 ? 8 : 4);         // raw units of a step: a tile's 256 K, half or a quarter of them
  static constexpr uint32_t RAW = 8;                                // two steps or more: a step's units are given back during the next; a slot is read by the same sets every time
  static constexpr uint32_t ACT = TN == 16 ? 3 : 2, ACT_BYTES = TN * BT_STEP * 4;
  static constexpr uint32_t SUB_BLOCKS = F16 ? 2 : 64 / TN, SUBS = 4 / SUB_BLOCKS;  // blocks of a pass: 64 columns of sums; passes per step
  static constexpr uint32_t OUT_BYTES = 2 * 16 * 128 * 4;
  static constexpr uint32_t BARS = 2 * RAW + 2 * ACT + 2 * BT_SETS;
  static constexpr size_t SMEM = 1024 + (size_t)RAW * BT_RAW_BYTES + ACT * ACT_BYTES + OUT_BYTES + BARS * 8 + 16 + 2 * TN * 4;
  static_assert(SMEM <= BT_SMEM_MAX && RAW % UNITS == 0 && (F16 || RAW >= 2 * UNITS), "shared memory plan");
};

struct BtArgs {
  CUtensorMap qs[3], d[3];
  GemvParams p;
  const uint8_t *image;
  const float *rowmul;
  float *part;        // [CTA][2][2 tiles][TN][128]
  uint32_t *tickets;  // [CTA]
  uint32_t n[3], tile_end[3], tiles, steps;
  int *error;
  // Runs of steps: column x of the grid's row y begins at step y * row + (x * run + min(x, longer)) * unit.
  uint32_t row, run, longer, unit;
};

__device__ __forceinline__ void bulk_load(void *smem_dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem_dst)), "l"(src), "r"(bytes),
               "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void sync_set(uint32_t set) { asm volatile("bar.sync %0, 128;" ::"r"(3 + set) : "memory"); }
__device__ __forceinline__ void sync_workers() { asm volatile("bar.sync 1, 512;" ::: "memory"); }

// One payload word -> exact integers q - 8 as fp16, two to a register, in the order of image_source().
__device__ __forceinline__ void int4_word(uint32_t w, uint32_t *o) {
  const uint32_t MAGIC = 0x64006400u, C1032 = 0x64086408u, SIXTEENTH = 0x2C002C00u, CM72 = 0xD480D480u;
  const uint32_t w8 = w >> 8;
  o[0] = hsub2_u(lop_and_or(w, 0x000F000Fu, MAGIC), C1032);
  o[1] = hsub2_u(lop_and_or(w8, 0x000F000Fu, MAGIC), C1032);
  o[2] = hfma2_u(lop_and_or(w, 0x00F000F0u, MAGIC), SIXTEENTH, CM72);
  o[3] = hfma2_u(lop_and_or(w8, 0x00F000F0u, MAGIC), SIXTEENTH, CM72);
}
__device__ __forceinline__ void int8_word(uint32_t w, uint32_t *o) {
  const uint32_t C1152 = 0x64806480u, t = w ^ 0x80808080u;
  o[0] = hsub2_u(__byte_perm(t, 0x64646464u, 0x5140), C1152);
  o[1] = hsub2_u(__byte_perm(t, 0x64646464u, 0x7362), C1152);
}

// The CTA whose run holds step s, of runs in one row of the grid.
__device__ __forceinline__ uint32_t run_of(const BtArgs &w, uint32_t s) {
  const uint32_t u = s / w.unit, head = w.longer * (w.run + 1);
  return u < head ? u / (w.run + 1) : w.longer + (u - head) / w.run;
}

struct TileAt {
  uint32_t seg, n0;
};
template <int EPI>
__device__ __forceinline__ TileAt tile_at(const BtArgs &w, uint32_t tile) {
  constexpr uint32_t ROWS = EPI == EPI_SWIGLU ? 64 : 128;
  TileAt r;
  r.seg = EPI != EPI_QKV || tile < w.tile_end[0] ? 0u : (tile < w.tile_end[1] ? 1u : 2u);
  r.n0 = (tile - (r.seg ? w.tile_end[r.seg - 1] : 0u)) * ROWS;  // one tile past the last is all out of range: copied as zeros, never stored
  return r;
}

// Rows of one finished pair of tiles out of shared memory, 16 activation rows from m_first: [tile][16][128 rows].
template <int EPI, int TN>
__device__ __forceinline__ void finish_pair(const BtArgs &w, uint32_t pair, uint32_t m_first, const float *buf, const float *factor, uint32_t tid) {
  const GemvParams &p = w.p;
  constexpr bool HALVES = EPI == EPI_SWIGLU || EPI == EPI_QKV;
  constexpr uint32_t LANES = HALVES ? 64 : 128, GROUPS = BT_WORKERS / LANES;
  const uint32_t j = tid % LANES, rows = p.M > m_first ? min(16u, p.M - m_first) : 0u;  // of this buffer
  if constexpr (!HALVES) {
    const uint32_t t = (tid / LANES) & 1, tile = pair * 2 + t, row = tile_at<EPI>(w, tile).n0 + j;
    if (tile >= w.tiles || row >= p.N) return;
    const float *col = buf + t * 16 * 128 + j;
    const size_t o = (size_t)m_first * p.N + row;
    factor += m_first;
    constexpr uint32_t U = 4;
    for (uint32_t m0 = tid / (2 * LANES); m0 < rows; m0 += U * GROUPS / 2) {
      float old[U];  // the residuals of four rows are on their way together
#pragma unroll
      for (uint32_t e = 0; e < U; ++e) {
        const uint32_t m = m0 + e * (GROUPS / 2);
        old[e] = EPI == EPI_RESIDUAL && m < rows ? __ldcg(p.resid + o + (size_t)m * p.N) : 0.f;
      }
#pragma unroll
      for (uint32_t e = 0; e < U; ++e) {
        const uint32_t m = m0 + e * (GROUPS / 2);
        if (m < rows) p.y[o + (size_t)m * p.N] = EPI == EPI_RESIDUAL ? old[e] + col[m * 128] * factor[m] : col[m * 128] * factor[m];
      }
    }
  } else {
    for (uint32_t i = tid / LANES; i < 2 * rows; i += GROUPS) {
      const uint32_t t = i >= rows, m = m_first + i - t * rows, tile = pair * 2 + t;
      if (tile >= w.tiles) continue;
      const TileAt at = tile_at<EPI>(w, tile);
      const float *col = buf + (t * 16 + m - m_first) * 128;
      const float f = factor[m];
      if (EPI == EPI_SWIGLU) {
        const uint32_t row = at.n0 + j;
        const float a = col[j] * f, b = col[j + 64] * f;
        if (row < p.N) p.y[(size_t)m * p.N + row] = (a / (1.0f + expf(-a))) * b;
      } else {
        const uint32_t half = p.Dh / 2, pos = reinterpret_cast<const uint32_t *>(factor)[TN + m];
        if (at.seg < 2) {
          const uint32_t in_head = j % half, lo = (j / half) * p.Dh + in_head, row = at.n0 + lo, head = row / p.Dh;
          if (row >= w.n[at.seg]) continue;  // whole heads
          const float a = col[lo] * f, b = col[lo + half] * f;
          float o0 = a, o1 = b;
          if (p.d_pos) {
            const float theta = (float)pos * powf(p.rope_base, -2.0f * (float)in_head / (float)p.Dh), c = cosf(theta), s = sinf(theta);
            o0 = a * c - b * s;
            o1 = a * s + b * c;
          }
          if (at.seg == 0) {
            float *q = p.q_out + (size_t)m * p.H * p.Dh + row;
            q[0] = o0;
            q[half] = o1;
          } else {
            if (p.k_out) {
              float *k = p.k_out + (size_t)m * p.Hkv * p.Dh + row;
              k[0] = o0;
              k[half] = o1;
            }
            if (p.k_cache && pos < p.max_seq) {  // a position past the cache is never written
              __half *k = p.k_cache + (((size_t)m * p.Hkv + head) * p.max_seq + pos) * p.Dh + in_head;
              k[0] = __float2half_rn(o0);
              k[half] = __float2half_rn(o1);
            }
          }
        } else {
#pragma unroll
          for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t row = at.n0 + j + 64 * h;
            if (row >= w.n[2]) continue;
            const float v = col[j + 64 * h] * f;
            if (p.v_out) p.v_out[(size_t)m * p.Hkv * p.Dh + row] = v;
            if (p.v_cache && pos < p.max_seq) p.v_cache[(((size_t)m * p.Hkv + row / p.Dh) * p.max_seq + pos) * p.Dh + row % p.Dh] = __float2half_rn(v);
          }
        }
      }
    }
  }
}

template <int FMT, int EPI, int TN>
__global__ void __launch_bounds__(BT_THREADS, 1) gemv_tc_kernel(const __grid_constant__ BtArgs w) {
  using P = BtPlan<FMT, TN>;
  constexpr bool Q4 = P::Q4, F16 = P::F16;
  constexpr uint32_t UNIT_BYTES = F16 ? BT_RAW_PAYLOAD : BT_RAW_BYTES;
  constexpr uint32_t RAW = P::RAW, ACT = P::ACT, UNITS = P::UNITS, SUBS = P::SUBS, SUB_BLOCKS = P::SUB_BLOCKS, SLAB = TN * 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *raw = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023), *act = raw + RAW * BT_RAW_BYTES;
  float *buf = reinterpret_cast<float *>(act + ACT * P::ACT_BYTES);
  uint64_t *raw_full = reinterpret_cast<uint64_t *>(reinterpret_cast<uint8_t *>(buf) + P::OUT_BYTES), *raw_empty = raw_full + RAW;
  uint64_t *act_full = raw_empty + RAW, *act_empty = act_full + ACT, *d_full = act_empty + ACT;  // [set], fp16: [set][slot]
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(d_full + 2 * BT_SETS);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1), *last_flag = abort_flag + 1;
  float *factor = reinterpret_cast<float *>(tmem_slot + 4);  // [TN], then positions [TN]
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t cta = blockIdx.y * gridDim.x + blockIdx.x, begin = blockIdx.y * w.row + (blockIdx.x * w.run + min(blockIdx.x, w.longer)) * w.unit;
  const uint32_t end = begin + (w.run + (blockIdx.x < w.longer ? 1 : 0)) * w.unit;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < RAW; ++s) {
      mbar_init(&raw_full[s], 1);
      mbar_init(&raw_empty[s], Q4 ? 8 : (F16 ? 1 : 4));
    }
    for (uint32_t s = 0; s < ACT; ++s) {
      mbar_init(&act_full[s], 1);
      mbar_init(&act_empty[s], BT_SETS);
    }
    for (uint32_t s = 0; s < 2 * BT_SETS; ++s) mbar_init(&d_full[s], 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BT_TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();

  const bool leader = elect_one();
  if (warp == 0) {
    pdl_wait();
    uint32_t s = 0, ph = 1, issued = 0;
    bool ok = true;
    for (uint32_t i = begin; i < end; ++i) {
      if (ok) ok = mbar_wait(&act_empty[s], ph, abort_flag, 700 + s);
      __syncwarp();
      if (leader && ok) {
        mbar_arrive_expect_tx(&act_full[s], P::ACT_BYTES);
        bulk_load(act + s * P::ACT_BYTES, w.image + (size_t)(i % w.steps) * P::ACT_BYTES, P::ACT_BYTES, &act_full[s]);
        ++issued;
      }
      if (++s == ACT) {
        s = 0;
        ph ^= 1;
      }
    }
    if (leader && *abort_flag) drain_copies(act_full, issued, ACT);
  } else if (warp == 2) {
    uint32_t u = 0, issued = 0;
    bool ok = true;
    for (uint32_t i = begin; i < end; ++i) {
      const uint32_t pair = i / w.steps, ks = i % w.steps;
      for (uint32_t v = 0; v < UNITS; ++v, ++u) {
        const uint32_t slot = u % RAW;
        const TileAt at = tile_at<EPI>(w, pair * 2 + (v & 1));
        if (u == RAW) pdl_wait();  // from here on the bounded waits depend on the predecessor's end
        uint8_t *dst = raw + slot * BT_RAW_BYTES;
        if (ok) ok = mbar_wait(&raw_empty[slot], ((u / RAW) & 1) ^ 1, abort_flag, 710 + slot);
        __syncwarp();
        if (leader && ok) {
          const int x = (int)((ks * (UNITS / 2) + (v >> 1)) * 128), kd = (int)(ks * BT_STEP_BLOCKS);
          mbar_arrive_expect_tx(&raw_full[slot], UNIT_BYTES);
          tma_load_2d(dst, &w.qs[at.seg], x, (int)at.n0, &raw_full[slot]);
          if (!F16) tma_load_2d(dst + BT_RAW_PAYLOAD, &w.d[at.seg], kd, (int)at.n0, &raw_full[slot]);
          if (EPI == EPI_SWIGLU) {
            tma_load_2d(dst + BT_RAW_PAYLOAD / 2, &w.qs[1], x, (int)at.n0, &raw_full[slot]);
            if (!F16) tma_load_2d(dst + BT_RAW_PAYLOAD + 64 * 16, &w.d[1], kd, (int)at.n0, &raw_full[slot]);
          }
          ++issued;
        }
      }
    }
    if (leader && *abort_flag) drain_copies(raw_full, issued, RAW);
  } else if (warp == 1) {  // what the end of every run needs of each activation row
    pdl_wait();
    if (lane < (int)w.p.M) {
      factor[lane] = __ldcg(w.rowmul + lane);
      if (EPI == EPI_QKV) reinterpret_cast<uint32_t *>(factor)[TN + lane] = w.p.d_pos ? __ldcg(w.p.d_pos + lane) : 0u;
    }
    asm volatile("bar.arrive 2, 544;" ::: "memory");
  } else if (warp >= (int)BT_SET_WARP0) {
    const uint32_t set = (uint32_t)(warp - BT_SET_WARP0) >> 2, t = set & 1, h = set >> 1, quad = warp & 3, row = quad * 32 + lane, x7 = row & 7;
    const uint32_t tid = threadIdx.x - 32 * BT_SET_WARP0;
    const uint32_t a_col = tmem + set * 64 + ((quad * 32) << 16), d_col = tmem + BT_D_COL + set * 64 + ((quad * 32) << 16);
    constexpr uint32_t idesc = instr_desc_f16(128, TN);
    const uint32_t act_lo = smem_desc_lo(smem_u32(act));
    const bool issuer = (warp & 3) == 0;
    uint32_t n = 0, as = 0, aph = 0;  // passes; activation stage and its phase
    bool ok = true, after = false, first = true;
    // fp16 weights are multiplied out of shared memory, 64 K of a tile at a time, a pass ahead of the reading of its sums.
    auto issue_f16 = [&](uint32_t step, uint32_t sub) {
      const uint32_t quarter = h + 2 * sub, u = (step - begin) * UNITS + quarter * 2 + t, slot = u % RAW;
      ok = __all_sync(0xffffffffu, ok && mbar_wait(&raw_full[slot], (u / RAW) & 1, abort_flag, 740 + slot));
      if (sub == 0) ok = __all_sync(0xffffffffu, ok && mbar_wait(&act_full[as], aph, abort_flag, 720 + as));
      if (leader && ok) {
        tc_fence_after();
        const uint32_t a = smem_desc_lo(smem_u32(raw)) + ((slot * BT_RAW_BYTES) >> 4), hi = act_lo + ((as * P::ACT_BYTES + quarter * SLAB) >> 4);
        const uint32_t lo = hi + ((4 * SLAB) >> 4);
#pragma unroll
        for (uint32_t b = 0; b < 2; ++b) {  // sums of 32 K like those of the other formats: one sum of 64 is cut off more often at full size
          const uint32_t d = tmem + set * 128 + sub * 64 + b * TN;
          umma_f16(d, a + b * 4, lo + b * 4, SMEM_DESC_HI_SW128, idesc, 0u);
          umma_f16(d, a + b * 4 + 2, lo + b * 4 + 2, SMEM_DESC_HI_SW128, idesc, 1u);
          umma_f16(d, a + b * 4, hi + b * 4, SMEM_DESC_HI_SW128, idesc, 1u);
          umma_f16(d, a + b * 4 + 2, hi + b * 4 + 2, SMEM_DESC_HI_SW128, idesc, 1u);
        }
        umma_commit(&d_full[set * 2 + sub]);
        umma_commit(&raw_empty[slot]);
        if (sub == 1) umma_commit(&act_empty[as]);
      }
      __syncwarp();
      if (sub == 1 && ++as == ACT) {
        as = 0;
        aph ^= 1;
      }
    };
    uint32_t v[32];                          // two blocks of this row, unpacked
    uint2 dw = make_uint2(0u, 0u), dw_next;  // scales of the step
    auto unit_of = [&](uint32_t step) { return (step - begin) * UNITS + (Q4 ? t : h * 2 + t); };
    auto open_unit = [&](uint32_t step) {
      const uint32_t u = unit_of(step);
      ok = __all_sync(0xffffffffu, ok && mbar_wait(&raw_full[u % RAW], (u / RAW) & 1, abort_flag, 740 + u % RAW));
      dw_next = *reinterpret_cast<const uint2 *>(raw + (u % RAW) * BT_RAW_BYTES + BT_RAW_PAYLOAD + row * 16 + h * 8);
    };
    auto unpack = [&](uint32_t step, uint32_t pair2) {  // blocks 2 pair2 and 2 pair2 + 1 of this set's half
      const uint8_t *pr = raw + (unit_of(step) % RAW) * BT_RAW_BYTES + row * 128;
#pragma unroll
      for (uint32_t c = 0; c < (Q4 ? 2u : 4u); ++c) {
        const uint4 q = *reinterpret_cast<const uint4 *>(pr + (((Q4 ? h * 4 + pair2 * 2 + c : pair2 * 4 + c) ^ x7) << 4));
        const uint32_t pw[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
          if (Q4)
            int4_word(pw[e], v + c * 16 + e * 4);
          else
            int8_word(pw[e], v + c * 8 + e * 2);
        }
      }
    };
    if constexpr (F16) {
      pdl_wait();
      if (issuer) issue_f16(begin, 0);
    } else {
      open_unit(begin);
      if (ok) unpack(begin, 0);
    }
    uint32_t i = begin;
    while (i < end) {
      const uint32_t pair = i / w.steps, k0 = i % w.steps, count = min(end - i, w.steps - k0);
      float2 acc[TN / 2];
#pragma unroll
      for (uint32_t j = 0; j < TN / 2; ++j) acc[j] = make_float2(0.f, 0.f);
#pragma unroll 1
      for (uint32_t k = 0; k < count; ++k, ++i) {
        if constexpr (F16) {
#pragma unroll
          for (uint32_t sub = 0; sub < 2; ++sub, ++n) {
            sync_set(set);  // the sums of the pass before have been read
            if (issuer) {
              if (sub == 0)
                issue_f16(i, 1);
              else if (i + 1 < end)
                issue_f16(i + 1, 0);
            }
            ok = __all_sync(0xffffffffu, ok && mbar_wait(&d_full[set * 2 + sub], (n >> 1) & 1, abort_flag, 750 + set));
            if (ok) {
              tc_fence_after();
#pragma unroll
              for (uint32_t c = 0; c < TN / 16; ++c) {
                uint32_t z0[16], z1[16];
                tmem_ld16(tmem + set * 128 + ((quad * 32) << 16) + sub * 64 + c * 16, z0);
                tmem_ld16(tmem + set * 128 + ((quad * 32) << 16) + sub * 64 + TN + c * 16, z1);
                tmem_ld_wait();
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                  acc[c * 8 + j].x += __uint_as_float(z0[2 * j]) + __uint_as_float(z1[2 * j]);
                  acc[c * 8 + j].y += __uint_as_float(z0[2 * j + 1]) + __uint_as_float(z1[2 * j + 1]);
                }
              }
              tc_fence_before();
            }
          }
          continue;
        }
        dw = dw_next;
#pragma unroll
        for (uint32_t sub = 0; sub < SUBS; ++sub, ++n) {
          if (ok) {
            tmem_st32(a_col, v);
            if (SUB_BLOCKS == 4) {
              unpack(i, 1);
              tmem_st32(a_col + 32, v);
            }
            tmem_st_wait();
            tc_fence_before();
          }
          if (!after) {  // bounded waits on what the predecessor holds up start after its end
            pdl_wait();
            after = true;
          }
          sync_set(set);
          if (issuer) {
            if (sub == 0) ok = __all_sync(0xffffffffu, ok && mbar_wait(&act_full[as], aph, abort_flag, 720 + as));
            if (leader && ok) {
              tc_fence_after();
#pragma unroll
              for (uint32_t b = 0; b < SUB_BLOCKS; ++b) {
                const uint32_t blk = h * 4 + sub * SUB_BLOCKS + b;
                const uint32_t hi = act_lo + ((as * P::ACT_BYTES + (blk >> 1) * SLAB + (blk & 1) * 64) >> 4), lo = hi + ((4 * SLAB) >> 4);
                const uint32_t a = tmem + set * 64 + b * 16, d = tmem + BT_D_COL + set * 64 + b * TN;
                umma_f16_ts(d, a, lo, SMEM_DESC_HI_SW128, idesc, 0u);
                umma_f16_ts(d, a + 8, lo + 2, SMEM_DESC_HI_SW128, idesc, 1u);
                umma_f16_ts(d, a, hi, SMEM_DESC_HI_SW128, idesc, 1u);
                umma_f16_ts(d, a + 8, hi + 2, SMEM_DESC_HI_SW128, idesc, 1u);
              }
              umma_commit(&d_full[set]);
              if (sub == SUBS - 1) umma_commit(&act_empty[as]);
            }
            __syncwarp();
          }
          // the next pass's first two blocks are unpacked while the tensor core works on this one
          if (sub + 1 < SUBS) {
            if (ok) unpack(i, 1);
          } else if (i + 1 < end) {
            open_unit(i + 1);
            if (ok) unpack(i + 1, 0);
          }
          ok = __all_sync(0xffffffffu, ok && mbar_wait(&d_full[set], n & 1, abort_flag, 750 + set));
          if (ok) {
            tc_fence_after();
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) {  // 16 columns of sums
              uint32_t z[16];
              tmem_ld16(d_col + c * 16, z);
              tmem_ld_wait();
              const uint32_t blk = sub * SUB_BLOCKS + c * 16 / TN, w2 = blk & 2 ? dw.y : dw.x, j0 = TN == 16 ? 0 : (c & 1) * 8;
              const float ds = __half2float(__ushort_as_half((unsigned short)(blk & 1 ? w2 >> 16 : w2 & 0xFFFFu)));
#pragma unroll
              for (uint32_t j = 0; j < 8; ++j)
                acc[j0 + j] = ffma2(make_float2(__uint_as_float(z[2 * j]), __uint_as_float(z[2 * j + 1])), make_float2(ds, ds), acc[j0 + j]);
            }
            tc_fence_before();
          }
        }
        // The unit is given back where its last value has been used (the scales), not behind its last load: see gemm_ts.cu.
        __syncwarp();
        if (lane == 0) mbar_arrive(&raw_empty[unit_of(i) % RAW]);
        if (++as == ACT) {
          as = 0;
          aph ^= 1;
        }
      }
      // ---- the run ends, or the row tile: the two halves of K meet, 16 activation rows at a time, then the CTAs that share the tile
      if (first) {
        asm volatile("bar.sync 2, 544;" ::: "memory");  // with warp 1: the factors are there
        first = false;
      }
      const bool whole = count == w.steps;
      float *mine = buf + t * 16 * 128 + row;
      float *part = w.part + ((size_t)(cta * 2 + (k0 == 0 ? 1 : 0)) * 2 + t) * TN * 128 + row;
#pragma unroll
      for (uint32_t g = 0; g < TN / 16; ++g) {
        if (h == 1) {
#pragma unroll
          for (uint32_t j = 0; j < 8; ++j) {
            mine[(2 * j) * 128] = acc[g * 8 + j].x;
            mine[(2 * j + 1) * 128] = acc[g * 8 + j].y;
          }
        }
        sync_workers();
        if (h == 0) {
          float *dst = whole ? mine : part + g * 16 * 128;
#pragma unroll
          for (uint32_t j = 0; j < 8; ++j) {
            const float a = acc[g * 8 + j].x + mine[(2 * j) * 128], b = acc[g * 8 + j].y + mine[(2 * j + 1) * 128];
            dst[(2 * j) * 128] = a;
            dst[(2 * j + 1) * 128] = b;
          }
          if (!whole && g + 1 == TN / 16) __threadfence();
        }
        sync_workers();
        if (whole) {
          finish_pair<EPI, TN>(w, pair, g * 16, buf, factor, tid);
          sync_workers();  // read before the buffer is written again
        }
      }
      if (!whole) {
        uint32_t c0 = blockIdx.y * gridDim.x, c1 = c0 + gridDim.x - 1;  // the CTAs that share the pair: a row of the grid, or out of the only one
        if (w.row == 0) c0 = run_of(w, pair * w.steps), c1 = run_of(w, (pair + 1) * w.steps - 1);
        if (tid == 0) *last_flag = atomicAdd(w.tickets + c0, 1u) == c1 - c0;
        sync_workers();
        if (*last_flag) {
          __threadfence();
          constexpr uint32_t MINE = TN / 2;  // both halves' threads: eight of every sixteen activation rows
          float sum[MINE];
#pragma unroll
          for (uint32_t j = 0; j < MINE; ++j) sum[j] = 0.f;
#pragma unroll(64 / MINE)
          for (uint32_t c = c0; c <= c1; ++c) {
            const float *src = w.part + ((size_t)(c * 2 + (c == c0 ? 1 : 0)) * 2 + t) * TN * 128 + h * 8 * 128 + row;
#pragma unroll
            for (uint32_t j = 0; j < MINE; ++j) sum[j] += __ldcg(src + (j / 8 * 16 + j % 8) * 128);
          }
#pragma unroll
          for (uint32_t g = 0; g < TN / 16; ++g) {
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) mine[(h * 8 + j) * 128] = sum[g * 8 + j];
            sync_workers();
            finish_pair<EPI, TN>(w, pair, g * 16, buf, factor, tid);
            sync_workers();
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncwarp();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) atomicCAS(w.error, 0, *abort_flag);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, BT_TMEM);
  }
}

// ---- the activations: fp16 pairs in the layout that the products read, and each row's factor ---------------------------------
// Per step of 256 K: four slabs of 64 K of the hi values, four of the lo values; a slab is [TN rows][128 bytes] under the 128-byte swizzle.
// Inside a block of Q4_0 the columns stand in the order in which a payload word's nibbles come out; zeros past K and past M.  One CTA per row,
// which keeps its share of up to IMG_HELD pieces of 8 columns in registers between the row's maximum and the conversion.
constexpr int IMG_THREADS = 1024, IMG_HELD = 4;

template <int FMT>
__device__ __forceinline__ void load_piece(const float *blk, uint32_t i, float (&v)[8]) {  // 8 columns of a block, as they stand in the image
  const float4 a = *reinterpret_cast<const float4 *>(blk + (FMT == GRETA_FMT_Q4_0 ? 4 * i : 8 * i));
  const float4 b = *reinterpret_cast<const float4 *>(blk + (FMT == GRETA_FMT_Q4_0 ? 16 + 4 * i : 8 * i + 4));
  if (FMT == GRETA_FMT_Q4_0) {
    v[0] = a.x, v[1] = a.z, v[2] = a.y, v[3] = a.w, v[4] = b.x, v[5] = b.z, v[6] = b.y, v[7] = b.w;
  } else {
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  }
}

template <int FMT>
__global__ void __launch_bounds__(IMG_THREADS) prep_image_kernel(const float *x, const float *__restrict__ gamma, float eps, uint32_t M, uint32_t K, uint32_t steps,
                                                                 float *rowmul, uint32_t *tickets, uint8_t *image) {
  __shared__ float red_max[IMG_THREADS / 32], red_ss[IMG_THREADS / 32];
  pdl_launch_dependents();
  const uint32_t m = blockIdx.x, TN = gridDim.x, pieces = steps * BT_STEP_BLOCKS * 4, live_pieces = m < M ? K / 8 : 0u;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float *xrow = x + (size_t)m * K;
  float held[IMG_HELD][8], amax = 0.f, ss = 0.f;
  pdl_wait();  // x comes from the previous kernel; the previous product has finished with the workspace
  auto take = [&](uint32_t u, float (&v)[8]) {  // piece u under the norm's weights, and its part of the sum of squares
    float g[8];
    load_piece<FMT>(xrow + (size_t)(u >> 2) * 32, u & 3, v);
    if (gamma) load_piece<FMT>(gamma + (size_t)(u >> 2) * 32, u & 3, g);
    float q = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      q = fmaf(v[j], v[j], q);
      if (gamma) v[j] *= g[j];
    }
    return q;
  };
  auto peak = [&](const float (&v)[8]) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      amax = fmaxf(amax, fabsf(v[j]));
      if (v[j] != v[j]) amax = INFINITY;
    }
  };
#pragma unroll
  for (int i = 0; i < IMG_HELD; ++i) {
    const uint32_t u = tid + i * IMG_THREADS;
    if (u < live_pieces) {
      ss += take(u, held[i]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) held[i][j] = 0.f;
    }
  }
#pragma unroll
  for (int i = 0; i < IMG_HELD; ++i) peak(held[i]);
  for (uint32_t u = tid + IMG_HELD * IMG_THREADS; u < live_pieces; u += IMG_THREADS) {
    float v[8];
    ss += take(u, v);
    peak(v);
  }
  if (m == 0 && tid < (int)BT_MAX_CTAS) tickets[tid] = 0;
  amax = warp_max(amax);
  ss = warp_sum(ss);
  if (lane == 0) {
    red_max[warp] = amax;
    red_ss[warp] = ss;
  }
  __syncthreads();
  amax = warp_max(red_max[lane]);
  ss = warp_sum(red_ss[lane]);
  float s = 1.f, is = 1.f;
  if (amax > 0.f && amax < INFINITY) {  // amax in [2^E, 2^(E+1)): scale by 2^(14-E)
    const int E = (int)(__float_as_uint(amax) >> 23) - 127;
    const int e = max(-100, min(100, 14 - E));
    s = __uint_as_float((uint32_t)(127 + e) << 23);
    is = __uint_as_float((uint32_t)(127 - e) << 23);
  }
  if (tid == 0) rowmul[m] = m < M ? is * (gamma ? rsqrtf(ss / (float)K + eps) : 1.f) : 0.f;
  auto put = [&](uint32_t u, const float (&v)[8]) {
    const uint32_t blk = u >> 2, step = blk / BT_STEP_BLOCKS, slab = (blk % BT_STEP_BLOCKS) >> 1, chunk = (blk & 1) * 4 + (u & 3);
    __half2 hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = v[2 * j] * s, b = v[2 * j + 1] * s;
      hi[j] = __floats2half2_rn(a, b);
      const float2 f = __half22float2(hi[j]);
      lo[j] = __floats2half2_rn(a - f.x, b - f.y);
    }
    uint8_t *dst = image + (size_t)step * TN * (BT_STEP * 4) + slab * TN * 128 + m * 128 + ((chunk ^ (m & 7)) << 4);
    *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(hi);
    *reinterpret_cast<uint4 *>(dst + 4 * TN * 128) = *reinterpret_cast<const uint4 *>(lo);
  };
#pragma unroll
  for (int i = 0; i < IMG_HELD; ++i) {
    const uint32_t u = tid + i * IMG_THREADS;
    if (u < pieces) put(u, held[i]);
  }
  for (uint32_t u = tid + IMG_HELD * IMG_THREADS; u < pieces; u += IMG_THREADS) {
    float v[8] = {};
    if (u < live_pieces) take(u, v);
    put(u, v);
  }
}

template <int FMT, int EPI, int TN>
int launch_tc(cudaStream_t stream, const BtArgs &a, dim3 grid) {
  using P = BtPlan<FMT, TN>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    GRETA_CUDA_TRY(cudaFuncSetAttribute(gemv_tc_kernel<FMT, EPI, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BT_SMEM_MAX));
    attr_set[dev] = true;
  }
  const GemvParams &p = a.p;
  GRETA_CUDA_TRY(launch_pdl(prep_image_kernel<FMT>, dim3(TN), dim3(IMG_THREADS), 0, stream, static_cast<const float *>(p.x), p.gamma, p.eps, p.M, p.K, a.steps,
                            const_cast<float *>(a.rowmul), a.tickets, const_cast<uint8_t *>(a.image)));
  if (int rc = launched("prep_image_kernel")) return rc;
  GRETA_CUDA_TRY(launch_pdl(gemv_tc_kernel<FMT, EPI, TN>, grid, dim3(BT_THREADS), P::SMEM, stream, a));
  return launched("gemv_tc_kernel");
}
template <int FMT, int EPI>
int launch_rows(cudaStream_t stream, const BtArgs &a, dim3 grid) {
  return a.p.M <= 16 ? launch_tc<FMT, EPI, 16>(stream, a, grid) : launch_tc<FMT, EPI, 32>(stream, a, grid);
}
template <int FMT>
int launch_epi(cudaStream_t stream, int epi, const BtArgs &a, dim3 grid) {
  switch (epi) {
    case EPI_PLAIN: return launch_rows<FMT, EPI_PLAIN>(stream, a, grid);
    case EPI_RESIDUAL: return launch_rows<FMT, EPI_RESIDUAL>(stream, a, grid);
    case EPI_SWIGLU: return launch_rows<FMT, EPI_SWIGLU>(stream, a, grid);
    default: return launch_rows<FMT, EPI_QKV>(stream, a, grid);
  }
}

}  // namespace

namespace greta {
int gemm_ts_error_word(int **word);  // gemm_ts.cu

size_t gemv_tc_workspace_bytes(uint32_t M, uint32_t K) {
  const size_t tn = M <= 16 ? 16 : 32, steps = (K + BT_STEP - 1) / BT_STEP;
  return BT_HEADER + steps * tn * (BT_STEP * 4) + (size_t)BT_MAX_CTAS * 2 * 2 * tn * 128 * 4;
}

bool gemv_tc_route(int fmt, uint32_t M, uint64_t rows, uint32_t K) {
  if (fmt != GRETA_FMT_Q4_0 && fmt != GRETA_FMT_Q8_0 && fmt != GRETA_FMT_F16) return false;
  const bool few = M <= 16 && (fmt == GRETA_FMT_F16 || (fmt == GRETA_FMT_Q4_0 && K > 512));
  const uint64_t least = M <= 8 && fmt != GRETA_FMT_Q8_0 ? BT_MIN_WEIGHTS_FEW_ROWS
                                                         : (K < BT_SHORT_K ? (few ? BT_MIN_WEIGHTS_SHORT_FEW : BT_MIN_WEIGHTS_SHORT) : BT_MIN_WEIGHTS);
  return M >= 1 && M <= 32 && K >= BT_STEP && rows * K >= least && rows * K < (1ull << 40) && encode_tiled();
}

bool gemv_tc_takes(int fmt, int epi, const void *params) {
  const GemvParams &p = *static_cast<const GemvParams *>(params);
  const uint64_t rows = epi == EPI_SWIGLU ? (uint64_t)2 * p.N : (epi == EPI_QKV ? (uint64_t)(p.H + 2 * p.Hkv) * p.Dh : p.N);
  return gemv_tc_route(fmt, p.M, rows, p.K) && (!p.gamma || aligned16(p.gamma));
}

// Into how many units of K steps a pair of row tiles is cut, every CTA taking an equal run of all units, and the CTAs.  Single steps in equal runs (parts = steps)
// balance best, but a run that ends inside a pair leaves parts of two pairs to be summed through the workspace, each as long as three steps, and every part of a
// pair costs its last CTA another read.  So also tried: every unit a CTA of its own, and whole pairs.  mma.sync form / equal runs only / as here, in a CUDA graph, us: 9 rows q4_0 23360 x 512 10.1 / 14.4 / 7.8, 5952 x 2048
// 13.4 / 13.2 / 10.9, 1600 x 8192 16.4 / 16.2 / 13.3, 8192 x 8192 31.9 / 23.2 / 20.5; 8 rows q8_0 18624 x 640 11.6 / 13.7 / 9.4; 9 rows fp16 15552 x 768
// 11.3 / 15.9 / 11.0; 32 rows q4_0 16384 x 4096 46.3 / 29.6 / 26.8.  Times in 10 ns, fitted to products of 16 to 3600 steps; a step of fp16 weights waits for its
// 128 KB (38 bytes/ns and SM), and in long runs of those the first meeting is hidden.
static uint32_t plan_shares(int fmt, uint32_t M, uint32_t steps, uint32_t pairs, uint32_t *ctas) {
  const uint32_t most = std::min((uint32_t)sm_count(), BT_MAX_CTAS), all = steps * pairs;
  const bool wide = M > 16, f16 = fmt == GRETA_FMT_F16;
  const uint64_t step = f16 ? 330 : (fmt == GRETA_FMT_Q4_0 ? 160 : 205) + (wide ? 100 : 0);
  const uint64_t meet = wide ? 660 : (f16 ? 650 : 430), part = wide ? 38 : 24, whole = wide ? 420 : (f16 ? 350 : 250);
  *ctas = most;
  // Long runs stay equal: there fewer CTAs cost the kernels around the product more than the meetings cost it (three parts of the pairs of 10240 x 8192, 16 rows: the
  // product 27.6 -> 26.8, the layer it stands in 353 -> 367; up to 8 steps a CTA, layers of widths 1536 to 8192: 1-6 % faster).
  if (all > 8 * most) return steps;
  const uint32_t deal = (pairs + most - 1) / most;  // pairs of a CTA that takes whole ones
  uint32_t parts = 1;
  *ctas = std::min(most, pairs);
  uint64_t best = (step * steps + whole) * deal;
  for (uint32_t m = 2; m <= steps && m * pairs <= most; ++m) {
    const uint64_t time = step * ((steps + m - 1) / m) + meet + part * m;
    if (time < best) best = time, parts = m, *ctas = m * pairs;
  }
  if (all > most) {
    const uint32_t run = (all + most - 1) / most, meetings = f16 && !wide && 2 * all > 5 * most ? 1 : 2;
    const uint64_t time = step * all / most + meetings * (meet + part * std::min(steps, (steps + run - 1) / run + 1)) + (run > 2 * steps ? whole * (run / steps - 1) : 0);
    if (time < best) parts = steps, *ctas = most;
  }
  return parts;
}

int gemv_tc(cudaStream_t stream, int fmt, int epi, const void *params, void *workspace) {
  const GemvParams &p = *static_cast<const GemvParams *>(params);
  BtArgs w{};
  w.p = p;
  w.steps = (p.K + BT_STEP - 1) / BT_STEP;
  const uint32_t nb = p.K / 32, tile_rows = epi == EPI_SWIGLU ? 64 : 128, planes = epi == EPI_QKV ? 3 : (epi == EPI_SWIGLU ? 2 : 1);
  const size_t row_bytes = (size_t)nb * (fmt == GRETA_FMT_Q4_0 ? 16 : (fmt == GRETA_FMT_Q8_0 ? 32 : 64));
  for (uint32_t i = 0; i < planes; ++i) {
    w.n[i] = epi == EPI_QKV ? (i == 0 ? p.H : p.Hkv) * p.Dh : p.N;
    if (i == 0 || epi == EPI_QKV) w.tiles += (w.n[i] + tile_rows - 1) / tile_rows;
    w.tile_end[i] = w.tiles;
    const cuuint64_t qd[2] = {row_bytes, w.n[i]}, qs[1] = {row_bytes}, dd[2] = {nb, w.n[i]}, ds[1] = {(cuuint64_t)d_row_stride(nb) * 2};
    const cuuint32_t qbox[2] = {128, tile_rows}, dbox[2] = {8, tile_rows}, one[2] = {1, 1};
    CUresult r = encode_tiled()(&w.qs[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t *>(p.w[i].qs), qd, qs, qbox, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS && fmt != GRETA_FMT_F16)
      r = encode_tiled()(&w.d[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(p.w[i].d), dd, ds, dbox, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
      set_error("batched gemv: cuTensorMapEncodeTiled failed with code %d", (int)r);
      return GRETA_ERR_INVALID_ARGS;
    }
  }
  const size_t tn = p.M <= 16 ? 16 : 32;
  uint8_t *ws = static_cast<uint8_t *>(workspace);
  w.rowmul = reinterpret_cast<const float *>(ws);
  w.tickets = reinterpret_cast<uint32_t *>(ws + 256);
  w.image = ws + BT_HEADER;
  w.part = reinterpret_cast<float *>(ws + BT_HEADER + (size_t)w.steps * tn * (BT_STEP * 4));
  const uint32_t pairs = (w.tiles + 1) / 2;
  uint32_t ctas;
  const uint32_t parts = plan_shares(fmt, p.M, w.steps, pairs, &ctas);
  dim3 grid(ctas);
  if (parts > 1 && parts * pairs == ctas) {  // a unit each: a row of the grid per pair
    grid = dim3(parts, pairs);
    w.row = w.steps, w.run = w.steps / parts, w.longer = w.steps % parts, w.unit = 1;
  } else {
    const uint32_t units = parts * pairs;
    w.row = 0, w.run = units / ctas, w.longer = units % ctas, w.unit = parts == 1 ? w.steps : 1;
  }
  if (int rc = gemm_ts_error_word(&w.error)) return rc;
  if (fmt == GRETA_FMT_F16) return launch_epi<GRETA_FMT_F16>(stream, epi, w, grid);
  return fmt == GRETA_FMT_Q4_0 ? launch_epi<GRETA_FMT_Q4_0>(stream, epi, w, grid) : launch_epi<GRETA_FMT_Q8_0>(stream, epi, w, grid);
}
}  // namespace greta
