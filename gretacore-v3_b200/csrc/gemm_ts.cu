// Prefill products of one layer over block-quantised weights, the weights going to the tensor cores through tensor memory:
//   out_i[M x N_i] = half(A[M x K]) * half(dequant(W_i[N_i x K]))^T, fp32 accumulation, for up to three W_i in one launch.
//
// The weight rows are the 128-row operand of tcgen05.mma and TN tokens its N dimension.  The weight operand is written to tensor
// memory by the threads that dequantise it, so it never passes through shared memory: with a weight tile in shared memory
// (gemm_tc.cu) a stage of 128 tokens x 64 K moves 74 KB through it (578 cycles against 380 of tensor-core time), and the per-thread
// copies of 16-byte weight pieces, 32 rows to an instruction, and the fence between the stores and the tensor core made that 950-1400
// cycles.  Here raw weights come by TMA, 256 (Q4_0) or 128 (Q8_0) elements of 128 rows at a time, and a stage of 128 K costs a thread
// its four blocks of one row: 4-8 shared loads, the half2 arithmetic and two tcgen05.st.
//
// Warp roles (768 threads, one persistent CTA per SM over tiles of 128 rows x TN tokens):
//   warp 0       TMA of the activations, two slabs of TN x 64 fp16 per stage, 128-byte swizzle;
//   warp 1       TMEM allocation, MMA issue (eight K = 16 per stage), commits;
//   warp 2       TMA of the raw weight units and their scales; starts before the kernel's predecessor has finished (weights do not
//                depend on it);
//   warps 4-19   dequantisation to exactly half((q - 8) * d): a set of four warps per weight slot in tensor memory, so up to four
//                dependent chains (load, arithmetic, wait, store, arrival) are under way at a time;
//   warps 20-23  epilogue out of TMEM, of the previous tile where two accumulators fit.
// A gate / up tile is 64 rows of either matrix: its accumulator has gate in lanes 0-63 and up in lanes 64-127 and the two meet through shared
// memory, so the tile costs what any other does (a tile of 128 rows of both needs two accumulators, which leaves half the weight slots: 115
// against 91 us at 512 tokens x 4096 x 2 x 11008).
// Measured alone with a cold L2 (median, launch and event overhead included; greta_cuda_gemm's kernel timed the same way behind the stroke), 512
// tokens, Q4_0: 3 x 4096 x 4096 52 / 120 us = 990 TFLOP/s, 4096 x 4096 29 / 43, 4096 x 11008 53 / 88, 2 x 11008 x 4096 with SwiGLU 92 / 114 without.
// 1531 tokens, Q8_0: 2 x 14336 x 4096 280 / 362 us = 1282 TFLOP/s (0.77 of the measured peak), 4096 x 14336 148 / 184.  What is left: the last
// tile's end (25 ns per token column) and waves that do not fill the SMs.
// Every wait is bounded: on a timeout the kernel raises a flag that all roles poll, drains, frees its tensor memory and returns;
// greta_cuda_gemm_status() reports it.
#include "gemm_dequant.cuh"
#include "greta_common.cuh"
#include "tc_device.cuh"

using namespace greta;

namespace {

constexpr uint32_t TS_RAW_UNITS = 4, TS_RAW_PAYLOAD = 128 * 128, TS_RAW_BYTES = TS_RAW_PAYLOAD + 128 * 16;
constexpr uint32_t TS_DEQ_WARP0 = 4, TS_EPI_WARP0 = TS_DEQ_WARP0 + 16, TS_THREADS = 32 * (TS_EPI_WARP0 + 4);
constexpr uint32_t TS_K = 2 * BK, TS_W_COLS = TS_K / 2;  // K elements of a stage; TMEM columns of its weights
constexpr uint32_t TS_ACT_MAX = 8, TS_W_MAX = 4, TS_TMEM = 512;
constexpr uint32_t TS_BARS = 2 * TS_RAW_UNITS + 2 * TS_ACT_MAX + 2 * TS_W_MAX + 4;
constexpr uint32_t TS_SWAP_LD = 33, TS_SWAP_BYTES = 64 * TS_SWAP_LD * 4;  // [64 rows][32 columns, padded]
constexpr size_t TS_SMEM_MAX = 232448, TS_SMEM_FIXED = (size_t)TS_RAW_UNITS * TS_RAW_BYTES + TS_SWAP_BYTES + 1024 + TS_BARS * 8 + 16;

struct TsArgs {
  CUtensorMap act, qs[3], d[3];
  float *out[3];
  uint32_t n[3], tile_end[3];  // rows of a segment; row tiles up to and with it
  uint32_t M, K, tiles, tok_tiles, tn, act_stages, w_slots, accs, idesc;
};

// The four epilogue warps.
__device__ __forceinline__ void sync_128() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
__device__ __forceinline__ bool all_of_128(bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)v)
      : "memory");
  return r != 0;
}

template <int FMT, int MODE>
__global__ void __launch_bounds__(TS_THREADS, 1) gemm_ts_kernel(const __grid_constant__ TsArgs w) {
  constexpr bool PAIR = MODE == GRETA_GEMM_SWIGLU_F16;
  constexpr uint32_t TILE_ROWS = PAIR ? TILE_N / 2 : TILE_N;  // rows of each matrix in a tile
  constexpr bool Q4 = FMT == GRETA_FMT_Q4_0;
  constexpr uint32_t SPU = Q4 ? 2 : 1;  // stages per raw unit (128 payload bytes of a row)
  extern __shared__ uint8_t smem_raw[];
  uint8_t *act = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t TN = w.tn, AS = w.act_stages, TS = w.w_slots, act_bytes = TN * (TS_K * 2);
  uint8_t *raw = act + (size_t)AS * act_bytes;
  float *swap = reinterpret_cast<float *>(raw + TS_RAW_UNITS * TS_RAW_BYTES);
  uint64_t *raw_full = reinterpret_cast<uint64_t *>(reinterpret_cast<uint8_t *>(swap) + TS_SWAP_BYTES), *raw_empty = raw_full + TS_RAW_UNITS;
  uint64_t *act_full = raw_empty + TS_RAW_UNITS, *act_empty = act_full + TS_ACT_MAX, *w_full = act_empty + TS_ACT_MAX, *w_empty = w_full + TS_W_MAX;
  uint64_t *acc_full = w_empty + TS_W_MAX, *acc_empty = acc_full + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t units = (w.K + TS_K * SPU - 1) / (TS_K * SPU), KT = units * SPU;  // raw units and stages of a tile; zeros past K

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < TS_RAW_UNITS; ++s) {
      mbar_init(&raw_full[s], 1);
      mbar_init(&raw_empty[s], SPU * 4);  // four warps read a stage
    }
    for (uint32_t s = 0; s < AS; ++s) {
      mbar_init(&act_full[s], 1);
      mbar_init(&act_empty[s], 1);
    }
    for (uint32_t s = 0; s < TS; ++s) {
      mbar_init(&w_full[s], 4);
      mbar_init(&w_empty[s], 1);
    }
    for (uint32_t b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&w.act) : "memory");
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TS_TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, tmem_w = tmem + TS_TMEM - TS * TS_W_COLS;
  pdl_launch_dependents();

  const bool leader = elect_one();
  if (warp == 0) {
    pdl_wait();
    uint32_t s = 0, ph = 1, issued = 0;
    bool ok = true;
    for (uint32_t t = blockIdx.x; t < w.tiles; t += gridDim.x) {
      const int m0 = (int)((t % w.tok_tiles) * TN);
      for (uint32_t kt = 0; kt < KT; ++kt) {
        uint8_t *dst = act + (size_t)s * act_bytes;
        if (ok) ok = mbar_wait(&act_empty[s], ph, abort_flag, 100 + s);
        __syncwarp();
        if (leader && ok) {
          mbar_arrive_expect_tx(&act_full[s], act_bytes);
          tma_load_2d(dst, &w.act, (int)(kt * TS_K), m0, &act_full[s]);
          tma_load_2d(dst + act_bytes / 2, &w.act, (int)(kt * TS_K + BK), m0, &act_full[s]);
          ++issued;
        }
        if (++s == AS) {
          s = 0;
          ph ^= 1;
        }
      }
    }
    if (leader && *abort_flag) drain_copies(act_full, issued, AS);
  } else if (warp == 2) {
    uint32_t u = 0, issued = 0;
    bool ok = true;
    for (uint32_t t = blockIdx.x; t < w.tiles; t += gridDim.x) {
      const uint32_t rt = t / w.tok_tiles, seg = PAIR ? 0u : (rt < w.tile_end[0] ? 0u : (rt < w.tile_end[1] ? 1u : 2u));
      const int n0 = (int)((rt - (seg ? w.tile_end[seg - 1] : 0)) * TILE_ROWS);
      for (uint32_t kq = 0; kq < units; ++kq, ++u) {
        const uint32_t slot = u % TS_RAW_UNITS;
        if (u == TS_RAW_UNITS) pdl_wait();  // from here on the bounded waits depend on the predecessor's end
        uint8_t *dst = raw + slot * TS_RAW_BYTES;
        const int kd = (int)((Q4 ? kq : kq / 2) * 8);  // the scales of 256 elements
        if (ok) ok = mbar_wait(&raw_empty[slot], ((u / TS_RAW_UNITS) & 1) ^ 1, abort_flag, 200 + slot);
        __syncwarp();
        if (leader && ok) {
          mbar_arrive_expect_tx(&raw_full[slot], TS_RAW_BYTES);
          tma_load_2d(dst, &w.qs[seg], (int)(kq * 128), n0, &raw_full[slot]);
          tma_load_2d(dst + TS_RAW_PAYLOAD, &w.d[seg], kd, n0, &raw_full[slot]);
          if (PAIR) {
            tma_load_2d(dst + TILE_ROWS * 128, &w.qs[1], (int)(kq * 128), n0, &raw_full[slot]);
            tma_load_2d(dst + TS_RAW_PAYLOAD + TILE_ROWS * 16, &w.d[1], kd, n0, &raw_full[slot]);
          }
          ++issued;
        }
      }
    }
    if (leader && *abort_flag) drain_copies(raw_full, issued, TS_RAW_UNITS);
  } else if (warp == 1) {
    const uint32_t a_lo0 = smem_desc_lo(smem_u32(act)), lg = TS == 4 ? 2 : 1;
    uint32_t s = 0, ph = 0, g = 0, it = 0;
    bool ok = true;
    pdl_wait();
    for (uint32_t t = blockIdx.x; t < w.tiles; t += gridDim.x, ++it) {
      const uint32_t b = w.accs == 2 ? (it & 1) : 0;
      if (ok) ok = mbar_wait(&acc_empty[b], ((w.accs == 2 ? it >> 1 : it) & 1) ^ 1, abort_flag, 300 + b);
      __syncwarp();
      for (uint32_t kt = 0; kt < KT; ++kt, ++g) {
        const uint32_t a_lo = a_lo0 + s * (act_bytes >> 4), slot = g & (TS - 1), d = tmem + b * TN, a = tmem_w + slot * TS_W_COLS;
        if (ok) ok = mbar_wait(&act_full[s], ph, abort_flag, 310 + s) && mbar_wait(&w_full[slot], (g >> lg) & 1, abort_flag, 320 + slot);
        __syncwarp();
        if (leader && ok) {
          tc_fence_after();
#pragma unroll
          for (uint32_t k16 = 0; k16 < TS_K / 16; ++k16)
            umma_f16_ts(d, a + k16 * 8, a_lo + (k16 / 4) * (act_bytes >> 5) + (k16 % 4) * 2, SMEM_DESC_HI_SW128, w.idesc, (kt | k16) ? 1u : 0u);
          umma_commit(&w_empty[slot]);
          umma_commit(&act_empty[s]);
        }
        if (++s == AS) {
          s = 0;
          ph ^= 1;
        }
      }
      if (leader && ok) umma_commit(&acc_full[b]);
    }
  } else if (warp >= (int)TS_DEQ_WARP0 && warp < (int)TS_EPI_WARP0) {
    // The set of a stage is its weight slot, and with whole units in every tile a raw slot is always read by the same sets: whoever waits on
    // a barrier has seen every phase of it, which a parity needs.
    const uint32_t set = (uint32_t)(warp - TS_DEQ_WARP0) >> 2, quad = warp & 3, row = quad * 32 + lane, x7 = row & 7;
    const uint32_t lg = TS == 4 ? 2 : 1;
    uint32_t u = 0, it = 0;
    bool ok = set < TS, after = false;
    for (uint32_t t = blockIdx.x; t < w.tiles && ok; t += gridDim.x, ++it) {
      for (uint32_t kq = 0; kq < units && ok; ++kq, ++u) {
        const uint32_t slot = u % TS_RAW_UNITS;
        for (uint32_t sub = 0; sub < SPU; ++sub) {
          const uint32_t g = it * KT + kq * SPU + sub;
          if ((g & (TS - 1)) != set) continue;
          if (!after && (g >= TS || u >= TS_RAW_UNITS)) {  // bounded waits on what the predecessor holds up start after its end
            pdl_wait();
            after = true;
          }
          ok = mbar_wait(&raw_full[slot], (u / TS_RAW_UNITS) & 1, abort_flag, 400 + slot);
          const uint8_t *st = raw + slot * TS_RAW_BYTES, *pr = st + row * 128;
          const uint2 dw = *reinterpret_cast<const uint2 *>(st + TS_RAW_PAYLOAD + row * 16 + (Q4 ? sub : kq & 1) * 8);
          uint32_t v[32];  // 64 fp16 of the row, ascending K; past K the copies filled payload, scales and activations with zeros
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint4 q[Q4 ? 2 : 4];
#pragma unroll
            for (int c = 0; c < (Q4 ? 2 : 4); ++c) q[c] = *reinterpret_cast<const uint4 *>(pr + (((Q4 ? sub * 4 + half * 2 + c : half * 4 + c) ^ x7) << 4));
#pragma unroll
            for (int hb = 0; hb < 2; ++hb) {
              const uint32_t w2 = half ? dw.y : dw.x, dh = hb ? (w2 >> 16) : (w2 & 0xFFFFu), d2 = dh | (dh << 16);
              if (Q4) {
                const uint32_t p[4] = {q[hb].x, q[hb].y, q[hb].z, q[hb].w};
#pragma unroll
                for (int i4 = 0; i4 < 4; ++i4) {
                  uint32_t lo[2], hi[2];
                  dq4_word(p[i4], d2, lo, hi);
                  v[hb * 16 + i4 * 2] = lo[0];
                  v[hb * 16 + i4 * 2 + 1] = lo[1];
                  v[hb * 16 + 8 + i4 * 2] = hi[0];
                  v[hb * 16 + 8 + i4 * 2 + 1] = hi[1];
                }
              } else {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                  const uint4 qq = q[Q4 ? 0 : hb * 2 + c];
                  const uint32_t p[4] = {qq.x, qq.y, qq.z, qq.w};
#pragma unroll
                  for (int i4 = 0; i4 < 4; ++i4) {
                    uint32_t o[2];
                    dq8_word(p[i4], d2, o);
                    v[hb * 16 + c * 8 + i4 * 2] = o[0];
                    v[hb * 16 + c * 8 + i4 * 2 + 1] = o[1];
                  }
                }
              }
            }
            if (half == 0) {
              ok = __all_sync(0xffffffffu, ok && mbar_wait(&w_empty[set], ((g >> lg) & 1) ^ 1, abort_flag, 410 + set));  // both waits, by the whole warp
              if (!ok) break;
              tc_fence_after();
            }
            tmem_st32(tmem_w + set * TS_W_COLS + half * 32 + ((quad * 32) << 16), v);
          }
          if (!ok) break;
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          // The raw unit is given back here, where every loaded value has been used, and not behind its last load: a load under way is not ahead
          // of the arrival, nor of the copy that the arrival lets loose (seen: single weight rows of a SwiGLU tile multiplied with the unit
          // that followed, in most prompts of more than 1000 tokens).
          if (lane == 0) {
            mbar_arrive(&w_full[set]);
            mbar_arrive(&raw_empty[slot]);
          }
        }
      }
    }
  } else if (warp >= (int)TS_EPI_WARP0) {
    const uint32_t quad = warp & 3;
    uint32_t it = 0;
    pdl_wait();
    for (uint32_t t = blockIdx.x; t < w.tiles; t += gridDim.x, ++it) {
      const uint32_t b = w.accs == 2 ? (it & 1) : 0, rt = t / w.tok_tiles, m0 = (t % w.tok_tiles) * TN;
      const uint32_t seg = PAIR ? 0u : (rt < w.tile_end[0] ? 0u : (rt < w.tile_end[1] ? 1u : 2u));
      const uint32_t in_tile = PAIR ? (quad & 1) * 32 + lane : quad * 32 + lane;
      const uint32_t N = w.n[seg], row = (rt - (seg ? w.tile_end[seg - 1] : 0)) * TILE_ROWS + in_tile, cols = min(TN, w.M - m0);
      const uint32_t src = tmem + b * TN + ((quad * 32) << 16), par = (w.accs == 2 ? it >> 1 : it) & 1;
      if (PAIR) {
        if (!all_of_128(mbar_wait_warp(&acc_full[b], par, abort_flag, 500 + b))) break;  // all four warps leave together: they meet at barriers below
        tc_fence_after();
        // Of 32 columns the gate warps hand over the last 16 and finish the first 16, the up warps the other way round.
        const bool up = quad >= 2;
        __half *o = reinterpret_cast<__half *>(w.out[0]) + (size_t)m0 * N + row;
        float *sw = swap + in_tile * TS_SWAP_LD;
#pragma unroll 1
        for (uint32_t c = 0; c < cols; c += 32) {
          uint32_t keep[16], give[16];
          __syncwarp();
          tmem_ld16(src + c + (up ? 0 : 16), give);
          tmem_ld16(src + c + (up ? 16 : 0), keep);
          tmem_ld_wait();
#pragma unroll
          for (uint32_t j = 0; j < 16; ++j) sw[(up ? 0 : 16) + j] = __uint_as_float(give[j]);
          sync_128();
          const uint32_t c0 = c + (up ? 16 : 0);
#pragma unroll
          for (uint32_t j = 0; j < 16; ++j) {
            const float other = sw[(up ? 16 : 0) + j], own = __uint_as_float(keep[j]), z = up ? other : own, u = up ? own : other;
            if (row < N && c0 + j < cols) o[(size_t)(c0 + j) * N] = __float2half_rn((z / (1.0f + expf(-z))) * u);
          }
          sync_128();  // read before the next 32 columns are handed over
        }
      } else {
        float *o = w.out[seg] + (size_t)m0 * N + row;
        float old[16];
        auto fetch = [&](uint32_t c) {
#pragma unroll
          for (uint32_t j = 0; j < 16; ++j) old[j] = row < N && c + j < cols ? o[(size_t)(c + j) * N] : 0.f;
        };
        if (MODE == GRETA_GEMM_ADD) fetch(0);  // the residual of the next 16 columns is on its way while these are stored
        if (!mbar_wait_warp(&acc_full[b], par, abort_flag, 500 + b)) break;
        tc_fence_after();
#pragma unroll 1
        for (uint32_t c = 0; c < cols; c += MODE == GRETA_GEMM_ADD ? 16 : 32) {
          __syncwarp();
          if (MODE == GRETA_GEMM_ADD) {
            uint32_t v[16];
            tmem_ld16(src + c, v);
            tmem_ld_wait();
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j) v[j] = __float_as_uint(old[j] + __uint_as_float(v[j]));
            fetch(c + 16);
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j)
              if (row < N && c + j < cols) o[(size_t)(c + j) * N] = __uint_as_float(v[j]);
          } else {
            uint32_t v[32];
            tmem_ld32(src + c, v);
            tmem_ld_wait();
#pragma unroll
            for (uint32_t j = 0; j < 32; ++j)
              if (row < N && c + j < cols) o[(size_t)(c + j) * N] = __uint_as_float(v[j]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[b]);
    }
  }
  tc_fence_before();
  __syncwarp();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TS_TMEM);
  }
}

uint32_t stages_of(uint32_t tn) { return (uint32_t)std::min<size_t>(TS_ACT_MAX, (TS_SMEM_MAX - TS_SMEM_FIXED) / ((size_t)tn * TS_K * 2)); }

// Tokens per tile: the width whose waves over the SMs take least.  A stage of 128 K takes 0.38 us at 64 tokens (the dequantising warps set
// the pace), 0.46 at 128, 0.53 at 192 (the tensor cores' measured rate), 0.80 at 256 (one accumulator, two activation stages);
// a tile's end costs about 1 us where the next tile's products cover it and 25 ns per column where they cannot.
uint32_t pick_tokens(uint32_t M, uint32_t row_tiles, uint32_t KT, uint32_t sms) {
  uint32_t best = 32;
  double least = 1e300;
  for (uint32_t tn = 32; tn <= 256; tn += 32) {
    const uint64_t tiles = (uint64_t)row_tiles * ((M + tn - 1) / tn), waves = (tiles + sms - 1) / sms;
    const double stage = tn <= 192 ? 0.31 + 0.0012 * tn : 0.0031 * tn, end = 0.025 * tn, covered = tn <= 192 ? 1.0 : end;
    const double cost = (double)waves * KT * stage + (double)(waves - 1) * covered + end;
    if (cost < least) {
      least = cost;
      best = tn;
    }
    if (tn >= M) break;
  }
  return best;
}

// Row tiles of `rows` weight rows, and the launch that they and M tokens make.
uint32_t row_tiles_of(uint32_t rows, int mode) {
  const uint32_t tile_rows = mode == GRETA_GEMM_SWIGLU_F16 ? TILE_N / 2 : TILE_N;
  return (rows + tile_rows - 1) / tile_rows;
}
struct TsPlan {
  uint32_t tn, accs, w_slots, act_stages, tok_tiles;
};
TsPlan plan_ts(uint32_t M, uint32_t K, uint32_t row_tiles) {
  TsPlan p;
  p.tn = pick_tokens(M, row_tiles, (K + 2 * TS_K - 1) / (2 * TS_K) * 2, (uint32_t)sm_count());
  p.accs = p.tn <= 192 ? 2 : 1;  // two accumulators and at least two weight slots
  p.w_slots = TS_TMEM - p.accs * p.tn >= 4 * TS_W_COLS ? 4 : 2;
  p.act_stages = stages_of(p.tn);
  p.tok_tiles = (M + p.tn - 1) / p.tn;
  return p;
}

template <int FMT, int MODE>
int launch_ts(cudaStream_t stream, const TsArgs &a, uint32_t sms, size_t smem) {
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    GRETA_CUDA_TRY(cudaFuncSetAttribute(gemm_ts_kernel<FMT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TS_SMEM_MAX));
    attr_set[dev] = true;
  }
  GRETA_CUDA_TRY(launch_pdl(gemm_ts_kernel<FMT, MODE>, dim3(std::min(a.tiles, sms)), dim3(TS_THREADS), smem, stream, a));
  return launched("gemm_ts_kernel");
}

}  // namespace

namespace greta {
int gemm_ts_status(int *code) {
  GRETA_CUDA_TRY(cudaMemcpyFromSymbol(code, g_gemm_error, sizeof(int)));
  return GRETA_OK;
}
int gemm_ts_error_word(int **word) {  // the current device's; the prompt's attention reports there too
  GRETA_CUDA_TRY(cudaGetSymbolAddress(reinterpret_cast<void **>(word), g_gemm_error));
  return GRETA_OK;
}
int gemm_ts_set_status(int code) {
  GRETA_CUDA_TRY(cudaMemcpyToSymbol(g_gemm_error, &code, sizeof(int)));
  return GRETA_OK;
}
}  // namespace greta

extern "C" int greta_cuda_gemm_segments_status(greta_stream_t stream, int *code) {
  GRETA_REQUIRE(code, "gemm_segments_status: null out pointer");
  GRETA_CUDA_TRY(cudaMemcpyFromSymbolAsync(code, g_gemm_error, sizeof(int), 0, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  return GRETA_OK;
}

extern "C" int greta_cuda_gemm_segments_route(uint32_t M, uint32_t K, const uint32_t *n, uint32_t n_segs, int mode, uint32_t *tile_tokens,
                                              uint32_t *accumulators, uint32_t *weight_slots, uint32_t *tiles) {
  GRETA_REQUIRE(n && n_segs >= 1 && n_segs <= 3 && tile_tokens && accumulators && weight_slots && tiles, "gemm_segments_route: bad argument");
  GRETA_REQUIRE(M && K && K % 32 == 0 && mode >= GRETA_GEMM_STORE && mode <= GRETA_GEMM_SWIGLU_F16, "gemm_segments_route: M=%u K=%u mode %d", M, K, mode);
  uint32_t row_tiles = 0;
  for (uint32_t i = 0; i < (mode == GRETA_GEMM_SWIGLU_F16 ? 1 : n_segs); ++i) row_tiles += row_tiles_of(n[i], mode);
  const TsPlan p = plan_ts(M, K, row_tiles);
  *tile_tokens = p.tn;
  *accumulators = p.accs;
  *weight_slots = p.w_slots;
  *tiles = row_tiles * p.tok_tiles;
  return GRETA_OK;
}

extern "C" int greta_cuda_gemm_segments(greta_stream_t stream, int fmt, const void *a_f16, uint32_t M, uint32_t K, const greta_gemm_segment *segs,
                                        uint32_t n_segs, int mode) {
  GRETA_REQUIRE(fmt == GRETA_FMT_Q4_0 || fmt == GRETA_FMT_Q8_0, "gemm_segments: format %d is not supported (Q4_0 or Q8_0)", fmt);
  GRETA_REQUIRE(mode >= GRETA_GEMM_STORE && mode <= GRETA_GEMM_SWIGLU_F16, "gemm_segments: mode %d", mode);
  GRETA_REQUIRE(segs && n_segs >= 1 && n_segs <= 3, "gemm_segments: %u segments (1 to 3)", n_segs);
  GRETA_REQUIRE(mode != GRETA_GEMM_SWIGLU_F16 || (n_segs == 2 && segs[0].n == segs[1].n), "gemm_segments: gate and up are two segments of one size");
  GRETA_REQUIRE(K % 32 == 0, "gemm_segments: K=%u is not a multiple of the block size 32", K);
  if (M == 0 || K == 0) return GRETA_OK;
  GRETA_REQUIRE(a_f16 && aligned16(a_f16), "gemm_segments: activations must be 16-byte aligned");
  EncodeTiledFn enc = encode_tiled();
  if (!enc) {
    set_error("gemm_segments: cuTensorMapEncodeTiled is not available from this driver");
    return GRETA_ERR_NOT_IMPLEMENTED;
  }
  const bool pair = mode == GRETA_GEMM_SWIGLU_F16;
  const uint32_t tile_rows = pair ? TILE_N / 2 : TILE_N, nb = K / 32, KT = (K + 2 * TS_K - 1) / (2 * TS_K) * 2, sms = (uint32_t)sm_count();
  const size_t row_bytes = (size_t)nb * payload_bytes(fmt);
  TsArgs w{};
  uint32_t row_tiles = 0;
  for (uint32_t i = 0; i < n_segs; ++i) {
    const greta_gemm_segment &g = segs[i];
    GRETA_REQUIRE(g.n > 0 && g.qs && g.d && (g.out || (pair && i == 1)), "gemm_segments: segment %u is empty or has a null pointer", i);
    GRETA_REQUIRE(aligned16(g.qs) && aligned16(g.d) && ((uintptr_t)g.out & 3) == 0, "gemm_segments: segment %u is misaligned", i);
    w.out[i] = static_cast<float *>(g.out);
    w.n[i] = g.n;
    if (!pair || i == 0) row_tiles += row_tiles_of(g.n, mode);
    w.tile_end[i] = row_tiles;
    const cuuint64_t qd[2] = {row_bytes, g.n}, qs[1] = {row_bytes}, dd[2] = {nb, g.n}, ds[1] = {(cuuint64_t)d_row_stride(nb) * 2};
    const cuuint32_t qbox[2] = {128, tile_rows}, dbox[2] = {8, tile_rows}, one[2] = {1, 1};
    CUresult r = enc(&w.qs[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(g.qs), qd, qs, qbox, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS)
      r = enc(&w.d[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(g.d), dd, ds, dbox, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
      set_error("gemm_segments: cuTensorMapEncodeTiled failed with code %d", (int)r);
      return GRETA_ERR_INVALID_ARGS;
    }
  }
  for (uint32_t i = n_segs; i < 3; ++i) w.tile_end[i] = row_tiles;
  const TsPlan plan = plan_ts(M, K, row_tiles);
  const uint32_t tn = plan.tn;
  w.M = M;
  w.K = K;
  w.tn = tn;
  w.tok_tiles = plan.tok_tiles;
  GRETA_REQUIRE((uint64_t)row_tiles * w.tok_tiles * KT < (1ull << 31), "gemm_segments: M=%u K=%u: too many tiles", M, K);
  w.tiles = row_tiles * w.tok_tiles;
  w.act_stages = plan.act_stages;
  w.accs = plan.accs;
  w.w_slots = plan.w_slots;
  w.idesc = instr_desc_f16(TILE_N, tn);
  const cuuint64_t ad[2] = {K, M}, as[1] = {(cuuint64_t)K * 2};
  const cuuint32_t abox[2] = {BK, tn}, one[2] = {1, 1};
  const CUresult r = enc(&w.act, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(a_f16), ad, as, abox, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("gemm_segments: cuTensorMapEncodeTiled failed with code %d", (int)r);
    return GRETA_ERR_INVALID_ARGS;
  }
  const size_t smem = TS_SMEM_FIXED + (size_t)w.act_stages * tn * TS_K * 2;
  cudaStream_t s = (cudaStream_t)stream;
  if (fmt == GRETA_FMT_Q4_0) {
    if (mode == GRETA_GEMM_STORE) return launch_ts<GRETA_FMT_Q4_0, GRETA_GEMM_STORE>(s, w, sms, smem);
    if (mode == GRETA_GEMM_ADD) return launch_ts<GRETA_FMT_Q4_0, GRETA_GEMM_ADD>(s, w, sms, smem);
    return launch_ts<GRETA_FMT_Q4_0, GRETA_GEMM_SWIGLU_F16>(s, w, sms, smem);
  }
  if (mode == GRETA_GEMM_STORE) return launch_ts<GRETA_FMT_Q8_0, GRETA_GEMM_STORE>(s, w, sms, smem);
  if (mode == GRETA_GEMM_ADD) return launch_ts<GRETA_FMT_Q8_0, GRETA_GEMM_ADD>(s, w, sms, smem);
  return launch_ts<GRETA_FMT_Q8_0, GRETA_GEMM_SWIGLU_F16>(s, w, sms, smem);
}
