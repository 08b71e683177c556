// Chunked form of the delta rules' scan, for portions.  With the names of delta_rule.cu, the tokens 0..15 of a chunk obey
//   c = KW S + P V - Q c,   o = RW S + R V - T c,   S <- W S + KD^T V - AKD^T c
// (rows KW_i = k_i W(0..i-1), RW_i = r_i W(0..i), KD_j = k_j W(j+1..15), AKD_j = ak_j W(j+1..15); P, Q strictly lower, R, T lower
// triangular), and since Q is strictly lower triangular
//   c = A S + B,   o = E S + F     with A = (1 + Q)^-1 KW,  B = (1 + Q)^-1 P V,  E = RW - T A,  F = R V - T B,
// which do not depend on S.  The gated form is the same with c = -d: KW_i = k_i W(0..i), Q_ij = (k_i W(j+1..i)) . bk_j, T_ij = (q_i
// W(j+1..i)) . bk_j, B = -(1 + Q)^-1 V, F = -T B and no KD.
//
// delta_chunk_prepare_kernel forms A, E, KD, AKD, W, B, F of every chunk side by side (a CTA per chunk and head); what is left to
// do one chunk after the other are four small products, which delta_chunk_scan_kernel runs on the tensor cores (mma.sync m16n8k16).
// fp32 is kept: every operand is the exact sum of three bf16 values (high, middle, low); of the nine products the three below 2^-24 of
// the whole are dropped, the high one and the others have accumulators of their own that start from zero in every chunk, and
// S <- W S + ... is an fp32 FMA.  No decay is ever divided by: pairs (i, j) run a product from j on.
//
// Bound by latency: a chunk is one chain of products, splits and a barrier (0.6 us alone, tensor cores busy 0.2 us of it), the preparation
// (8600 instructions of a warp per chunk and head) runs beside it.  2048 tokens, 32 heads 64 x 64: 285 us token by token, 154 here; 1337 tokens, 16 heads
// 128 x 128: 238 and 106.  Error against 64 bits, 2-norm: 1.36e-7 and 1.16e-7 of the outputs (slow decays 3.8e-7 and 2.1e-7), gated 1.24e-7 and 1.12e-7.
// Operands as pairs of tf32 values took the same time and were less exact than fp32 (1.66e-7).
#include <algorithm>

#include "delta_scan.cuh"

using namespace greta;

namespace {

constexpr int CT = 16;             // tokens of a chunk
// Below this the token-by-token scan is as fast (32 heads 64 x 64: 17 against 19 us at 64 tokens, 27 against 21 at 128).
constexpr uint32_t MIN_TOKENS = 80;
// Tokens that are prepared together, while the ones before them are walked.  The kernels alternate, prepare 0, scan 0, prepare 1, scan 1, ..,
// over two halves of the scratch.  A scan lets its successor start once its own wait is over; prepare j > 0 then runs beside scan j - 1 without
// waiting for it (scan j - 2, which read its half, has ended: scan j - 1 waited for prepare j - 1, and that for scan j - 2), and only its first CTA
// waits for scan j - 1, at its end, so that the end of prepare j implies that of scan j - 1.  What other kernels of this chain may have
// read before is loaded past L1.
// 2048 tokens, us with 256 / 512 / 768 / 1024 tokens (in a graph, inputs in L2): general form, heads of 64: 8 heads 90 / 84 / 85 / 84, 32 heads 193 / 151 / 144 / 143, 64 heads
// 307 / 281 / 290 / 282; heads of 128: 8 heads 139 / 134 / 142 / 147, 16 heads 229 / 214 / 215 / 214, 64 heads 849 / 892 / 873 / 878; gated, heads of 128: 8 heads
// 118 / 116 / 118 / 118, 16 heads 185 / 162 / 153 / 146, 64 heads 629 / 574 / 560 / 554.  Between 512 and 1024 there is little to choose.
constexpr uint32_t SLICE = 768;

__host__ __device__ constexpr uint32_t pad16(uint32_t v) { return (v + 15u) & ~15u; }

// Scratch of a chunk and head, in words: rows A | E | (KD) | -AKD as bf16 triples in the order in which the scan's lanes read them (a
// fragment is 8 tokens or rows x 16: per lane high 2, middle 2; then per lane low 2), W; then per group of 16 value columns (V: per lane high
// 4, middle 4, low 4 of a 16 x 16 fragment) | B | F.
constexpr int FRAG = 192;
template <int DP, bool GATED>
struct ChunkCfg {
  static constexpr int KP = DP / 16, WARPS = 4, SL = KP / WARPS, THREADS = WARPS * 32 + 64;  // a warp of the scan owns SL x 16 rows; two copy and write o
  static constexpr int ROWS = GATED ? 3 : 4, ARRAY = 2 * KP * FRAG, SHARED = ROWS * ARRAY + DP, VF = GATED ? 0 : 384, CG = VF + 512;
  static constexpr int STAGES = DP == 128 && !GATED ? 3 : 4;
  static constexpr size_t SCAN_SMEM = (size_t)(STAGES * (SHARED + CG) + 4 * WARPS * 256) * 4;
  // prepare: k and r (then A and E), w, (a), v, the pairs' triangles, KD | -AKD
  static constexpr int PREP_THREADS = 2 * DP, LD1 = DP + 16, LD2 = DP + 8, TRI = GATED ? 2 : 4, WR = GATED ? 1 : 2;
  __host__ __device__ static constexpr uint32_t ldv(uint32_t V) { return pad16(V) + 4; }
  __host__ __device__ static constexpr uint32_t rates(uint32_t V) { return !GATED && ldv(V) < DP ? DP : ldv(V); }  // rows of removal rates, then B
  __host__ __device__ static constexpr size_t prep_floats(uint32_t V) {
    return 2 * CT * LD1 + CT * DP + CT * rates(V) + CT * ldv(V) + TRI * CT * CT + WR * CT * LD2 + CT;
  }
  __host__ __device__ static constexpr uint32_t chunk_floats(uint32_t V) { return SHARED + pad16(V) / 16 * CG; }
};

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ float4 ldg4(const float *p) { return __ldcg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ void st4(float *p, const float4 &v) { *reinterpret_cast<float4 *>(p) = v; }
// Two fp32 values as the sums of three bf16 values each, packed.
struct Triple {
  uint32_t h, m, l;
  __device__ __forceinline__ void set(float x, float y) {
    h = pack(x, y);
    x -= __uint_as_float(h << 16), y -= __uint_as_float(h & 0xffff0000u);
    m = pack(x, y);
    l = pack(x - __uint_as_float(m << 16), y - __uint_as_float(m & 0xffff0000u));
  }
  __device__ __forceinline__ static uint32_t pack(float x, float y) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
    return r;
  }
};
// Left operand of 16 rows x 16.  Two tiles held as accumulators (c0, c1: row g, columns 2t, 2t+1; c2, c3: row g+8) are that of the next product.
struct Left {
  uint4 h, m, l;
  __device__ __forceinline__ void put(int i, float x, float y) {
    Triple v;
    v.set(x, y);
    (&h.x)[i] = v.h, (&m.x)[i] = v.m, (&l.x)[i] = v.l;
  }
  __device__ __forceinline__ void set(const float (&p)[4], const float (&q)[4]) { put(0, p[0], p[1]), put(1, p[2], p[3]), put(2, q[0], q[1]), put(3, q[2], q[3]); }
  __device__ __forceinline__ void load(const float *p, int lane) {
    const uint4 *q = reinterpret_cast<const uint4 *>(p) + lane;
    h = q[0], m = q[32], l = q[64];
  }
  __device__ __forceinline__ void store(float *p, int lane) const {
    uint4 *q = reinterpret_cast<uint4 *>(p) + lane;
    q[0] = h, q[32] = m, q[64] = l;
  }
};
// Two fp32 values side by side in a 64-bit register: one instruction for both.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 join2(float x, float y) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 split2(f32x2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ float sum2(f32x2 a) {
  const float2 v = split2(a);
  return v.x + v.y;
}
__device__ __forceinline__ float dot8(const f32x2 (&a)[4], const f32x2 (&b)[4]) {
  return sum2(fma2(a[3], b[3], fma2(a[2], b[2], fma2(a[1], b[1], mul2(a[0], b[0])))));
}
// N = 4 or 2 values over a group of L lanes: lane l receives the total of value l / (L / N).
template <int N, int L>
__device__ __forceinline__ float group_sum(const float (&v)[N], int l) {
  float x = v[0], y = v[N / 2 - 1];
  int m = L / 2;
  const bool up = l & m;
  if (N == 4) {
    x = (up ? v[N / 2] : v[0]) + __shfl_xor_sync(0xffffffffu, up ? v[0] : v[N / 2], m);
    y = (up ? v[N - 1] : v[1]) + __shfl_xor_sync(0xffffffffu, up ? v[1] : v[N - 1], m);
    const bool up2 = l & (m / 2);
    x = (up2 ? y : x) + __shfl_xor_sync(0xffffffffu, up2 ? x : y, m / 2);
    m /= 4;
  } else {
    x = (up ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, up ? v[0] : v[1], m);
    m /= 2;
  }
  for (; m > 0; m >>= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
  return x;
}

template <int DP, bool GATED>
__global__ void __launch_bounds__(2 * DP) delta_chunk_prepare_kernel(const __grid_constant__ ScanArgs a, uint32_t t0, uint32_t t_end, float *scratch, int vec) {
  using C = ChunkCfg<DP, GATED>;
  extern __shared__ __align__(16) float sm[];
  const uint32_t h = blockIdx.x, hk = h / a.per, D = a.dim, V = a.vdim, VP = pad16(V), LV = C::ldv(V), first = t0 + blockIdx.y * CT;
  const int n = (int)min((uint32_t)CT, t_end - first), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float *sk = sm, *sr = sk + CT * C::LD1, *sw = sr + CT * C::LD1, *sa = sw + CT * DP, *sv = sa + CT * C::rates(V), *tri = sv + CT * C::ldv(V);
  float *sd = tri + C::TRI * CT * CT, *sb = sd + C::WR * CT * C::LD2;  // sb: write strengths
  float *out = scratch + ((size_t)blockIdx.y * a.heads + h) * C::chunk_floats(V);
  pdl_launch_dependents();
  if (!t0) pdl_wait();

  // Tokens behind the portion's end leave the state as it is (w = 1, everything else 0); rows past dim are zero.
  const float *gk = a.k + (size_t)first * a.ld_k + (size_t)hk * D, *gr = a.r + (size_t)first * a.ld_r + (size_t)hk * D;
  const float *gw = a.w + (size_t)first * a.ld_w + (size_t)h * D, *gv = a.v + (size_t)first * a.ld_v + (size_t)h * V;
  const float *ga = a.a + (size_t)first * a.ld_a + (GATED ? (size_t)h : (size_t)h * D);
  if (vec) {
    for (int i = tid; i < CT * DP / 4; i += C::PREP_THREADS) {
      const int t = i / (DP / 4), e = i % (DP / 4) * 4;
      const bool on = t < n && e < (int)D;
      float4 k = make_float4(0.f, 0.f, 0.f, 0.f), r = k, w = k, x = k;
      if (e < (int)D) w = make_float4(1.f, 1.f, 1.f, 1.f);
      if (on) {
        k = ldg4(gk + (size_t)t * a.ld_k + e), r = ldg4(gr + (size_t)t * a.ld_r + e), w = ldg4(gw + (size_t)t * a.ld_w + e);
        if (!GATED) x = ldg4(ga + (size_t)t * a.ld_a + e);
      }
      st4(sk + t * C::LD1 + e, k), st4(sr + t * C::LD1 + e, r), st4(sw + t * DP + e, w);
      if (!GATED) st4(sa + t * DP + e, x);
    }
    for (int i = tid; i < CT * (int)VP / 4; i += C::PREP_THREADS) {
      const int t = i / (VP / 4), e = i % (VP / 4) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < n && e < (int)V) v = ldg4(gv + (size_t)t * a.ld_v + e);
      st4(sv + t * LV + e, v);
    }
  } else {
    for (int i = tid; i < CT * DP; i += C::PREP_THREADS) {
      const int t = i / DP, e = i % DP;
      const bool on = t < n && e < (int)D;
      sk[t * C::LD1 + e] = on ? __ldcg(gk + (size_t)t * a.ld_k + e) : 0.f;
      sr[t * C::LD1 + e] = on ? __ldcg(gr + (size_t)t * a.ld_r + e) : 0.f;
      sw[t * DP + e] = on ? __ldcg(gw + (size_t)t * a.ld_w + e) : e < (int)D ? 1.f : 0.f;
      if (!GATED) sa[t * DP + e] = on ? __ldcg(ga + (size_t)t * a.ld_a + e) : 0.f;
    }
    for (int i = tid; i < CT * (int)VP; i += C::PREP_THREADS) {
      const int t = i / VP, e = i % VP;
      sv[t * LV + e] = t < n && e < (int)V ? __ldcg(gv + (size_t)t * a.ld_v + e) : 0.f;
    }
  }
  if (GATED && tid < CT) sb[tid] = tid < n ? __ldcg(ga + (size_t)tid * a.ld_a) : 0.f;
  __syncthreads();
  const int g = lane >> 2, t = lane & 3;
  if constexpr (!GATED)  // V as the scan multiplies it: words 2 (token / 8) + column / 8 of lane (column % 8, token % 8 / 2)
    for (uint32_t q = warp; q < VP / 16; q += C::PREP_THREADS / 32) {
      const float *v = sv + 2 * t * LV + q * 16 + g;
      Left x;
      x.put(0, v[0], v[LV]), x.put(1, v[8], v[LV + 8]), x.put(2, v[8 * LV], v[9 * LV]), x.put(3, v[8 * LV + 8], v[9 * LV + 8]);
      x.store(out + C::SHARED + q * C::CG, lane);
    }

  // Pairs: LPJ lanes carry what token j writes (eight rows each) through the tokens i behind it, decaying it on the way.
  {
    constexpr int LPJ = DP / 8, JW = 32 / LPJ;
    const int j = warp * JW + lane / LPJ, l = lane % LPJ, e0 = l * 4, e1 = DP / 2 + l * 4;
    auto load8 = [&](f32x2(&x)[4], const float *row) {
      const ulonglong2 p = *reinterpret_cast<const ulonglong2 *>(row + e0), q = *reinterpret_cast<const ulonglong2 *>(row + e1);
      x[0] = p.x, x[1] = p.y, x[2] = q.x, x[3] = q.y;
    };
    auto store8 = [&](float *row, const f32x2(&x)[4]) {
      *reinterpret_cast<ulonglong2 *>(row + e0) = make_ulonglong2(x[0], x[1]);
      *reinterpret_cast<ulonglong2 *>(row + e1) = make_ulonglong2(x[2], x[3]);
    };
    f32x2 kj[4], akj[4], p[4], pa[4];
    load8(kj, sk + j * C::LD1);
    if (GATED) {
      const f32x2 beta = join2(sb[j], sb[j]);
#pragma unroll
      for (int e = 0; e < 4; ++e) akj[e] = mul2(beta, kj[e]);
    } else {
      load8(akj, sa + j * DP);
      float kk = dot8(kj, kj);
#pragma unroll
      for (int m = LPJ / 2; m > 0; m >>= 1) kk += __shfl_xor_sync(0xffffffffu, kk, m);
      kk = 1.f / (kk + 1e-6f);
      const f32x2 inv2 = join2(kk, kk);
#pragma unroll
      for (int e = 0; e < 4; ++e) akj[e] = mul2(mul2(akj[e], kj[e]), inv2);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) p[e] = pa[e] = 0;
    constexpr int N = GATED ? 2 : 4;
    float *at = tri + (l / (LPJ / N)) * CT * CT + j;
    const bool writes = l % (LPJ / N) == 0;
    auto token = [&](int i, bool edge) {  // edge: the warp's own tokens, of which one is j
      f32x2 w[4], k[4], r[4];
      load8(w, sw + i * DP);
      load8(k, sk + i * C::LD1);
      load8(r, sr + i * C::LD1);
      const bool here = edge && i == j;
      float x[N];
      if constexpr (GATED) {
#pragma unroll
        for (int e = 0; e < 4; ++e) pa[e] = mul2(pa[e], w[e]);
        x[0] = dot8(k, pa);
#pragma unroll
        for (int e = 0; e < 4; ++e) pa[e] = here ? akj[e] : pa[e];
        x[1] = dot8(r, pa);
      } else {
        x[0] = dot8(k, p), x[1] = dot8(k, pa);
#pragma unroll
        for (int e = 0; e < 4; ++e) p[e] = mul2(p[e], w[e]), pa[e] = mul2(pa[e], w[e]);
#pragma unroll
        for (int e = 0; e < 4; ++e) p[e] = here ? kj[e] : p[e], pa[e] = here ? akj[e] : pa[e];
        x[N - 2] = dot8(r, p), x[N - 1] = dot8(r, pa);
      }
      const float s = group_sum<N, LPJ>(x, l);
      if (writes) at[i * CT] = s;
    };
#pragma unroll
    for (int i = 0; i < JW; ++i) token(warp * JW + i, true);
#pragma unroll 2
    for (int i = warp * JW + JW; i < CT; ++i) token(i, false);
    constexpr f32x2 SIGNS = 0x8000000080000000ull;
#pragma unroll
    for (int e = 0; e < 4; ++e) pa[e] ^= SIGNS;
    if (!GATED) store8(sd + j * C::LD2, p);
    store8(sd + (C::WR - 1) * CT * C::LD2 + j * C::LD2, pa);
  }
  __syncthreads();

  const float *P = tri, *Q = tri + (GATED ? 0 : CT * CT), *R = tri + 2 * CT * CT, *T = tri + (GATED ? 1 : 3) * CT * CT;
  // Row of a triangle times x[0 .. N-1].  From zero and in four sums: added to the large term one by one they would round sixteen times at its size.
  auto row_dot = [](const float *row, const float(&x)[CT], int N) {
    f32x2 y0 = 0, y1 = 0;
    float odd = 0.f;
#pragma unroll
    for (int q = 0; q < CT; q += 4)
      if (q < N) {
        const ulonglong2 c = *reinterpret_cast<const ulonglong2 *>(row + q);
        if (q + 2 <= N) y0 = q ? fma2(c.x, join2(x[q], x[q + 1]), y0) : mul2(c.x, join2(x[q], x[q + 1]));
        if (q + 4 <= N) y1 = q ? fma2(c.y, join2(x[q + 2], x[q + 3]), y1) : mul2(c.y, join2(x[q + 2], x[q + 3]));
        if (q + 1 == N) odd = split2(c.x).x * x[q];
        if (q + 3 == N) odd = split2(c.y).x * x[q + 2];
      }
    float s = N >= 2 ? sum2(y0) : 0.f;
    if (N >= 4) s += sum2(y1);
    return N & 1 ? s + odd : s;
  };
  if (tid < DP) {  // a row of the state per thread: A and E take the places of k and r
    float x[CT], cum = 1.f;
#pragma unroll
    for (int i = 0; i < CT; ++i) {
      const float w = sw[i * DP + tid], k = sk[i * C::LD1 + tid], before = cum;
      cum *= w;
      x[i] = k * (GATED ? cum : before) - row_dot(Q + i * CT, x, i);
      sk[i * C::LD1 + tid] = x[i];
      sr[i * C::LD1 + tid] = sr[i * C::LD1 + tid] * cum - row_dot(T + i * CT, x, i + 1);
    }
    out[C::ROWS * C::ARRAY + tid] = cum;
  } else {  // a value column per thread
#pragma unroll 1
    for (uint32_t c = tid - DP; c < VP; c += DP) {
      asm volatile("" ::: "memory");  // the triangles are read again for every column: kept in registers they would spill
      float v[CT], b[CT], f[CT];
#pragma unroll
      for (int i = 0; i < CT; ++i) v[i] = sv[i * LV + c];
#pragma unroll
      for (int i = 0; i < CT; ++i) {
        if constexpr (GATED) {
          b[i] = -v[i] - row_dot(Q + i * CT, b, i);
          f[i] = -row_dot(T + i * CT, b, i + 1);
        } else {
          b[i] = row_dot(P + i * CT, v, i) - row_dot(Q + i * CT, b, i);
          f[i] = row_dot(R + i * CT, v, i + 1) - row_dot(T + i * CT, b, i + 1);
        }
      }
#pragma unroll
      for (int i = 0; i < CT; ++i) sa[i * LV + c] = b[i], sv[i * LV + c] = f[i];
    }
  }
  __syncthreads();
  for (uint32_t q = warp; q < VP / 4; q += C::PREP_THREADS / 32) {  // B and F of a group: per token tile and lane two tokens of columns g, g + 8
    const float *y = (q & 2 ? sv : sa) + ((q & 1) * 8 + 2 * t) * LV + (q >> 2) * 16 + g;
    st4(out + C::SHARED + (q >> 2) * C::CG + C::VF + ((q & 3) * 32 + lane) * 4, make_float4(y[0], y[LV], y[8], y[LV + 8]));
  }
#pragma unroll
  for (int arr = 0; arr < C::ROWS; ++arr)
#pragma unroll
    for (int n = 0; n < 2 * C::KP / (C::PREP_THREADS / 32); ++n) {  // a fragment per warp
      const int q = n * (C::PREP_THREADS / 32) + warp;
      Triple x, y;
      if (arr < 2) {
        const float4 v = ld4((arr ? sr : sk) + (q / C::KP * 8 + g) * C::LD1 + q % C::KP * 16 + t * 4);
        x.set(v.x, v.y), y.set(v.z, v.w);
      } else {
        const float *d = sd + (arr - 2) * CT * C::LD2 + 2 * t * C::LD2 + (q >> 1) * 16 + (g >> 1) * 4 + (q & 1) * 2 + (g & 1);
        x.set(d[0], d[C::LD2]), y.set(d[8 * C::LD2], d[9 * C::LD2]);
      }
      uint32_t *o = reinterpret_cast<uint32_t *>(out) + arr * C::ARRAY + q * FRAG;
      *reinterpret_cast<uint4 *>(o + lane * 4) = make_uint4(x.h, y.h, x.m, y.m);
      *reinterpret_cast<uint2 *>(o + 128 + lane * 2) = make_uint2(x.l, y.l);
    }
  if (t0 && !blockIdx.x && !blockIdx.y) pdl_wait();
}

// ---- the walk over the chunks
// D = A B + C, or (from zero) A B
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint4 &a, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16_zero(float (&c)[4], const uint4 &a, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "f"(0.f));
}
struct Right {
  uint4 hm;
  uint2 l;
  __device__ __forceinline__ void load(const float *frag, int lane) {
    hm = *reinterpret_cast<const uint4 *>(frag + lane * 4);
    l = *reinterpret_cast<const uint2 *>(frag + 128 + lane * 2);
  }
};
struct Acc {  // high products; middle ones; the rest
  float h[4], m[4], l[4];
  __device__ __forceinline__ float sum(int i) const { return h[i] + (m[i] + l[i]); }
};
// Two tiles side by side: products of one tile wait for one another less often.  HIGH, REST: from zero, else added.
template <bool HIGH, bool REST>
__device__ __forceinline__ void mma_triples(Acc (&c)[2], const Left &a, const Right (&b)[2]) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (HIGH) mma_bf16_zero(c[i].h, a.h, b[i].hm.x, b[i].hm.y);
    else mma_bf16(c[i].h, a.h, b[i].hm.x, b[i].hm.y);
    if (REST) {
      mma_bf16_zero(c[i].m, a.h, b[i].hm.z, b[i].hm.w);
      mma_bf16_zero(c[i].l, a.h, b[i].l.x, b[i].l.y);
    } else {
      mma_bf16(c[i].m, a.h, b[i].hm.z, b[i].hm.w);
      mma_bf16(c[i].l, a.h, b[i].l.x, b[i].l.y);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    mma_bf16(c[i].m, a.m, b[i].hm.x, b[i].hm.y);
    mma_bf16(c[i].l, a.m, b[i].hm.z, b[i].hm.w);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) mma_bf16(c[i].l, a.l, b[i].hm.x, b[i].hm.y);
}

// Grid (heads, groups of 16 value columns).  Each of the first four warps holds SL slabs of 16 rows of the group's state, transposed, a slab as
// two accumulator tiles (tile p, lane (g, t): rows 16 slab + 4 t + 2 p + {0, 1}, columns g and g + 8); the warps' parts of c and o meet in
// shared memory.  Two more warps copy the chunks in and write o, eight tokens each.
// One barrier per chunk: in front of it every warp has put down its parts of c and, of the chunk before, of o, and finished with that chunk.
template <int DP, bool GATED>
__global__ void __launch_bounds__(ChunkCfg<DP, GATED>::THREADS) delta_chunk_scan_kernel(const __grid_constant__ ScanArgs a, uint32_t t0, uint32_t t_end, const float *scratch,
                                                                                      float *o_buf) {
  using C = ChunkCfg<DP, GATED>;
  constexpr int STAGE = C::SHARED + C::CG, ST = C::STAGES, W = C::WARPS, SL = C::SL;
  extern __shared__ __align__(16) float sm[];
  float *ex_c = sm + ST * STAGE, *ex_o = ex_c + 2 * W * 256;  // [2][warp][token tile][lane][4]
  const uint32_t h = blockIdx.x, c0 = blockIdx.y * 16, V = a.vdim, chunks = (t_end - t0 + CT - 1) / CT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  pdl_wait();
  pdl_launch_dependents();

  if (warp >= W) {
    const int i = warp - W, tid = threadIdx.x - W * 32;
    const size_t step = (size_t)a.heads * C::chunk_floats(V);
    const float *src = scratch + (size_t)h * C::chunk_floats(V) + tid * 4, *src_g = src + C::SHARED + blockIdx.y * C::CG;
    auto stage = [&](uint32_t c) {
      if (c < chunks) {
        float *dst = sm + (c % ST) * STAGE + tid * 4;
#pragma unroll
        for (int e = 0; e < C::SHARED; e += 256)
          if (e + 256 <= C::SHARED || tid * 4 + e < C::SHARED) cp16(dst + e, src + c * step + e);
#pragma unroll
        for (int e = 0; e < C::CG; e += 256)
          if (e + 256 <= C::CG || tid * 4 + e < C::CG) cp16(dst + C::SHARED + e, src_g + c * step + e);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int c = 0; c < ST - 1; ++c) stage(c);
    asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
    __syncthreads();
    float4 F = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t ch = 0; ch <= chunks; ++ch) {
      asm volatile("cp.async.wait_group %0;" ::"n"(ST - 3) : "memory");  // the next chunk is there
      const float4 f = F;
      if (ch < chunks) F = ld4(sm + (ch % ST) * STAGE + C::SHARED + C::VF + 256 + (i * 32 + lane) * 4);
      __syncthreads();
      stage(ch + ST - 1);  // into the place of the chunk before: every warp has passed its last read of it
      if (!ch) continue;
      const float *xo = ex_o + ((ch - 1) & 1) * W * 256 + (i * 32 + lane) * 4;  // o of the chunk before
      const float4 p = ld4(xo), q = ld4(xo + 256), r = ld4(xo + 512), u = ld4(xo + 768);
      const float y[4] = {f.x + ((p.x + r.x) + (q.x + u.x)), f.y + ((p.y + r.y) + (q.y + u.y)), f.z + ((p.z + r.z) + (q.z + u.z)), f.w + ((p.w + r.w) + (q.w + u.w))};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t row = t0 + (ch - 1) * CT + i * 8 + 2 * t + (e & 1), col = c0 + g + (e >> 1) * 8;
        if (row < t_end && col < V) o_buf[((size_t)row * a.heads + h) * V + col] = y[e];
      }
    }
    return;
  }

  float *state = a.state + ((size_t)a.slot * a.heads + h) * V * DP + 16 * SL * warp + 4 * t;
  float s[SL][2][4];
  const bool fresh = a.pos0 + t0 == 0;
#pragma unroll
  for (int k = 0; k < SL; ++k) {
    float4 u = make_float4(0.f, 0.f, 0.f, 0.f), v = u;
    if (!fresh && c0 + g < V) u = ldg4(state + (size_t)(c0 + g) * DP + 16 * k);
    if (!fresh && c0 + g + 8 < V) v = ldg4(state + (size_t)(c0 + g + 8) * DP + 16 * k);
    s[k][0][0] = u.x, s[k][0][1] = u.y, s[k][1][0] = u.z, s[k][1][1] = u.w;
    s[k][0][2] = v.x, s[k][0][3] = v.y, s[k][1][2] = v.z, s[k][1][3] = v.w;
  }
  __syncthreads();
  for (uint32_t ch = 0; ch < chunks; ++ch) {
    const float *b = sm + (ch % ST) * STAGE, *bc = b + C::SHARED;
    float *xc = ex_c + (ch & 1) * W * 256, *xo = ex_o + (ch & 1) * W * 256;
    Left S[SL];
    Acc d[SL][2];
    Right r[2];
    float hi[2][4];
    Acc x[2];
    auto times_state = [&](int array) {  // this warp's part of A S or E S
#pragma unroll
      for (int k = 0; k < SL; ++k) {
        r[0].load(b + array * C::ARRAY + (warp * SL + k) * FRAG, lane), r[1].load(b + array * C::ARRAY + (C::KP + warp * SL + k) * FRAG, lane);
        if (k == 0)
          mma_triples<true, true>(x, S[k], r);
        else
          mma_triples<true, false>(x, S[k], r);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) hi[i][e] = k ? hi[i][e] + x[i].h[e] : x[i].h[e];
      }
    };
    auto put = [&](float *to) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = hi[i][e] + (x[i].m[e] + x[i].l[e]);
        st4(to + ((warp * 2 + i) * 32 + lane) * 4, make_float4(y[0], y[1], y[2], y[3]));
      }
    };
#pragma unroll
    for (int k = 0; k < SL; ++k) S[k].set(s[k][0], s[k][1]);
    times_state(0);
    if constexpr (!GATED) {  // KD^T V
      Left v;
      v.load(bc, lane);
#pragma unroll
      for (int k = 0; k < SL; ++k) {
        const float *f = b + 2 * C::ARRAY + (warp * SL + k) * 2 * FRAG;
        r[0].load(f, lane), r[1].load(f + FRAG, lane);
        mma_triples<true, true>(d[k], v, r);
      }
    }
    put(xc);
    const float4 B0 = ld4(bc + C::VF + lane * 4), B1 = ld4(bc + C::VF + 128 + lane * 4);
    __syncthreads();
    float4 part[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int w = 0; w < W; ++w) part[i][w] = ld4(xc + ((w * 2 + i) * 32 + lane) * 4);
    times_state(1);
    float c[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {  // B last, the parts in pairs: fewer roundings at the size of the sum
      const float4 p = part[i][0], q = part[i][1], u = part[i][2], v = part[i][3], B = i ? B1 : B0;
      c[i][0] = B.x + ((p.x + u.x) + (q.x + v.x)), c[i][1] = B.y + ((p.y + u.y) + (q.y + v.y));
      c[i][2] = B.z + ((p.z + u.z) + (q.z + v.z)), c[i][3] = B.w + ((p.w + u.w) + (q.w + v.w));
    }
    Left cl;
    cl.set(c[0], c[1]);
#pragma unroll
    for (int k = 0; k < SL; ++k) {  // - AKD^T c
      const float *f = b + (C::ROWS - 1) * C::ARRAY + (warp * SL + k) * 2 * FRAG;
      r[0].load(f, lane), r[1].load(f + FRAG, lane);
      mma_triples<GATED, GATED>(d[k], cl, r);
    }
    put(xo);
#pragma unroll
    for (int k = 0; k < SL; ++k) {
      const float4 w = ld4(b + C::ROWS * C::ARRAY + 16 * (warp * SL + k) + 4 * t);
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const float w0 = p ? w.z : w.x, w1 = p ? w.w : w.y;
#pragma unroll
        for (int e = 0; e < 4; ++e) s[k][p][e] = fmaf(e & 1 ? w1 : w0, s[k][p][e], d[k][p].sum(e));
      }
    }
  }
  __syncthreads();  // the last chunk's o
#pragma unroll
  for (int k = 0; k < SL; ++k) {
    if (c0 + g < V) st4(state + (size_t)(c0 + g) * DP + 16 * k, make_float4(s[k][0][0], s[k][0][1], s[k][1][0], s[k][1][1]));
    if (c0 + g + 8 < V) st4(state + (size_t)(c0 + g + 8) * DP + 16 * k, make_float4(s[k][0][2], s[k][0][3], s[k][1][2], s[k][1][3]));
  }
}

template <int DP, bool GATED>
int run(cudaStream_t st, const ScanArgs &a, float *o_buf, float *scratch) {
  using C = ChunkCfg<DP, GATED>;
  constexpr size_t ALONE = 118 * 1024;  // as launch_scan: a grid that fits the SMs takes one each
  const size_t prep = C::prep_floats(a.vdim) * 4;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    GRETA_CUDA_TRY(cudaFuncSetAttribute(delta_chunk_prepare_kernel<DP, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(C::prep_floats(256) * 4)));
    GRETA_CUDA_TRY(cudaFuncSetAttribute(delta_chunk_scan_kernel<DP, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)std::max(C::SCAN_SMEM, ALONE)));
    attr_set[dev] = true;
  }
  const dim3 grid(a.heads, pad16(a.vdim) / 16);
  const size_t smem = grid.x * grid.y <= (uint32_t)sm_count() ? std::max(C::SCAN_SMEM, ALONE) : C::SCAN_SMEM;
  const int vec = scan_vec(a, GATED);
  for (uint32_t t = 0; t < a.T; t += SLICE) {
    const uint32_t end = std::min(a.T, t + SLICE);
    float *half = scratch + (t / SLICE & 1 ? (size_t)(SLICE / CT) * a.heads * C::chunk_floats(a.vdim) : 0);
    GRETA_CUDA_TRY(launch_pdl(delta_chunk_prepare_kernel<DP, GATED>, dim3(a.heads, (end - t + CT - 1) / CT), dim3(C::PREP_THREADS), prep, st, a, t, end, half, vec));
    if (int rc = launched("delta_chunk_prepare_kernel")) return rc;
    GRETA_CUDA_TRY(launch_pdl(delta_chunk_scan_kernel<DP, GATED>, grid, dim3(C::THREADS), smem, st, a, t, end, half, o_buf));
    if (int rc = launched("delta_chunk_scan_kernel")) return rc;
  }
  return GRETA_OK;
}

}  // namespace

namespace greta {

size_t chunk_scan_bytes(uint32_t heads, uint32_t dim, uint32_t vdim, bool gated, uint32_t T) {
  const uint32_t dp = dim32(dim);
  if ((dp != 64 && dp != 128) || T < MIN_TOKENS) return 0;
  const uint32_t rows = gated ? (dp == 64 ? ChunkCfg<64, true>::chunk_floats(vdim) : ChunkCfg<128, true>::chunk_floats(vdim))
                              : (dp == 64 ? ChunkCfg<64, false>::chunk_floats(vdim) : ChunkCfg<128, false>::chunk_floats(vdim));
  return (size_t)((std::min(T, 2 * SLICE) + CT - 1) / CT) * heads * rows * 4;
}

int chunk_scan(cudaStream_t s, const ScanArgs &a, bool gated, float *o_buf, float *scratch) {
  const bool narrow = dim32(a.dim) == 64;
  if (gated) return narrow ? run<64, true>(s, a, o_buf, scratch) : run<128, true>(s, a, o_buf, scratch);
  return narrow ? run<64, false>(s, a, o_buf, scratch) : run<128, false>(s, a, o_buf, scratch);
}

}  // namespace greta
