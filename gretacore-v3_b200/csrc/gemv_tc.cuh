// Batched products on tcgen05 (gemv_tc.cu), as gemv_batch.cu's entry points call them.
#pragma once
#include "greta_common.cuh"

constexpr uint32_t BT_MAX_CTAS = 160;
constexpr size_t BT_HEADER = 1024;  // row factors, then tickets
// Smallest products (weights) that go through tcgen05; below, launch and the meeting of CTAs cost more than gemv_batch.cu takes.  In a CUDA graph, both sides, us:
// 16 rows 1024 x 512 q4_0 9.1 / 8.2, 1024 x 1024 9.5 / 11.7; 32 rows of q8_0 11.3 / 11.2, 12.3 / 16.9.  Up to 8 rows the mma.sync form holds out longer, except
// where its weights are 8 bits wide (8 rows 1024 x 1024 9.4 / 12.7): 8 rows of q4_0 6144 x 4096 15.5 / 13.3, 8192 x 8192 23.1 / 26.1; fp16 4096 x 4096 16.1 / 13.3,
// 6144 x 4096 18.7 / 19.3.  Rows of one or two K steps leave few CTAs and nothing to stream while the others meet: a step of 13 sequences at width 512,
// whose only product this large is 3648 x 512, took 145 against 142 us, at width 1024 170 against 200.
constexpr uint64_t BT_MIN_WEIGHTS = 1ull << 20, BT_MIN_WEIGHTS_FEW_ROWS = 1ull << 25, BT_MIN_WEIGHTS_SHORT = 1ull << 22;
constexpr uint32_t BT_SHORT_K = 640;

namespace greta {
size_t gemv_tc_workspace_bytes(uint32_t M, uint32_t K);
bool gemv_tc_route(int fmt, uint32_t M, uint64_t rows, uint32_t K);  // by formats and sizes alone
// `params` is the GemvParams of the product (a type of its own in every file that includes gemv_device.cuh).
bool gemv_tc_takes(int fmt, int epi, const void *params);
int gemv_tc(cudaStream_t stream, int fmt, int epi, const void *params, void *workspace);
}  // namespace greta
