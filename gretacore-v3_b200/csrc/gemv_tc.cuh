// Batched products on tcgen05 (gemv_tc.cu), as gemv_batch.cu's entry points call them.
#pragma once
#include "greta_common.cuh"

constexpr uint32_t BT_MAX_CTAS = 160;
constexpr size_t BT_HEADER = 1024;  // row factors, then tickets
// Smallest products (weights) that go through tcgen05; below, launch and the meeting of CTAs cost more than gemv_batch.cu takes.  In a CUDA graph, mma.sync form / this
// one, us: 9 rows 1664 x 640 q4_0 8.5 / 8.8, 1408 x 768 9.0 / 8.9, 1024 x 1024 11.0 / 9.0; q8_0 1664 x 640 11.0 / 8.8; fp16 10.3 / 10.3; 32 rows q4_0 13.7 / 12.1.
// Up to 8 rows the mma.sync form holds out longer, except where its weights are 8 bits wide (8 rows q8_0 1664 x 640 10.0 / 8.7): 8 rows of q4_0 8256 x 4096 13.1 / 13.9,
// 11712 x 4096 22.0 / 17.9; fp16 8256 x 4096 19.0 / 20.8, 11712 x 4096 33.2 / 24.7.
// Below 640 columns it does, too: 9 rows q4_0 7360 x 288 7.1 / 7.7, 14592 x 288 7.7 / 7.8, 8192 x 512 9.2 / 7.7, but 7808 x 544 8.7 / 9.1, 10368 x 576 9.5 / 9.1;
// fp16 8192 x 512 8.5 / 9.0, 16448 x 512 9.3 / 9.4, 7808 x 544 10.1 / 10.3; 32 rows q8_0 7360 x 288 9.8 / 10.7, 16384 x 256 10.2 / 8.6.
constexpr uint64_t BT_MIN_WEIGHTS = 1ull << 20, BT_MIN_WEIGHTS_FEW_ROWS = 36ull << 20, BT_MIN_WEIGHTS_SHORT = 4ull << 20, BT_MIN_WEIGHTS_SHORT_FEW = 6ull << 20;
constexpr uint32_t BT_SHORT_K = 640;

namespace greta {
size_t gemv_tc_workspace_bytes(uint32_t M, uint32_t K);
bool gemv_tc_route(int fmt, uint32_t M, uint64_t rows, uint32_t K);  // by formats and sizes alone
// `params` is the GemvParams of the product (a type of its own in every file that includes gemv_device.cuh).
bool gemv_tc_takes(int fmt, int epi, const void *params);
int gemv_tc(cudaStream_t stream, int fmt, int epi, const void *params, void *workspace);
}  // namespace greta
