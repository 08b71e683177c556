// Drives BlockScheduler from C++ where the C interface does not reach: buffers that it exposes and the tensor-parallel hooks.  The first
// argument names the check; exits non-zero when it fails.  Built by gretacore-v3_b200/csrc/Makefile (target scheduler_test) and run by
// tests/test_scheduler_gpu.py.
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "gcore/inference/block_scheduler.hpp"
#include "greta_cuda.h"

using namespace gcore::inference;
using gcore::rt::GretaDataType;

static std::string g_err;
static int complain(const std::string &what) {
  fprintf(stderr, "%s: %s\n", what.c_str(), g_err.c_str());
  return 1;
}

static ModelConfig small() {
  ModelConfig c;
  c.dim = 512; c.num_heads = 8; c.num_heads_kv = 4; c.num_layers = 2; c.vocab_size = 1000; c.hidden_dim = 1536; c.head_dim = 64; c.max_seq_len = 160;
  c.rope_base = 10000.0f; c.rms_eps = 1e-5f;
  c.weight_type = GretaDataType::Q4_0; c.lm_head_type = GretaDataType::FP16;
  return c;
}
static std::vector<int32_t> prompt(size_t n) {
  std::vector<int32_t> t(n);
  for (size_t i = 0; i < n; ++i) t[i] = (int32_t)((i * 7919 + 13) % 1000);
  return t;
}
static bool start(BlockScheduler &s, const ModelConfig &c) {
  return s.init(c, &g_err) && s.allocate_weights(&g_err) && s.load_synthetic_weights(5, &g_err) && s.allocate_activations(1, c.max_seq_len, &g_err);
}
static std::vector<float> rows_of(gcore::rt::cuda::Buffer &b, size_t n) {
  std::vector<float> v(n);
  if (!b.copy_to_host(v.data(), n * 4, &g_err)) v.clear();
  return v;
}

// get_norm_out() after a prompt: fp32 rows of the last layer's feed-forward norm, on either side of 32 rows, after forward() and after
// execute_layer().  With a norm weight of one a row's root mean square is one.
static int norm_out() {
  const ModelConfig c = small();
  BlockScheduler s;
  if (!start(s, c)) return complain("start");
  std::vector<float> ones(c.dim, 1.0f);
  for (size_t l = 0; l < c.num_layers; ++l)
    if (!s.set_layer_tensor(l, LayerTensor::FFN_NORM, ones.data(), ones.size() * 4, &g_err)) return complain("set_layer_tensor");
  const std::vector<int32_t> t = prompt(150);
  std::vector<float> few;
  for (size_t n : {(size_t)32, (size_t)33, (size_t)150}) {
    for (int layer = -1; layer < 1; ++layer) {
      if (!s.forward(t.data(), 0, n, &g_err)) return complain("forward");
      if (layer >= 0 && (!s.execute_layer(layer, 0, n, t.data(), &g_err) || !s.stream() || (s.stream()->synchronize(), false))) return complain("execute_layer");
      const std::vector<float> v = rows_of(s.get_norm_out(), n * c.dim);
      if (v.empty()) return complain("get_norm_out");
      for (size_t r = 0; r < n; ++r) {
        double ss = 0;
        for (size_t i = 0; i < c.dim; ++i) ss += (double)v[r * c.dim + i] * v[r * c.dim + i];
        if (!(std::fabs(std::sqrt(ss / c.dim) - 1) < 1e-2)) {
          fprintf(stderr, "%zu rows, layer %d: row %zu has rms %g\n", n, layer, r, std::sqrt(ss / c.dim));
          return 1;
        }
      }
      if (layer < 0 && n == 32) few = v;
      if (layer < 0 && n > 32) {  // the same rows through fp16 products
        double worst = 0;
        for (size_t i = 0; i < few.size(); ++i) worst = std::fmax(worst, std::fabs((double)few[i] - v[i]));
        if (!(worst < 2e-2)) return fprintf(stderr, "%zu rows differ from 32 by %g\n", n, worst), 1;
      }
    }
  }
  return 0;
}

// A bounded wait of a layer's kernels that gave up (its code is written by the host here) fails finish(), once; without such kernels nothing is asked.
static int gave_up() {
  ModelConfig c = small();
  c.max_seq_len = 600;
  BlockScheduler s;
  if (!start(s, c)) return complain("start");
  const std::vector<int32_t> t = prompt(600);
  if (!s.forward(t.data(), 0, 520, &g_err)) return complain("forward");
  const size_t portions[][2] = {{0, 40}, {520, 8}, {520, 32}};  // products with bounded waits; the attention alone
  for (const auto &p : portions) {
    if (!s.execute_layer(0, p[0], p[1], t.data(), &g_err) || greta_cuda_gemm_set_status(31) != GRETA_OK) return complain("execute_layer");
    std::string err;
    if (s.finish(&err) || err.find("31") == std::string::npos) return complain("finish passed, or hid the code: " + err);
    if (!s.execute_layer(0, p[0], p[1], t.data(), &g_err) || !s.finish(&g_err)) return complain("the code was reported twice");
  }
  return s.execute_layer(0, 0, 8, t.data(), &g_err) && s.finish(&g_err) ? 0 : complain("few rows");
}

// Buffer::copy_rows_to_host: rows apart on the device, together on the host; nothing beyond the buffer's end.
static int copy_rows() {
  gcore::rt::cuda::Buffer dev, pinned, none;
  if (!dev.allocate(40, gcore::rt::cuda::BufferUsage::DeviceOnly, GretaDataType::INT8, &g_err) ||
      !pinned.allocate(40, gcore::rt::cuda::BufferUsage::HostVisible, GretaDataType::INT8, &g_err))
    return complain("allocate");
  char src[40], got[40];
  for (int i = 0; i < 40; ++i) src[i] = (char)i;
  for (auto *b : {&dev, &pinned}) {
    if (!b->copy_to_device(src, 40, &g_err) || !b->copy_rows_to_host(got, 14, 12, 3, &g_err)) return complain("copy_rows_to_host");
    for (int r = 0; r < 3; ++r)
      if (std::memcmp(got + 12 * r, src + 14 * r, 12) != 0) return complain("rows differ");
    if (b->copy_rows_to_host(got, 14, 13, 3, nullptr) || b->copy_rows_to_host(got, 8, 8, 6, nullptr)) return complain("copied beyond the end");
    if (!b->copy_rows_to_host(got, 14, 0, 3, &g_err) || !b->copy_rows_to_host(got, 14, 12, 0, &g_err)) return complain("an empty copy");
  }
  return none.copy_rows_to_host(got, 4, 4, 1, nullptr) ? complain("copied from a buffer that holds nothing") : 0;
}

// The prompt of a tensor-parallel model, two ranks as two threads on one GPU: the all-reduce hook waits for its own stream, and the ranks meet
// on the host (no kernel waits for another rank's).  Hidden rows and logits against the same model on one rank, on either side of 32 rows and
// behind an earlier portion.
struct Meeting {
  std::mutex m;
  std::condition_variable cv;
  std::vector<float> sum;
  int arrived = 0, round = 0;
  void add(std::vector<float> &v) {
    std::unique_lock<std::mutex> lock(m);
    if (arrived == 0) sum.assign(v.size(), 0.0f);
    for (size_t i = 0; i < v.size(); ++i) sum[i] += v[i];
    const int now = round;
    if (++arrived == 2) {
      arrived = 0;
      ++round;
      cv.notify_all();
    } else if (!cv.wait_for(lock, std::chrono::seconds(60), [&] { return round != now; })) {
      std::fprintf(stderr, "the other rank did not come\n");
      std::exit(1);
    }
    v = sum;
  }
};
static int tensor_parallel() {
  const ModelConfig c = small();
  const std::vector<int32_t> t = prompt(150);
  const size_t parts[] = {20, 40, 90};
  struct Result {
    std::vector<std::vector<float>> hidden, logits;
    std::string err;
    bool ok = false;
  } one, two[2];
  Meeting meet;
  auto run = [&](ModelConfig k, Result *out) {
    BlockScheduler s;
    if (!(s.init(k, &out->err) && s.allocate_weights(&out->err) && s.load_synthetic_weights(5, &out->err) && s.allocate_activations(1, k.max_seq_len, &out->err))) return;
    if (k.tp_size > 1)
      s.set_all_reduce([&](float *buf, size_t count, cudaStream_t stream) {
        std::vector<float> v(count);
        if (greta_cuda_stream_synchronize((greta_stream_t)stream) != GRETA_OK || greta_cuda_memcpy_d2h_sync(v.data(), buf, count * 4) != GRETA_OK) return 1;
        meet.add(v);
        return greta_cuda_memcpy_h2d_sync(buf, v.data(), count * 4) == GRETA_OK ? 0 : 1;
      });
    size_t pos = 0;
    for (size_t n : parts) {
      if (!s.forward(t.data() + pos, pos, n, &out->err)) return;
      pos += n;
      std::vector<float> h(n * k.dim), z(k.vocab_size);
      if (!s.get_hidden_state().copy_to_host(h.data(), h.size() * 4, &out->err) || !s.get_logits().copy_to_host(z.data(), z.size() * 4, &out->err)) return;
      out->hidden.push_back(std::move(h));
      out->logits.push_back(std::move(z));
    }
    out->ok = true;
  };
  run(c, &one);
  std::vector<std::thread> ranks;
  for (uint32_t r = 0; r < 2; ++r) {
    ModelConfig k = c;
    k.tp_size = 2;
    k.tp_rank = r;
    ranks.emplace_back(run, k, &two[r]);
  }
  for (auto &th : ranks) th.join();
  for (const Result *r : {&one, &two[0], &two[1]})
    if (!r->ok) return fprintf(stderr, "%s\n", r->err.c_str()), 1;
  for (size_t p = 0; p < 3; ++p)
    for (const Result &r : two) {
      const std::vector<float> *pairs[2][2] = {{&one.hidden[p], &r.hidden[p]}, {&one.logits[p], &r.logits[p]}};
      for (auto &ab : pairs) {
        double worst = 0, top = 0;
        for (size_t i = 0; i < ab[0]->size(); ++i) {
          worst = std::fmax(worst, std::fabs((double)(*ab[0])[i] - (*ab[1])[i]));
          top = std::fmax(top, std::fabs((double)(*ab[0])[i]));
        }
        // fp32 sums in another order; above 32 rows a value may round to the next fp16 (2^-11) on the way into a product
        if (!(worst <= (parts[p] > 32 || p ? 1e-3 : 1e-5) * top)) return fprintf(stderr, "portion %zu: %g of %g\n", p, worst, top), 1;
      }
    }
  return 0;
}

int main(int argc, char **argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  const int rc = what == "norm_out" ? norm_out() : what == "copy_rows" ? copy_rows() : what == "gave_up" ? gave_up() : what == "tensor_parallel" ? tensor_parallel() : 2;
  printf("%s: %s\n", what.c_str(), rc ? "FAIL" : "PASS");
  return rc;
}
