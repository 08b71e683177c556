"""Batched products that go through tcgen05 (a million weights or more, with workspace): row tiles and K steps that are not whole, both widths of the
activation operand (16 and 32 rows), row tiles shared by many CTAs and shares that end inside a pair of tiles, every epilogue and weight format.
Bars as in test_batch_gpu.py: 2e-5 (observed about 3e-7), exact integer weights and activations of at least 22 bits, summed in fp32."""
import ctypes as C

import numpy as np
import pytest

from _support import load_package, make_blocks, max_abs_rel
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TIGHT = 2e-5


@pytest.fixture(scope="module")
def g():
    pkg = load_package()
    pkg.build()
    pkg.ffi.require_device()
    return pkg.ffi


class _Weight:
    """A [N x K] weight of `name` on the device, and the oracle's product with it."""

    def __init__(self, g, rng, name, N, K):
        self.N, self.K = N, K
        if name == "f16":
            self.bits = rng.normal(0, 0.02, (N, K)).astype(np.float16).view(np.uint16)
            self.fmt, self.held = g.FMT_F16, g.DeviceBuffer.from_numpy(self.bits)
            self.qs, self.d = self.held.ptr, None
            self.product = lambda x: O.gemm_f16w(x, self.bits, N, K)
        else:
            self.fmt, ofmt = (g.FMT_Q4_0, O.FMT_Q4_0) if name == "q4_0" else (g.FMT_Q8_0, O.FMT_Q8_0)
            self.blocks = make_blocks(rng, ofmt, N, K)
            self.held = g.Weight(self.blocks, self.fmt, N, K)
            self.qs, self.d = self.held.qs.ptr, self.held.d.ptr
            self.product = lambda x: O.gemv(x, self.blocks, ofmt, N, K)


def _ws(g, M, K):
    b = g.DeviceBuffer(g.cuda().greta_cuda_gemv_batch_workspace_bytes(M, K))
    b.fill(0xFF)  # nothing in it may be taken for zeros
    return b


def _out(g, n):
    b = g.DeviceBuffer(n * 4)
    b.fill(0xFF)
    return b


@pytest.mark.parametrize("name", ["q4_0", "q8_0", "f16"])
@pytest.mark.parametrize("M,N,K", [(9, 1100, 1056), (16, 130, 8256), (17, 8100, 544), (32, 2051, 2080), (32, 131, 33024), (2, 4700, 7232), (1, 4700, 7232)])
def test_products(g, name, M, N, K):
    lib, rng = g.cuda(), np.random.default_rng(M + N + K)
    w = _Weight(g, rng, name, N, K)
    x = (rng.normal(0, 1, (M, K)) * rng.uniform(0.01, 30.0, (M, 1))).astype(np.float32)
    gamma, resid = rng.normal(1, 0.2, K).astype(np.float32), rng.normal(0, 1, (M, N)).astype(np.float32)
    xd, gd, rd, ws, y = g.DeviceBuffer.from_numpy(x), g.DeviceBuffer.from_numpy(gamma), g.DeviceBuffer.from_numpy(resid), _ws(g, M, K), _out(g, M * N)
    g.check(lib.greta_cuda_gemv_batch(None, w.fmt, xd.ptr, None, 0.0, w.qs, w.d, None, y.ptr, M, N, K, 0, ws.ptr))
    got, want = y.download(np.float32).reshape(M, N), w.product(x)
    for m in range(M):
        assert max_abs_rel(got[m], want[m]) < TIGHT, m
    first = got.copy()
    g.check(lib.greta_cuda_gemv_batch(None, w.fmt, xd.ptr, None, 0.0, w.qs, w.d, None, y.ptr, M, N, K, 0, ws.ptr))
    assert np.array_equal(y.download(np.float32).reshape(M, N), first)  # whoever finishes a shared row tile adds in the same order
    g.check(lib.greta_cuda_gemv_batch(None, w.fmt, xd.ptr, gd.ptr, 1e-5, w.qs, w.d, rd.ptr, y.ptr, M, N, K, 0, ws.ptr))
    got, want = y.download(np.float32).reshape(M, N), w.product(O.rmsnorm(x, gamma, 1e-5)).astype(np.float64) + resid
    for m in range(M):
        assert max_abs_rel(got[m], want[m]) < TIGHT, m
    x[M // 2, 7] = np.inf  # stays in its row
    xd2 = g.DeviceBuffer.from_numpy(x)
    g.check(lib.greta_cuda_gemv_batch(None, w.fmt, xd2.ptr, None, 0.0, w.qs, w.d, None, y.ptr, M, N, K, 0, ws.ptr))
    got = y.download(np.float32).reshape(M, N)
    assert not np.isfinite(got[M // 2]).any()
    others = [m for m in range(M) if m != M // 2]
    assert np.array_equal(got[others], first[others])


# Whole pairs of row tiles, one or two to a CTA; pairs in parts that do not divide their K steps; equal runs; few rows above the line of their own.
@pytest.mark.parametrize("name", ["q4_0", "q8_0", "f16"])
@pytest.mark.parametrize("M,N,K", [(9, 23400, 512), (12, 40001, 544), (32, 5900, 2080), (16, 1700, 8192), (10, 24000, 1312), (5, 5300, 7232)])
def test_shares(g, name, M, N, K):
    lib, rng = g.cuda(), np.random.default_rng(M + N + K)
    w = _Weight(g, rng, name, N, K)
    assert lib.greta_cuda_gemv_batch_route(w.fmt, M, N, K) == 1
    x = rng.normal(0, 1, (M, K)).astype(np.float32)
    xd, ws, y = g.DeviceBuffer.from_numpy(x), _ws(g, M, K), _out(g, M * N)
    first = None
    for _ in range(3):
        g.check(lib.greta_cuda_gemv_batch(None, w.fmt, xd.ptr, None, 0.0, w.qs, w.d, None, y.ptr, M, N, K, 0, ws.ptr))
        got = y.download(np.float32).reshape(M, N)
        first = got.copy() if first is None else first
        assert np.array_equal(got, first)
    want = w.product(x)
    for m in range(M):
        assert max_abs_rel(got[m], want[m]) < TIGHT, m


@pytest.mark.parametrize("name", ["q4_0", "q8_0"])
@pytest.mark.parametrize("M,D,F", [(16, 1056, 1001), (32, 2080, 450), (8, 8192, 2100)])
def test_gate_and_up(g, name, M, D, F):
    lib, rng = g.cuda(), np.random.default_rng(M + D + F)
    w1, w3 = _Weight(g, rng, name, F, D), _Weight(g, rng, name, F, D)
    x, gamma = rng.normal(0, 1, (M, D)).astype(np.float32), rng.normal(1, 0.1, D).astype(np.float32)
    xd, gd, ws, y = g.DeviceBuffer.from_numpy(x), g.DeviceBuffer.from_numpy(gamma), _ws(g, M, D), _out(g, M * F)
    g.check(lib.greta_cuda_fused_ffn_front_batch(None, w1.fmt, xd.ptr, gd.ptr, 1e-5, w1.qs, w1.d, w3.qs, w3.d, y.ptr, M, D, F, ws.ptr))
    xn = O.rmsnorm(x, gamma, 1e-5)
    got, want = y.download(np.float32).reshape(M, F), O.silu_mul(w1.product(xn), w3.product(xn))
    for m in range(M):
        assert max_abs_rel(got[m], want[m]) < TIGHT, m


@pytest.mark.parametrize("name", ["q4_0", "q8_0"])
@pytest.mark.parametrize("M,H,Hkv,Dh,D", [(17, 5, 1, 64, 4128), (9, 3, 3, 128, 1056), (32, 16, 2, 128, 768)])
def test_queries_keys_and_values(g, name, M, H, Hkv, Dh, D):
    """Segments that end inside a tile of 128 rows; rotation and cache rows at every sequence's own position, one of them past the cache."""
    lib, rng = g.cuda(), np.random.default_rng(M + H)
    max_seq = 40
    pos = rng.integers(0, max_seq, M).astype(np.uint32)
    pos[1] = max_seq + 3
    wq, wk, wv = (_Weight(g, rng, name, n * Dh, D) for n in (H, Hkv, Hkv))
    x, gamma = rng.normal(0, 1, (M, D)).astype(np.float32), rng.normal(1, 0.1, D).astype(np.float32)
    xd, gd, pd, ws, q_out = g.DeviceBuffer.from_numpy(x), g.DeviceBuffer.from_numpy(gamma), g.DeviceBuffer.from_numpy(pos), _ws(g, M, D), _out(g, M * H * Dh)
    kc, vc = (g.DeviceBuffer(M * Hkv * max_seq * Dh * 2, zero=True) for _ in range(2))
    g.check(lib.greta_cuda_fused_rmsnorm_qkv_rope_kv_batch(None, wq.fmt, xd.ptr, gd.ptr, 1e-5, wq.qs, wq.d, wk.qs, wk.d, wv.qs, wv.d, q_out.ptr, None, None,
                                                           kc.ptr, vc.ptr, pd.ptr, M, H, Hkv, Dh, max_seq, 10000.0, D, ws.ptr))
    got_q = q_out.download(np.float32).reshape(M, H * Dh)
    got_k, got_v = (O.f16_bits_to_f32(c.download(np.uint16)).reshape(M, Hkv, max_seq, Dh) for c in (kc, vc))
    for m in range(M):
        xn = O.rmsnorm(x[m:m + 1], gamma, 1e-5)
        assert max_abs_rel(got_q[m], O.rope(wq.product(xn), 1, H, Dh, 10000.0, int(pos[m])).ravel()) < 5e-4
        if pos[m] >= max_seq:
            assert not got_k[m].any() and not got_v[m].any()
            continue
        assert max_abs_rel(got_k[m, :, pos[m]].ravel(), O.rope(wk.product(xn), 1, Hkv, Dh, 10000.0, int(pos[m])).ravel()) < 1e-3
        assert max_abs_rel(got_v[m, :, pos[m]].ravel(), wv.product(xn).ravel()) < 1e-3
        assert not np.delete(got_k[m], pos[m], axis=1).any() and not np.delete(got_v[m], pos[m], axis=1).any()
    k_out, v_out = _out(g, M * Hkv * Dh), _out(g, M * Hkv * Dh)
    g.check(lib.greta_cuda_fused_rmsnorm_qkv_rope_kv_batch(None, wq.fmt, xd.ptr, None, 0.0, wq.qs, wq.d, wk.qs, wk.d, wv.qs, wv.d, q_out.ptr, k_out.ptr, v_out.ptr,
                                                           None, None, None, M, H, Hkv, Dh, max_seq, 10000.0, D, ws.ptr))
    for buf, w in ((q_out, wq), (k_out, wk), (v_out, wv)):
        assert max_abs_rel(buf.download(np.float32).reshape(M, -1), w.product(x)) < TIGHT


def test_products_on_two_streams(g):
    """Each stream with a workspace of its own, captured into a graph on the second: the results of the default stream."""
    lib, rng, M, N, K = g.cuda(), np.random.default_rng(8), 16, 6000, 2080
    w = _Weight(g, rng, "q4_0", N, K)
    assert lib.greta_cuda_gemv_batch_route(w.fmt, M, N, K) == 1
    xd = g.DeviceBuffer.from_numpy(rng.normal(0, 1, (M, K)).astype(np.float32))
    call = lambda stream, ws, y: g.check(lib.greta_cuda_gemv_batch(stream, w.fmt, xd.ptr, None, 0.0, w.qs, w.d, None, y.ptr, M, N, K, 0, ws.ptr))
    ws, y = _ws(g, M, K), _out(g, M * N)
    call(None, ws, y)
    want = y.download(np.float32)
    streams, spaces, outs = [C.c_void_p(), C.c_void_p()], [_ws(g, M, K) for _ in range(2)], [_out(g, M * N) for _ in range(2)]
    graph, ready = C.c_void_p(), C.c_void_p()
    for s in streams:
        g.check(lib.greta_cuda_stream_create(C.byref(s)))
    g.check(lib.greta_cuda_device_synchronize())
    g.check(lib.greta_cuda_graph_capture_begin(streams[1]))
    call(streams[1], spaces[1], outs[1])
    g.check(lib.greta_cuda_graph_capture_end(streams[1], C.byref(graph)))
    g.check(lib.greta_cuda_graph_instantiate(graph, C.byref(ready)))
    for _ in range(8):
        call(streams[0], spaces[0], outs[0])
        g.check(lib.greta_cuda_graph_launch(ready, streams[1]))
    for s in streams:
        g.check(lib.greta_cuda_stream_synchronize(s))
    for o in outs:
        assert np.array_equal(o.download(np.float32), want)
    g.check(lib.greta_cuda_graph_exec_destroy(ready))
    g.check(lib.greta_cuda_graph_destroy(graph))
    for s in streams:
        g.check(lib.greta_cuda_stream_destroy(s))


def test_a_batch_reports_a_product_that_gave_up(g):
    """The code of a bounded wait that gave up is written by the host here; reading the ids fails with it, once."""
    pkg = load_package()
    cfg = dict(dim=1024, num_heads=8, num_heads_kv=4, num_layers=1, vocab=500, hidden_dim=2080, head_dim=128, max_seq=32, rope_base=1e4, rms_eps=1e-5)
    m = pkg.model.Model(cfg, weight_fmt=g.FMT_Q8_0, batch=2)
    m.load_synthetic(4)
    m.begin_decode(np.array([3, 4], np.int32), np.zeros(2, np.uint32))
    m.decode_step()
    g.check(g.cuda().greta_cuda_gemm_set_status(123))
    with pytest.raises(RuntimeError, match="gave up.*123"):
        m.read_generated(1)
    assert np.asarray(m.read_generated(1)).shape == (2, 1)
    m.close()


def _fmt(g, fmt):
    return g.FMT_Q4_0 if fmt == "q4_0" else g.FMT_Q8_0


@pytest.mark.parametrize("fmt", ["q4_0", "q8_0"])
@pytest.mark.parametrize("n", [2, 9, 17, 32])
def test_a_short_prompt_equals_its_tokens_one_by_one(g, fmt, n):
    """Prompts of 2 to 32 tokens take the batched products (tcgen05 from 9 rows on with 4-bit weights, always with 8-bit ones); a token at a time takes the
    single-row kernels.  Apart: fp32 sums in another order, then the fp16 cache of two layers.  A wait that gave up fails the prompt, once."""
    pkg = load_package()
    cfg = dict(dim=1024, num_heads=8, num_heads_kv=4, num_layers=2, vocab=1000, hidden_dim=2080, head_dim=128, max_seq=64, rope_base=1e4, rms_eps=1e-5)
    m = pkg.model.Model(cfg, weight_fmt=_fmt(g, fmt))
    m.load_synthetic(5)
    prompt = pkg.model.synth_tokens(5, 40, cfg["vocab"])
    for first in (0, 3):  # from the start of the sequence, and behind three tokens
        if first:
            m.forward(prompt[:first], 0)
        whole = np.array(m.forward(prompt[first:first + n], first))
        for i in range(first + n):
            one = np.array(m.forward(prompt[i:i + 1], i))
        assert np.linalg.norm(whole - one) < 2e-3 * np.linalg.norm(one)
    waits = n > 8 or fmt == "q8_0"
    assert bool(g.cuda().greta_cuda_gemv_batch_route(_fmt(g, fmt), n, 2 * cfg["hidden_dim"], cfg["dim"])) == waits
    if waits:
        g.check(g.cuda().greta_cuda_gemm_set_status(77))
        with pytest.raises(RuntimeError, match="gave up.*77"):
            m.forward(prompt[:n], 0)
        m.forward(prompt[:n], 0)
    m.close()
