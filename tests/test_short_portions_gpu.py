"""Portions of 8 to 32 tokens that end behind 512 positions: their attention is the one on tcgen05, whose waits are bounded, while the products of a model
this small have no such waits.  And what a batch's steps leave to be read besides their ids."""
import numpy as np
import pytest

from _support import load_package

pytestmark = pytest.mark.gpu


def _cfg(**kw):
    return dict(dict(dim=512, num_heads=8, num_heads_kv=4, num_layers=2, vocab=1000, hidden_dim=1056, head_dim=64, max_seq=600, rope_base=1e4, rms_eps=1e-5), **kw)


@pytest.mark.parametrize("first,n", [(505, 8), (520, 17), (568, 32)])
def test_a_short_portion_behind_512_positions(first, n):
    """Equals its tokens one by one (fp32 sums in another order, then the fp16 cache of two layers); a code that a wait left, written by the host here, fails
    the call, once."""
    pkg = load_package()
    g, cfg = pkg.ffi, _cfg()
    fmt = g.FMT_Q4_0
    assert g.cuda().greta_cuda_attn_prefill_route(n, first, 64) == 1
    assert not any(g.cuda().greta_cuda_gemv_batch_route(fmt, n, rows, k) for rows, k in ((1024, 512), (512, 512), (2112, 512), (512, 1056)))
    m = pkg.model.Model(cfg, weight_fmt=fmt)
    m.load_synthetic(6)
    prompt = pkg.model.synth_tokens(6, 600, cfg["vocab"])
    m.forward(prompt[:first], 0)
    whole = np.array(m.forward(prompt[first:first + n], first))
    for i in range(first, first + n):
        one = np.array(m.forward(prompt[i:i + 1], i))
    assert np.linalg.norm(whole - one) < 2e-3 * np.linalg.norm(one)
    g.check(g.cuda().greta_cuda_gemm_set_status(55))
    with pytest.raises(RuntimeError, match="gave up.*55"):
        m.forward(prompt[first:first + n], first)
    assert np.array_equal(m.forward(prompt[first:first + n], first), whole)
    m.close()


@pytest.mark.parametrize("read", ["logits", "hidden", "sample"])
def test_what_a_batch_leaves_is_asked_for(read):
    pkg = load_package()
    g, cfg = pkg.ffi, _cfg(dim=1024, num_heads=16, hidden_dim=2080, max_seq=32)
    m = pkg.model.Model(cfg, weight_fmt=g.FMT_Q8_0, batch=2)
    m.load_synthetic(4)
    out = np.empty(cfg["vocab"], np.float32)

    def ask():
        if read == "logits":
            return m.h.greta_model_get_logits(m.handle, out.ctypes.data, out.size)
        if read == "hidden":
            return m.h.greta_model_get_hidden(m.handle, out.ctypes.data, 0, 500)
        return m.h.greta_model_sample_greedy(m.handle, out.ctypes.data)

    m.begin_decode(np.array([3, 4], np.int32), np.zeros(2, np.uint32))
    m.decode_step()
    assert ask() == 0
    m.decode_step()
    g.check(g.cuda().greta_cuda_gemm_set_status(66))
    assert ask() != 0 and b"gave up" in m.h.greta_host_last_error()
    assert ask() == 0
    m.close()


def test_a_host_driven_batch_brings_the_code_with_its_ids():
    pkg = load_package()
    g, cfg = pkg.ffi, _cfg(dim=1024, num_heads=16, hidden_dim=2080, max_seq=32)
    m = pkg.model.Model(cfg, weight_fmt=g.FMT_Q8_0, batch=5)
    m.load_synthetic(4)
    first, pos = np.arange(5, dtype=np.int32), np.zeros(5, np.uint32)
    ids, _ = m.decode_e2e(first, pos, 6)
    m.begin_decode(first, pos)
    for _ in range(6):
        m.decode_step()
    assert np.array_equal(ids, m.read_generated(6))
    g.check(g.cuda().greta_cuda_gemm_set_status(88))
    with pytest.raises(RuntimeError, match="gave up.*88"):
        m.decode_e2e(first, pos, 1)
    assert np.array_equal(m.decode_e2e(first, pos, 6)[0], ids)
    m.close()
