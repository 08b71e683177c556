"""Model-level parity: logits and greedy token ids of the C++ host layer (BlockScheduler / Generator
on the CUDA kernels) against the CPU oracle, on a small Llama-shaped model with seeded synthetic
weights.  Token ids must be identical; logits within the matmul tolerance."""
import ctypes as C

import numpy as np
import pytest

from _support import load_package, max_abs_rel
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SMALL = dict(dim=256, num_heads=4, num_heads_kv=2, num_layers=2, vocab=1000, hidden_dim=768, head_dim=64, max_seq=96,
             rope_base=10000.0, rms_eps=1e-5)
SMALL_MHA = dict(dim=512, num_heads=4, num_heads_kv=4, num_layers=3, vocab=2000, hidden_dim=1536, head_dim=128, max_seq=64,
                 rope_base=10000.0, rms_eps=1e-5)


@pytest.fixture(scope="module")
def pkg():
    p = load_package()
    p.build()
    p.ffi.require_device()
    return p


@pytest.mark.parametrize("cfg,fmt_name", [(SMALL, "q4_0"), (SMALL_MHA, "q4_0"), (SMALL, "q8_0")])
def test_logits_and_greedy_tokens_match_oracle(pkg, cfg, fmt_name):
    gfmt, ofmt = (pkg.ffi.FMT_Q4_0, O.FMT_Q4_0) if fmt_name == "q4_0" else (pkg.ffi.FMT_Q8_0, O.FMT_Q8_0)
    seed = 3
    weights = pkg.model.synth_weights(cfg, seed, gfmt)
    prompt = pkg.model.synth_tokens(seed, 20, cfg["vocab"])
    m = pkg.model.Model(cfg, weight_fmt=gfmt)
    m.load_synthetic(seed)
    ref = O.Model(cfg, weights, ofmt)

    # prefill (20 tokens: the GEMV route, x kept in fp32) then single-token steps
    lg = m.forward(prompt, 0)
    lo, xo = ref.forward(prompt, 0)
    assert max_abs_rel(m.hidden(len(prompt) - 1), xo) < 2e-5
    assert max_abs_rel(lg, lo) < 2e-5
    assert int(np.argmax(lg)) == O.argmax(lo)[0]
    tok = int(np.argmax(lg))
    for step in range(4):
        lg = m.forward(np.array([tok], np.int32), len(prompt) + step)
        lo, _ = ref.forward(np.array([tok], np.int32), len(prompt) + step)
        assert max_abs_rel(lg, lo) < 2e-5
        assert int(np.argmax(lg)) == O.argmax(lo)[0]
        tok = int(np.argmax(lg))
    m.close()


def test_generate_on_device_loop_matches_oracle(pkg):
    """Generator::generate_tokens: prefill + the graph-captured decode loop with device-side token
    feedback gives the oracle's greedy ids, step for step."""
    cfg, seed, n_new = SMALL, 5, 24
    weights = pkg.model.synth_weights(cfg, seed)
    prompt = pkg.model.synth_tokens(seed, 16, cfg["vocab"])
    m = pkg.model.Model(cfg)
    m.load(weights)                      # the explicit-tensor route (set_layer_tensor / set_global_tensor)
    ids, stats = m.generate(prompt, n_new)
    want, gaps = O.Model(cfg, weights).generate(prompt, n_new)
    assert min(gaps) > 1e-6, "a near-tie in the oracle's logits makes this seed unusable"
    assert ids == want
    assert stats["generated_tokens"] == n_new and stats["decode_ms"] > 0
    # a second generation on the same model (graph replay, cache overwritten) gives the same ids
    ids2, _ = m.generate(prompt, n_new)
    assert ids2 == want
    # and so does a model filled by load_synthetic (same bytes, generated inside the host layer)
    m2 = pkg.model.Model(cfg)
    m2.load_synthetic(seed)
    assert m2.generate(prompt, n_new)[0] == want
    m.close()
    m2.close()


def test_long_prompt_takes_the_tensor_core_route_and_matches_oracle(pkg):
    """A prompt of more than 32 tokens runs the projections through the tcgen05 GEMM (operands rounded to
    fp16, as the reference's M > 32 route does); logits and the following greedy ids equal the oracle's."""
    cfg, seed = SMALL_MHA, 11
    weights = pkg.model.synth_weights(cfg, seed)
    prompt = pkg.model.synth_tokens(seed, 45, cfg["vocab"])
    m = pkg.model.Model(cfg)
    m.load_synthetic(seed)
    ref = O.Model(cfg, weights)
    lg = m.forward(prompt, 0)
    lo, xo = ref.forward(prompt, 0)
    assert max_abs_rel(m.hidden(len(prompt) - 1), xo) < 1e-4
    assert max_abs_rel(lg, lo) < 1e-4
    ids, _ = m.generate(prompt, 12)
    want, gaps = ref.generate(prompt, 12)
    assert min(gaps) > 1e-5
    assert ids == want
    m.close()


@pytest.mark.parametrize("tokens,fmt_name", [(257, "q4_0"), (1531, "q8_0"), (3001, "q4_0")])
def test_whole_prompts_give_the_same_bits_every_time(pkg, tokens, fmt_name):
    """One prompt on one model and on a fresh one, kernels started ahead of their predecessor's end and not (greta_cuda_set_pdl): hidden rows and logits
    are the same bits.  The feed-forward products of the longer prompts are up to 25 tiles per CTA, so every ring in them is reused many times."""
    cfg = dict(dim=2048, num_heads=16, num_heads_kv=4, num_layers=2, vocab=1000, hidden_dim=14336, head_dim=128, max_seq=tokens, rope_base=500000.0, rms_eps=1e-5)
    gfmt = pkg.ffi.FMT_Q4_0 if fmt_name == "q4_0" else pkg.ffi.FMT_Q8_0
    prompt = pkg.model.synth_tokens(17, tokens, cfg["vocab"])
    lib, first = pkg.ffi.cuda(), None
    try:
        for _ in range(2):
            m = pkg.model.Model(cfg, weight_fmt=gfmt)
            m.load_synthetic(17)
            for pdl in (0, 1, 1, 1):
                pkg.ffi.check(lib.greta_cuda_set_pdl(pdl))
                got = [m.forward(prompt, 0), np.stack([m.hidden(i) for i in range(tokens)])]
                first = first or got
                for a, b in zip(first, got):
                    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (pdl, int((a != b).any(-1).sum()))
            m.close()
    finally:
        lib.greta_cuda_set_pdl(1)


def test_prompt_buffers_are_those_that_the_route_uses(pkg):
    """The feed-forward's fp32 `up` rows and the products' workspace belong to routes that a long prompt does not take: only `gate` is held for every row."""
    pkg.ffi.cuda()
    cudart = C.CDLL("libcudart.so.12")   # the one that the library is linked to

    def free_bytes():
        free, total = C.c_size_t(), C.c_size_t()
        assert cudart.cudaMemGetInfo(C.byref(free), C.byref(total)) == 0
        return free.value

    cfg = dict(SMALL, hidden_dim=8192, max_seq=8192)
    S, D, ql, kvl = cfg["max_seq"], cfg["dim"], 256, 128
    pkg.model.Model(cfg).close()         # what the process holds once
    before = free_bytes()
    m = pkg.model.Model(cfg)
    held = before - free_bytes()
    weights = 2 * (2 * D * ql + 2 * D * kvl + 3 * D * cfg["hidden_dim"]) * 18 // 32 + 4 * cfg["vocab"] * D
    rows = 4 * S * (cfg["hidden_dim"] + 2 * D + 2 * ql + 2 * kvl) + 2 * 2 * S * kvl * 2
    assert held < weights + rows + (100 << 20), held   # 100 MB: allocation granularity and small buffers; `up` alone would be 268
    m.close()


def test_forward_reports_a_product_that_gave_up(pkg):
    """A bounded wait that gave up in a prompt's products leaves a code on the device; forward() fails with it, once, and the next prompt is as before.
    The code is written by the host here."""
    lib, code = pkg.ffi.cuda(), C.c_int(-1)
    m = pkg.model.Model(SMALL)
    m.load_synthetic(4)
    prompt = pkg.model.synth_tokens(4, 40, SMALL["vocab"])
    first = m.forward(prompt, 0)
    pkg.ffi.check(lib.greta_cuda_gemm_set_status(123))
    assert lib.greta_cuda_gemm_status(C.byref(code)) == 0 and code.value == 123
    m.forward(prompt[:32], 0)                            # no product of that kind in it
    with pytest.raises(RuntimeError, match="gave up.*123"):
        m.forward(prompt, 0)
    assert lib.greta_cuda_gemm_status(C.byref(code)) == 0 and code.value == 0
    assert np.array_equal(m.forward(prompt, 0), first)
    m.close()


@pytest.mark.parametrize("chunks", [(40, 40), (40, 10), (12, 45, 3)])
def test_chunked_prefill_attends_to_the_cache(pkg, chunks):
    """A prompt fed in several forward() calls: every chunk after the first starts at pos0 > 0, its queries attend to
    the cache rows of the earlier chunks (tensor-core route for chunks of more than 32 tokens, GEMV route below).
    Logits after the last chunk and the greedy ids that follow equal the oracle's on the whole prompt."""
    cfg, seed = SMALL, 21
    weights = pkg.model.synth_weights(cfg, seed)
    prompt = pkg.model.synth_tokens(seed, sum(chunks), cfg["vocab"])
    m = pkg.model.Model(cfg)
    m.load_synthetic(seed)
    ref = O.Model(cfg, weights)
    pos = 0
    for n in chunks:
        lg = m.forward(prompt[pos:pos + n], pos)
        pos += n
    lo, xo = ref.forward(prompt, 0)
    assert max_abs_rel(m.hidden(chunks[-1] - 1), xo) < 1e-4
    assert max_abs_rel(lg, lo) < 1e-4
    tok = int(np.argmax(lg))
    assert tok == O.argmax(lo)[0]
    m.begin_decode(tok, pos)
    for _ in range(6):
        m.decode_step()
    got = m.read_generated(6)
    want, gaps = ref.generate(prompt, 7)
    assert min(gaps) > 1e-5
    assert [tok] + got == want
    m.close()


def test_decode_loop_is_refused_past_the_cache(pkg):
    """The device-side loop advances the position by itself: the host refuses the step that would read or write a
    cache row that does not exist, and generation requests that cannot fit are refused up front."""
    cfg = dict(SMALL, max_seq=24)
    prompt = pkg.model.synth_tokens(2, 20, cfg["vocab"])
    m = pkg.model.Model(cfg)
    m.load_synthetic(2)
    tok = int(np.argmax(m.forward(prompt, 0)))
    m.begin_decode(tok, 20)
    for _ in range(4):                       # positions 20..23 exist
        m.decode_step()
    with pytest.raises(pkg.ffi.GretaError, match="exceeds max_seq_len"):
        m.decode_step()                      # position 24 does not
    assert len(m.read_generated(4)) == 4
    with pytest.raises(pkg.ffi.GretaError, match="exceeds max_seq_len"):
        m.generate(prompt, 6)                # 20 + 5 decode steps do not fit in 24 rows
    assert len(m.generate(prompt, 5)[0]) == 5
    with pytest.raises(pkg.ffi.GretaError):
        m.begin_decode(tok, 24)
    m.close()


def test_generation_stops_at_the_end_of_sequence_id(pkg):
    """generate_tokens ends with the first end-of-sequence id it samples (the reference's loop breaks on its
    tokenizer's id); the ids before it are the ones an unbounded run produces."""
    cfg, seed = SMALL, 5
    prompt = pkg.model.synth_tokens(seed, 16, cfg["vocab"])
    m = pkg.model.Model(cfg)
    m.load_synthetic(seed)
    full, _ = m.generate(prompt, 40)
    for stop_at in (0, 7, 17, 33):           # inside the first chunk of the device loop, on a chunk boundary, later
        eos = full[stop_at]
        first = full.index(eos)
        assert m.generate_until(prompt, 40, eos) == full[:first + 1]
    assert m.generate_until(prompt, 40, cfg["vocab"] + 5) == full      # an id that never comes: runs to max_tokens
    m.close()


@pytest.mark.parametrize("cfg,batch", [(SMALL, 5), (SMALL_MHA, 3), (SMALL, 16)])
def test_batched_decode_matches_the_oracle_sequence_by_sequence(pkg, cfg, batch):
    """A batch of sequences decoding in step (weights streamed once per step for all of them): every sequence's greedy ids
    equal the oracle's for that sequence alone.  Prompts of different lengths, so every sequence sits at its own position."""
    seed, n_new = 31, 10
    weights = pkg.model.synth_weights(cfg, seed)
    ref = O.Model(cfg, weights)
    lens = [8 + 3 * (b % 5) for b in range(batch)]
    prompts = [pkg.model.synth_tokens(seed, lens[b], cfg["vocab"], stream=(1 << 40) + b) for b in range(batch)]
    m = pkg.model.Model(cfg, batch=batch)
    m.load_synthetic(seed)
    first = []
    for b in range(batch):                       # prefill, one sequence at a time
        m.set_sequence(b)
        first.append(int(np.argmax(m.forward(prompts[b], 0))))
    m.begin_decode(first, lens)
    for _ in range(n_new - 1):
        m.decode_step()
    got = m.read_generated(n_new - 1)
    for b in range(batch):
        want, gaps = ref.generate(prompts[b], n_new)
        assert min(gaps) > 1e-6
        assert [first[b]] + got[b].tolist() == want, b
    # the host-driven loop (ids up and down every step) gives the same ids
    ids, _ = m.decode_e2e(first, lens, n_new - 1)
    assert np.array_equal(ids, got)
    m.close()


def test_batched_70b_shape_ids_equal_the_stored_oracle_ids(pkg):
    """The tensor-parallel scaling workload's shape (hidden 8192, 64 / 8 heads of 128, FFN 28672, vocab 128256, rope base
    500000) at 2 layers, 16 sequences with their own 48-token prompts, 8 greedy ids each: equal to the oracle's ids stored
    in tests/golden/model_ids.npz (tests/golden/make_model_ids.py)."""
    import os
    from _support import ROOT
    from gretacore_v3_b200.model import LLAMA3_70B
    gold = np.load(os.path.join(ROOT, "tests", "golden", "model_ids.npz"))
    name = "llama3_70b_l2_seed4_b16"
    want, gaps, prompts, seed = gold[name + ".ids"], gold[name + ".gaps"], gold[name + ".prompts"], int(gold[name + ".seed"])
    cfg = dict(LLAMA3_70B, num_layers=2, max_seq=64)
    assert [cfg[k] for k in ("dim", "num_heads", "num_heads_kv", "num_layers", "vocab", "hidden_dim", "head_dim", "max_seq")] == list(gold[name + ".shape"])
    B = want.shape[0]
    for b in range(B):
        assert np.array_equal(prompts[b], pkg.model.synth_tokens(seed, prompts.shape[1], cfg["vocab"], stream=(1 << 40) + b))
    m = pkg.model.Model(cfg, batch=B)
    m.load_synthetic(seed)
    ids = m.generate_batch(prompts, want.shape[1])
    m.close()
    bad = [(b, int(np.argmax(ids[b] != want[b]))) for b in range(B) if not np.array_equal(ids[b], want[b])]
    print(f"70B shape x 2 layers, batch {B}: smallest top-2 logit gap of the oracle {gaps.min():.3e}; sequences that differ: {bad}")
    assert not bad


def test_persistent_decode_step_gives_the_same_ids(pkg, monkeypatch):
    """GRETA_PERSISTENT_STEP=1: all layers of a decode step in one persistent kernel (grid barriers between the
    phases) - same greedy ids as the oracle and as the operator-by-operator graph."""
    cfg, seed, n_new = SMALL_MHA, 13, 20
    weights = pkg.model.synth_weights(cfg, seed)
    prompt = pkg.model.synth_tokens(seed, 18, cfg["vocab"])
    want, gaps = O.Model(cfg, weights).generate(prompt, n_new)
    assert min(gaps) > 1e-6
    monkeypatch.setenv("GRETA_PERSISTENT_STEP", "1")
    m = pkg.model.Model(cfg)
    m.load_synthetic(seed)
    assert m.generate(prompt, n_new)[0] == want
    assert m.generate(prompt, n_new)[0] == want      # barrier generation counter carries over between launches
    m.close()
    monkeypatch.setenv("GRETA_PERSISTENT_STEP", "0")
    m = pkg.model.Model(cfg)
    m.load_synthetic(seed)
    assert m.generate(prompt, n_new)[0] == want
    m.close()


def test_forward_rejects_bad_ranges(pkg):
    m = pkg.model.Model(SMALL)
    m.load_synthetic(1)
    with pytest.raises(pkg.ffi.GretaError):
        m.forward(np.zeros(SMALL["max_seq"] + 1, np.int32), 0)
    with pytest.raises(pkg.ffi.GretaError):
        m.forward(np.zeros(4, np.int32), SMALL["max_seq"] - 2)
    m.close()
