"""Prefill attention over more than 512 keys (tcgen05) against float64."""
import ctypes as C

import numpy as np
import pytest

from _support import load_package

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    return load_package().ffi


@pytest.mark.parametrize("S,pos0,H,Hkv,Dh,gain", [(513, 0, 2, 2, 128, 1.0), (8, 505, 4, 1, 64, 1.0), (640, 0, 2, 1, 64, 1.0), (300, 467, 3, 3, 128, 1.0),
                                                  (16, 700, 4, 2, 128, 1.0), (769, 0, 2, 1, 128, 8.0), (128, 513, 1, 1, 64, 8.0), (1100, 0, 1, 1, 128, 1.0)])
def test_prefill_attention_above_512_keys(g, S, pos0, H, Hkv, Dh, gain):
    """Tile edges of queries and keys, rows behind the last key that are no numbers, maxima that grow from tile to tile (gain); fp16 output is the
    rounded fp32 output.  Tolerance: pairs of fp16 keep 22 bits of queries and probabilities, sums are cut at 24 bits up to 8 times per 128 keys."""
    rng = np.random.default_rng(S + Dh)
    n, ms = pos0 + S, pos0 + S + 9
    dev = lambda a: g.DeviceBuffer.from_numpy(np.ascontiguousarray(a))
    q = (rng.normal(0, gain, (S, H, Dh)) * np.linspace(0.2, 1, S)[:, None, None]).astype(np.float32)
    k, v = (rng.normal(0, 1, (Hkv, ms, Dh)).astype(np.float16) for _ in range(2))
    k *= np.linspace(0.1, 1, ms).astype(np.float16)[None, :, None]
    k[:, n:], v[:, n:] = np.nan, np.nan
    dq, dk, dv = dev(q), dev(k.view(np.uint16)), dev(v.view(np.uint16))
    o, o2, o16 = (dev(np.zeros((S, H, Dh), np.float32)) for _ in range(3))
    lib, scale, code = g.cuda(), Dh ** -0.5, C.c_int(-1)
    g.check(lib.greta_cuda_attn_prefill(None, dq.ptr, dk.ptr, dv.ptr, o.ptr, S, pos0, H, Hkv, Dh, ms, scale))
    g.check(lib.greta_cuda_attn_prefill_f16(None, dq.ptr, dk.ptr, dv.ptr, o16.ptr, o2.ptr, S, pos0, H, Hkv, Dh, ms, scale))
    g.check(lib.greta_cuda_gemm_segments_status(None, C.byref(code)))
    g.check(lib.greta_cuda_device_synchronize())
    assert code.value == 0
    got = o.download(np.float32).reshape(S, H, Dh)
    assert (o16.download(np.uint16)[:S * H * Dh] == got.astype(np.float16).view(np.uint16).reshape(-1)).all()
    hidden = np.arange(n)[None] > pos0 + np.arange(S)[:, None]
    for h in range(H):
        s = q[:, h].astype(np.float64) @ k[h // (H // Hkv), :n].astype(np.float64).T * scale
        s[hidden] = -np.inf
        w = np.exp(s - s.max(1, keepdims=True))
        want = (w / w.sum(1, keepdims=True)) @ v[h // (H // Hkv), :n].astype(np.float64)
        err = np.abs(got[:, h] - want).max() / want.std()
        assert err < 2e-5 * gain, err


@pytest.mark.parametrize("S,pos0,H,Hkv,Dh,at", [(700, 0, 2, 1, 128, (5, 130, 255, 256, 640)), (300, 467, 2, 2, 64, (470, 511, 512, 766)), (40, 600, 4, 2, 128, (10, 605, 639)),
                                                (130, 511, 1, 1, 64, (511, 512, 639, 640))])
def test_values_that_are_no_finite_numbers_reach_no_earlier_row(g, S, pos0, H, Hkv, Dh, at):
    """Infinities and NaNs in single columns of value rows `at`: rows in front of them are what they are with zeros there, up to the order of their
    sums (tolerance as above); so are, to the bit, the columns without any; the rows that see them are no finite numbers in those columns."""
    rng = np.random.default_rng(S + Dh)
    n, ms = pos0 + S, pos0 + S + 3
    q = rng.normal(0, 1, (S, H, Dh)).astype(np.float32)
    k, v = (rng.normal(0, 1, (Hkv, ms, Dh)).astype(np.float16) for _ in range(2))
    bad = np.zeros((Hkv, ms, Dh), bool)
    for i, j in enumerate(at):
        bad[i % Hkv, j, (7 * i) % Dh] = bad[Hkv - 1, j, Dh - 1 - i] = True
    clean, dirty = v.copy(), v.copy()
    clean[bad], dirty[bad] = 0, rng.choice(np.array([np.inf, -np.inf, np.nan], np.float16), int(bad.sum()))
    out = []
    for x in (clean, dirty):
        dq, dk, dv = (g.DeviceBuffer.from_numpy(np.ascontiguousarray(a)) for a in (q, k.view(np.uint16), x.view(np.uint16)))
        o = g.DeviceBuffer(S * H * Dh * 4)
        g.check(g.cuda().greta_cuda_attn_prefill(None, dq.ptr, dk.ptr, dv.ptr, o.ptr, S, pos0, H, Hkv, Dh, ms, Dh ** -0.5))
        g.check(g.cuda().greta_cuda_device_synchronize())
        out.append(o.download(np.float32).reshape(S, H, Dh))
    assert np.isfinite(out[0]).all()
    sees = np.stack([np.stack([bad[h // (H // Hkv), :pos0 + i + 1].any(0) for h in range(H)]) for i in range(S)])  # [S][H][Dh]
    assert not np.isfinite(out[1][sees]).any()
    spared = ~bad.any(1)[np.arange(H) // (H // Hkv)]  # [H][Dh]
    assert np.array_equal(out[1][:, spared], out[0][:, spared])
    assert np.abs(out[1] - out[0])[~sees].max() < 2e-5 * out[0].std()


@pytest.mark.parametrize("S,Dh,most", [(700, 128, 5.0e4), (530, 64, 6.5e4)])
def test_queries_near_the_end_of_fp16(g, S, Dh, most):
    """Queries whose largest |q * scale| is `most`, below 65504, against small keys.  Scores reach about 30: 22-bit queries leave weights 1e-5 open."""
    rng = np.random.default_rng(S)
    q, k = rng.normal(0, 1, (S, 1, Dh)).astype(np.float32), (rng.normal(0, 1, (S, Dh)) * 2.0 ** -14).astype(np.float16)
    v, scale = rng.normal(0, 1, (S, Dh)).astype(np.float16), Dh ** -0.5
    q = (q * (most / scale / np.abs(q).max())).astype(np.float32)
    dq, dk, dv = (g.DeviceBuffer.from_numpy(a) for a in (q, k.view(np.uint16), v.view(np.uint16)))
    o = g.DeviceBuffer(S * Dh * 4)
    g.check(g.cuda().greta_cuda_attn_prefill(None, dq.ptr, dk.ptr, dv.ptr, o.ptr, S, 0, 1, 1, Dh, S, scale))
    g.check(g.cuda().greta_cuda_device_synchronize())
    s = q[:, 0].astype(np.float64) @ k.astype(np.float64).T * scale
    assert 10 < np.abs(s).max() < 60
    s[np.arange(S)[None] > np.arange(S)[:, None]] = -np.inf
    w = np.exp(s - s.max(1, keepdims=True))
    want = (w / w.sum(1, keepdims=True)) @ v.astype(np.float64)
    assert np.abs(o.download(np.float32).reshape(S, Dh) - want).max() < 1e-4 * want.std()


def test_a_tile_of_scores_of_minus_infinity(g):
    """The first 150 keys score minus infinity (both halves of the split query have the sign for it): rows behind them attend to the rest."""
    S, Dh, rng = 600, 64, np.random.default_rng(1)
    q, k, v = rng.normal(0, 1, (S, 1, Dh)).astype(np.float32), rng.normal(0, 1, (S, Dh)).astype(np.float16), rng.normal(0, 1, (S, Dh)).astype(np.float16)
    scale = Dh ** -0.5
    first = next(x for x in np.linspace(1, 2, 99, dtype=np.float32) if (f := np.float32(x * np.float32(np.float32(scale) * np.float32(1.4426950408889634)))) > np.float32(np.float16(f)))
    q[:, 0, 0], k[:150, 0], k[150:, 0] = first, -np.inf, 0
    dq, dk, dv = (g.DeviceBuffer.from_numpy(a) for a in (q, k.view(np.uint16), v.view(np.uint16)))
    o = g.DeviceBuffer(S * Dh * 4)
    g.check(g.cuda().greta_cuda_attn_prefill(None, dq.ptr, dk.ptr, dv.ptr, o.ptr, S, 0, 1, 1, Dh, S, scale))
    g.check(g.cuda().greta_cuda_device_synchronize())
    s = q[150:, 0].astype(np.float64) @ k[150:].astype(np.float64).T * scale
    s[np.arange(S - 150)[None] > np.arange(S - 150)[:, None]] = -np.inf
    w = np.exp(s - s.max(1, keepdims=True))
    want = (w / w.sum(1, keepdims=True)) @ v[150:].astype(np.float64)
    assert np.abs(o.download(np.float32).reshape(S, Dh)[150:] - want).max() < 2e-5 * want.std()
