"""The chunked form of the delta rules' scan at the edges of its chunks, slices, column groups and head sizes, against float64."""
import ctypes as C

import numpy as np
import pytest

from _hybrid import O
from _latent import L
from _support import load_package

pytestmark = pytest.mark.gpu
# Sums of at most 128 rows and 16 tokens in fp32, and as many roundings of the operands: 288 x 2^-24 of the largest output.
TOL = 288 * 2.0 ** -24


@pytest.fixture(scope="module")
def g():
    return load_package().ffi


def dev(g, a):
    return g.DeviceBuffer.from_numpy(np.ascontiguousarray(a, np.float32))


def run(g, lib, gated, x, cuts, chunked, pad, state_bytes):
    """o of the tokens, portion by portion, through one of the two forms."""
    T, H, d = x["w"].shape
    V, G = x["v"].shape[2], x["k"].shape[1]
    rows = lambda a: a.reshape(T, -1)
    state = dev(g, np.full(state_bytes // 4, 1e3))
    got, pos = [], 0
    for n in cuts:
        part = lambda a: rows(a)[pos:pos + n]
        u = np.concatenate([part(x[c]) for c in (("r", "k", "v") if gated else ("r", "k", "v", "a"))] + [np.zeros((n, pad))], 1)
        ud, wd, ad, o = dev(g, u), dev(g, part(x["w"])), dev(g, part(x["a"])), g.DeviceBuffer(n * H * V * 4)
        at = lambda i: ud.ptr + 4 * i * H * d
        if gated:
            s = g.GatedDelta(H, G, d, V, 1, 1, 1, 1e-5, wd.ptr, 4, None, None, ad.ptr, H, None, state.ptr, None, 1, 1, None, None, None, None, ud.ptr,
                             u.shape[1], wd.ptr, None, H * d, H * V)
            need = lib.greta_cuda_gated_delta_scan_scratch_bytes(H, d, V, n)
            plain, through = lib.greta_cuda_gated_delta_scan, lib.greta_cuda_gated_delta_scan_chunked
        else:
            s = g.DeltaRule(H, d, 1, u.shape[1], 1e-5, at(0), at(1), at(2), at(3), None, wd.ptr, H * d, None, 1, None, None, None, state.ptr)
            need = lib.greta_cuda_delta_scan_scratch_bytes(H, d, n)
            plain, through = lib.greta_cuda_delta_scan, lib.greta_cuda_delta_scan_chunked
        r = g.Rows(n, 0, pos, None)
        if chunked:
            assert need > 0
            scratch = dev(g, np.full(need // 4, np.nan))
            g.check(through(None, C.byref(s), C.byref(r), o.ptr, scratch.ptr, need), "chunked")
        else:
            g.check(plain(None, C.byref(s), C.byref(r), o.ptr), "scan")
        g.check(lib.greta_cuda_device_synchronize(), "sync")
        got.append(o.download(np.float32, n * H * V).reshape(n, H, V))
        pos += n
    return np.concatenate(got)


def inputs(rng, T, H, G, d, V, gated):
    f = lambda *s: rng.normal(size=s).astype(np.float32)
    x = {"r": f(T, G, d), "k": f(T, G, d), "v": f(T, H, V), "w": np.exp(-0.6 * O.sigmoid(f(T, H, d) * 4)).astype(np.float32)}
    x["w"][7] = 0                                             # forgets everything: nothing may be divided by a decay
    x["w"][11:15] = 1
    if gated:
        x["r"] /= d ** 0.5 * np.linalg.norm(x["r"], axis=2, keepdims=True)
        x["k"] /= np.linalg.norm(x["k"], axis=2, keepdims=True)
        x["a"] = O.sigmoid(2 * f(T, H)).astype(np.float32)
    else:
        x["a"] = O.sigmoid(f(T, H, d)).astype(np.float32)
        x["k"][5] = 0
        x["k"][6] *= 1e-4
    return x


def want(x, gated):
    y = {k: v.astype(np.float64) for k, v in x.items()}
    return L.gated_scan(y["r"], y["k"], y["v"], y["w"], y["a"])[0] if gated else O.delta_scan(y["r"], y["k"], y["v"], y["w"], y["a"])[0]


# heads, query / key heads, head sizes, portions, floats behind a row (1: no row starts on 16 bytes)
CASES = [(False, 2, 2, 64, 64, [80, 97], 0), (False, 1, 1, 40, 40, [96, 81], 1), (False, 2, 2, 128, 128, [111], 0), (False, 1, 1, 97, 97, [80], 3),
         (False, 1, 1, 64, 64, [768, 768, 83], 4), (False, 1, 1, 33, 33, [1553], 0),
         (True, 2, 1, 128, 128, [95, 80], 0), (True, 3, 3, 64, 17, [83], 1), (True, 4, 2, 100, 56, [128, 80], 0), (True, 1, 1, 128, 256, [1544], 0),
         (True, 2, 2, 52, 200, [769], 0)]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_chunked_scan_is_as_exact_as_the_other(g, case):
    gated, H, G, d, V, cuts, pad = CASES[case]
    lib = g.cuda()
    x = inputs(np.random.default_rng(case), sum(cuts), H, G, d, V, gated)
    bytes_ = lib.greta_cuda_gated_delta_state_bytes(H, d, V) if gated else lib.greta_cuda_delta_state_bytes(H, d)
    w = want(x, gated)
    for chunked in (False, True):
        got = run(g, lib, gated, x, cuts, chunked, pad, bytes_)
        assert np.abs(got - w).max() <= TOL * np.abs(w).max(), (chunked, np.abs(got - w).max() / np.abs(w).max())


def test_tokens_in_front_of_a_nan_do_not_see_it(g):
    lib = g.cuda()
    x = inputs(np.random.default_rng(1), 96, 2, 2, 64, 64, False)
    clean = run(g, lib, False, x, [96], True, 0, lib.greta_cuda_delta_state_bytes(2, 64))
    x["v"][41, 0, 3] = x["k"][42, 1, 5] = np.nan
    got = run(g, lib, False, x, [96], True, 0, lib.greta_cuda_delta_state_bytes(2, 64))
    assert np.array_equal(got[:41, 0], clean[:41, 0]) and np.array_equal(got[:42, 1], clean[:42, 1])
    assert np.isnan(got[41:, 0, 3]).any() and np.array_equal(got[:, 0, :3], clean[:, 0, :3])


def test_sizes_without_the_chunked_form_ask_for_no_scratch(g):
    lib = g.cuda()
    assert lib.greta_cuda_delta_scan_scratch_bytes(2, 64, 79) == 0 and lib.greta_cuda_delta_scan_scratch_bytes(2, 32, 512) == 0
    assert lib.greta_cuda_delta_scan_scratch_bytes(2, 96, 512) == 0 and lib.greta_cuda_gated_delta_scan_scratch_bytes(2, 256, 64, 512) == 0
    assert lib.greta_cuda_delta_scan_scratch_bytes(2, 64, 4096) == lib.greta_cuda_delta_scan_scratch_bytes(2, 64, 1536)
