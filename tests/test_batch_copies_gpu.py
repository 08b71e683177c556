"""The batched matmul on prepared activations waits for the activations of a cell as well as for its weights: with the caches cold and few rows,
cells are multiplied faster than the next cell's activations arrive."""
import numpy as np
import pytest

from _support import load_package, make_blocks
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(8, 32000, 4096), (1, 32000, 2048), (16, 32000, 4096)])
def test_activations_have_landed_before_they_are_read(M, N, K):
    g = load_package().ffi
    lib, rng = g.cuda(), np.random.default_rng(M)
    w = (rng.standard_normal((N, K), dtype=np.float32) * 0.02).astype(np.float16)
    rows = np.arange(0, N, 97)
    flush = g.DeviceBuffer(256 << 20)
    dw, y = g.DeviceBuffer.from_numpy(w.view(np.uint16)), g.DeviceBuffer(M * N * 4)
    ws = g.DeviceBuffer(lib.greta_cuda_gemv_batch_workspace_bytes(M, K))
    for i in range(4):                                        # other activations each time: what lay there before does not do
        x = rng.standard_normal((M, K), dtype=np.float32)
        dx = g.DeviceBuffer.from_numpy(x)
        flush.fill(i)
        g.check(lib.greta_cuda_gemv_batch(None, g.FMT_F16, dx.ptr, None, 0.0, dw.ptr, None, None, y.ptr, M, N, K, 0, ws.ptr))
        g.check(lib.greta_cuda_device_synchronize())
        want = x.astype(np.float64) @ w[rows].astype(np.float64).T
        got = y.download(np.float32).reshape(M, N)[:, rows]
        # K products of exact weights and 22-bit activations, summed in fp32 over at most 128 blocks and 8 slices
        assert np.abs(got - want).max() < 2e-5 * np.abs(want).max(), i
    for b in (flush, dw, y, ws):
        b.free()


# The products above go through tcgen05; these take the kernel whose copies the wait is for: slices forced, or sizes whose route says so.  Formats and row counts
# differ in the depth of its rings.
@pytest.mark.parametrize("M,N,K,slices", [(8, 16000, 4096, 1), (16, 16000, 4096, 2), (24, 8000, 4096, 1), (3, 8000, 4096, 8), (16, 8000, 2048, 4), (8, 7000, 4096, 0)])
@pytest.mark.parametrize("fmt", ["f16", "q4_0", "q8_0"])
def test_the_same_without_tcgen05(fmt, M, N, K, slices):
    g = load_package().ffi
    lib, rng = g.cuda(), np.random.default_rng(M + slices)
    if fmt == "f16":
        w = (rng.standard_normal((N, K), dtype=np.float32) * 0.02).astype(np.float16)
        held, code, product = g.DeviceBuffer.from_numpy(w.view(np.uint16)), g.FMT_F16, lambda x: x.astype(np.float64) @ w[::97].astype(np.float64).T
        qs, d = held.ptr, None
    else:
        code, ofmt = (g.FMT_Q4_0, O.FMT_Q4_0) if fmt == "q4_0" else (g.FMT_Q8_0, O.FMT_Q8_0)
        blocks = make_blocks(rng, ofmt, N, K)
        few = np.ascontiguousarray(blocks.reshape(N, -1)[::97]).reshape(-1)
        held, product = g.Weight(blocks, code, N, K), lambda x: O.gemv(x, few, ofmt, len(range(0, N, 97)), K)
        qs, d = held.qs.ptr, held.d.ptr
    if not slices and lib.greta_cuda_gemv_batch_route(code, M, N, K):
        pytest.skip("this format takes tcgen05 here")
    flush, y = g.DeviceBuffer(256 << 20), g.DeviceBuffer(M * N * 4)
    ws = g.DeviceBuffer(lib.greta_cuda_gemv_batch_workspace_bytes(M, K))
    for i in range(4):
        x = rng.standard_normal((M, K), dtype=np.float32)
        dx = g.DeviceBuffer.from_numpy(x)
        flush.fill(i)
        g.check(lib.greta_cuda_gemv_batch(None, code, dx.ptr, None, 0.0, qs, d, None, y.ptr, M, N, K, slices, ws.ptr))
        g.check(lib.greta_cuda_device_synchronize())
        got, want = y.download(np.float32).reshape(M, N)[:, ::97], product(x)
        assert np.abs(got - want).max() < 2e-5 * np.abs(want).max(), i
