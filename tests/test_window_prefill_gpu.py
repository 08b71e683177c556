"""Windowed prefill attention where tiles of keys lie wholly inside what every row sees (the short path), beside those that do not: windows and kept
positions that end inside tiles, a ring that wraps inside a tile, distances beyond the table of logarithms, and every bucket of head sizes."""
import numpy as np
import pytest

from _support import load_package, max_abs_rel
from test_hybrid_gpu import Attn, attn_oracle, head_params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    pkg = load_package()
    pkg.build()
    pkg.ffi.require_device()
    return pkg.ffi


@pytest.mark.parametrize("H,G,dim,vdim,window,keep,cuts", [
    (4, 2, 64, 64, 200, 70, [500, 199]),       # kept positions end inside the second tile; the ring wraps in the second portion
    (2, 1, 128, 72, 321, 0, [330, 330]),
    (2, 2, 64, 40, 0, 0, [2200]),              # no window: distances beyond the table
    (1, 1, 136, 200, 2500, 3, [1300, 1203]),   # a window wider than the table
    (3, 1, 16, 16, 64, 64, [64, 65, 300])])
@pytest.mark.parametrize("bias", [True, False])
def test_tiles_inside_and_at_the_edges(g, H, G, dim, vdim, window, keep, cuts, bias):
    rng = np.random.default_rng(dim + window)
    T, p = sum(cuts), head_params(rng, H)
    if not bias:
        p = dict(p, r1=np.zeros(H, np.float32))
    raw = rng.normal(size=(T, (H + G) * dim + G * vdim)).astype(np.float32)
    want = attn_oracle(raw, H, G, dim, vdim, None, window, keep, 0.4, 6.0, p)
    at, pos, got = Attn(g, H, G, dim, vdim, 0, window, keep, T, max(cuts), 0.4, 6.0, p, None, "f16"), 0, []
    if not bias:
        at.a.r1 = at.a.r2 = None
    for n in cuts:
        got.append(at.portion(raw[pos:pos + n], pos, mma=True))
        pos += n
    assert max_abs_rel(np.concatenate(got), want) < 3e-3  # fp16 queries, keys, values and weights: as in test_hybrid_gpu
