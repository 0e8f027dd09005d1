"""GPU parity of the context splits of the decode attention: the last CTA of a head group merges the splits' partial rows, one warp per head.
Sizes at the rule's edges: one split per 256 tokens at most, 32 splits at most, an even number of pages per split, sequences much shorter than
the longest one (splits without a page), more heads in a group than warps.  Bound as in test_gpu_attention.py: 3e-3 of the float64 attention
over the same cache."""
import numpy as np
import pytest

from oracle import kv
from tests.test_gpu_attention import ROPE, _check_pages, _mk, _run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("B,Hq,Hkv,lens", [
    (1, 4, 1, [513]),              # the shortest context that splits
    (1, 4, 1, [8200]),             # 32 splits of an even number of pages
    (3, 8, 2, [2049, 1, 640]),     # splits without pages
    (2, 16, 1, [1300, 1281]),      # two head groups of eight: two heads per merging warp
    (5, 10, 2, [1500, 64, 65, 900, 1472]),  # five heads: an uneven share per merging warp
])
def test_split_contexts(dev, bits, B, Hq, Hkv, lens):
    rng = np.random.default_rng(sum(lens) + bits)
    kp, vp, bt, q, k, v = _mk(rng, B, Hq, Hkv, lens, bits)
    out, k_gpu, v_gpu = _run_gpu(dev, kp, vp, bt, q, k, v, lens, bits)
    exact = kv.decode_attention(q, k, v, kp, vp, bt, lens, ROPE, faithful=False).astype(np.float32)
    _check_pages(kp, vp, k_gpu, v_gpu, bt, lens)
    got = out.astype(np.float32)
    assert np.isfinite(got).all()
    assert np.abs(got - exact).max() <= 3e-3 * max(1.0, float(np.abs(exact).max()))
