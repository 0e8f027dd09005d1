"""GPU parity of the context splits of the decode attention: the last CTA of a head group merges the splits' partial rows, one warp per head.
Sizes at the rule's edges: one split per 256 tokens at most, 32 splits at most, sequences much shorter than the longest one (splits without a page),
more heads in a group than warps.  Bound as in test_gpu_attention.py: 3e-3 of the float64 attention
over the same cache."""
import numpy as np
import pytest
import torch

from oracle import kv
from tests.test_gpu_attention import ROPE, _check_pages, _mk, _run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("B,Hq,Hkv,lens", [
    (1, 4, 1, [513]),              # the shortest context that splits
    (1, 4, 1, [8200]),             # 32 splits
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


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("B,Hq,Hkv,ctx", [(1, 4, 1, 513), (4, 32, 8, 8000), (3, 8, 2, 2049), (5, 32, 8, 6000), (9, 32, 8, 4000), (2, 16, 1, 3000), (28, 8, 8, 1100), (37, 8, 8, 1100),
                                          (38, 8, 8, 1100), (1, 8, 8, 512)])
def test_splits_fill_the_machine(dev, bits, B, Hq, Hkv, ctx):
    """How far a warp walks bounds how much the V product loses: its accumulator holds 1024 times the weights' sum beside the codes, and every 16-token
    step rounds the whole of it.  So the number of splits is part of the result's precision: what fills four blocks per multiprocessor, rounded up, for
    both page formats, and no fewer.  The partial rows that the splits leave in the work space tell it."""
    from qserve_b200 import backend as b

    rng = np.random.default_rng(B + ctx)
    lens = [ctx] + [int(n) for n in rng.integers(1, ctx + 1, B - 1)]
    ws = b.attention_workspace(dev, B, Hq, 128)
    rows = ws[256 * 1024:256 * 1024 + B * Hq * 32 * 130 * 4].view(torch.float32)  # behind the counters: [sequence][head][split][130]
    rows.fill_(float("nan"))
    kp, vp, bt, q, k, v = _mk(rng, B, Hq, Hkv, lens, bits, pages=64)  # the sequences share pages: only the splits' number matters here
    _run_gpu(dev, kp, vp, bt, q, k, v, lens, bits)
    assert b.attention_workspace(dev, B, Hq, 128).data_ptr() == ws.data_ptr()
    blocks = B * Hkv * -(-(Hq // Hkv) // 8)
    slots = 4 * torch.cuda.get_device_properties(dev).multi_processor_count
    want = min(32, -(-ctx // 256), -(-slots // blocks)) if 2 * blocks <= slots and ctx > 512 else 0
    assert int((~rows.isnan()).sum()) == B * Hq * want * 130


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("lens", [[2049, 1980, 1700, 1500, 1100, 650, 300, 70, 1], [4097, 4000, 3300, 2900, 2500, 2100], [8193, 7000, 6500, 6000]])
def test_every_number_of_splits_with_pages(dev, bits, lens):
    """The merge takes eight splits' rows at a time: sequences of one call that leave it one to nine, 11 to 17 and 23 to 32 of them."""
    rng = np.random.default_rng(sum(lens) + bits)
    B, Hq, Hkv = len(lens), 4, 1
    kp, vp, bt, q, k, v = _mk(rng, B, Hq, Hkv, lens, bits)
    out, _, _ = _run_gpu(dev, kp, vp, bt, q, k, v, lens, bits)
    exact = kv.decode_attention(q, k, v, kp, vp, bt, lens, ROPE, faithful=False).astype(np.float32)
    got = out.astype(np.float32)
    assert np.isfinite(got).all()
    assert np.abs(got - exact).max() <= 3e-3 * max(1.0, float(np.abs(exact).max()))
