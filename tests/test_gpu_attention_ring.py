"""GPU parity of the decode attention's rings over walks of many slices: enough sequences that no context is split, a few of them long, so that a warp runs
through its ring more than 32 slices and fetches its page pointers again (INT8: the keys' ahead of the values').  Bound as in test_gpu_attention.py: 3e-3
of the float64 attention over the same cache."""
import numpy as np
import pytest
import torch

from oracle import kv
from tests.test_gpu_attention import ROPE, _mk, _run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("long", [[4033, 4097], [4225, 8321], [8257, 4161]])
def test_walks_past_a_batch_of_pointers(dev, bits, long):
    rng = np.random.default_rng(sum(long) + bits)
    B, H = 38, 8  # 304 blocks: more than half of what the chip holds, so no splits
    lens = long + [int(n) for n in rng.integers(1, 200, B - len(long))]
    need = [(n + 63) // 64 for n in lens]
    kp, vp, bt, q, k, v = _mk(rng, B, H, H, lens, bits, pages=1 + sum(need))
    own = 1 + rng.permutation(sum(need))  # every sequence has pages of its own
    for b, n in enumerate(need):
        bt[b, :n] = own[sum(need[:b]):sum(need[:b]) + n]
    out, _, _ = _run_gpu(dev, kp, vp, bt, q, k, v, lens, bits)
    exact = kv.decode_attention(q, k, v, kp, vp, bt, lens, ROPE, faithful=False).astype(np.float32)
    got = out.astype(np.float32)
    assert np.isfinite(got).all()
    assert np.abs(got - exact).max() <= 3e-3 * max(1.0, float(np.abs(exact).max()))


@pytest.mark.parametrize("ctx", [1, 33, 64, 65, 190, 300, 512])
def test_whole_slices_and_halves(dev, ctx):
    """INT8 calls of up to three blocks per multiprocessor fetch whole slices, larger ones halves: the same sequences give the same bits in either."""
    rng = np.random.default_rng(ctx)
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    few, H = 5, 8
    many = 3 * sms // H + 1
    lens = ([ctx, 1, max(1, ctx - 63), ctx // 2 + 1, ctx] * (-(-many // few)))[:many]
    kp, vp, bt, q, k, v = _mk(rng, many, H, H, lens, 8, pages=1 + sum((n + 63) // 64 for n in lens))
    own, at = 1 + rng.permutation(sum((n + 63) // 64 for n in lens)), 0
    for b, n in enumerate(lens):
        bt[b, :(n + 63) // 64] = own[at:at + (n + 63) // 64]
        at += (n + 63) // 64
    halves, k1, v1 = _run_gpu(dev, kp, vp, bt, q, k, v, lens, 8)
    whole, _, _ = _run_gpu(dev, kp, vp, bt[:few], q[:few], k[:few], v[:few], lens[:few], 8)
    assert np.isfinite(halves.astype(np.float32)).all() and np.array_equal(whole.view(np.uint16), halves[:few].view(np.uint16))
