"""GPU parity of the decode attention's rings over walks of many slices: enough sequences that no context is split, a few of them long, so that a warp runs
through its ring more than 32 slices and fetches its page pointers again (INT8: the keys' ahead of the values').  Bound as in test_gpu_attention.py: 3e-3
of the float64 attention over the same cache."""
import numpy as np
import pytest

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
