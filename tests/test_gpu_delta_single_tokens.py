"""The delta rule over a step of single tokens, whose convolution shifts each sequence's state while it reads it, against the same tokens in a step that also has
a longer run and leaves the states to a kernel of their own: the same bits of outputs, recurrent states and convolution states, for heads that fill a warp's
lanes and heads that do not, every number of taps with a walk of its own and others, and sequences younger than the convolution."""
import pytest
import torch

from .test_gpu_long_runs import BF, F32, GatedDelta

pytestmark = pytest.mark.gpu
POS0 = [0, 1, 2, 3, 9, 40]


@pytest.mark.parametrize("dtype", [BF, F32])
@pytest.mark.parametrize("taps", [2, 3, 4, 6])
@pytest.mark.parametrize("H,G,D,Dv", [(4, 2, 128, 128), (4, 1, 96, 64), (2, 2, 128, 40), (3, 1, 36, 132)])
def test_bits_of_a_step_with_a_run(dtype, taps, H, G, D, Dv):
    n, got = len(POS0), []
    for more in (0, 1):
        layer = GatedDelta(5, dtype, n + 1, H, G, D, Dv)
        layer.taps, layer.conv_w, layer.conv = taps, layer.rand(layer.C, taps) * 0.5, layer.rand(n + 1, taps - 1, layer.C)
        slots = list(range(n + 1))[::-1]
        for slot, pos in zip(slots, POS0):
            layer.conv[slot, :max(0, taps - 1 - pos)] = 0.0  # ahead of the sequence
        proj = layer.rand(n + 2, layer.W).to(dtype)
        lens, pos0 = [1] * n + [2] * more, POS0 + [5] * more
        prep, _, out = layer.step(proj[:sum(lens)], lens, pos0, slots[:n + more])
        used = slots[:n]
        got.append((prep[:n], out[:n], layer.state[used], layer.conv[used]))
        assert torch.isfinite(prep[:n]).all()
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n", [511, 512, 515, 700, 2049])
def test_bits_of_walks_over_several_sequences(n):
    """From 512 tokens on a lane walks several of them, from 2048 on 16: tokens of different sequences, each of which shifts a state of its own."""
    got = []
    for more in (0, 1):
        layer = GatedDelta(6, BF, n + 1, 2, 1, 32, 40)
        layer.conv = layer.rand(n + 1, 3, layer.C)
        slots, pos = list(range(n + 1))[::-1], [(7 * i) % 11 for i in range(n)]
        for slot, a in zip(slots, pos):
            layer.conv[slot, :max(0, 3 - a)] = 0.0  # ahead of the sequence
        proj = layer.rand(n + 2, layer.W).to(BF)
        prep, _, out = layer.step(proj[:n + 2 * more], [1] * n + [2] * more, pos + [5] * more, slots[:n + more])
        used = slots[:n]
        got.append((prep[:n], out[:n], layer.state[used], layer.conv[used]))
        assert torch.isfinite(prep[:n]).all()
    for a, b in zip(*got):
        assert torch.equal(a, b)
