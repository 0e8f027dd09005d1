"""Group scales: blocks whose dequantised range is a byte's take one multiply-add per four weights, others the 32-bit multiply and the bytewise add.  Ranges on
both sides of the line (15 s + (z ^ 128) = 255 and 256), products past a byte, and blocks of one kind beside blocks of the other: bit-exact against the oracle."""
import numpy as np
import pytest
import torch

from oracle import ops, w4a8
from tests.util import np_of, to_dev

pytestmark = pytest.mark.gpu


def _range(rng, groups, n, top):
    """s, z with 15 s + (z ^ 128) = top in every channel"""
    s = rng.integers(1, 18, (groups, n))
    up = top - 15 * s
    s, up = np.where((up < 0) | (up > 255), 1, s), np.where((up < 0) | (up > 255), top - 15, up)
    return s, up ^ 128


@pytest.mark.parametrize("kind", ["edge", "past", "one_past", "any"])
@pytest.mark.parametrize("M,N,K", [(7, 256, 896), (40, 128, 1024), (100, 384, 512), (513, 2048, 640)])
def test_ranges(dev, kind, M, N, K):
    import qserve_backend.qgemm_w4a8_per_group as op

    rng = np.random.default_rng(M + N + len(kind))
    groups = K // 128
    s, z = _range(rng, groups, N, 256 if kind == "past" else 255)
    if kind == "one_past":  # one channel of every other group, the others beside it on the line
        c = rng.integers(0, N, groups)
        sp, zp = _range(rng, groups, N, 256)
        for k in range(0, groups, 2):
            s[k, c[k]], z[k, c[k]] = sp[k, c[k]], zp[k, c[k]]
    if kind == "any":
        s, z = rng.integers(0, 256, (groups, N)), rng.integers(0, 256, (groups, N))
    s, z = (t.astype(np.uint8).view(np.int8) for t in (s, z))
    qw = rng.integers(-128, 128, (N, K // 2)).astype(np.int8)
    s1 = (rng.random(N) * 1e-3 + 1e-4).astype(np.float16)
    aq, sa, _ = ops.quant_per_token(rng.standard_normal((M, K)).astype(np.float16))
    out_o, acc_o = w4a8.gemm_w4a8_per_group(aq, qw, z, s, s1, sa, return_acc=True)
    out = torch.full((M, N), float("nan"), dtype=torch.half, device=dev)
    acc = torch.zeros((M, N), dtype=torch.int32, device=dev)
    op.gemm_forward_cuda(*(to_dev(t, dev) for t in (aq, qw, z, s, s1, sa)), out, _acc_out=acc)
    assert np.array_equal(np_of(acc), acc_o)
    assert np.array_equal(np_of(out).view(np.uint16), out_o.view(np.uint16))


@pytest.mark.parametrize("kind", ["edge", "past", "one_past"])
@pytest.mark.parametrize("M,N,K", [(393, 9728, 512), (192, 19200, 512)])
def test_ranges_over_rounds(dev, kind, M, N, K):
    """76 and 75 tiles of 256 tokens on 74 pairs: the kernel with warps of its own for the epilogue, which unpacks while they store."""
    test_ranges(dev, kind, M, N, K)
