"""Tiles of CTA pairs with 128 to 256 tokens: what the tile's tokens are follows the number of rounds, the result does not.  Against the same rows in pieces
of at most 100 or 64 tokens, which take the single-CTA tiles: the same bits, for the sizes that calls with short K get (per channel 128, 192 and 256 tokens,
group scales 256, W8A8 160 and 256; every size in test_gpu_gemm.py), ragged last tiles, one and several tiles per pair, and where pairs begin."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["chn", "grp", "w8"])
@pytest.mark.parametrize("M,N", [(512, 4096), (600, 4096), (700, 4096), (890, 4096), (1000, 4096), (2500, 4096), (130, 28672), (200, 28672), (250, 28672), (1301, 6144), (4500, 4096)])
def test_bits_of_small_tiles(dev, mode, M, N):
    same_bits_in_pieces(dev, mode, M, N, 640 if mode != "chn" else 512, 100)


@pytest.mark.parametrize("mode", ["chn", "grp", "w8"])
@pytest.mark.parametrize(
    "M,N,K", [(64, 9728, 2048), (65, 9728, 2048), (96, 9728, 2048), (128, 18688, 2176), (65, 9472, 2048), (129, 4096, 1024), (257, 2560, 640), (257, 4096, 2048), (300, 12288, 1024),
              (512, 2048, 8064), (512, 2048, 8192), (520, 512, 1024), (1100, 4096, 1024), (2048, 256, 2048)])
def test_bits_where_pairs_take_over(dev, mode, M, N, K):
    same_bits_in_pieces(dev, mode, M, N, K, 64)


def same_bits_in_pieces(dev, mode, M, N, K, most):
    import qserve_backend.qgemm_w4a8_per_chn as chn
    import qserve_backend.qgemm_w4a8_per_group as grp
    import qserve_backend.qgemm_w8a8 as w8

    g = torch.Generator(device=dev).manual_seed(M + N)
    ints = lambda lo, hi, *s: torch.randint(lo, hi, s, dtype=torch.int8, device=dev, generator=g)
    half = lambda n, s: torch.rand(n, device=dev, generator=g).add(0.5).mul(s).half()
    x, w = ints(-128, 128, M, K), ints(-128, 128, N, K if mode == "w8" else K // 2)
    ws, xs, wz, xsum, s2, z2 = half(N, 2e-3), half(M, 1e-2), half(N, 1e-2), half(M, 1.0), ints(1, 17, K // 128, N), ints(-120, 1, K // 128, N)
    got = []
    for piece in (M, most):
        out = torch.full((M, N), float("nan"), dtype=torch.half, device=dev)
        for a in range(0, M, piece):
            r = slice(a, a + piece)
            if mode == "chn":
                chn.gemm_forward_cuda(x[r], w, ws, xs[r], wz, xsum[r], out[r])
            elif mode == "grp":
                grp.gemm_forward_cuda(x[r], w, z2, s2, ws, xs[r], out[r])
            else:
                w8.w8a8_gemm_forward_cuda(x[r], w, ws, xs[r], out[r])
        assert torch.isfinite(out.float()).all()
        got.append(out)
    assert torch.equal(*got)
