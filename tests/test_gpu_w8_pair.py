"""W8A8 products against 64-bit sums (exact) and the epilogue's fp32 arithmetic, bit for bit: tiles of CTA pairs (one and several per pair, an odd number of
K stages, ragged tokens), 128-token tiles with two CTAs per multiprocessor, with one, and split, around the limits between them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [
    (512, 256, 512), (513, 512, 640),                        # split, above 512 tokens as well
    (1000, 4096, 1152), (600, 4096, 640),                    # pairs: tiles of 256 tokens, of 160
    (2100, 4096, 512), (3000, 8192, 512), (4500, 8192, 640),  # several tiles per pair: two, six and eight
    (129, 28672, 512), (300, 28672, 640), (400, 6144, 512),  # pairs below 512 tokens
    (128, 28672, 640), (65, 19200, 512),                     # two CTAs per multiprocessor
    (300, 6144, 512), (200, 6144, 640), (100, 12800, 512),   # one
    (100, 4096, 4096), (128, 6144, 1152), (66, 128, 2048),   # split
    (64, 6144, 640), (33, 28672, 512), (1, 128, 128), (17, 256, 384),
    (300, 16256, 6144), (500, 12416, 6144), (300, 16256, 6016), (520, 16256, 6144),  # an odd number of channel tiles: one and two CTAs per multiprocessor
])
def test_against_64_bits(dev, M, N, K):
    import qserve_backend.qgemm_w8a8 as w8

    g = torch.Generator(device=dev).manual_seed(M + N + K)
    x, w = (torch.randint(-128, 128, s, dtype=torch.int8, device=dev, generator=g) for s in ((M, K), (N, K)))
    ws, xs = (torch.rand(n, device=dev, generator=g).add(0.5).mul(s).half() for n, s in ((N, 2e-3), (M, 1e-2)))
    out = torch.full((M, N), float("nan"), dtype=torch.half, device=dev)
    w8.w8a8_gemm_forward_cuda(x, w, ws, xs, out)
    acc = (x.double() @ w.double().t()).float()  # whole numbers below 2^53, then rounded to fp32 once
    assert torch.equal(out, (acc * (ws.float()[None] * xs.float()[:, None])).half())
