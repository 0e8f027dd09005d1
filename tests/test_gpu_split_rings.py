"""Calls that split K take rings of their own depths, by mode, tokens and depth of K: fewer stages than a ring has, exactly as many, many times over, half a
stage at the end, tile counts on both sides of where a ring is chosen.  INT32 partial sums are exact: the bits of the unsplit launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["chn", "grp", "w8"])
@pytest.mark.parametrize("M", [3, 32, 50, 128])
@pytest.mark.parametrize("tiles,K", [(2, 512), (8, 896), (16, 6144), (17, 6016), (19, 7168), (24, 4096), (25, 2176), (26, 2048), (33, 4096), (33, 4224), (48, 4096), (74, 1152)])
def test_bits_of_the_unsplit_launch(dev, mode, M, tiles, K):
    import qserve_backend.qgemm_w4a8_per_chn as chn
    import qserve_backend.qgemm_w4a8_per_group as grp
    import qserve_backend.qgemm_w8a8 as w8
    from qserve_b200._lib import lib

    N = tiles * 128
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    ints = lambda lo, hi, *s: torch.randint(lo, hi, s, dtype=torch.int8, device=dev, generator=g)
    half = lambda n, s: torch.rand(n, device=dev, generator=g).add(0.5).mul(s).half()
    x, w = ints(-128, 128, M, K), ints(-128, 128, N, K if mode == "w8" else K // 2)
    ws, xs, wz, xsum, s2, z2 = half(N, 2e-3), half(M, 1e-2), half(N, 1e-2), half(M, 1.0), ints(1, 17, K // 128, N), ints(-120, 1, K // 128, N)
    got = []
    try:
        for split in (0, 1):
            lib.qs_gemm_force_split(split)
            out = torch.full((M, N), float("nan"), dtype=torch.half, device=dev)
            if mode == "chn":
                chn.gemm_forward_cuda(x, w, ws, xs, wz, xsum, out)
            elif mode == "grp":
                grp.gemm_forward_cuda(x, w, z2, s2, ws, xs, out)
            else:
                w8.w8a8_gemm_forward_cuda(x, w, ws, xs, out)
            assert torch.isfinite(out.float()).all()
            got.append(out)
    finally:
        lib.qs_gemm_force_split(0)
    assert torch.equal(*got)
