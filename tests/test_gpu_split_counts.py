"""Tile counts around the number of clusters that the device holds at a time: the split over K changes there (8, 4, 2), the result does not.  The INT32
partial sums are exact, so every split gives the bits of the unsplit launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["chn", "grp", "w8"])
@pytest.mark.parametrize("M", [16, 50, 100])
@pytest.mark.parametrize("tiles", [15, 16, 18, 33, 34, 37])
def test_bits_at_the_number_of_clusters(dev, mode, M, tiles):
    import qserve_backend.qgemm_w4a8_per_chn as chn
    import qserve_backend.qgemm_w4a8_per_group as grp
    import qserve_backend.qgemm_w8a8 as w8
    from qserve_b200._lib import lib

    N, K = tiles * 128, 2432
    g = torch.Generator(device=dev).manual_seed(M + N)
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
