"""CTA pairs that take several tiles each: with warps of their own for the epilogue (tiles of 256 tokens, or more than two rounds), whose accumulators wait in
registers while the next tile's products run, and without.  Odd and even numbers of stages, ragged last tiles: the bits of the same rows in small pieces."""
import pytest

from tests.test_gpu_pair_tiles import same_bits_in_pieces

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["chn", "grp"])
@pytest.mark.parametrize("M,N,K", [(2400, 4096, 2048), (1700, 4096, 1024), (4736, 4096, 2176), (3001, 4096, 640), (257, 28672, 512), (230, 19200, 1152), (230, 19200, 8064)])
def test_bits_over_rounds(dev, mode, M, N, K):
    same_bits_in_pieces(dev, mode, M, N, K, 64)
