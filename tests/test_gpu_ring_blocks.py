"""Single tokens of the hybrid decoders' attention: numbers of tokens around the lines between the instances with three and with four blocks per SM (444 and 666
blocks on 148 SMs) have the bits of the general tensor-core kernel, with one share of the keys and with several, and with every option in the instance of four."""
import pytest
from .test_gpu_ring_attention import _run

pytestmark = pytest.mark.gpu
POS = [0, 15, 16, 47, 63, 64, 300]


@pytest.mark.parametrize("maps", [1, 2])
@pytest.mark.parametrize("n", [55, 56, 64, 73, 74, 111, 112, 148, 166, 167])
def test_around_the_lines(dev, n, maps):
    _run(dev, 16, 4, maps, [POS[i % 7] + i for i in range(n)])


@pytest.mark.parametrize("maps", [1, 2])
@pytest.mark.parametrize("kw", [dict(chunk=100), dict(window=70), dict(window=90, keep=130), dict(sinks=True), dict(slopes=True), dict(softcap=5.0),
                                dict(gate="wide", window=33, keep=64, slopes=True), dict(scale=-0.1)], ids=str)
def test_options_with_four_blocks(dev, maps, kw):
    _run(dev, 8, 4, maps, [POS[i % 7] + i for i in range(150)], **kw)
