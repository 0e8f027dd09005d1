"""The hybrid decoders' stream update without a norm behind it: every choice of summands, rows of one word to several blocks, one row to many, and rows that are
not on 16-byte boundaries (the general kernel).  The sum of the summands, from zero, is added to the stream: the bits of the same additions in torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("T,W", [(1, 4), (3, 512), (5, 516), (2, 1020), (7, 1024), (64, 1028), (3000, 2048), (33, 5000), (9, 1022)])
@pytest.mark.parametrize("dt", [BF, F32])
@pytest.mark.parametrize("one,two,bias", [("st", None, False), ("f32", None, True), (None, "st", False), ("f32", "f32", True), ("st", "f32", False), (None, None, True),
                                          (None, None, False)])
def test_bits(dev, T, W, dt, one, two, bias):
    from qserve_b200._lib import check, lib

    g = torch.Generator(device=dev).manual_seed(T * W)
    r = lambda *s: torch.randn(*s, device=dev, generator=g)
    kind = {"st": dt, "f32": F32}
    x, a1, a2, b = r(T + 1, W), r(T, W).to(kind[one]) if one else None, r(T, W).to(kind[two]) if two else None, r(W) if bias else None
    x[0, :2] = -0.0
    want = x.clone()
    if one or two or bias:
        u = torch.zeros(T, W, device=dev)
        for a in (a1, a2, b):
            if a is not None:
                u = u + a.float()
        want[:T] += u
    p = lambda t: None if t is None else t.data_ptr()
    check(lib.qs_hyb_stream_update_norm(None, None, x.data_ptr(), None, p(a1), int(one == "f32"), p(a2), int(two == "f32"), p(b), None, None, 0, 1e-5, T, W,
                                        0 if dt == BF else 1, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(x.view(torch.int32), want.view(torch.int32))
