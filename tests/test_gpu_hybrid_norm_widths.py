"""The hybrid decoders' norms over rows whose words a thread holds (one, two or four of 16 bytes, the last of them whole or for some of the threads) and over
wider rows that are read again, against 64 bits.  The stream's additions and the joined rows are exact; a norm's bound adds up its roundings of 2^-24: a
row's sum 31 (20 terms of a thread, ten levels of the block's tree, the square's own), half of that behind the root with the division and eps ahead of it, and
one each for the root, its reciprocal, the difference to the mean and the products: 22, taken as 32; the mean's own 31 count by the row's mean magnitude.
bfloat16, eight bits long, rounds the result by half a unit of the last of them, 2^-8 of it at most."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32
WIDTHS = [512, 516, 1020, 1024, 1028, 2048, 2052, 4096, 4100, 5000]
T, EPS = 5, 1e-5
U = 2.0 ** -24


def _p(t):
    return None if t is None else t.data_ptr()


def _near(got, want, size, dtype):
    bound = 32 * U * size
    if dtype == BF:
        bound = bound + (want.abs() + bound) * 2.0 ** -8
    worst = ((got.double() - want).abs() / bound).max()
    assert worst <= 1, float(worst)


@pytest.mark.parametrize("dtype", [F32, BF])
@pytest.mark.parametrize("width", WIDTHS)
def test_rms_norm(dev, dtype, width):
    from qserve_b200._lib import check, lib

    g = torch.Generator(device=dev).manual_seed(width)
    r = lambda *s: torch.randn(*s, device=dev, generator=g)
    x, add, w1, w2 = r(T, width) + 0.5, r(T, width).to(dtype), r(width) * 0.3, r(width) * 0.3
    for use_add, two in ((True, True), (False, True), (True, False), (False, False)):
        xs, o1, o2 = x.clone(), *(torch.full((T, width), float("nan"), dtype=dtype, device=dev) for _ in range(2))
        check(lib.qs_hyb_rms_norm(o1.data_ptr(), _p(o2 if two else None), xs.data_ptr(), _p(add if use_add else None), w1.data_ptr(), _p(w2 if two else None), 1.0, EPS,
                                  T, width, 0 if dtype == BF else 1, torch.cuda.current_stream().cuda_stream))
        want = x + add.float() if use_add else x
        assert torch.equal(xs, want)
        n = want.double() / (want.double().pow(2).mean(-1, keepdim=True) + EPS).sqrt()
        for o, w in ((o1, w1), (o2, w2))[:1 + two]:
            y = n * (1.0 + w.double())
            _near(o, y, y.abs() + n.abs() * U, dtype)  # (1 + w is rounded once more)


@pytest.mark.parametrize("dtype", [F32, BF])
@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("width", WIDTHS)
def test_stream_norm(dev, dtype, kind, width):
    from qserve_b200._lib import check, lib

    g = torch.Generator(device=dev).manual_seed(width + kind)
    r = lambda *s: torch.randn(*s, device=dev, generator=g)
    x, x0, w, b, ab = r(T, width) + 0.7, r(T, width), r(width), r(width), r(width)
    for one, two, bias, cat, shift in ((F32, dtype, True, True, True), (dtype, None, False, False, True), (None, F32, False, True, False), (None, None, True, False, True),
                                       (None, None, False, True, False), (None, None, False, False, True)):
        a1, a2 = (None if t is None else r(T, width).to(t) for t in (one, two))
        xs, h, joined = x.clone(), torch.full((T, width), float("nan"), dtype=dtype, device=dev), torch.full((T, 2 * width), float("nan"), dtype=dtype, device=dev)
        check(lib.qs_hyb_stream_update_norm(h.data_ptr(), _p(joined if cat else None), xs.data_ptr(), x0.data_ptr(), _p(a1), int(one == F32), _p(a2), int(two == F32),
                                            _p(ab if bias else None), w.data_ptr(), _p(b if kind == 2 and shift else None), kind, EPS, T, width, 0 if dtype == BF else 1,
                                            torch.cuda.current_stream().cuda_stream))
        u = torch.zeros(T, width, device=dev)
        for a in (a1, a2, ab if bias else None):
            if a is not None:
                u = u + a.float()
        want = x + u
        assert torch.equal(xs, want)
        if cat:
            assert torch.equal(joined, torch.cat([want, x0], -1).to(dtype))
        v = want.double()
        c = v - v.mean(-1, keepdim=True) if kind == 2 else v
        s = 1.0 / (c.pow(2).mean(-1, keepdim=True) + EPS).sqrt()
        y = c * s * w.double()
        size = y.abs() + (v.abs().mean(-1, keepdim=True) * s * w.double().abs() if kind == 2 else 0)  # (the mean's own roundings)
        if kind == 2 and shift:
            y, size = y + b.double(), size + b.double().abs()
        _near(h, y, size, dtype)
