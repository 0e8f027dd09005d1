"""The 16-byte row kernels of the hybrid decoders (embedding, rotary append, delta-rule preparation and read-out, combination of the maps) against
the general kernels, which rows of an odd stride still take: the same numbers in, the same numbers out up to the order of a head's sum."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _s():
    return torch.cuda.current_stream().cuda_stream


def _i(x, dev):
    return torch.tensor(x, dtype=torch.int32, device=dev)


def _batch(lens, pos0, dev):
    """Flat batch tables: entry, position per token; start, length, slot, first position per entry."""
    ent = [e for e, n in enumerate(lens) for _ in range(n)]
    pos = [p + k for n, p in zip(lens, pos0) for k in range(n)]
    start = [sum(lens[:e]) for e in range(len(lens))]
    return _i(ent, dev), _i(pos, dev), _i(start, dev), _i(lens, dev), _i(list(range(len(lens)))[::-1], dev), _i(pos0, dev)


def _strided(x, extra):
    """x in rows `extra` elements further apart."""
    out = torch.zeros(x.shape[0], x.shape[1] + extra, dtype=x.dtype, device=x.device)
    out[:, :x.shape[1]] = x
    return out


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("W,copies,pair", [(4, 1, True), (36, 3, False), (256, 1, True), (516, 2, True), (2052, 1, True), (4096, 1, False)])
def test_embedding(dev, W, copies, pair, dtype):
    from qserve_b200._lib import check, lib

    g = torch.Generator(device=dev).manual_seed(W)
    table, pt = (torch.randn(n, W, device=dev, generator=g).to(dtype) for n in (50, 14))
    tok, prev = _i([3, 49, 0, 7], dev), _i([-1, 3, 49, 0], dev)
    out = torch.empty(4, copies, W, device=dev)
    check(lib.qs_hyb_embed(out.data_ptr(), tok.data_ptr(), prev.data_ptr(), table.data_ptr(), pt.data_ptr() if pair else None, 4, W, 13, 31, 5, 1.5, copies,
                           0 if dtype == BF else 1, _s()))
    rows = torch.where(prev < 0, 13, (prev.long() * 31 + tok.long() * 5) % 13)
    want = table[tok.long()].double() * 1.5 + (pt[rows].double() if pair else 0.0)
    assert (out - want[:, None]).abs().max() <= 2 ** -22 * want.abs().max()  # two fp32 roundings


@pytest.mark.parametrize("H,G,maps,D,Dv,rot", [(4, 2, 2, 128, 128, 64), (3, 1, 1, 64, 8, 64), (2, 2, 2, 24, 40, 8), (16, 4, 1, 128, 128, 0)])
def test_rope_append(dev, H, G, maps, D, Dv, rot):
    from qserve_b200._lib import check, lib

    lens, pos0, page = [5, 1, 70], [0, 130, 3], 16
    ent, pos, _, _, slot, _ = _batch(lens, pos0, dev)
    T, W = sum(lens), (H + G) * maps * D + G * Dv
    g = torch.Generator(device=dev).manual_seed(T + D)
    x = torch.randn(T, W, device=dev, generator=g).to(BF)
    freq = torch.rand(max(rot // 2, 1), device=dev, generator=g)
    table = torch.randperm(30, device=dev, generator=g).view(3, 10).to(torch.int32)
    got = []
    for extra in (8 - W % 8, 9 - W % 8):  # whole 16-byte words, then the general kernel
        p = _strided(x, extra)
        k, v = (torch.zeros(30, page, G, n, dtype=BF, device=dev) for n in (maps * D, Dv))
        tok_slot = slot[ent.long()].contiguous()
        check(lib.qs_hyb_rope_append(p.data_ptr(), p.stride(0), tok_slot.data_ptr(), pos.data_ptr(), table.data_ptr(), 10, k.data_ptr(), v.data_ptr(),
                                     freq.data_ptr(), 1.1, T, H, G, maps, D, Dv, rot, page, 0, _s()))
        got.append((p[:, :W].float(), k.float(), v.float()))
    for a, b in zip(*got):
        assert ((a - b).abs() <= 2 ** -8 * b.abs() + 1e-6).all()  # at most the last bit of a bfloat16 number
        assert (a != b).float().mean() < 1e-3
    assert torch.equal(got[0][2], got[1][2])


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("H,G,D,Dv,taps,lens,pos0", [
    (4, 2, 128, 128, 4, [17, 1, 3, 50], [0, 9, 2, 0]),   # portions that begin inside the convolution's memory
    (2, 1, 64, 128, 2, [33, 4], [0, 1]),
    (6, 2, 20, 36, 3, [2, 40], [0, 0]),                  # idle lanes
    (2, 2, 128, 64, 1, [5, 6], [0, 3]),
    (2, 1, 32, 128, 7, [9, 1], [2, 0]),                  # taps without a window in registers
    (2, 1, 128, 128, 4, [700], [0]),                     # runs of several tokens per block
])
def test_delta_preparation_and_read_out(dev, H, G, D, Dv, taps, lens, pos0, dtype):
    from qserve_b200._lib import check, lib

    ent, pos, start, ln, slot, p0 = _batch(lens, pos0, dev)
    T, E, C = sum(lens), len(lens), 2 * G * D + H * Dv
    W = C + H * Dv + 2 * H
    g = torch.Generator(device=dev).manual_seed(T + D)
    r = lambda *s: torch.randn(*s, device=dev, generator=g)
    x, cw, cst, S0 = r(T, W).to(dtype), r(C, taps), r(E, max(taps - 1, 1), C), r(E, H, D, Dv) * 0.2
    alog, dtb, nw = r(H) * 0.5, r(H) * 0.5, 1 + r(Dv) * 0.1
    got = []
    for extra in (8 - W % 8, 9 - W % 8):
        p, cs, S = _strided(x, extra), cst.clone(), S0.clone()
        prep, o, out = torch.zeros(T, C + 2 * H, device=dev), torch.zeros(T, H * Dv, device=dev), torch.zeros(T, H * Dv, device=dev, dtype=dtype)
        check(lib.qs_hyb_gated_delta(out.data_ptr(), H * Dv, prep.data_ptr(), o.data_ptr(), p.data_ptr(), p.stride(0), cw.data_ptr(), cs.data_ptr(), S.data_ptr(),
                                     alog.data_ptr(), dtb.data_ptr(), nw.data_ptr(), ent.data_ptr(), pos.data_ptr(), start.data_ptr(), ln.data_ptr(),
                                     slot.data_ptr(), p0.data_ptr(), T, E, H, G, D, Dv, taps, 1e-6, 1e-5, 0 if dtype == BF else 1, _s()))
        got.append((prep, out.float(), cs))
    close = lambda a, b, tol: ((a - b).norm() / b.norm()).item() <= tol
    assert close(got[0][0], got[1][0], 1e-6) and torch.equal(got[0][2], got[1][2])  # fp32: the order of a head's sum of squares
    assert close(got[0][1], got[1][1], 1e-5 if dtype == torch.float32 else 2e-3)   # bfloat16: a last bit here and there
