"""Prompt tiles of the hybrid decoders' attention on tcgen05 (heads of 128 numbers, an even number of query heads per key / value head, pages of whole
64-key blocks) against the plain CUDA-core kernel over the same cache, which works one token at a time in fp32: every mask and option, portions that
begin inside a tile, a page or a window, tiles with few rows, and cells past a portion's end that hold NaN."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _run(dev, H, G, maps, lens, pos0, page, D=128, chunk=0, window=0, keep=0, sinks=False, slopes=False, softcap=0.0, gate=None, scale=None, seed=0, spoil=True, tiles_only=False):
    from qserve_b200._lib import AttnExtra, check, lib
    from qserve_b200.hybrid import StepBatch

    g = torch.Generator(device=dev).manual_seed(seed + sum(lens))
    r = lambda *s: torch.randn(*s, device=dev, generator=g)
    E, T = len(lens), sum(lens)
    blocks = [-(-(p + n) // page) for n, p in zip(lens, pos0)]
    table = torch.zeros(E, max(blocks), dtype=torch.int32, device=dev)
    ids = torch.randperm(sum(blocks), device=dev, generator=g).to(torch.int32)
    at = 0
    for e, n in enumerate(blocks):
        table[e, :n] = ids[at:at + n]
        at += n
    k, v = r(sum(blocks), page, G, maps * D).to(BF), r(sum(blocks), page, G, D).to(BF)
    if spoil:  # whatever lies behind a sequence's last position
        for e, (n, p) in enumerate(zip(lens, pos0)):
            end = (p + n) % page
            if end:
                k[table[e, blocks[e] - 1].long(), end:] = float("nan")
                v[table[e, blocks[e] - 1].long(), end:] = float("nan")
    W = H * maps * D
    q = r(T, W + (H * D if gate else 0)).to(BF)
    b = StepBatch.build([(e, p, -1, [1] * n) for e, (n, p) in enumerate(zip(lens, pos0))], table, dev)
    sk = r(H) if sinks else None
    sl = 2.0 ** (-8.0 * torch.arange(1, H + 1, device=dev) / H) if slopes else None
    gp = q.data_ptr() + W * 2 if gate else None
    ex = ctypes.byref(AttnExtra(keep, sl.data_ptr() if slopes else None, gp, q.stride(0), 1 if gate == "wide" else 0, softcap))
    scale = scale if scale is not None else D ** -0.5
    scratch = torch.full((int(lib.qs_hyb_attention_scratch_floats(T, H, G, maps, D)),), float("nan"), device=dev)
    p = lambda t: None if t is None else t.data_ptr()
    s = torch.cuda.current_stream().cuda_stream
    outs = []
    for fast in (True, False):
        out = torch.zeros(T, H * D, dtype=BF, device=dev)
        if fast:
            check(lib.qs_hyb_attention_fast(out.data_ptr(), out.stride(0), q.data_ptr(), q.stride(0), k.data_ptr(), v.data_ptr(), p(b.tok_slot), p(b.tok_pos),
                                            table.data_ptr(), table.shape[1], p(b.tile_entry), p(b.tile_row0), b.n_tiles, p(b.long_tokens), b.n_long,
                                            None if tiles_only else p(b.short_tokens), 0 if tiles_only else b.n_short, p(b.entry_start), p(b.entry_len), p(b.entry_slot), p(b.entry_pos0),
                                            scratch.data_ptr(), H, G, maps, D, D, scale, 0.35, 0.8, 1e-5, 1 if maps == 2 else 0, page, chunk, window, p(sk), ex, 0, s))
        else:
            check(lib.qs_hyb_attention(out.data_ptr(), out.stride(0), q.data_ptr(), q.stride(0), k.data_ptr(), v.data_ptr(), p(b.tok_slot), p(b.tok_pos),
                                       table.data_ptr(), table.shape[1], T, H, G, maps, D, D, scale, 0.35, 0.8, 1e-5, 1 if maps == 2 else 0, page, chunk,
                                       window, p(sk), ex, 0, s))
        outs.append(out.float())
    if tiles_only:
        assert 0 < b.n_long < T
        outs = [o[b.long_tokens.long()] for o in outs]
    assert torch.isfinite(outs[1]).all() and torch.isfinite(outs[0]).all()
    # both kernels are fp32 up to the output's rounding: one bfloat16 unit, plus fp32 noise next to zero
    assert ((outs[0] - outs[1]).abs() <= 2 ** -7 * outs[1].abs() + 3e-4).all(), (outs[0] - outs[1]).abs().max()
    assert ((outs[0] - outs[1]).norm() / outs[1].norm()) < 2e-3


@pytest.mark.parametrize("H,G,maps,lens,pos0,page", [
    (4, 2, 2, [64], [0], 64),                     # one whole tile
    (2, 1, 1, [16, 17, 63, 65, 128, 129], [0] * 6, 64),
    (8, 2, 2, [200, 90], [0, 37], 64),            # a portion that begins inside a page
    (4, 1, 1, [40, 3, 100], [1000, 64, 191], 128),  # beside a short portion (single-token kernel)
    (16, 4, 2, [300], [5], 192),
    (6, 1, 1, [70], [0], 64),                     # six heads of one group
])
def test_causal(dev, H, G, maps, lens, pos0, page):
    _run(dev, H, G, maps, lens, pos0, page)


@pytest.mark.parametrize("kw", [dict(chunk=100), dict(window=70), dict(window=1), dict(window=64, keep=5), dict(window=90, keep=130), dict(sinks=True),
                                dict(slopes=True), dict(softcap=5.0), dict(softcap=50.0, slopes=True, window=150), dict(sinks=True, chunk=64), dict(gate="head"),
                                dict(gate="wide", window=33, keep=64, slopes=True), dict(scale=2.5)], ids=str)
def test_options(dev, kw):
    _run(dev, 4, 2, 1, [150, 66, 400], [0, 129, 31], 64, **kw)
    if not set(kw) & {"gate"}:
        _run(dev, 4, 2, 2, [90], [200], 128, **kw)


@pytest.mark.parametrize("H,G,page,D,scale", [(3, 3, 64, 128, None), (4, 2, 48, 128, None), (4, 2, 64, 64, None), (4, 2, 64, 128, -0.1)])
def test_shapes_that_stay_on_the_general_tiles(dev, H, G, page, D, scale):
    _run(dev, H, G, 1, [130], [7], page, D=D, scale=scale)


def test_tiles_without_the_short_portions(dev):
    """A call that lists the tiles of a mixed step alone: its token rows go past the number of rows it lists."""
    _run(dev, 4, 2, 2, [3, 9, 130, 1, 70], [0, 70, 5, 640, 0], 64, tiles_only=True)


def test_the_longest_tiles_start_first(dev):
    """Shapes that stay on the general tiles (three query heads per key/value head): a list of tiles by how many positions they see is faster than the same
    list backwards (1.2 to 1.4 times; the other way about where the kernel starts with the first of the list), and every order gives the same bits."""
    from qserve_b200._lib import check, lib
    from qserve_b200.hybrid import StepBatch

    H, G, lens, page, D = 6, 2, [2048, 1843, 1570, 1297], 64, 128
    g, E, T, blocks = torch.Generator(device=dev).manual_seed(5), len(lens), sum(lens), 32
    table = torch.arange(E * blocks, dtype=torch.int32, device=dev).view(E, blocks)
    r = lambda *s: torch.randn(*s, device=dev, generator=g).to(BF)
    q, k, v, out = r(T, H * D), r(E * blocks, page, G, D), r(E * blocks, page, G, D), torch.zeros(T, H * D, dtype=BF, device=dev)
    b = StepBatch.build([(e, 0, -1, [1] * n) for e, n in enumerate(lens)], table, dev)
    scratch = torch.zeros(int(lib.qs_hyb_attention_scratch_floats(T, H, G, 1, D)), device=dev)
    p, us, outs = lambda t: t.data_ptr(), [], []
    for te, tr in ((b.seen_entry, b.seen_row0), (b.seen_entry.flip(0).contiguous(), b.seen_row0.flip(0).contiguous())):
        took = []
        for _ in range(6):
            a, e = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(5):
                check(lib.qs_hyb_attention_fast(p(out), out.stride(0), p(q), q.stride(0), p(k), p(v), p(b.tok_slot), p(b.tok_pos), p(table), blocks, p(te), p(tr),
                                                b.n_tiles, p(b.long_tokens), b.n_long, None, 0, p(b.entry_start), p(b.entry_len), p(b.entry_slot), p(b.entry_pos0),
                                                p(scratch), H, G, 1, D, D, D ** -0.5, 0.0, 1.0, 1e-5, 0, page, 0, 0, None, None, 0,
                                                torch.cuda.current_stream().cuda_stream))
            e.record()
            e.synchronize()
            took.append(a.elapsed_time(e))
        us.append(min(took) * 200)
        outs.append(out.clone())
    assert torch.equal(*outs)
    assert us[0] < 0.95 * us[1], us
