"""Single tokens of the hybrid decoders' attention: the kernel with a ring per warp (heads of 128 + 128 numbers, up to eight query rows per key/value head,
pages of whole 16-key slices) has the bits of the general tensor-core kernel, which takes the same cells when they are addressed through pages of 24:
both maps or one, every number of rows, positions around slices, tiles and pages, one token (many shares, some without keys) to many, every option, and
cells past the position that hold NaN."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
D = 128


def _run(dev, H, G, maps, pos, keep=0, chunk=0, window=0, slopes=False, sinks=False, softcap=0.0, gate=None, scale=D ** -0.5):
    from qserve_b200._lib import AttnExtra, check, lib
    from qserve_b200.hybrid import StepBatch

    g = torch.Generator(device=dev).manual_seed(sum(pos) + H + maps)
    r = lambda *s: torch.randn(*s, device=dev, generator=g)
    E, blocks = len(pos), max(pos) // 48 + 1
    table = torch.randperm(E * blocks, device=dev, generator=g).to(torch.int32).view(E, blocks)
    k, v = r(E * blocks, 48, G, maps * D).to(BF), r(E * blocks, 48, G, D).to(BF)
    for e, n in enumerate(pos):
        k[table[e, n // 48].long(), n % 48 + 1:] = float("nan")
        v[table[e, n // 48].long(), n % 48 + 1:] = float("nan")
    W = H * maps * D
    q = r(E, W + (H * D if gate else 0)).to(BF)
    sk, sl = (r(H) if sinks else None), (2.0 ** (-8.0 * torch.arange(1, H + 1, device=dev) / H) if slopes else None)
    p = lambda t: None if t is None else t.data_ptr()
    ex = ctypes.byref(AttnExtra(keep, p(sl), q.data_ptr() + W * 2 if gate else None, q.stride(0), 1 if gate == "wide" else 0, softcap))
    halves = torch.stack([2 * table, 2 * table + 1], 2).flatten(1).contiguous()
    outs = []
    for page, tab in ((48, table.contiguous()), (24, halves)):
        b = StepBatch.build([(e, n, -1, [1]) for e, n in enumerate(pos)], tab, dev)
        assert b.n_tiles == 0 and b.n_short == E
        scratch = torch.full((int(lib.qs_hyb_attention_scratch_floats(E, H, G, maps, D)),), float("nan"), device=dev)
        out = torch.zeros(E, H * D, dtype=BF, device=dev)
        check(lib.qs_hyb_attention_fast(p(out), out.stride(0), p(q), q.stride(0), p(k), p(v), p(b.tok_slot), p(b.tok_pos), p(tab), tab.shape[1], p(b.tile_entry),
                                        p(b.tile_row0), 0, p(b.long_tokens), 0, p(b.short_tokens), E, p(b.entry_start), p(b.entry_len), p(b.entry_slot),
                                        p(b.entry_pos0), p(scratch), H, G, maps, D, D, scale, 0.35, 0.8, 1e-5, 1 if maps == 2 else 0, page, chunk, window, p(sk),
                                        ex, 0, torch.cuda.current_stream().cuda_stream))
        outs.append(out)
    assert torch.isfinite(outs[0].float()).all() and torch.equal(*outs)


POS = [0, 14, 15, 16, 47, 48, 62, 63, 64, 95, 127, 300, 767]


@pytest.mark.parametrize("H,G,maps", [(16, 4, 2), (4, 1, 2), (3, 1, 2), (2, 2, 2), (8, 1, 1), (5, 1, 1), (12, 3, 1), (4, 4, 1)])
@pytest.mark.parametrize("pos", [[0], [1500], POS, [40 + i * 7 for i in range(90)]], ids=["first", "shares", "edges", "many"])
def test_bits_of_the_general_kernel(dev, H, G, maps, pos):
    _run(dev, H, G, maps, pos)


@pytest.mark.parametrize("maps", [1, 2])
@pytest.mark.parametrize("kw", [dict(chunk=100), dict(window=70), dict(window=1), dict(window=64, keep=5), dict(window=90, keep=130), dict(sinks=True),
                                dict(slopes=True), dict(softcap=5.0), dict(softcap=50.0, slopes=True, window=150), dict(gate="head"),
                                dict(gate="wide", window=33, keep=64, slopes=True), dict(scale=2.5), dict(scale=-0.1)], ids=str)
def test_options(dev, maps, kw):
    _run(dev, 8, 2, maps, POS, **kw)
