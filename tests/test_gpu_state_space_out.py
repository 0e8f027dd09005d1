"""Read-out of the state space layer (gate, unit RMS in equal parts of the row, gain) in 64 bits over the scan's own outputs: parts of up to 512 numbers take a
warp each in steps of many, larger ones and rows that do not start on a 16-byte boundary a block: parts of one word, of a part of the lanes, of several words per lane, the
largest, and the first that is larger; a number of parts that does not fill the last block.  Errors: bfloat16 results (8 significant bits) round by up to
2^-8 of themselves, and their silu goes by the special-function unit (2^-21); in 32 bits a sum of n squares, exponential, division and root add up to fewer than 16 units of 2^-24."""
import pytest
import torch

from .test_gpu_long_runs import BF, DEV, F32, StateSpace, _tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [BF, F32])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("H,Dv,parts", [(1, 4, 1), (2, 64, 1), (3, 44, 1), (8, 64, 2), (8, 64, 1), (16, 64, 1), (16, 64, 2), (9, 64, 3), (5, 100, 1), (4, 132, 1)])
def test_against_64_bits(dtype, shift, H, Dv, parts):
    against_64_bits(dtype, shift, H, Dv, parts, [33, 4])


@pytest.mark.parametrize("dtype", [BF, F32])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("H,Dv,parts", [(1, 4, 1), (3, 44, 1), (8, 64, 2), (8, 64, 1), (9, 64, 3), (4, 132, 1)])
def test_steps_of_many_parts(dtype, shift, H, Dv, parts):
    """As many (token, part) pairs as 16 per multiprocessor, and a few more: fewer take a block each whatever their size."""
    per = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    against_64_bits(dtype, shift, H, Dv, parts, [per // parts - 4, 8])


def against_64_bits(dtype, shift, H, Dv, parts, lens):
    from qserve_b200._lib import check, lib

    pos0, p = [0, 7], lambda t: t.data_ptr()
    T, inner = sum(lens), H * Dv
    layer = StateSpace(3, dtype, 2, max(H, 2), 1, 16, Dv)  # (decays are set for two heads)
    C = inner + 32
    conv_w, conv_b, conv = layer.rand(C, 4), layer.rand(C), layer.rand(2, 3, C)
    state, norm = layer.rand(2, H, 16, Dv), torch.empty(inner + 1, device=DEV)[shift:shift + inner].copy_(1 + 0.1 * layer.rand(inner))
    proj = layer.rand(T, (inner + C + H + 7) // 8 * 8).to(dtype)
    tab, _ = _tables(lens, pos0, [1, 0])
    prep, o, out = layer.buffers(T, int(lib.qs_hyb_state_space_prep_floats(H, 1, 16, Dv)), inner)
    check(lib.qs_hyb_state_space(p(out), inner, p(prep), p(o), p(proj), proj.stride(0), p(conv_w), p(conv_b), p(conv), p(state), p(layer.a_log), p(layer.dt_bias),
                                 p(layer.skip), p(norm), parts, 0.7, *map(p, tab), T, 2, H, 1, 16, Dv, 4, 1e-5, layer.dt, layer.stream()))
    y = o.double() * torch.nn.functional.silu(proj[:, :inner].double())
    y = y.view(T, parts, -1)
    want = (y * 0.7 * torch.rsqrt((y * y).mean(-1, keepdim=True) + 1e-5)).flatten(1) * norm.double()
    assert ((out.double() - want).abs() <= (2.0 ** -8 + 2.0 ** -18 if dtype is BF else 2.0 ** -20) * want.abs() + 1e-30).all()
