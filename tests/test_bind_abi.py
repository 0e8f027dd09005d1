"""The C ABI's functions behind the CPython binding: as many arguments as the ctypes declarations have, the same numbers handed on, and what is no address or
no number refused with TypeError."""
import re

import numpy
import pytest
import torch

from qserve_b200 import _bind
from qserve_b200._lib import SIGNATURES, lib

NAMES = sorted(n for n in dir(_bind) if n.startswith("qs_"))


@pytest.mark.parametrize("name", NAMES)
def test_arguments_of_the_declaration(name):
    with pytest.raises(TypeError) as e:
        getattr(_bind, name)()
    assert int(re.search(r"expected (\d+) arguments", str(e.value)).group(1)) == len(SIGNATURES[name][1])


def _refused(f, args):
    rc = f(*args)
    return rc, lib.qs_last_error()


@pytest.mark.parametrize("change", [{}, {11: -5}, {11: (1 << 32) + 7}, {14: 64, 15: 1}, {15: -1e300}, {3: -(1 << 62)}, {0: None}, {0: (1 << 64) - 16}, {12: True}], ids=str)
def test_numbers_as_ctypes_hands_them_on(change):
    args = [16, 16, 16, 384, 384, 384, 16, 128, 16, 1, 4, 4, 3, 2, 96, 0.5, None]  # 3 heads over 2, heads of 96: refused ahead of any call of CUDA
    for i, v in change.items():
        args[i] = v
    got = [_refused(f, args) for f in (_bind.qs_prefill_attention, lib.qs_prefill_attention)]
    assert got[0] == got[1] and got[0][0] != 0


class _Index:
    def __init__(self, v):
        self.v = v

    def __index__(self):
        return self.v


@pytest.mark.parametrize("kind", [numpy.int32, numpy.int64, numpy.uint8, torch.tensor, _Index], ids=lambda k: k.__name__)
@pytest.mark.parametrize("at", [3, 9, 12, 14])
def test_whatever_has_an_index_is_an_integer(kind, at):  # sizes that a program read out of an array
    args = [16, 16, 16, 384, 384, 384, 16, 128, 16, 1, 4, 4, 3, 2, 96, 0.5, None]
    args[at] = kind(args[at] % 256)
    got = [_refused(f, args) for f in (_bind.qs_prefill_attention, lib.qs_prefill_attention)]
    assert got[0] == got[1] and got[0][0] != 0


def test_an_index_that_raises():
    args = [16, 16, 16, 384, 384, 384, 16, 128, 16, 1, 4, 4, 3, 2, torch.tensor([96, 96]), 0.5, None]
    with pytest.raises(TypeError, match="index"):  # (torch's own words)
        _bind.qs_prefill_attention(*args)


@pytest.mark.parametrize("at,value", [(0, numpy.int64(16)), (0, torch.tensor(16)), (9, numpy.float32(1)), (9, torch.tensor(1.5)), (0, "x"), (0, 1.5), (3, 1.5), (3, None), (9, "1"), (15, "0.5"), (15, None), (16, b"")])
def test_what_is_no_number_is_refused(at, value):
    args = [16, 16, 16, 384, 384, 384, 16, 128, 16, 1, 4, 4, 3, 2, 96, 0.5, None]
    args[at] = value
    with pytest.raises(TypeError):
        _bind.qs_prefill_attention(*args)
