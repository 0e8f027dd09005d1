"""Tiles of a step's prompt portions: listed once entry by entry, as the recurrent layers walk them, and once by how many positions they see."""
import torch

from qserve_b200.hybrid import StepBatch


def test_tiles_by_what_they_see():
    entries = [(0, 0, -1, [1] * 200), (1, 130, 5, [2] * 70), (2, 40, 6, [3]), (3, 0, -1, [4] * 64), (4, 500, 7, [5] * 16)]
    host, sizes = StepBatch.pack(entries)
    b = StepBatch.view(host, sizes, torch.zeros(5, 12, dtype=torch.int32))
    tiles = list(zip(b.tile_entry.tolist(), b.tile_row0.tolist()))
    assert tiles == [(0, 0), (0, 64), (0, 128), (0, 192), (1, 0), (1, 64), (3, 0), (4, 0)] and b.n_tiles == 8
    seen = list(zip(b.seen_entry.tolist(), b.seen_row0.tolist()))
    assert seen == [(0, 0), (3, 0), (0, 64), (0, 128), (1, 0), (0, 192), (1, 64), (4, 0)]
    assert StepBatch.pack([(0, 9, 1, [2])])[1][2] == 0
