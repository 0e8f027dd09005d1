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


def test_a_batch_made_of_its_tables():
    """A step's tables may come from a caller's own code, which knows the tiles in one order: the arguments keep their places, and the attention layers
    take that order."""
    entries = [(0, 0, -1, [1] * 70), (1, 40, 6, [3])]
    host, sizes = StepBatch.pack(entries)
    b = StepBatch.view(host, sizes, torch.zeros(2, 2, dtype=torch.int32))
    own = StepBatch(b.n_tokens, b.n_entries, b.tokens, b.prev, b.tok_slot, b.tok_pos, b.tok_entry, b.entry_start, b.entry_len, b.entry_slot, b.entry_pos0,
                    b.block_table, b.n_tiles, b.n_long, b.n_short, b.tile_entry, b.tile_row0, b.long_tokens, b.short_tokens, 64, [(0, 0, 70)])
    assert own.page_size == 64 and own.long_spans == [(0, 0, 70)] and own.context() is not None
    assert own.seen_entry is b.tile_entry and own.seen_row0 is b.tile_row0
    assert StepBatch.view(*StepBatch.pack([(0, 9, 1, [2])]), b.block_table).seen_entry is not None
