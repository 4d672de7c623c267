"""How the partial tiles of a split GEMM meet, from shapes alone: sending them pays only while a tile has few rows."""
import pytest

from sharq_b200 import _lib

REGISTERS, BLOCKS, PULL = 0, 1, 2
KINDS = [(1, 1), (1, 0), (0, 1)]


def _form(tile_n, kind, rows, k, splits):
    return _lib.lib().sharq_gemm_exchange(tile_n, *kind, rows, k, splits)


@pytest.mark.parametrize("tile_n", [128, 256])
@pytest.mark.parametrize("kind", KINDS)
def test_tiles_of_more_than_80_rows_are_read_behind_the_barrier(tile_n, kind):
    for splits in range(2, 9):
        for k in range(512 * splits, 512 * splits + 256 * 24, 256):
            assert all(_form(tile_n, kind, rows, k, splits) == PULL for rows in (81, 96, 127, 128))
            assert all(_form(tile_n, kind, rows, k, splits) == REGISTERS for rows in (1, 31, 32))


@pytest.mark.parametrize("kind", KINDS)
def test_block_copies_are_used_wherever_four_ctas_share_a_narrow_tile(kind):
    """The receiving slot is any of the ring's: no number of K stages falls back."""
    for splits in range(2, 9):
        for k in range(512 * splits, 512 * splits + 256 * 40, 256):
            want = BLOCKS if splits >= 4 else PULL
            assert all(_form(128, kind, rows, k, splits) == want for rows in (33, 48, 64))


def test_wide_tiles_without_room_for_the_blocks_are_read():
    assert _form(256, (1, 1), 64, 18944, 8) == PULL and _form(256, (1, 1), 33, 18944, 8) == BLOCKS


def test_other_arguments():
    assert [_form(*a) for a in ((512, (1, 1), 1, 1024, 2), (128, (0, 0), 1, 1024, 2), (128, (1, 1), 129, 1024, 2), (128, (1, 1), 1, 1024, 9))] == [-1] * 4


@pytest.mark.parametrize("kind", KINDS)
def test_the_line_rises_with_the_ctas_of_a_tile(kind):
    for splits in range(4, 9):
        forms = [[_form(128, kind, rows, k, splits) for k in range(512 * splits, 512 * splits + 256 * 40, 256)] for rows in (48 + 4 * splits, 49 + 4 * splits)]
        assert BLOCKS in forms[0] and set(forms[1]) == {PULL}  # the room for the blocks depends on the slots, K
