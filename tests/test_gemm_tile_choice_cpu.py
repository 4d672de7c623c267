"""The tile width that the automatic choice takes, from shapes alone."""
import pytest

from sharq_b200 import _lib

SMS = 148


def _tile(m, n, k, split, sms=SMS):
    return _lib.lib().sharq_gemm_tile_n(m, n, k, split, sms)


def test_long_k_takes_wide_tiles_only_where_k_is_split():
    assert _tile(384, 3584, 18944, 1) == 256
    assert _tile(384, 3584, 18944, 0) == 128  # 42 CTAs would run the K loop that 84 can share
    assert _tile(384, 3584, 16384, 1) == 128  # the crossover


# an odd number of 128-wide column tiles: 147, 145 and 143 narrow tiles fit the GPU, the 75 to 77 wide ones leave no second CTA each
@pytest.mark.parametrize("m,n", [(384, 49 * 128), (640, 29 * 128), (1408, 13 * 128 - 8)])
def test_wide_tiles_that_leave_no_room_for_a_split_are_not_taken(m, n):
    assert _tile(m, n, 18944, 1) == 128


def test_wide_tiles_are_split_whenever_they_are_taken_for_a_long_k():
    taken = 0
    for m in range(129, 1400, 61):
        for n in range(136, 12000, 104):
            tile = _tile(m, n, 18944, 1)
            if tile == 256:
                taken += 1
                assert 2 * (-(-m // 128) * -(-n // 256)) <= SMS
            assert _tile(m, n, 18944, 0) != 256
    assert taken > 50


def test_a_row_of_tiles():
    assert [_tile(m, 4096, 4096, s) for m in (1, 128) for s in (0, 1)] == [128] * 4
    assert _tile(32, 28672, 4096, 1) == 256 and _tile(32, 128, 4096, 1) == 128 and _tile(2048, 4096, 4096, 1) == 512
