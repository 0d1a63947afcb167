"""How contractions are cut into tiles and shares of K, decided on the host: no GPU needed."""
import ctypes as C

import pytest

from myea_b200 import capi


def _split(tiles, chunks, pairs):
    out = [C.c_int() for _ in range(3)]
    assert capi.load().myea_b200_split_plan(tiles, chunks, pairs, *[C.byref(x) for x in out]) == 0
    return [x.value for x in out]


@pytest.mark.parametrize("pairs", [74, 66])
def test_split_tiles_cover_k_with_eight_shares_at_most(pairs):
    for tiles in list(range(1, 2 * pairs + 2)):
        for chunks in list(range(1, 40)) + [48, 63, 64, 65, 128, 1000]:
            whole, run, clusters = _split(tiles, chunks, pairs)
            if run == 0:
                assert whole == tiles and clusters == min(tiles, pairs)
                continue
            units = (tiles - whole) * chunks
            assert whole % pairs == 0 and 0 < tiles - whole < pairs
            assert run < chunks                        # a run touches two tiles at most
            assert run * clusters >= units and clusters <= pairs
            assert 8 * run >= chunks                   # the last of a tile's pairs adds up the partial sums of all others


@pytest.mark.parametrize("tiles,chunks,run", [(32, 32, 16), (32, 16, 8), (25, 8, 4), (15, 9, 3), (1, 128, 16), (2, 64, 8), (4, 32, 4), (4, 64, 8), (4, 20, 3), (40, 16, 9)])
def test_tiles_of_a_single_wave_are_cut_into_equal_shares_where_these_are_hardly_longer(tiles, chunks, run):
    assert _split(tiles, chunks, 74)[1] == run
