"""The row ranges of the tensor-core residual kernel's work units."""
import pytest

from jaxns_gb300.engine import residual_row_tiles


@pytest.mark.parametrize("tiles,rs", [([(1, 1)], 1), ([(2, 8)], 1), ([(2, 38)], 1), ([(2, 39)], 2), ([(4, 32)], 2),
                                      ([(2, 32)] * 8, 4), ([(2, 32)] * 10, 6), ([(3, 64)] * 8, 12),
                                      # twelve uneven problems of up to 16384 rows
                                      ([(7, 128), (6, 55), (6, 65), (6, 37), (4, 37), (6, 99), (2, 87), (5, 36), (5, 90), (4, 43),
                                        (6, 38), (4, 25)], 6)])
def test_measured_choices(tiles, rs):
    assert residual_row_tiles(tiles, 152) == rs


@pytest.mark.parametrize("runs", [1, 3, 12, 100])
def test_no_other_range_leaves_a_twelfth_less_on_the_fullest_cta(runs):
    for ct in (1, 2, 5):
        for rt in (1, 7, 32, 128):
            tiles = [(ct, max(1, rt - r % 5)) for r in range(runs)]
            rs = residual_row_tiles(tiles, 152)
            longest = max(r for _, r in tiles)
            load = lambda q: -(-sum(c * -(-r // q) for c, r in tiles) // 152) * (0.5 + -(-min(q, longest) // 2))
            if rs == 1:
                assert sum(c * r for c, r in tiles) <= 76
            else:
                assert rs % 2 == 0 and 2 <= rs <= 16 and all(11 * load(rs) <= 12 * load(q) for q in range(2, 17, 2))
