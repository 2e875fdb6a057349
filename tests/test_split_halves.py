"""The halves of a split ensemble (model._halves): no more Legendre tiles than
needed, and no imbalance that saves none."""
import pytest

from my_swampe_gb300.model import _halves


@pytest.mark.parametrize("M,precision,scheme,tile", [(42, "fp64", 0, 4), (63, "fp64", 2, 2), (106, "fp64", 0, 1),
                                                     (42, "fast", 0, 8), (106, "fast", 0, 8), (63, "fast", 2, 1)])
def test_halves(M, precision, scheme, tile):
    for B in range(2, 300):
        a, b = _halves(M, B, precision, scheme)
        assert a + b == B and min(a, b) >= 1
        total = lambda h: -(-h // tile) + -(-(B - h) // tile)  # noqa: E731
        assert total(a) == min(map(total, range(1, B)))
        if total(B // 2) == total(a):
            assert max(a, b) < 2 * min(a, b) or abs(a - b) <= 1


def test_small_ensembles_of_the_finest_grid():
    assert [_halves(106, B, "fast", 0) for B in (10, 12, 15, 16, 21)] == [(5, 5), (6, 6), (8, 7), (8, 8), (8, 13)]
    assert _halves(106, 5, "fp64", 0) == (2, 3) and _halves(42, 13, "fp64", 0) == (8, 5)
