"""The FP32 division without special cases (srs_div_in_range) against the IEEE
division: equal for every numerator significand over a sample of denominators at
the corners of its exponent range, and for every quotient of the logarithm."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ea,eb", [(0, 0), (-60, 59), (59, -60), (-60, -60), (59, 59)])
def test_division_is_correctly_rounded(srs, ea, eb):
    # spread over the significands, and next to both ends
    for first, step, n in ((5, 16411, 480), (0, 1, 16), (2 ** 23 - 16, 1, 16)):
        assert srs.division_check(first, step, n, ea, eb) == (0, 0, 0)


def test_range_is_checked(srs):
    for ea, eb in ((-61, 0), (0, 60)):
        with pytest.raises(srs.SrsError) as e:
            srs.division_check(0, 1, 1, ea, eb)
        assert e.value.status == -1
