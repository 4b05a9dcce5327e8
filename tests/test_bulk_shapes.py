"""The tile shapes of the bulk interval that a program may choose (no GPU is touched)."""
import pytest


@pytest.mark.parametrize("precision", [32, 64])
def test_six_shapes_can_be_chosen(rm, precision):
    keep = rm.bulk_shape(precision)
    try:
        assert len(rm.bulk_shapes(precision)) >= 6
        for k in range(6):
            rm.set_bulk_shape(precision, k)
            assert rm.bulk_shape(precision) == k
        with pytest.raises(rm.RmpcdError):
            rm.set_bulk_shape(precision, len(rm.bulk_shapes(precision)))
    finally:
        rm.set_bulk_shape(precision, keep)


@pytest.mark.parametrize("precision", [32, 64])
def test_the_automatic_choice_can_be_read_and_put_back(rm, precision):
    keep = rm.bulk_shape(precision)
    try:
        rm.set_bulk_shape(precision, -1)
        automatic = rm.bulk_shape(precision)
        assert automatic == -1
        rm.set_bulk_shape(precision, 1)
        rm.set_bulk_shape(precision, automatic)
        assert rm.bulk_shape(precision) == -1
        with pytest.raises(rm.RmpcdError):
            rm.set_bulk_shape(precision, -2)
    finally:
        rm.set_bulk_shape(precision, keep)
