"""A wrong number of source parameters is a ValueError, before any device is needed."""
import numpy as np
import pytest


@pytest.mark.parametrize("count", [0, 1, 5, 6, 7, 11, 13])
def test_wrong_number_of_parameters(count):
    from bbhx_b200.utils.arrays import param_rows

    with pytest.raises(ValueError, match="12 source parameters"):
        param_rows(tuple(np.ones((count, 3))))
