"""Masks that are no uint8 arrays: every form converts as astype(uint8) does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["nested list", "int64", "float64", "bool list"])
def test_values_outside_of_a_byte_wrap(cuda, form):
    from stonewall.fields import Flags, Grid
    mask = np.zeros((5, 3, 4), np.int64)
    mask[1, 1, 1], mask[2, 0, 3], mask[3, 2, 2], mask[:, :, 0] = 1, 257, 512, 2
    given = {"nested list": mask.tolist(), "int64": mask, "float64": (mask % 256).astype(float),
             "bool list": (mask > 0).tolist()}[form]
    want = np.asarray(given).astype(np.uint8)
    f = Flags(Grid(5, 3, 4), given)
    np.testing.assert_array_equal(f.host, want)
