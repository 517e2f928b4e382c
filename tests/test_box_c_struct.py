"""The C struct of a box whose dimensions or flags were set from numpy values (no GPU)."""

import numpy as np
import pytest

from freud_gb300 import box


@pytest.mark.parametrize("kind", [int, float, np.int64, np.int32, np.uint8, np.float32, np.array])
def test_dimensions_of_any_number(kind):
    b = box.Box(3.0, 4.0, 5.0, 0.1, 0.2, 0.3)
    b.dimensions = kind(3)
    assert b.is2D is False and b._c_box().is2D == 0 and b._c_box().Lz == 5.0
    b.dimensions = kind(2)
    assert b.is2D is True and b._c_box().is2D == 1 and b._c_box().Lz == 0.0
    b.periodic_x = np.bool_(False)
    b.periodic_y = np.int64(1)
    c = b._c_box()
    assert (c.periodic_x, c.periodic_y, c.periodic_z) == (0, 1, 1)
    b.periodic = np.zeros(3)
    assert b._c_box().periodic_z == 0
