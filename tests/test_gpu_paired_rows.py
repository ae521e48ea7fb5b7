"""Float-float strings of one to one and a half waves of strips, whose strips are
longer than the most rows or, where a column cannot be cut so, shorter: steps
against the C oracle."""
import pytest

import test_gpu_strips

pytestmark = pytest.mark.gpu


# on 152 SMs, which hold 1,216 strips: 20 rows, 17, 24, 8 of 16
@pytest.mark.parametrize("nx,ny,images", [(33, 40, 210), (64, 50, 160), (31, 24, 620), (35, 16, 620)])
@pytest.mark.parametrize("mc,uniform,delta", [(False, True, 0.0), (True, True, 0.1), (True, False, 0.1)])
def test_steps(nx, ny, images, mc, uniform, delta):
    test_gpu_strips.test_strip_steps(nx, ny, images, mc, False, uniform, delta, True, "paired")
