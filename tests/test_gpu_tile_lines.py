"""The 2D hydro step on both sides of the lines between its tiles: 6 x 14 cells up
to 296 CTAs, 6 x 30 up to 444, or up to 740 where 16 x 24 would take more than 296."""
import pytest

import test_gpu_tiles as tiles

pytestmark = pytest.mark.gpu


# 296 and 304 CTAs of 6 x 14; 444 and 456 of 6 x 30 (210 of 16 x 24); 708 (330); 740 (320) and 760
@pytest.mark.parametrize("nx,ny", [(222, 112), (223, 112), (222, 360), (223, 360), (350, 350), (120, 1110), (121, 1111)])
@pytest.mark.parametrize("walls", [False, True])
def test_lines(nx, ny, walls):
    tiles.test_tiles_equal_the_restatement(nx, ny, walls)
