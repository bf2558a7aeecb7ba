"""Units of the fused Toeplitz x stage that end in a short one: a strip's coils in
two units of two and one (two units per block), and of nine and eight (eight units
per block while a unit keeps eight coils), against the unfused stage."""
import pytest

import test_gpu_toeplitz as toeplitz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("img,grid,nch,nb", [
    ((16, 64, 40), (32, 128, 80), 3, 2),      # 1280 strips
    ((16, 64, 48), (32, 128, 96), 17, 3),     # 2304 strips
])
def test_split_strips(gpu_lib, cgs, img, grid, nch, nb):
    toeplitz.test_toeplitz_units_of_the_fused_stage(gpu_lib, cgs, img, grid, nch, nb)
