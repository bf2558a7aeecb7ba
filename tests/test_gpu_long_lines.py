"""The quad x passes on lines of 352 to 512 points (codelets of more than 16
points, stages taken in two turns, input rows in two copies) against coil planes
and the tiled spreading, bit for bit."""
import pytest

import test_gpu_quad_grid as quads

pytestmark = pytest.mark.gpu

CASES = [
    ((301, 16, 12), (352, 32, 24), 6, 4.25),   # first stage in one turn, second in two
    ((192, 16, 12), (384, 32, 24), 4, 4.0),
    ((270, 16, 12), (384, 32, 24), 3, 4.0),
    ((224, 16, 12), (448, 32, 24), 3, 4.0),    # half-pruned
    ((301, 16, 12), (448, 32, 24), 9, 4.25),
    ((256, 16, 12), (512, 32, 24), 4, 4.0),
    ((257, 16, 12), (512, 32, 24), 6, 4.0),    # input rows in two copies, one row over
    ((512, 16, 12), (512, 32, 24), 3, 4.25),   # the whole line
]


@pytest.mark.parametrize("img,grid,nch,kb_w", CASES)
@pytest.mark.parametrize("pruned", [True, False])
def test_forward_pass(gpu_lib, cgs, img, grid, nch, kb_w, pruned):
    quads.test_quads_equal_coil_planes_bitwise(gpu_lib, cgs, img, grid, nch, kb_w, pruned)


@pytest.mark.parametrize("img,grid,nch,kb_w", CASES)
@pytest.mark.parametrize("compensated", [False, True])
def test_adjoint_pass(gpu_lib, cgs, img, grid, nch, kb_w, compensated):
    quads.test_sliced_gather_equals_tiled_kernel_bitwise(gpu_lib, cgs, img, grid, nch, kb_w, compensated)
