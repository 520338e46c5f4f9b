"""The tcgen05 convolutions where their rings start again: blocks that walk several z columns (more
input planes than barriers, more output planes than accumulators, column ends inside the ring), and
grids of one partial tile with one or two planes."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

# (cin, cout): one of each split of the output channels and of each ring depth
SHAPES = [(16, 16), (16, 48), (32, 96), (48, 16), (64, 64), (96, 32)]


@pytest.mark.parametrize("grid", [(328, 120, 40), (121, 250, 23), (9, 17, 1), (7, 16, 2)])
@pytest.mark.parametrize("shape", SHAPES)
def test_conv_rings(gpu_lib, shape, grid):
    """Against the mma.sync form on the same BF16 inputs: the FP32 sums differ only in order, so the
    BF16 outputs agree to a rounding step (2^-8 relative, doubled) of the output scale."""
    cin, cout = shape
    nx, ny, nz = grid
    diff, ref = C.c_double(), C.c_double()
    rc = gpu_lib.frehg_unet_conv_check(cin, cout, cin, 0, cout, 0, nx, ny, nz, 1, 23,
                                       C.byref(diff), C.byref(ref))
    assert rc == 0, gpu_lib.frehg_last_error()
    assert ref.value > 0.0
    assert diff.value <= 2.0 ** -7 * ref.value, (diff.value, ref.value)
