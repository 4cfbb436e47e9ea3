"""The occupancy report of the persistent tile kernel."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_occupancy_is_of_the_kernel_that_runs(tq):
    """FP64 tiles of 256 with ib = 32 run one CTA per SM, with the strips' digit planes in shared memory."""
    from tileqr import _lib
    ctas, smem = ctypes.c_int(0), ctypes.c_int(0)
    assert _lib.lib().tqr_tile_dag_occupancy(8, 0, ctypes.byref(ctas), ctypes.byref(smem)) == 0
    assert ctas.value == 1 and smem.value > 200 * 1024
