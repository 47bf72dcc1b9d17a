"""Which calls of the dynamic NVFP4 quantiser are sent to the one-launch kernel: the rule of csrc/quantize_nvfp4.cu itself, on a device of
148 SMs, through the debug-hook build (no GPU needed)."""
import pytest

from tests.helpers import takes_one_launch

N25 = 2 ** 25


@pytest.mark.parametrize("shape,asked", [
    ((666, 4096), False), ((1000, 4096), False), ((1000, 4800), True), ((1000, 5120), True), ((2048, 4096), True), ((2049, 4096), False),
    ((4096, 4096), False), ((4097, 4096), True), ((8192, 4096), True), ((8193, 4096), False), ((32768, 8192), False),
    ((1, 4096, 40, 128), False), ((1100000, 16), True), ((40000, 128), True), ((100000, 8), True), ((33000, 1000), True), ((1000000, 24), True),
])
def test_rows_by_their_tiles(shape, asked):
    assert takes_one_launch(shape, len(shape) - 2, len(shape) - 1) == asked


@pytest.mark.parametrize("shape,asked", [
    ((64, 48, 1024), True), ((64, 42, 1024), False), ((64, 16, 1024), False), ((40, 16, 1024), False), ((4096, 4, 2048), False), ((8192, 8, 512), False),
    ((1, N25 - 64), False), ((1, N25 - 8), False), ((256, 16, 4104), False), ((600, 30, 1024), False), ((256, 64, 1032), True), ((500, 64, 1032), True),
    ((130, 65, 2048), True), ((200, 65, 2048), False), ((300, 100, 1024), True), ((327, 100, 1024), True), ((128, 129, 1024), True),
    ((2, 3, 129, 40000), False),
])
def test_rows_that_leave_most_of_a_tile_empty(shape, asked):
    """two launches where the tiles would be padding: 16 rows a matrix took 7.8 us for 6.8, four 553 for 215, one 2200 for 791"""
    assert takes_one_launch(shape, len(shape) - 2, len(shape) - 1) == asked


@pytest.mark.parametrize("shape,cross,reduce", [((1, 16, 400, 128), 3, 1), ((1, 75600, 40, 128), 3, 1), ((8, 4000), 1, 0), ((4000, 8), 1, 0)])
@pytest.mark.parametrize("swizzle", [False, True])
def test_columns(shape, cross, reduce, swizzle):
    assert takes_one_launch(shape, cross, reduce, swizzle)
