"""Layers that the masked form and the kernel for long rows leave to the kernel that is named for them: few channels of many samples,
whose clusters would walk them for several times as long, and more channels of a few vectors a thread than two waves of clusters hold."""
import pytest

FWD, BWD, FWD_RES, BWD_RES = (0, False), (1, False), (0, True), (1, True)


@pytest.mark.parametrize("shape,call,named", [
    ((97106, 1, 1, 81), FWD, "plain"), ((93078, 1, 1, 146), BWD, "plain"), ((130265, 1, 1, 47), FWD_RES, "plain"), ((154066, 1, 1, 113), BWD_RES, "plain"),
    ((179444, 3, 1, 5), BWD_RES, "plain"), ((40523, 1, 1, 46), BWD_RES, "plain"),
    ((110600, 1, 1, 165), FWD, "tiled"), ((2705, 2, 1, 818), FWD, "tiled"), ((2705, 2, 1, 818), BWD, "tiled"), ((2705, 2, 1, 818), FWD_RES, "tiled"),
    ((3967, 3, 1, 209), BWD_RES, "tiled"), ((4096, 3, 1, 243), BWD, "tiled"),
    ((119, 12, 1, 3886), FWD_RES, "tiled"), ((392, 12, 1, 1225), FWD_RES, "tiled"), ((33, 25, 1, 6426), BWD, "tiled"), ((1057, 8, 1, 650), FWD, "tiled"),
    ((4, 2048, 1, 435), FWD, "register"), ((4, 2048, 1, 435), FWD_RES, "register"), ((1, 2048, 1, 1218), BWD, "register"), ((1, 1409, 1, 2746), FWD, "register")])
def test_stays_with_the_kernel_named_for_it(shape, call, named):
    from anode_b200 import ops
    direction, residual = call
    assert ops.serving_kernel(shape, direction, residual=residual) == named
    assert ops.launched_kernel(shape, direction, residual=residual) == named


@pytest.mark.parametrize("shape,call,launched", [
    ((4096, 3, 7, 7), BWD, "stream"), ((2374, 147, 1, 83), BWD_RES, "stream"), ((4160, 7, 1, 33), FWD, "stream"), ((1403, 355, 1, 131), FWD, "stream"), ((1826, 159, 1, 179), BWD, "stream"),
    ((32, 42, 11, 680), FWD, "long"), ((3, 1199, 1, 2091), FWD, "long"), ((1993, 4, 1, 307), BWD, "stream"), ((1, 3, 1, 262144), FWD, "long"), ((41, 6, 64, 64), BWD, "long"), ((3, 512, 1, 2003), BWD_RES, "long"), ((3, 1023, 1, 1467), BWD_RES, "long")])
def test_goes_where_it_is_faster(shape, call, launched):
    from anode_b200 import ops
    assert ops.launched_kernel(shape, call[0], residual=call[1]) == launched


@pytest.mark.parametrize("shape,call,launched", [
    ((207, 54, 1, 262), BWD, "stream"), ((169, 32, 1, 254), BWD_RES, "stream"), ((22, 450, 1, 262), FWD_RES, "stream"), ((156, 32, 1, 262), BWD_RES, "long"),
    ((496, 20, 1, 253), FWD, "long"), ((197, 44, 1, 270), BWD, "long"), ((183, 46, 1, 350), FWD_RES, "long")])
def test_the_smaller_estimate_of_the_two(shape, call, launched):
    from anode_b200 import ops
    assert ops.launched_kernel(shape, call[0], residual=call[1]) == launched
