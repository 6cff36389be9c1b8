"""Which convolutions run on the image and which gathered is a rule on their sizes."""
import pytest

from necklace_b200 import _lib

pytestmark = pytest.mark.skipif(not _lib.available(), reason="native library not built")


def _route(N, H, W, C, Cout, k, stride):
    return _lib.value("nkb_conv_route", N, H, W, C, Cout, k, k, stride, k // 2)


def test_pixels_enough_and_64_channels_run_on_the_image():
    for C, hw in ((64, 56), (128, 28), (256, 14), (512, 7)):
        assert _route(256, hw, hw, C, C, 3, 1) == 3
    for C, hw in ((128, 56), (256, 28), (512, 14)):
        assert _route(256, hw, hw, C, C, 3, 2) == 3
        assert _route(256, hw, hw, 2 * C, 4 * C, 1, 2) == 3
    assert _route(33, 40, 53, 64, 128, 3, 1) == 3


def test_few_pixels_with_a_long_contraction_are_gathered():
    # a handful of tiles, each running through taps x channels; the GEMM of the gathered form
    # has slices
    assert _route(8, 14, 14, 512, 512, 3, 2) == 0
    assert _route(1, 28, 28, 512, 512, 3, 1) == 0
    assert _route(1, 7, 7, 512, 512, 5, 1) == 0


def test_few_channels_are_gathered():
    assert _route(128, 56, 56, 8, 64, 3, 1) == 0
    assert _route(64, 28, 28, 8, 8, 5, 1) == 0


def test_what_the_kernels_cannot_take():
    for bad in ((1, 8, 8, 12, 8, 3, 1), (1, 8, 8, 8, 12, 3, 1), (1, 8, 8, 8, 8, 3, 3),
                (0, 8, 8, 8, 8, 3, 1), (1, 1, 1, 8, 8, 4, 1)):
        N, H, W, C, Cout, k, s = bad
        assert _lib.value("nkb_conv_route", N, H, W, C, Cout, k, k, s, 0) == -3
