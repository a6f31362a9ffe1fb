"""Which convolutions ask for the scratch of the two-term products (host arithmetic: runs without a GPU)."""
import ctypes

import pytest


@pytest.fixture
def scratch(monkeypatch):
    from mytorch_b200.backends.cuda.env import LIBRARY_PATH

    fn = ctypes.CDLL(LIBRARY_PATH).mtb_conv2d_workspace_bytes
    fn.restype = ctypes.c_longlong

    def both(*args):
        """(bytes asked for, bytes without those products)"""
        asked = fn(*args)
        monkeypatch.setenv("MTB_DISABLE_TC_SPLIT", "1")
        without = fn(*args)
        monkeypatch.delenv("MTB_DISABLE_TC_SPLIT")
        return asked, without

    return both


def test_taken_where_they_pay(scratch):
    asked, without = scratch(32, 48, 37, 37, 3, 3, 1, 1, 1, 1, 82)
    assert asked > without


def test_weight_gradients_over_few_pixels_are_not_taken(scratch):
    asked, without = scratch(1, 1500, 6, 6, 7, 7, 1, 1, 3, 3, 470)  # no other direction of it is taken either
    assert asked == without


def test_scratch_is_bounded(scratch):
    """64 MB of packed activations an operand or one image of at most 256 MB, a packed filter of at most 256 MB, and planes of
    sums only where a weight gradient is added up from several."""
    header = 4 * 3 * 1024
    # forward and data gradient of 2000 -> 470, 7x7 would pack 370 MB of filter; its weight gradient over one image is written in one piece
    asked, without = scratch(1, 2000, 11, 11, 7, 7, 1, 1, 3, 3, 470)
    assert without < asked == header + 121 * (63 + 15) * 256
