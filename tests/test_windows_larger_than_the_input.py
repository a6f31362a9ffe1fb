"""A filter or window that does not fit the padded input has no output: every entry point says so, whatever its stride
(one that is short by less than a stride has an output extent of 1 where the division rounds towards zero)."""
import pytest

from mytorch_b200.backends.cuda.env import LIBRARY_PATH, NativeError, _binding

POINTER = 1 << 20  # never dereferenced: the calls are refused before anything is enqueued


@pytest.mark.parametrize("cin,cout", [(32, 32), (64, 128), (8, 12), (3, 64)])
@pytest.mark.parametrize("h,w,kh,kw,s,p", [(64, 64, 65, 3, 2, 0), (64, 64, 3, 67, 4, 1), (64, 63, 66, 66, 2, 0), (64, 64, 70, 70, 1, 1)])
def test_refused(cin, cout, h, w, kh, kw, s, p):
    _binding.load(LIBRARY_PATH, NativeError)
    lib, dims = _binding, (8, cin, h, w, kh, kw, s, s, p, p)
    conv = (*dims, cout)
    room = max(lib.conv2d_workspace_bytes(*conv), 1 << 20)
    end = (POINTER, room, None)
    calls = [lambda: lib.conv2d_forward_f32(*conv, POINTER, POINTER, None, POINTER, 0, *end),
             lambda: lib.conv2d_bn_forward_f32(*conv, POINTER, POINTER, None, None, None, POINTER, POINTER, 1e-5, None, 0, POINTER, *end),
             lambda: lib.conv2d_dgrad_f32(*conv, POINTER, POINTER, POINTER, *end),
             lambda: lib.conv2d_dgrad_add_f32(*conv, POINTER, POINTER, 2 * POINTER, POINTER, *end),
             lambda: lib.conv2d_wgrad_f32(*conv, POINTER, POINTER, POINTER, *end),
             lambda: lib.max_pool2d_forward_f32(*dims, POINTER, POINTER, None, None),
             lambda: lib.max_pool2d_backward_f32(*dims, POINTER, None, POINTER, POINTER, POINTER, None)]
    for call in calls:
        with pytest.raises(NativeError, match="is larger than the padded"):
            call()


def test_packing_a_window_larger_than_the_input():
    _binding.load(LIBRARY_PATH, NativeError)
    with pytest.raises(NativeError, match="is larger than the padded"):
        _binding.pack_patches_f32(64, 3, 64, 4, 1, 5, 1, 2, 0, 0, POINTER, POINTER, None)
