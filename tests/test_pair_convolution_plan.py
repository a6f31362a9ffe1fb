"""Memory of the convolution kernel that works in pairs of SMs, as the host plans it (no GPU)."""
import ctypes


def test_copies_and_descriptors_stay_inside_their_stage():
    from mytorch_b200.backends.cuda.env import LIBRARY_PATH

    lib = ctypes.CDLL(LIBRARY_PATH)
    lib.mtb_conv2d_pair_plan_f32.argtypes = [ctypes.c_int] * 11 + [ctypes.POINTER(ctypes.c_int)]
    out = (ctypes.c_int * 18)()
    taken = 0
    for w in list(range(1, 130)) + [190, 254, 255, 300]:
        for h in (1, 7, 56):
            for cin in (32, 64, 96, 128, 160):
                for cout in (16, 32, 72, 64, 96, 128, 256):
                    assert lib.mtb_conv2d_pair_plan_f32(5, cin, h, w, 3, 3, 1, 1, 1, 1, cout, out) == 0
                    for kc, nout, o in ((cin, cout, 0), (cout, cin, 9)):
                        form, smem, stage, wfirst, wlast, rfirst, rlast, rows, tmem = out[o:o + 9]
                        assert form == 0 or (kc % 32 == 0 and 64 <= kc <= 128 and nout % 16 == 0 and nout >= 64)
                        if form:
                            taken += 1
                            assert form in (1, 2) and smem <= 227 * 1024 - 4096 and stage % 1024 == 0
                            assert 0 <= wfirst < wlast <= stage and 0 <= rfirst < rlast <= stage and rows <= 32 and tmem <= 512
                            assert smem >= 1024 + 2 * stage + kc // 32 * 9 * 4096
    assert taken > 5000
    for bad in ((5, 5, 1, 1, 2, 2), (3, 3, 2, 2, 1, 1), (3, 3, 1, 1, 0, 0), (3, 3, 1, 2, 1, 1), (3, 1, 1, 1, 1, 0)):
        assert lib.mtb_conv2d_pair_plan_f32(5, 64, 32, 32, *bad, 64, out) == 0 and out[0] == out[9] == 0
