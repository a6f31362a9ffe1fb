"""No SM may hold CTAs of two of the kernels by pairs of SMs: they wait for tensor memory without a limit, holding what the other CTA of the pair has got (no GPU)."""
import ctypes


def test_two_never_fit_one_sm():
    from mytorch_b200.backends.cuda.env import LIBRARY_PATH

    smem = ctypes.CDLL(LIBRARY_PATH).mtb_conv2d_pair_smem_bytes
    smem.argtypes, smem.restype = [ctypes.c_int] * 12, ctypes.c_longlong
    seen = [0, 0, 0]
    for w in list(range(1, 130)) + [190, 254]:
        for h in (1, 7, 56):
            for cin in (64, 96, 128):
                for cout in (36, 48, 64, 96, 128):
                    for direction in range(3):
                        for n in (3, 3000):
                            own = smem(n, cin, h, w, 3, 3, 1, 1, 1, 1, cout, direction)
                            # 228 KB a SM, of which a CTA takes 1 KB beside its own; at most 227 KB a CTA, 4 of which are left to static variables
                            assert own == 0 or 2 * (own + 1024) > 228 * 1024 and own <= 223 * 1024
                            seen[direction] += own > 0
    assert min(seen) > 500
    assert smem(3, 64, 7, 7, 5, 5, 1, 1, 2, 2, 64, 2) == 0
