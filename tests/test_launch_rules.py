"""Launch rules on the host side of the CUDA library, called without a GPU."""
import ctypes

import pytest

CANDIDATES = (8, 16, 32, 64)  # z-planes that sclet_tune tries
SMS = 152


def _symbol(sg, name, restype, *args):
    f = getattr(sg.lib(), name)
    f.restype, f.argtypes = restype, args
    return f


@pytest.mark.parametrize("tensors", [False, True])
def test_tuned_planes_fill_the_gpu_as_the_default_does(tensors, sclet_lib):
    """The default shape is one of the tuner's candidates, and no candidate
    leaves SMs without the four CTAs that a finer march would give them."""
    planes = _symbol(sclet_lib, "_ZN5sclet13rhs_ac_planesEiibxi", ctypes.c_int, ctypes.c_int, ctypes.c_int,
                     ctypes.c_bool, ctypes.c_longlong, ctypes.c_int)
    for n in (8, 12, 36, 52, 68, 101, 196, 516, 1028):
        for runs in (1, 2, 7, 300):
            tiles = -(-(n - 2) ** 2 // 256) * runs
            tried = [planes(n, c, tensors, tiles, runs) for c in CANDIDATES]
            assert planes(n, 0, tensors, tiles, runs) in tried, (n, runs)
            most = tiles * -(-n // 2)
            for zc in tried:
                assert zc >= 2 and tiles * -(-n // zc) >= min(4 * SMS, most), (n, runs, zc)
