"""The triage network's entries refuse activations that are not 16-byte aligned before any
device work: the kernels copy and store them 16 bytes at a time.  No call here needs a GPU."""
import ctypes

import pytest

from msceer_gb300 import _lib, build


@pytest.fixture(scope="module")
def lib():
    build.build_library()
    return _lib.load()


ADDR = 0x7F0000000000  # never read


def _p(off=0):
    return ctypes.c_void_p(ADDR + off)


@pytest.mark.parametrize("off", [2, 8, 14])
@pytest.mark.parametrize("which", [0, 1, 2], ids=["features", "act1", "act2"])
def test_misaligned_activations_are_refused(lib, which, off):
    o = [off if q == which else 0 for q in range(3)]
    dims = _lib.dims_arg((4, 4, 4))
    rc = lib.msc_triage_forward_3d(_p(o[0]), dims, _p(), _p(o[1]), _p(o[2]), _p(), None)
    assert rc < 0 and b"aligned" in lib.msc_triage_last_error_string()
    rc = lib.msc_triage_backward_3d(_p(o[0]), _p(o[1]), _p(o[2]), _p(), _p(), dims, _p(), ctypes.c_float(1.0), _p(),
                                    _p(), None)
    assert rc < 0 and b"aligned" in lib.msc_triage_last_error_string()
