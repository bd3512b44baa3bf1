"""Which grids the grouped band FFT (csrc/fft_band.cuh) takes, on the host: a plane it accepts fits a
CTA's 227 KiB of shared memory together with the 224 bytes of masks that its first pass keeps beside the
tile."""

import ctypes as C

import pytest


class PlaneGeom(C.Structure):  # csrc/kernels.h
    _fields_ = [(n, C.c_int) for n in ("N1", "N2", "N3", "g1min", "n1", "g2min", "n2", "g3min", "n3", "maxcnt")] + [
        ("grouped", C.c_bool), ("order", C.c_int)]


def supported(n2, n3):
    from pawpyseed_gb300 import _lib

    f = _lib.lib()._ZN5pawpy18fft_band_supportedERKNS_9PlaneGeomE
    f.restype, f.argtypes = C.c_bool, [C.POINTER(PlaneGeom)]
    return f(C.byref(PlaneGeom(12, n2, n3, -2, 5, -2, 5, -2, 5, 13, True, 0)))


@pytest.mark.parametrize("n2,n3", [(216, 132), (130, 220), (110, 260), (66, 432)])
def test_planes_that_do_not_fit_beside_the_masks_are_left_out(n2, n3):
    # the tile alone, rows of an odd number of values, leaves less than the twiddles and masks need
    assert 8 * n2 * (n3 | 1) < 227 * 1024
    assert not supported(n2, n3)


@pytest.mark.parametrize("n2,n3", [(168, 168), (165, 168), (54, 72), (14, 15)])
def test_planes_that_fit_are_taken(n2, n3):
    assert supported(n2, n3)
