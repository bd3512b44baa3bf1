"""The rules by which the library holds more on the device than a call needs, as host functions of sizes,
and the calls that follow them."""

import ctypes as C

import pytest

GB = 1 << 30


def rule(name, restype, *argtypes):
    from pawpyseed_gb300 import _lib

    f = getattr(_lib.lib(), name)
    f.restype, f.argtypes = restype, list(argtypes)
    return f


def test_real_space_wavefunctions_leave_half_of_the_device_free():
    keeps = rule("_ZN5pawpy16keeps_real_spaceExxx", C.c_bool, C.c_longlong, C.c_longlong, C.c_longlong)
    assert keeps(71 * GB, 270 * GB, 280 * GB)
    assert keeps(130 * GB, 270 * GB, 280 * GB)
    assert not keeps(131 * GB, 270 * GB, 280 * GB)
    assert not keeps(1, 100 * GB, 280 * GB)


@pytest.mark.gpu
def test_basis_larger_than_that_is_prepared_without_them():
    """4,096 bands on 168^3, a grid of the grouped band FFT: 155 GB of real-space wavefunctions."""
    from pawpyseed_gb300 import _lib
    from test_gpu_fft_grouped import wavefunction

    wf, _ = wavefunction((168, 168, 168), 8.0, nband=4096, gamma=True)
    wf.check_c_projectors()
    assert _lib.lib().pawpy_gpu_prepare_basis(wf.wf_ptr, 1) == 0
    _lib.check()


@pytest.mark.gpu
def test_smaller_basis_on_such_a_grid_keeps_them():
    from pawpyseed_gb300 import _lib
    from test_gpu_fft_grouped import wavefunction

    wf, _ = wavefunction((14, 15, 16), 60.0)
    wf.check_c_projectors()
    assert _lib.lib().pawpy_gpu_prepare_basis(wf.wf_ptr, 1) == 1
    _lib.check()
