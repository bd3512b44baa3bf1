"""The rules by which the library holds more on the device than a call needs, as host functions of sizes,
and the calls that follow them."""

import ctypes as C

import numpy as np
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


def test_contractions_of_one_launch_stay_within_its_grid_and_workspace():
    group = rule("_ZN5pawpy15grouped_batchesEiix", C.c_int, C.c_int, C.c_int, C.c_longlong)
    assert group(8, 64, 64 * 32 * 32 * 8) == 8
    assert group(1100, 64, 64 * 4 * 8) == 1023  # x 64 splits: 65,472 of 65,535
    assert group(70000, 1, 0) == 65535
    assert group(100, 5, 5 * 512 * 512 * 8) == 25
    assert group(3, 2, 2 * 8192 * 8192 * 8) == 1


@pytest.mark.gpu
def test_realspace_projections_of_more_than_a_thousand_k_points():
    """1,100 k-points of a contraction in 64 splits: more than one launch's grid holds. Bound: both sides'
    states in FP32 and the contraction over 32,768 points, 1e-5 as the other real-space projections."""
    from pawpyseed_gb300.projector import Projector
    from test_gpu_fft_grouped import wavefunction

    wf, _ = wavefunction((16, 16, 16), 20.0, nk=1100, nband=2, seed=3)
    basis, _ = wavefunction((16, 16, 16), 20.0, nk=1100, nband=3, seed=3)
    out = Projector(wf, basis, method="realspace").project_all()
    vol, n3 = abs(np.linalg.det(wf.structure.lattice)), 32**3
    for k in (0, 600, 1022, 1023, 1099):
        S = np.array([wf.get_state_realspace(b, k, 0, dim=(32, 32, 32)).ravel() for b in range(2)])
        R = np.array([basis.get_state_realspace(b, k, 0, dim=(32, 32, 32)).ravel() for b in range(3)])
        assert np.abs(out[:, k::1100] - S @ R.conj().T * vol / n3).max() <= 1e-5


def test_scratch_of_the_real_space_functions_follows_the_free_memory():
    pieces = rule("_ZN5pawpy14scratch_piecesExxxx", C.c_int, C.c_longlong, C.c_longlong, C.c_longlong, C.c_longlong)
    MB, many = 1 << 20, 1 << 62
    # 16 band grids of 216 MB: all on a free device, nine of them in 8 GB, four (1 GiB) where little is free
    assert pieces(16, 216 * MB, many, 270 * GB) == 16
    assert pieces(16, 216 * MB, many, 8 * GB) == 9
    assert pieces(16, 216 * MB, many, 1 * GB) == 4
    assert pieces(16, 1100 * MB, many, 2 * GB) == 1
    # k-points of 500 MB: at most 8 GB of them
    assert pieces(100, 500 * MB, 8 * GB, 270 * GB) == 16
    # little scratch is taken whatever is free
    assert pieces(16, 64 * MB, many, 0) == 16


DENSITY = """
import numpy as np, torch
from test_gpu_fft_grouped import wavefunction
from pawpyseed_gb300 import _lib, synth, vaspio
from pawpyseed_gb300.wavefunction import Wavefunction
st, _ = synth.structures(0)
cr = vaspio.CoreRegion(synth.potcar_text(["A"]))
w = dict(encut=30.0, kpts=np.array([[0.1, 0.2, 0.3]]), nband=32, nspin=1, dim=(16, 16, 16))
data = synth.wavefunction_data(st, w, 3)
data["occs"] = np.asarray([[[float(b % 2 == 0) for b in range(32)]]]).reshape(np.asarray(data["occs"]).shape)
wf = Wavefunction.from_arrays(st, cr, (16, 16, 16), data)
wf.get_realspace_density(dim=(18, 18, 18))
wf.get_state_realspace(0, 0, 0, dim=(216, 216, 216))  # the sphere tables of the grid
_lib.lib().pawpy_gpu_synchronize()
free = torch.cuda.mem_get_info()[0]
wf.get_realspace_density(dim=(216, 216, 216))
_lib.lib().pawpy_gpu_synchronize()
print((free - torch.cuda.mem_get_info()[0]) // (8 * 216**3))
"""


@pytest.mark.gpu
def test_density_of_separate_bands_holds_one_grid_at_a_time():
    """16 occupied bands, none beside another: the grids the call adds to the pool (one band's and its density
    fit in what the state before it left there) are fewer than a few, not 16."""
    import os
    import subprocess
    import sys

    from conftest import ROOT

    env = dict(os.environ, PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests")]))
    r = subprocess.run([sys.executable, "-c", DENSITY], capture_output=True, text=True, env=env, cwd=ROOT)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout.split()[-1]) <= 4


@pytest.mark.gpu
def test_state_on_a_grid_whose_bloch_factors_are_tabulated_in_slabs():
    """270 x 256 x 252 points (a table of 279 MB) against every other point's grid, where it is built whole: the
    same values at the same points, 1e-5 of the largest as the other states."""
    from test_gpu_fft_grouped import wavefunction

    wf, _ = wavefunction((16, 16, 16), 60.0)
    fine = wf.get_state_realspace(3, 1, 0, dim=(270, 256, 252))[::2, ::2, ::2]
    coarse = wf.get_state_realspace(3, 1, 0, dim=(135, 128, 126))
    assert np.abs(fine - coarse).max() <= 1e-5 * np.abs(coarse).max()
    rf = wf.get_realspace_density(dim=(270, 256, 252))[::2, ::2, ::2]
    rc = wf.get_realspace_density(dim=(135, 128, 126))
    assert np.abs(rf - rc).max() <= 1e-5 * np.abs(rc).max()
