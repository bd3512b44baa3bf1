"""Real-space functions on grids with a length that does not split into two groups (210 = 2 x 3 x 5 x 7,
245 = 5 x 7 x 7): states against the grid of every other point, overlaps against the sums over the states
where the rows are padded (a number of points that is no multiple of 16), and a batch of bands in as many
launches as one band.

Bounds: FP32 transforms and sums, 1e-5 of the largest value."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_states_on_every_other_point_agree():
    from test_gpu_fft_grouped import wavefunction

    wf, _ = wavefunction((16, 16, 16), 60.0)
    fine = wf.get_state_realspace(3, 1, 0, dim=(210, 28, 36))[::2, ::2, ::2]
    coarse = wf.get_state_realspace(3, 1, 0, dim=(105, 14, 18))
    assert np.abs(fine - coarse).max() <= 1e-5 * np.abs(coarse).max()


def test_overlaps_with_padded_rows():
    from pawpyseed_gb300.projector import Projector
    from test_gpu_fft_grouped import wavefunction

    wf, basis = wavefunction((16, 16, 16), 60.0, seed=3)[0], wavefunction((16, 16, 16), 60.0, seed=3)[0]
    dim = (245, 15, 15)
    pr = Projector(wf, basis, method="realspace")
    vol, n3 = abs(np.linalg.det(wf.structure.lattice)), int(np.prod(dim))
    assert n3 % 16
    out = pr._single_band_projection_realspace(2, dim=dim)
    for k in range(2):
        s = wf.get_state_realspace(2, k, 0, dim=dim).ravel()
        R = np.array([basis.get_state_realspace(b, k, 0, dim=dim).ravel() for b in range(basis.nband)])
        assert np.abs(out[k::2] - R.conj() @ s * vol / n3).max() <= 1e-5


@pytest.mark.parametrize("dim", [(210, 16, 16), (245, 15, 15)])
def test_a_batch_of_bands_takes_no_more_launches_than_two(dim):
    from pawpyseed_gb300 import _lib
    from test_gpu_fft_grouped import wavefunction

    L, g = _lib.lib(), np.array(dim, dtype=np.int32)
    count = {}
    for nband in (2, 13):
        wf = wavefunction((16, 16, 16), 60.0, nk=1, nband=nband)[0]
        basis = wavefunction((16, 16, 16), 60.0, nk=1, nband=nband)[0]
        wf.check_c_projectors()
        basis.check_c_projectors()
        out = np.zeros(nband * nband, dtype=np.complex128)
        for _ in range(2):  # tables first
            L.pawpy_gpu_launch_count(1)
            L.pawpy_gpu_project_realspace_all(out, wf.wf_ptr, basis.wf_ptr, g, wf.nums, wf.coords, basis.nums,
                                              basis.coords)
            _lib.check()
            count[nband] = L.pawpy_gpu_launch_count(0)
    assert count[2] == count[13]
