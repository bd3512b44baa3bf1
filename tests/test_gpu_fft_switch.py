"""A grouped band FFT on plane lists that were made while PAWPY_GPU_FFT=generic chose the stage-by-stage form:
the positions in its tile are made when it first runs. Bound: the overlaps of two forms, 1e-5 each of FP64."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [(28, 28, 28), (25, 33, 35)])
def test_grouped_form_after_lists_of_the_other(dim, monkeypatch):
    from pawpyseed_gb300 import _lib
    from pawpyseed_gb300.projector import Projector
    from test_gpu_fft_grouped import wavefunction

    def overlaps(lists):
        pair = [wavefunction(dim, 150.0, seed=3)[0] for _ in range(2)]
        # with the transform deferred, the setup makes the lists only
        _lib.lib().pawpy_gpu_set_host_projections(0)
        try:
            monkeypatch.setenv("PAWPY_GPU_FFT", lists)
            for w in pair:
                w.check_c_projectors()
            monkeypatch.setenv("PAWPY_GPU_FFT", "")
            return Projector(*pair).project_all()
        finally:
            _lib.lib().pawpy_gpu_set_host_projections(1)

    plain, late = overlaps(""), overlaps("generic")
    assert np.abs(plain).max() > 0.5
    assert np.abs(late - plain).max() <= 2e-5
