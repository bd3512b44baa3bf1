"""The grouped line FFT in stage order repeats the stage-by-stage form operation for operation: the FP32 projector
coefficients of the two are equal bit for bit, at fixed and run-time lengths, groups of one stage and of
several, and every radix. (90^3 repeats the register kernels instead.)"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,encut,gamma", [
    ((14, 15, 16), 60.0, False), ((28, 28, 28), 200.0, False), ((26, 21, 27), 150.0, True), ((25, 33, 35), 150.0, False),
    ((49, 26, 32), 150.0, False), ((42, 98, 40), 200.0, False), ((54, 64, 72), 200.0, False), ((100, 100, 100), 200.0, True),
])
def test_projections_of_the_two_forms_are_equal(dim, encut, gamma, monkeypatch):
    from test_gpu_fft_grouped import projections, wavefunction

    monkeypatch.delenv("PAWPY_GPU_FFT", raising=False)
    mine = projections(wavefunction(dim, encut, gamma=gamma)[0])
    monkeypatch.setenv("PAWPY_GPU_FFT", "generic")
    assert np.array_equal(mine, projections(wavefunction(dim, encut, gamma=gamma)[0]))
