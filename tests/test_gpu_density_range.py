"""Densities of wavefunctions far from unit norm: coefficients times a power of two scale every single-precision
value exactly, so the FP64 density scales by its square; |psi|^2 reaches 1e-37 and 1e40, beyond what
single precision holds. Bound: the FP64 sum of the squares of equal single-precision values, 1e-11 of the
largest (the sum over bands is allowed 1e-13)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def density(factor, nband, dim):
    from pawpyseed_gb300 import synth, vaspio
    from pawpyseed_gb300.wavefunction import Wavefunction

    st, _ = synth.structures(0)
    cr = vaspio.CoreRegion(synth.potcar_text(["A"]))
    w = dict(encut=40.0, kpts=np.array([[0.0, 0.0, 0.0], [0.1, -0.2, 0.3]]), nband=nband, nspin=1, dim=(16, 16, 16))
    data = synth.wavefunction_data(st, w, 5)
    data["occs"] = np.ones_like(np.asarray(data["occs"]))
    data["coeffs"] = [np.asarray(c) * np.float32(factor) for c in data["coeffs"]]
    return Wavefunction.from_arrays(st, cr, (16, 16, 16), data).get_realspace_density(dim=dim)


@pytest.mark.parametrize("nband", [2, 3, 17])
@pytest.mark.parametrize("power", [-60, -20, 20, 70])
def test_density_scales_with_the_square(power, nband):
    dim = (18, 20, 21)
    base, scaled = density(1.0, nband, dim), density(2.0**power, nband, dim)
    assert base.max() > 0 and np.all(np.isfinite(scaled))
    assert np.abs(scaled * 4.0**-power - base).max() <= 1e-11 * base.max()
