"""Result arrays of complex128 values that lie at 8 modulo 16 bytes (a view into a record or a mapped
file; the type needs 8): every entry point that writes such an array gives the values it gives in an
aligned one, which are written by the device in place where it can reach host memory."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def placed(n, off):
    """n zeros of complex128 whose address is off modulo 16."""
    raw = np.zeros(16 * n + 32, dtype=np.uint8)
    at = (off - raw.ctypes.data) % 16
    v = raw[at:at + 16 * n].view(np.complex128)
    assert v.ctypes.data % 16 == off
    return v


@pytest.mark.parametrize("method", ["aug_real", "aug_recip"])
def test_projections_into_an_array_at_8_modulo_16(method, workload_dirs):
    from pawpyseed_gb300 import _lib
    from pawpyseed_gb300.projector import Projector
    from pawpyseed_gb300.wavefunction import Wavefunction

    dirs = workload_dirs("cfg1s")
    basis, wf = Wavefunction.from_directory(dirs["basis"]), Wavefunction.from_directory(dirs["defect"])
    pr = Projector(wf, basis, method=method)
    L, n = _lib.lib(), basis.nband * basis.nwk * basis.nspin
    got = {}
    for off in (0, 8):
        pseudo, total = placed(n, off), placed(n, off)
        L.pseudoprojection(pseudo, basis.wf_ptr, wf.wf_ptr, 1, 0)
        _lib.check()
        # the augmentation terms are added to what the array holds
        total[:] = pseudo
        pr._add_augmentation_terms(total, 1, False)
        every = placed(wf.nband * n, off)
        L.pawpy_gpu_project_all(every, basis.wf_ptr, wf.wf_ptr, len(pr.M_R), len(pr.N_R), len(pr.N_S),
                                len(pr.N_RS_R), *pr._lists(), 0)
        _lib.check()
        got[off] = pseudo.copy(), total.copy(), every.copy()
    for a, b in zip(got[0], got[8]):
        assert np.abs(a).max() > 0
        assert np.array_equal(a, b)


def test_realspace_projections_into_an_array_at_8_modulo_16(realspace_dirs):
    from pawpyseed_gb300 import _lib
    from pawpyseed_gb300.projector import Projector
    from pawpyseed_gb300.wavefunction import Wavefunction

    basis, wf = Wavefunction.from_directory(realspace_dirs["basis"]), Wavefunction.from_directory(realspace_dirs["defect"])
    Projector(wf, basis, method="realspace")
    L, n, g = _lib.lib(), basis.nband * basis.nwk * basis.nspin, np.array([20, 18, 21], dtype=np.int32)
    got = {}
    for off in (0, 8):
        one, every = placed(n, off), placed(wf.nband * n, off)
        L.project_realspace_state(one, 1, wf.wf_ptr, basis.wf_ptr, g, wf.nums, wf.coords, basis.nums, basis.coords)
        _lib.check()
        L.pawpy_gpu_project_realspace_all(every, wf.wf_ptr, basis.wf_ptr, g, wf.nums, wf.coords, basis.nums,
                                          basis.coords)
        _lib.check()
        got[off] = one.copy(), every.copy()
    for a, b in zip(got[0], got[8]):
        assert np.abs(a).max() > 0
        assert np.array_equal(a, b)
