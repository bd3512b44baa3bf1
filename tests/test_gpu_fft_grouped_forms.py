"""The grouped band FFT in the forms that test_gpu_fft_grouped.py does not reach: the second pass that writes
whole grids (resident basis, defect grids), the second pass on planes issued at setup when a switch has changed
the form since, and the densities' tiles of 2, 4 and 16 bands, full and partial, of consecutive and separate bands.

Bounds: overlaps 1e-5 of FP64 for each of two forms; with the same kernels behind both, 2e-6 (the split-BF16
contraction in another tiling); densities 1e-5 of the largest value, as the other real-space tests."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [((28, 28, 28), 150.0), ((25, 33, 35), 150.0), ((56, 56, 56), 150.0), ((54, 64, 72), 200.0)]


def pair(dim, encut, nband):
    """Basis and defect (one atom displaced: both structures' smoothed waves are projected) at two k-points."""
    from pawpyseed_gb300 import synth, vaspio
    from pawpyseed_gb300.wavefunction import Wavefunction

    cr = vaspio.CoreRegion(synth.potcar_text(["A"]))
    w = dict(encut=encut, kpts=np.array([[0.11, -0.23, 0.31], [0.0, 0.0, 0.0]]), nband=nband, nspin=1, dim=dim)
    return [Wavefunction.from_arrays(st, cr, dim, synth.wavefunction_data(st, w, seed))
            for seed, st in enumerate(synth.structures(0))]


@pytest.mark.parametrize("dim,encut", GRIDS)
@pytest.mark.parametrize("nband", [5, 17])
def test_whole_grids_match_the_stage_by_stage_form(dim, encut, nband, monkeypatch):
    from pawpyseed_gb300 import _lib
    from pawpyseed_gb300.projector import Projector

    L = _lib.lib()

    def overlaps(resident):
        basis, wf = pair(dim, encut, nband)
        basis.check_c_projectors()
        assert L.pawpy_gpu_prepare_basis(basis.wf_ptr, int(resident)) == int(resident)
        return Projector(wf, basis).project_all()

    L.pawpy_gpu_set_sphere_contraction(2)
    try:
        monkeypatch.setenv("PAWPY_GPU_DEFECT_GRID", "1")
        mine = overlaps(True)
        monkeypatch.setenv("PAWPY_GPU_DEFECT_GRID", "0")
        monkeypatch.setenv("PAWPY_GPU_FFT", "generic")
        ref = overlaps(False)
    finally:
        L.pawpy_gpu_set_sphere_contraction(1)
    assert np.abs(ref).max() > 0
    assert np.abs(mine - ref).max() <= 2e-5


@pytest.mark.parametrize("dim,encut,switch", [
    ((90, 90, 90), 60.0, ("PAWPY_GPU_XPICK_TC", "1")), ((90, 90, 90), 60.0, ("PAWPY_GPU_FFT", "generic")),
    ((28, 28, 28), 150.0, ("PAWPY_GPU_FFT", "generic")), ((25, 33, 35), 150.0, ("PAWPY_GPU_FFT", "generic")),
])
def test_second_pass_follows_planes_issued_at_setup(dim, encut, switch, monkeypatch):
    from pawpyseed_gb300 import _lib
    from pawpyseed_gb300.projector import Projector

    L = _lib.lib()

    def launches(f):
        L.pawpy_gpu_synchronize()
        _lib.kernel_stats(reset=True)
        L.pawpy_gpu_profile(1)
        try:
            f()
            L.pawpy_gpu_synchronize()
        finally:
            L.pawpy_gpu_profile(0)
        s = _lib.kernel_stats(reset=True)
        return {k: s[k][1] if k in s else 0 for k in ("fft_planes", "fft_x_pick")}

    def overlaps(late):
        monkeypatch.setenv("PAWPY_GPU_EARLY_FFT", "1")
        monkeypatch.delenv(switch[0], raising=False)
        basis, wf = pair(dim, encut, 5)
        basis.check_c_projectors()
        # with the basis's grids resident, the defect's passes are the only ones
        assert L.pawpy_gpu_prepare_basis(basis.wf_ptr, 1) == 1
        first = launches(wf.check_c_projectors)
        assert first["fft_planes"] > 0 and first["fft_x_pick"] == 0
        if late:
            monkeypatch.setenv(*switch)
        out = []
        second = launches(lambda: out.append(Projector(wf, basis).project_all()))
        assert second["fft_planes"] == 0 and second["fft_x_pick"] > 0
        return out[0]

    _lib.set_precision("bf16x3")
    L.pawpy_gpu_set_host_projections(0)
    try:
        plain, late = overlaps(False), overlaps(True)
    finally:
        L.pawpy_gpu_set_host_projections(1)
        _lib.set_precision("fp32")
    assert np.abs(plain).max() > 0
    assert np.abs(late - plain).max() <= 2e-6


@pytest.mark.parametrize("occupied", [
    [0, 1, 2], [0, 1, 2, 3], list(range(5)), list(range(15)), list(range(17)), list(range(33)), [0, 2, 4, 5, 6, 7, 20, 31, 32],
])
def test_densities_in_tiles_of_every_width(occupied):
    import oracle as orc

    from pawpyseed_gb300 import synth, vaspio
    from pawpyseed_gb300.wavefunction import Wavefunction

    st, _ = synth.structures(0)
    cr = vaspio.CoreRegion(synth.potcar_text(["A"]))
    w = dict(encut=40.0, kpts=np.array([[0.0, 0.0, 0.0], [0.1, -0.2, 0.3]]), nband=33, nspin=1, dim=(16, 16, 16))
    data = synth.wavefunction_data(st, w, 5)
    occ = np.zeros_like(np.asarray(data["occs"], dtype=np.float64)).reshape(2, 33)
    occ[:, occupied] = np.linspace(0.3, 1.0, len(occupied))
    data["occs"] = occ.reshape(np.asarray(data["occs"]).shape)
    rho = Wavefunction.from_arrays(st, cr, (16, 16, 16), data).get_realspace_density(dim=(18, 20, 21))
    ow = orc.OracleWavefunction(data=data, struct=st, cr=cr, dim=(16, 16, 16))
    ow.setup_projectors()
    truth = ow.ae_chg_density((18, 20, 21))
    assert truth.max() > 0
    assert np.abs(rho - truth).max() <= 1e-5 * truth.max()


def test_real_space_overlaps_in_batches_of_bands_and_k_points():
    """120 basis bands on 216^3, transformed in batches of 1 GiB of planes, the grids of one k-point (9.7 GB) at
    a time: each value is the sum over its states."""
    from pawpyseed_gb300.projector import Projector
    from test_gpu_fft_grouped import wavefunction

    dim = (216, 216, 216)
    basis = wavefunction((24, 24, 24), 200.0, nk=2, nband=120, seed=3)[0]
    wf = wavefunction((24, 24, 24), 200.0, nk=2, nband=1, seed=3)[0]
    out = Projector(wf, basis, method="realspace")._single_band_projection_realspace(0, dim=dim)
    vol = abs(np.linalg.det(wf.structure.lattice))
    for k in (0, 1):
        s = wf.get_state_realspace(0, k, 0, dim=dim).ravel()
        for b in (0, 110, 111, 119):
            r = basis.get_state_realspace(b, k, 0, dim=dim).ravel()
            assert abs(out[2 * b + k] - np.vdot(r, s) * vol / 216**3) <= 1e-5
