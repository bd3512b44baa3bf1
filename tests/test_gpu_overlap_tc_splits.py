"""Tensor-core contractions of one shape and several lengths in one process: the split that was chosen for a long K
must fit the workspace of a shorter one (lengths up to 4,096 share a choice). Bounds: as the other precision
tests, rows of unit norm, 1e-5 of FP64 (split BF16) and 5e-3 (TF32)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("bf16x3", 1e-5), ("tf32", 5e-3)])
@pytest.mark.parametrize("M,N,nz", [(24, 40, 1), (131, 70, 2)])
def test_short_lengths_after_a_long_one(M, N, nz, prec, tol):
    from pawpyseed_gb300 import _lib

    rng = np.random.default_rng(M + N)

    def rows(n, k):
        x = rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k))
        return (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.complex64)

    for k in (4090, 2050, 700, 300, 130, 64, 16, 3900):
        As, Bs = [rows(M, k) for _ in range(nz)], [rows(N, k) for _ in range(nz)]
        out = _lib.overlap_matrix(As, Bs, prec)
        for z in range(nz):
            truth = Bs[z].astype(np.complex128) @ As[z].astype(np.complex128).conj().T
            assert np.abs(out[z] - truth).max() <= tol
