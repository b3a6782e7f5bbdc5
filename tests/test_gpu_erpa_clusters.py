"""The refined ERPA form on a spectrum with more clusters of close eigenvalues than the block kernels
have blocks (304 block solves, 64 rows of blocks in the products): each walks its list further.
Tolerances of the clustered spectra: 1e-9 of the largest element with FP64 products and two iterations,
1e-7 with FP64TC5 products."""
import numpy as np
import pytest

from .test_gpu_erpa_refined import erpa_identity_plus, planted_spectrum, yyT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-9), ("fp64tc5", 1e-7)])
def test_more_clusters_than_blocks(gpu_lib, precision, tol):
    M, _ = planted_spectrum(800, 21, [(s, [0.0, 1e-9]) for s in range(100, 800, 2)])
    w, U = np.linalg.eigh(M)
    om = np.sqrt(np.abs(w))
    ref = yyT(U / np.sqrt(2 * np.where(w > 1e-6, om, 1.0))[None, :], np.where(w > 1e-6, om, w))
    Y, e, st = erpa_identity_plus(M, "refined", precision)
    assert st["fallbacks"] == 0 and 2 <= st["max_cluster"] <= 8, st
    assert np.abs(yyT(Y, e) - ref).max() < tol * np.abs(ref).max()
