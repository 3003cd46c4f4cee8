"""The mixed form's FP32 solve on thread-block clusters (block rows and columns in the clusters' shared
memory) against the one-CTA solve of the same launch kind: the same operations in the same order, so the
same bits; sizes at the edges of the blocks, of the owners' rounds (16, 32 blocks) and of what fits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from ufednl_gb300 import fednl

    fednl.load()
    return fednl


@pytest.mark.parametrize("d", [321, 352, 353, 511, 512, 513, 544, 800, 1023, 1024, 1025, 1120, 1248, 1249, 1312])
def test_cluster_solves_equal_one_cta(gpu, d):
    rng = np.random.default_rng(d)
    q, _ = np.linalg.qr(rng.standard_normal((d, d)))
    H = (q * np.geomspace(1.0, 1e-4, d)) @ q.T
    H = np.ascontiguousarray((H + H.T) / 2).ravel()
    g = rng.standard_normal(d)
    ref = gpu.cholesky_option_b_solve32(H, d, d, 1e-3, g, grid=7)          # too few CTAs for the clusters
    assert np.isfinite(ref).all()
    for grid in (0, 32, 61, 152, -16, -8):
        np.testing.assert_array_equal(gpu.cholesky_option_b_solve32(H, d, d, 1e-3, g, grid=grid), ref, err_msg=str(grid))
