"""The FP64 cooperative solve around its panels, tiles and slabs (dimensions at and beside multiples of 8
and 32, one and many CTAs, more panel columns per CTA than its slab) against the oracle bit for bit, and
the shift update and merge for words that every client or no client selected."""
import numpy as np
import pytest

from ufednl_gb300 import datagen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from ufednl_gb300 import build, fednl
    build.build()
    fednl.load()
    return fednl


@pytest.mark.parametrize("d", [1, 2, 7, 8, 31, 32, 33, 39, 40, 41, 47, 63, 64, 65, 71, 96, 97, 128, 200, 340, 512])
def test_solve_sizes(gpu, oracle, d):
    rng = np.random.default_rng(d)
    lda = (d + 3) // 4 * 4
    a = rng.standard_normal((d + 8, d))
    H = np.zeros((d, lda))
    H[:, :d] = a.T @ a / (d + 8) + 1e-3 * np.eye(d)
    g = rng.standard_normal(d)
    got = gpu.cholesky_option_b_solve(H.reshape(-1), d, lda, 0.05, g)
    x = np.linalg.solve(H[:, :d] + 0.05 * np.eye(d), g)
    np.testing.assert_allclose(got, x, rtol=1e-9, atol=1e-9 * np.abs(x).max())
    prob = datagen.dense_problem(80 + d, d, [7, 5], 1e-2) if d > 1 else None
    if prob is not None and d <= 128:
        U = d * (d + 1) // 2
        fed = gpu.FedNL(prob, "identity", U, 1.0, feature_format=2)
        orc = oracle.FedNL(prob, "identity", U, 1.0, workers=1, threads=1)
        for _ in range(2):
            fed.round()
            orc.round()
            np.testing.assert_array_equal(fed.x(), orc.x())
        fed.close()
        orc.close()


@pytest.mark.parametrize("comp,alpha", [("topk", 1.0), ("topk", 0.75), ("randk", 0.3), ("natural", 8 / 9)])
@pytest.mark.parametrize("clients", [3, 31, 32, 33, 70])
def test_merge_words(gpu, oracle, comp, alpha, clients):
    """k small: the first words kept by nearly all clients, the last by hardly any."""
    prob = datagen.binary_problem(91, 25, [12 + c % 7 for c in range(clients)], 0.2, 1e-2)
    fed = gpu.FedNL(prob, comp, 40, alpha)
    orc = oracle.FedNL(prob, comp, 40, alpha, workers=1, threads=1)
    for _ in range(3):
        fed.round()
        orc.round()
        np.testing.assert_array_equal(fed.x(), orc.x())
        # column-major, the upper triangle is current (rows i <= column j: numpy's lower one)
        np.testing.assert_array_equal(np.tril(fed.H().reshape(25, -1)[:, :25]), np.tril(orc.H().reshape(25, -1)[:, :25]))
        for c in (0, clients // 2, clients - 1):
            np.testing.assert_array_equal(fed.shift(c), orc.shift(c))
    fed.close()
    orc.close()
