"""The shuffle behind RandK and the FedNL-PP sampler where its form changes: one step, every place
drawn, the largest shared-memory scratch and the smallest one in global memory, targets that meet
often (k near the number of places); bit-exact against the oracle."""
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


@pytest.mark.parametrize("d,k", [(1, 1), (2, 1), (2, 3), (3, 6), (23, 255), (23, 257), (200, 16384), (200, 16385),
                                 (181, 16471)])
def test_randk_edges(gpu, oracle, d, k):
    lda = (d + 3) // 4 * 4
    states = np.array([7, 123, 0xFFFFFFFF], dtype=np.uint32)
    ref = [np.array([s], dtype=np.uint32) for s in states]
    for _ in range(2):
        got = gpu.generate_randk_items_in_upper_triangular_part(states, d, lda, k)
        for c in range(3):
            np.testing.assert_array_equal(got[c], oracle.randk(ref[c], d, lda, k))
            assert states[c] == ref[c][0]


@pytest.mark.parametrize("clients,tau", [(1, 1), (33, 33), (300, 7), (17000, 16500)])
def test_pp_sampler_edges(gpu, oracle, clients, tau):
    prob = datagen.binary_problem(31, 3, [2] * clients, 0.5, 1e-2)
    fed = gpu.FedNL(prob, "randseqk", 3, 0.5, clients_per_round=tau)
    orc = oracle.FedNL(prob, "randseqk", 3, 0.5, workers=1, threads=1, clients_per_round=tau)
    for _ in range(2):
        fed.round()
        orc.round()
        np.testing.assert_array_equal(fed.selected(), orc.selected())
        np.testing.assert_array_equal(fed.x(), orc.x())
    fed.close()
    orc.close()


@pytest.mark.parametrize("d,k", [(4, 1), (4, 10), (60, 1830), (60, 600)])
def test_randk_philox_edges(gpu, oracle, d, k):
    """One position, every position, and a draw spread over a whole cluster."""
    prob = datagen.binary_problem(32, d, [9, 14, 11], 0.4, 1e-2)
    U = d * (d + 1) // 2
    fed = gpu.FedNL(prob, "randk_philox", k, k / U)
    orc = oracle.FedNL(prob, "randk_philox", k, k / U, workers=1, threads=1)
    for _ in range(2):
        fed.round()
        orc.round()
        for c in range(3):
            np.testing.assert_array_equal(fed.message(c)[0], orc.message(c)[0])
    fed.close()
    orc.close()
