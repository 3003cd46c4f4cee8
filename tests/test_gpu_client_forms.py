"""The client oracle of {0,1} features as one kernel and as two, each on clients of several words of 64 samples
(the order of the word sums, the intercept's own warp), against the oracle bit for bit; and where each is taken:
two only with more clients than resident CTAs and few samples a client."""
import numpy as np
import pytest

from ufednl_gb300 import datagen

pytestmark = pytest.mark.gpu


LARGE = [63, 64, 65, 128, 129, 200, 300]      # beside clients of few samples


def _one(fed):
    names = [n for n, _ in fed.profile_kernels(1, 0)]
    assert ("k_client_binary" in names) != ("k_grad_binary" in names)
    return "k_client_binary" in names


@pytest.mark.parametrize("clients,small,per_round,one", [
    (60, 4, 0, True),             # resident at once
    (4200, 4, 0, False),          # more than resident anywhere, mean below 16 samples
    (4200, 4, 65, False),
    (4200, 17, 0, True),          # as many, mean above 16
])
def test_forms_and_where_they_are_taken(gpu, oracle, clients, small, per_round, one):
    d = 21
    ns = [LARGE[c // 6 % len(LARGE)] if c % 6 == 5 and c < 60 else small if small > 16 else 1 + c % small
          for c in range(clients)]
    prob = datagen.binary_problem(29, d, ns, 0.3, 1e-2)
    kw = {"clients_per_round": per_round} if per_round else {}
    fed = gpu.FedNL(prob, "randseqk", d, 0.5, **kw)
    orc = oracle.FedNL(prob, "randseqk", d, 0.5, workers=1, threads=1, **kw)
    for _ in range(3):
        fed.run(1)
        orc.round()
        np.testing.assert_array_equal(fed.x(), orc.x())
        np.testing.assert_array_equal(fed.grad(), orc.grad())
    assert _one(fed) == one
    fed.close()
    orc.close()


def test_many_clients_of_many_samples_stay_one_kernel(gpu):
    prob = datagen.binary_problem(31, 70, [100] * 1700, 0.3, 1e-2)
    fed = gpu.FedNL(prob, "randseqk", 70, 0.5)
    assert _one(fed)
    fed.close()
