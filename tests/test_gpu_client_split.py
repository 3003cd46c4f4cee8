"""The client oracle of {0,1} features as one kernel (a CTA per client) and as two (past the clients whose
CTAs are resident at once: 1621 at d = 70 on 152 SMs), against the oracle bit for bit; partial
participation with its sampler and true gradient on a branch of the round's graph."""
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


@pytest.mark.parametrize("clients,per_round", [(1500, 0), (1700, 0), (1700, 65)])
def test_one_kernel_and_two(gpu, oracle, clients, per_round):
    d = 70
    prob = datagen.binary_problem(17, d, [1 + c % 5 for c in range(clients)], 0.3, 1e-2)
    kw = {"clients_per_round": per_round} if per_round else {}
    fed = gpu.FedNL(prob, "randseqk", d, 0.5, **kw)
    orc = oracle.FedNL(prob, "randseqk", d, 0.5, workers=1, threads=1, **kw)
    for _ in range(3):
        fed.run(1)
        orc.round()
        np.testing.assert_array_equal(fed.x(), orc.x())
        np.testing.assert_array_equal(fed.grad(), orc.grad())
    fed.close()
    orc.close()
