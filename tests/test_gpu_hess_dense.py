"""The dense FP64 Hessian where its shapes change: one position, one warp's rows cut by U, columns split
between CTAs, sample counts around the batch of 16 and its groups of four; bit-exact against the oracle
through whole rounds (messages, shifts, iterates), plain and FedNL-PP."""
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


CASES = [(2, [1, 3]), (15, [16, 17, 15]), (16, [4, 33, 5]), (31, [1, 64, 19]), (33, [48, 47, 2]), (91, [21, 40]),
         (72, [3 + c % 19 for c in range(30)])]


@pytest.mark.parametrize("comp", ["topk", "identity"])
@pytest.mark.parametrize("d,ns", CASES, ids=[f"d{c[0]}-n{len(c[1])}" for c in CASES])
def test_dense_rounds_vs_oracle(gpu, oracle, d, ns, comp):
    prob = datagen.dense_problem(41 + d, d, ns, 1e-2)
    U = d * (d + 1) // 2
    k = U if comp == "identity" else min(2 * d, U)
    fed = gpu.FedNL(prob, comp, k, 1.0, feature_format=2)
    orc = oracle.FedNL(prob, comp, k, 1.0, workers=1, threads=1)
    for _ in range(3):
        fed.round()
        orc.round()
        np.testing.assert_array_equal(fed.x(), orc.x())
        assert fed.l() == orc.l()
        for c in range(0, len(ns), max(1, len(ns) // 5)):
            ig, vg = fed.message(c)
            io, vo = orc.message(c)
            np.testing.assert_array_equal(ig, io)
            np.testing.assert_array_equal(vg, vo)
            np.testing.assert_array_equal(fed.shift(c), orc.shift(c))
    fed.close()
    orc.close()


def test_dense_pp_vs_oracle(gpu, oracle):
    prob = datagen.dense_problem(47, 33, [5, 17, 18, 4, 20, 33], 1e-2)
    fed = gpu.FedNL(prob, "natural", 1, 8 / 9, clients_per_round=4, feature_format=2)
    orc = oracle.FedNL(prob, "natural", 33 * 34 // 2, 8 / 9, workers=1, threads=1, clients_per_round=4)
    for _ in range(4):
        fed.round()
        orc.round()
        np.testing.assert_array_equal(fed.x(), orc.x())
        assert fed.l() == orc.l()
    fed.close()
    orc.close()
