"""The cooperative solve's back substitution with a CTA per group of blocks and with fewer CTAs than groups
(many problems in one launch: a CTA then takes several groups, one after the other), against the round's
own solve bit for bit; and a solution of which every entry is a NaN, which ends like any other."""
import numpy as np
import pytest

from ufednl_gb300 import datagen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from ufednl_gb300 import fednl

    fednl.load()
    return fednl


@pytest.mark.parametrize("problems", [2, 60, 170])
@pytest.mark.parametrize("d", [33, 128, 129, 290])
def test_groups_and_ctas(gpu, d, problems):
    prob = datagen.dense_problem(d, d, [9, 6], 1e-2)
    make = lambda: gpu.FedNL(prob, "topk", d, 1.0, feature_format=2)
    ref = make()
    ref.run(1)
    live = [make() for _ in range(problems)]
    for p in live:
        p.client_phase()
    gpu.solve_batch(live)
    for p in (live[0], live[problems // 2], live[-1]):
        np.testing.assert_array_equal(p.x(), ref.x())
    for p in live + [ref]:
        p.close()


def test_solution_of_nans(gpu):
    d = 140
    H = np.eye(d)
    g = np.full(d, np.nan)
    assert np.isnan(gpu.cholesky_option_b_solve(H.reshape(-1), d, d, 0.1, g)).all()
