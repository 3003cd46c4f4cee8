"""The reference-order solve where its panels, blocks of eight rows and substitution change shape (one row,
fewer than eight, exact multiples of eight and of the 32-row panel, a panel's last columns, several own
columns per CTA), bit for bit against the oracle; a matrix that is not positive definite, at pivots in
different places, ends the round with its status and leaves x."""
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


@pytest.mark.parametrize("d", [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 39, 40, 41, 63, 64, 65, 72, 96, 97, 129, 200,
                               257])
def test_ref_solve_sizes(gpu, oracle, d):
    prob = datagen.dense_problem(60 + d, d, [9, 14, 5], 1e-2) if d > 1 else \
        datagen.Problem(1, np.array([3, 4], np.int32), np.ones((7, 1)), np.array([1., -1, 1, 1, -1, 1, 1]), 1e-2)
    U = d * (d + 1) // 2
    fed = gpu.FedNL(prob, "identity", U, 1.0, order="reference", feature_format=2)
    orc = oracle.FedNL(prob, "identity", U, 1.0, workers=1, threads=1, ref_order=True)
    for _ in range(3):
        gg, go = fed.round(), orc.round()
        assert gg == go or abs(gg - go) <= 1e-14 * go
        np.testing.assert_array_equal(fed.x(), orc.x())
        assert fed.l() == orc.l()
    fed.close()
    orc.close()


@pytest.mark.parametrize("d,scale", [(5, 0), (20, 3), (33, 12), (70, 40), (70, 66)])
@pytest.mark.parametrize("order", ["reference", "fixed"])
def test_not_positive_definite(gpu, order, d, scale):
    """lambda < 0 with `scale` large features: the first negative pivot is the first small one."""
    rng = np.random.default_rng(d + scale)
    a = rng.standard_normal((40, d)) * np.where(np.arange(d) < scale, 300.0, 1e-3)[None, :]
    y = np.where(rng.random(40) < 0.5, 1.0, -1.0)
    prob = datagen.Problem(d, np.array([20, 20], np.int32), a, y, -1e-2)
    fed = gpu.FedNL(prob, "identity", 1, 1.0, order=order, feature_format=2)
    with pytest.raises(gpu.FedNLError) as e:
        fed.round()
    assert e.value.code == -4
    np.testing.assert_array_equal(fed.x(), np.zeros(d))
    fed.close()
