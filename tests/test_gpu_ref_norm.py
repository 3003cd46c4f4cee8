"""The reference order's norm beside the heap walk (its ring of columns) past the columns that are loaded a step
ahead, at partial steps, and where the ring does not fit beside the heap and a kernel of its own runs: TopK and
TopLEK runs against the oracle bit for bit."""
import numpy as np
import pytest

from ufednl_gb300 import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,k,comp,own_kernel", [
    (97, 194, "toplek", False), (130, 520, "topk", False), (400, 1600, "toplek", False),
    (301, 9000, "toplek", True), (301, 9000, "topk", True), (403, 8500, "toplek", True),
])
def test_norm_in_the_reference_order(gpu, oracle, d, k, comp, own_kernel):
    prob = datagen.binary_problem(11 + d, d, [70, 129, 40], 0.1, 1e-2)
    fed = gpu.FedNL(prob, comp, k, 1.0, order="reference")
    orc = oracle.FedNL(prob, comp, k, 1.0, workers=1, threads=1, ref_order=True)
    for _ in range(3):
        gg, go = fed.round(), orc.round()
        assert abs(gg - go) <= 1e-14 * go        # the oracle sums ||g||^2 in its own order
        np.testing.assert_array_equal(fed.x(), orc.x())
        assert fed.l() == orc.l()
    assert ("k_frob_ref" in [n for n, _ in fed.profile_kernels(1, 0)]) == own_kernel
    fed.close()
    orc.close()
