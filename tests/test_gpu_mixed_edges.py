"""The mixed engine's kernels at the sizes where their splits can go wrong: margins with one and with two
samples a thread, gradients of an odd number of features and of ragged clients, the Gram epilogue's whole
and partial chunks, and selections with many equal differences."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from ufednl_gb300 import fednl

    fednl.load()
    return fednl


@pytest.mark.parametrize("d", [65, 127, 128, 1025])
def test_margins_one_and_two_samples_a_thread(gpu, d):
    """The same clients once (too few blocks of 128 samples for two samples a thread) and repeated until
    they get them: the mean gradient is the same mean of the same per-client gradients, so the norms agree
    to the rounding of FP64 sums (480 terms: 480 2^-53 < 1e-13), and with the FP64 engine's to 1e-10, the
    bound of the float-float sums."""
    from ufednl_gb300 import datagen

    ns = [1, 31, 255, 256, 257, 385]
    one = datagen.dense_problem_fp32(7, d, ns, 1e-3)
    rep = 80 if d < 1000 else 60
    many = datagen.Problem(d, np.tile(one.n_samples, rep), np.tile(one.features, (rep, 1)), np.tile(one.labels, rep), one.lam)
    assert sum((n + 127) // 128 for n in ns) * rep >= 3 * 152
    g = []
    for p in (one, many):
        e = gpu.MixedFedNL(p, d, 0.1)
        g.append(e.run(1)[0])
        e.close()
    p64 = datagen.Problem(d, one.n_samples, one.features.astype(np.float64), one.labels, one.lam)
    e = gpu.FedNL(p64, "randk_philox", d, 0.1, feature_format=2)
    g64 = e.run(1)[0]
    e.close()
    assert abs(g[0] - g[1]) <= 1e-13 * g[0]
    assert abs(g[0] - g64) <= 1e-10 * g64


@pytest.mark.parametrize("d,k", [(66, 300), (129, 1000), (130, 5000), (258, 9000), (400, 3)])
def test_topk_with_equal_differences(gpu, d, k):
    """Columns in equal triples: every difference off the blocks' diagonals appears several times, so the
    threshold is shared; the lower positions are kept (one CTA a client, clusters of 2 and of 8)."""
    from ufednl_gb300 import datagen

    p = datagen.dense_problem_fp32(9, d, [70, 129], 1e-3)
    p = datagen.Problem(d, p.n_samples, np.ascontiguousarray(p.features[:, (np.arange(d) // 3) * 3]), p.labels, p.lam)
    mx = gpu.MixedFedNL(p, k, 1.0, compressor="topk")
    ties = 0
    for _ in range(3):
        mx.run(1)
        for c in range(2):
            mag, sel = np.abs(mx.diff(c)), mx.selection(c)
            order = np.lexsort((np.arange(len(mag)), -mag))
            np.testing.assert_array_equal(np.sort(order[:k]), sel)
            ties += mag[order[k - 1]] == mag[order[k]]
    assert ties > 0 or k < 10
    mx.close()
