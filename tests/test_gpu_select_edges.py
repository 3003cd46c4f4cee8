"""TopK / TopLEK where the selection kernel's forms change: heaps around the 21 entries whose top is kept
in registers and around the chunks of 32 extractions, scans that start inside a row of 32 or at a chunk of
entries, rows whose bound ties with the root (equal magnitudes, zeros, magnitudes that share their upper
word), and a bitmap too large for shared memory; bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from ufednl_gb300 import build, fednl
    build.build()
    fednl.load()
    return fednl


def _mats(d, lda, kind, seed):
    rng = np.random.default_rng(seed)
    out = []
    for t in range(3):
        if kind == "ties":
            m = rng.integers(-3, 4, size=(d, d)) * 0.25
        elif kind == "upper":          # magnitudes that differ in their lower words only
            m = (1.0 + rng.integers(0, 40, size=(d, d)) * 2.0**-50) * rng.choice([-1.0, 1.0], size=(d, d))
        elif kind == "sparse":
            m = rng.standard_normal((d, d)) * (rng.random((d, d)) < 0.05)
        elif kind == "falling":        # few replacements, then many
            m = rng.standard_normal((d, d)) * np.linspace(0.1, 3.0, d)[None, :]
        else:
            m = rng.standard_normal((d, d))
        m = np.triu(m) + np.triu(m, 1).T
        full = np.zeros((d, lda))
        full[:, :d] = m.T
        out.append(full.reshape(-1))
    return np.stack(out)


@pytest.mark.parametrize("kind", ["cont", "ties", "upper", "sparse", "falling"])
@pytest.mark.parametrize("d,k", [(40, 20), (40, 21), (40, 22), (40, 32), (40, 33), (40, 53), (40, 54), (40, 64),
                                 (40, 65), (40, 127), (40, 128), (40, 129), (64, 31), (91, 700), (730, 300)])
def test_select_edges(gpu, oracle, d, k, kind):
    lda = (d + 3) // 4 * 4
    mats = _mats(d, lda, kind, 7 * d + k)
    got = gpu.get_topk_from_upper_diagonal_part(mats, d, lda, k)
    for t in range(len(mats)):
        np.testing.assert_array_equal(got[t], oracle.topk(mats[t], d, lda, k))
    ws, st = np.array([1234], dtype=np.uint32), np.array([1234], dtype=np.uint32)
    got = gpu.get_toplek_from_upper_diagonal_part(mats, d, lda, k, ws)
    for t in range(len(mats)):
        np.testing.assert_array_equal(got[t], oracle.toplek(mats[t], d, lda, k, st))
    assert ws[0] == st[0]
