"""A component of the solution that overflows stays alone: the FP64 back substitution's lanes past a top block of
fewer than 32 rows take part in the warp's operations and must not carry that row's infinity into the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [3, 33, 34, 35, 36, 38, 63, 64, 66, 131, 301])
def test_an_infinite_first_component(gpu, oracle, d):
    H = np.eye(d)
    H[0, 0] = 1e-300
    H[0, d - 1] = H[d - 1, 0] = 1e-160
    g = np.ones(d)
    g[d - 1] = 1e200
    dx = gpu.cholesky_option_b_solve(H, d, d, 0.0, g)
    np.testing.assert_array_equal(dx, oracle.cholesky_solve(H, d, d, 0.0, g)[1])
    assert dx[0] == -np.inf and np.all(np.isfinite(dx[1:]))
