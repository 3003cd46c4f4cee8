"""A wait inside a solve that runs out gives FEDNL_ETIMEOUT and leaves the iterate as it was: the FP64 back
substitution with its blocks in one CTA and over several, and the FP32 solves on one cluster (d up to 512) and
on two of a grid.  The waits are cut to nothing; every one still ends by itself."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp32,d", [(0, 64), (0, 129), (0, 301), (0, 1024), (-1, 69), (-1, 301),
                                    (1, 350), (1, 512), (1, 640), (1, 1024)])
def test_x_stays_when_a_wait_runs_out(gpu, fp32, d):
    for _ in range(3):
        assert gpu.selftest_lost_wait(d, fp32, -1) == (-5, 0)
        assert gpu.selftest_lost_wait(d, fp32, 0) == (0, d)


@pytest.mark.parametrize("d", [640, 1024])
def test_a_grid_that_got_no_clusters_solves_without(gpu, d):
    """As a profiler may replay it: no store into another CTA of a cluster, and no wait for one."""
    assert gpu.selftest_lost_wait(d, 2, -1) == (0, d)


@pytest.mark.parametrize("fp32,d", [(0, 1), (0, 31), (-1, 20), (1, 31), (1, 301)])
def test_solves_without_such_waits(gpu, fp32, d):
    assert gpu.selftest_lost_wait(d, fp32, -1) == (0, d)
