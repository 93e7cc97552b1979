"""The cluster sizes of the dGN engine: within the hardware's and the ranks'
limits, one problem on up to 16 CTAs, many problems within one wave of SMs."""
import pytest

from tensorfox_gb300.gauss_newton import auto_cluster


@pytest.mark.parametrize("dims,R", [((2, 2, 2), 1), ((4, 4, 4), 3), ((10, 10, 10), 10), ((21, 22, 23), 9),
                                    ((30, 30, 30), 30), ((50, 50, 50), 50), ((90, 70, 60), 8), ((8, 8, 8, 8), 20)])
@pytest.mark.parametrize("problems", [1, 2, 10, 100, 5000])
def test_cluster_sizes(dims, R, problems):
    c = auto_cluster(dims, R, problems)
    n = 1
    for d in dims:
        n *= d
    assert 1 <= c <= min(16, R)
    assert c <= (16 if n * R >= 100000 else 8)
    # a batch takes no more CTAs than SMs unless its problems' own work asks for them
    assert c * problems <= 152 or c <= max(1, n * R * len(dims) // 1200000)
    if problems == 1:
        assert c == min(R, 16 if n * R >= 100000 else 8)
