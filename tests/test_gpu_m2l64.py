"""The plain method's class products (FP64) against the oracle, alone and in a forest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the products sum a pair's terms and a target's pairs in another order than the
# oracle: two FP64 sums of some hundred terms each
TOL = 1e-12


@pytest.mark.parametrize("P,n,ncrit,dist,least", [(6, 90007, 8, "cube", 3000000), (8, 60013, 16, "plummer", 1000000),
                                                  (10, 40021, 24, "cube", 400000)])
def test_products_equal_the_oracle_and_the_forest(ex, oracle, datasets, P, n, ncrit, dist, least):
    x = getattr(datasets, dist)(n, seed=P)
    small = datasets.cube(900, seed=3)  # pair by pair in the same forest
    with ex.Fmm(P=P, theta=0.4, ncrit=ncrit, precision=ex.FP64) as f:
        f.set_bodies(x)
        f.solve()
        a = f.results()
        assert f.info()["n_m2l"] >= least
        f.set_systems([small, x, small])
        f.solve()
        r = f.system_results()
        f.set_bodies(small)
        f.solve()
        assert np.array_equal(r[1], a) and np.array_equal(r[0], f.results())
    ref = oracle.solve(x, P=P, theta=0.4, ncrit=ncrit).trg
    for k in (slice(0, 1), slice(1, 4)):
        assert np.linalg.norm(a[:, k] - ref[:, k]) < TOL * np.linalg.norm(ref[:, k])
