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


@pytest.mark.parametrize("shift", [0.0, 1e3, 1e6])
def test_displaced_boxes_keep_the_centers_offset(ex, oracle, datasets, shift):
    """The tree rounds every cell's center, by an ulp of the coordinates a level; a class's operator
    stands for pairs at its integer offset only to 2^-48 of the separation, and the others go pair
    by pair.  Bound: that, times the few degrees that carry the field (a gradient one more), plus
    FP64 sums in another order (some thousand terms, 2^-53 sqrt(1000) = 4e-15)."""
    x = datasets.cube(40021, seed=10)
    x[:, :3] += shift
    with ex.Fmm(P=10, theta=0.4, ncrit=24, precision=ex.FP64) as f:
        f.set_bodies(x)
        f.solve()
        got = f.results()
        assert f.info()["n_m2l"] >= 400000
    ref = oracle.solve(x, P=10, theta=0.4, ncrit=24).trg
    for k, bound in ((slice(0, 1), 2e-14), (slice(1, 4), 1e-13)):
        assert np.linalg.norm(got[:, k] - ref[:, k]) < bound * np.linalg.norm(ref[:, k])


def test_a_large_forest_keeps_every_systems_bits(ex, datasets):
    """Whether a system takes the products goes by its own pairs alone: here the forest's
    contributions would be 18 GB together."""
    x = datasets.cube(40021, seed=10)
    kw = dict(P=10, theta=0.4, ncrit=24, precision=ex.FP64)
    with ex.Fmm(**kw) as f:
        f.set_bodies(x)
        f.solve()
        solo = f.results()
        pairs = f.info()["n_m2l"]
    assert pairs >= 400000
    count = int(18e9 / (8 * 112 * pairs)) + 1
    with ex.Fmm(**kw) as f:
        f.set_systems([x] * count)
        f.solve()
        assert f.info()["n_m2l"] == count * pairs
        for r in f.system_results():
            assert np.array_equal(r, solo)


@pytest.mark.parametrize("P,n,ncrit,dist", [(6, 90007, 8, "cube"), (8, 60013, 16, "plummer"), (10, 40021, 24, "cube")])
def test_the_workspace_changes_no_bit(ex, datasets, P, n, ncrit, dist):
    x = getattr(datasets, dist)(n, seed=P)
    kw = dict(P=P, theta=0.4, ncrit=ncrit, precision=ex.FP64)
    out = []
    for work in (None, 200 << 20, 1 << 20):  # one piece, a few, as many as there are
        with ex.Fmm(**kw) as f:
            if work:
                f.set_m2l_workspace(work)
            f.set_bodies(x)
            f.solve()
            out.append((f.results(), f.device_bytes()))
    assert np.array_equal(out[1][0], out[0][0]) and np.array_equal(out[2][0], out[0][0])
    assert out[2][1] < out[1][1] < out[0][1]
    with ex.Fmm(**kw) as f, pytest.raises(ex.FmmError):
        f.set_m2l_workspace(0)


@pytest.mark.parametrize("P", [8, 10])
def test_few_pairs_a_class_go_pair_by_pair(ex, datasets, P):
    """1.6M pairs in 51,000 offset classes: an operator for each would take 1.7 to 5 GB and longer
    than the pairs themselves."""
    x = datasets.plummer(150000, seed=5)
    out = []
    for _ in range(2):
        with ex.Fmm(P=P, theta=0.3, ncrit=128, precision=ex.FP64) as f:
            f.set_bodies(x)
            f.solve()
            assert f.info()["n_m2l"] >= 1500000
            out.append(f.results())
            assert f.device_bytes() < 1000e6
    assert np.array_equal(*out)
