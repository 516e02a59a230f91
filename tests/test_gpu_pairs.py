"""Pair kernels on the GPU against the oracle's direct sum: the direct sum at the
edges of its target blocks and source tiles, and the P2P kernels at the edges of
their lane groups, segments and divided leaves (a tree of one leaf is P2P alone)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# FP64: sums of up to a few thousand terms of either sign, each within a few ulp
TOL64 = 1e-13
# mixed: FP32 products (2^-24, the reciprocal square root 2^-22) of two-float
# separations, summed with compensation; 1e-6 is the form's stated precision
TOL32 = 1e-6


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("nt,ns,images", [(1, 1, 0), (1, 257, 0), (128, 255, 0), (129, 256, 0), (300, 1031, 0),
                                          (257, 513, 0), (5, 40, 1), (130, 65, 1)])
def test_direct_block_and_tile_edges(ex, oracle, nt, ns, images):
    rng = np.random.default_rng(nt * 1009 + ns)
    t, s = rng.uniform(-1, 1, (nt, 4)), rng.uniform(-1, 1, (ns, 4))
    s[0, :3] = t[0, :3] if ns > 1 else s[0, :3]  # one pair at distance zero
    got = ex.direct(t, s, images=images, theta=0.4)
    assert _rel(got, oracle.direct(t, s, images=images, theta=0.4)) < TOL64


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [2, 7, 8, 9, 12, 13, 16, 17, 24, 25, 32, 33, 49, 64, 65, 70, 97, 130, 257, 1000])
def test_one_leaf_is_the_direct_sum(ex, oracle, n, mixed):
    x = np.random.default_rng(n).uniform(-1, 1, (n, 4))
    if n > 8:
        x[3, :3] = x[7, :3]  # coincident bodies: no contribution
    with ex.Fmm(P=4, ncrit=1024, precision=ex.MIXED if mixed else ex.FP64) as f:
        f.set_bodies(x)
        f.solve()
        got = f.results()
        again = f.solve() or f.results()
    ref = oracle.direct(x, x)
    assert _rel(got[:, 0], ref[:, 0]) < (TOL32 if mixed else TOL64)
    assert _rel(got[:, 1:], ref[:, 1:]) < (TOL32 if mixed else TOL64)
    assert np.array_equal(got, again)  # divided leaves add in a fixed order


@pytest.mark.parametrize("d", [1e-100, 1e-150, 1e-155])
def test_tiny_distances_keep_their_weight(ex, d):
    """The squared distance down to a subnormal number (1e-310, good to about 1e-14 of itself)."""
    got = ex.direct(np.zeros((1, 4)), np.array([[d, 0.0, 0.0, 1.0], [0.0, 0.0, 0.0, 5.0]]))
    assert abs(got[0, 0] * d - 1.0) < 1e-10


@pytest.mark.parametrize("missing", ["targets", "sources", "results"])
def test_direct_refuses_a_null_array(ex, missing):
    a = {k: np.ones((300, 4)) for k in ("targets", "sources", "results")}
    ptr = {k: None if k == missing else v.ctypes.data for k, v in a.items()}
    t, s, r = (ptr[k] for k in ("targets", "sources", "results"))
    assert ex.lib().exafmm_direct(t, 300, s, 300, 0, 0.4, 1.0, r) != 0
    assert ex.lib().exafmm_direct_range(t, 300, s, 300, 0, 1.0, r) != 0
    cycle = np.ones(3)
    assert ex.lib().exafmm_direct_cutoff(ctypes.c_void_p(t), ctypes.c_longlong(300), ctypes.c_void_p(s),
                                         ctypes.c_longlong(300), 0, ctypes.c_void_p(cycle.ctypes.data),
                                         ctypes.c_double(1.0), ctypes.c_void_p(r)) != 0
    got = ex.direct(a["targets"], a["sources"])  # the next call is untouched
    assert np.all(got == 0)


@pytest.mark.parametrize("charge", [np.inf, np.nan])
def test_coincident_bodies_drop_any_charge(ex, oracle, charge):
    """A pair at distance zero has no weight whatever its charge: a body whose charge is not
    finite leaves itself and the bodies at its own point alone."""
    x = np.random.default_rng(5).uniform(-1, 1, (200, 4))
    x[3, :3] = x[7, :3]
    x[90, :3] = x[7, :3]
    bad = x.copy()
    bad[7, 3] = charge
    x[7, 3] = 0.0
    at, other = [3, 7, 90], 50
    ref = oracle.direct(x, x)
    with ex.Fmm(P=4, ncrit=256) as f:  # one leaf: P2P alone
        f.set_bodies(bad)
        f.solve()
        solved = f.results()
    for got in (ex.direct(bad, bad), solved):
        assert _rel(got[at], ref[at]) < TOL64
        assert not np.isfinite(got[other, 0])


@pytest.mark.parametrize("ns", [1, 300])
def test_a_small_charge_very_near_does_not_overflow(ex, ns):
    """q / r^2 is taken as (q / r) / r / r: 1 / r^2 alone would overflow at this distance."""
    d, q = 1e-155, 1e-200
    s = np.zeros((ns, 4))
    s[0] = [d, 0.0, 0.0, q]
    t = np.zeros((1, 4))
    with ex.Fmm(P=4, ncrit=512) as f:
        f.set_bodies(np.concatenate([t, s[:1], [[1.0, 1.0, 1.0, 0.0]]]))
        f.solve()
        solved = f.results()[:1]
    for got in (ex.direct(t, s), solved):
        assert abs(got[0, 0] * d / q - 1.0) < 1e-10
        assert abs(got[0, 1] * d * d / q - 1.0) < 1e-10


def test_reciprocal_distance_error(ex):
    """1/r of one pair against the exact quotient, over r from 1e-150 to 1e150.  The distances have
    26 bits, so that r^2 is exact.  Bound: the last addition rounds once, 2^-53, and e = 1 - r^2 y0^2
    carries the rounding of r^2 y0, which counts half; the cubic term is below 2^-56 for the 20 bits
    of y0 (a seed of 18 would do)."""
    rng = np.random.default_rng(11)
    n = 100000
    m = rng.integers(1 << 25, 1 << 26, n)
    d = np.ldexp(m.astype(np.float64), rng.integers(-500, 474, n))
    t = np.zeros((n, 4))
    t[:, 0] = d
    got = ex.direct(t, np.array([[0.0, 0.0, 0.0, 1.0]]))[:, 0]
    err = np.abs(got.astype(np.longdouble) * d.astype(np.longdouble) - 1)
    print(f"largest error {float(err.max()):.3g}")
    assert float(err.max()) < 1.5 * 2.0 ** -53 + 2.0 ** -56
