"""The kernel method's tree kernel where its layout changes: point counts around a pass (256 >> n
points) and a group, at every order's first level; the zeroed vertex (the last one) at any place in
time, equal times, vertices later than X, X on either branch; and points handed to the pivoted
LU next to others. Against the CPU oracle, |gpu - cpu| <= 1e-12 of the point's sum of |terms|."""
import numpy as np
import pytest

from keldy_b200 import capi
from tests.test_gpu_wick_tree import one_sided_models, window_models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10])
def test_point_counts_places_and_branches(ctx, oracle, golden, n):
    le, gr = golden["table_beta20_lesser"], golden["table_beta20_greater"]
    gm, om = ctx.model(10.0, le, gr, 0.4), oracle.model(10.0, le, gr, 0.4)
    rng = np.random.default_rng(60 + n)
    per_pass = 32 if n <= 3 else max(1, 256 >> n)
    counts = {1, per_pass + 1, 33} if n <= 6 else {1, per_pass + 1, 17} if n <= 8 else {2}
    for k, count in enumerate(sorted(counts)):
        X = (6.0, 0, (n + k) % 2, 0, 0)
        t = rng.random((count, n)) * 10.0
        if n > 1:
            t[::2, n - 1] = t[::2, 0]  # the zeroed vertex at another one's time
        t[-1, 0] = X[0]
        got, dom = gm.integrand_kernel(X, t)
        want, odom, sc = oracle.integrand_kernel(om, X, t)
        assert np.array_equal(dom, odom)
        assert np.all(np.abs(got - want).max(axis=(1, 2)) <= 1e-12 * np.maximum(sc, 1e-300)), (n, count)


@pytest.mark.parametrize("n", [1, 3, 4, 6])
def test_guarded_points_among_others(ctx, oracle, n):
    """A table whose g(0) is small but not zero for some copies: every point of it goes to the
    pivoted LU; in one call with an ordinary model's item, both sums equal the oracle's."""
    t = np.linspace(-10, 10, 2001)
    le = 1j * t * np.exp(-t * t / 8) + 0.2 * np.sin(t)
    odd = (le, -np.conj(le[::-1]))
    le2 = 0.5j * np.exp(-np.abs(t)) + 0.1 * np.sin(t) * np.exp(-np.abs(t))
    plain = (le2, -np.conj(le2))
    X = (10.0, 0, 0, 0, 0)
    chain = [(capi.WARPER_PLASMA_UV, 10.0, 0.0), (capi.WARPER_EXPONENTIAL, 10.0, 1.0)]
    items = [dict(model=ctx.model(10.0, *m), rng=ctx.sobol(n), chain=chain, A=X, order=n, k_first=5, n_points=151)
             for m in (odd, plain)]
    for (s, npt, nd, bins, cnt, drop), m in zip(capi.integrate_kernel(ctx, items, 7, 1.0, 9.0), (odd, plain)):
        ws, onp, ond, sc, ob, oc, od = oracle.integrate_kernel(oracle.model(10.0, *m), X, chain, n, 151, 7, 1.0, 9.0, seed=4)
        assert (npt, nd, drop) == (onp, ond, od) and np.array_equal(cnt, oc)
        assert np.abs(bins - ob).max() <= 1e-12 * sc and abs(s - ws) <= 1e-12 * sc


@pytest.mark.parametrize("interp", [1, 3])
@pytest.mark.parametrize("tmax,mesh", [(9.0, 1001), (11.0, 2001), (10.0, 2001)])
def test_window_upper_end(ctx, oracle, tmax, mesh, interp):
    """Vertices at 0 and t_max, X at t_max: 2 t_max / delta may round above the last mesh point's number."""
    gm, om, _ = window_models(ctx, oracle, tmax, mesh, interp)
    rng = np.random.default_rng(4)
    for n in (1, 2, 4, 7, 9):
        t = rng.random((3, n)) * tmax
        t[0, 0], t[1, n - 1] = 0.0, tmax
        t[2, [0, n - 1]] = 0.0, tmax if n > 1 else 0.0
        for X in ((tmax, 0, 0, 0, 0), (tmax, 0, 1, 0, 0)):
            got, dom = gm.integrand_kernel(X, t)
            want, odom, sc = oracle.integrand_kernel(om, X, t)
            assert np.array_equal(dom, odom)
            assert np.all(np.abs(got - want).max(axis=(1, 2)) <= 1e-12 * np.maximum(sc, 1e-300)), n


@pytest.mark.parametrize("n", [1, 3, 6, 9])
def test_points_outside_with_any_jacobian(ctx, golden, n):
    """Points outside the domain add nothing, whatever their Jacobian (exp(u_max / w) overflows here, the
    times are -infinity)."""
    gm = ctx.model(10.0, golden["table_beta20_lesser"], golden["table_beta20_greater"])
    item = dict(model=gm, rng=ctx.sobol(n), chain=[(capi.WARPER_EXPONENTIAL, 10.0, 0.01)], A=(10.0, 0, 0, 0, 0), order=n,
                k_first=1, n_points=100)
    (s, npt, nd, bins, cnt, drop), = capi.integrate_kernel(ctx, [item], 7, 1.0, 9.0)
    assert (s, npt, nd, drop) == (0, 100, 0, 0) and not bins.any() and not cnt.any()
    (s, npt, nd), = [r[:3] for r in capi.integrate_kernel_single_omega(ctx, [item], 0.3)]
    assert (s, npt, nd) == (0, 100, 0)


@pytest.mark.parametrize("ratio,small", [(1e-1, "lesser"), (1e-1, "greater"), (1e-5, "lesser")])
def test_nearly_empty_and_full_levels(ctx, oracle, ratio, small):
    """(At a ratio of 1e-5 the other way the elimination without pivoting itself is off by 1e-12.)"""
    gm, om = one_sided_models(ctx, oracle, ratio, small)
    for n in (1, 2, 3, 4, 5, 6, 7, 8, 9):
        t = np.random.default_rng(n).random((40 if n < 8 else 8, n)) * 10.0
        X = (10.0, 0, 0, 0, 0) if n % 2 else (6.0, 0, 1, 0, 0)
        got, dom = gm.integrand_kernel(X, t)
        want, odom, sc = oracle.integrand_kernel(om, X, t)
        assert np.array_equal(dom, odom) and np.all(np.abs(got - want).max(axis=(1, 2)) <= 1e-12 * sc), n


@pytest.mark.parametrize("n", [1, 2, 4, 7])
@pytest.mark.parametrize("npts", [1, 15, 17, 100])
def test_models_whose_spins_differ(ctx, oracle, golden, n, npts):
    """Every point goes to the pivoted LU, set up 16 at a time: sums, bins and values."""
    tables = [golden[f"table_{k}_{s}"] for k in ("beta20", "T0") for s in ("lesser", "greater")]
    gm, om = ctx.model(10.0, *tables[:2], 0.0, *tables[2:]), oracle.model(10.0, *tables[:2], 0.0, *tables[2:])
    X = (10.0, 0, 0, 0, 0)
    chain = [(capi.WARPER_PLASMA_UV, 10.0, 0.0), (capi.WARPER_INVERSE, 10.0, 2.0)]
    item = dict(model=gm, rng=ctx.sobol(n), chain=chain, A=X, order=n, k_first=5, n_points=npts)
    (s, npt, nd, bins, cnt, drop), = capi.integrate_kernel(ctx, [item], 7, 1.0, 9.0)
    ws, onp, ond, sc, ob, oc, od = oracle.integrate_kernel(om, X, chain, n, npts, 7, 1.0, 9.0, seed=4)
    assert (npt, nd, drop) == (onp, ond, od) and np.array_equal(cnt, oc)
    assert np.abs(bins - ob).max() <= 1e-12 * sc and abs(s - ws) <= 1e-12 * sc
    t = np.random.default_rng(n).random((npts, n)) * 10.0
    t[::3, 0] *= -1.0
    got, dom = gm.integrand_kernel(X, t)
    want, odom, sc = oracle.integrand_kernel(om, X, t)
    assert np.array_equal(dom, odom) and np.all(np.abs(got - want).max(axis=(1, 2)) <= 1e-12 * sc)


@pytest.mark.parametrize("n,count", [(1, 40), (2, 1), (3, 33), (5, 70)])
def test_values_of_guarded_points(ctx, oracle, n, count):
    """Every point of the domain goes to the pivoted LU (g(0) = 0) after the tree has counted them."""
    t = np.linspace(-10, 10, 2001)
    le = 1j * t * np.exp(-t * t / 8) + 0.2 * np.sin(t)
    tables = le, -np.conj(le[::-1])
    gm, om = ctx.model(10.0, *tables), oracle.model(10.0, *tables)
    u = np.random.default_rng(n).random((count, n)) * 10.0
    u[1::4, 0] *= -1.0
    for X in ((10.0, 0, 0, 0, 0), (6.0, 0, 1, 0, 0)):
        got, dom = gm.integrand_kernel(X, u)
        want, odom, sc = oracle.integrand_kernel(om, X, u)
        assert np.array_equal(dom, odom) and np.all(np.abs(got - want).max(axis=(1, 2)) <= 1e-12 * sc)
