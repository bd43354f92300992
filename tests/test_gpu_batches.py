"""Batches and groups of the integration where the kernels' schedule branches: the search of a chunk's
item over one, two and three rounds of 32, items without points among others, ordinary items beside
items whose points all go to the pivoted LU (their pass follows only when the sums count some), and
groups of several quads of passes at every compiled order. A batch's sums are those of separate
calls, bit for bit; against the CPU oracle, |gpu - cpu| <= 1e-12 of the sum of |terms|."""
import numpy as np
import pytest

from keldy_b200 import capi

pytestmark = pytest.mark.gpu

INVERSE = [(capi.WARPER_PLASMA_UV, 10.0, 0.0), (capi.WARPER_INVERSE, 10.0, 2.0)]  # few points in the domain above order 8
EXPONENTIAL = [(capi.WARPER_PLASMA_UV, 10.0, 0.0), (capi.WARPER_EXPONENTIAL, 10.0, 1.0)]
A, B = (10.0, 0, 0, 0, 0), (10.0, 0, 1, 0, 0)


def _tables(kind):
    t = np.linspace(-10, 10, 2001)
    if kind == "guarded":  # g(0) = 0: a zero pivot at every point
        le = 1j * t * np.exp(-t * t / 8) + 0.2 * np.sin(t)
    else:
        le = 0.5j * np.exp(-np.abs(t)) + 0.1 * np.sin(t) * np.exp(-np.abs(t))
    return le, -np.conj(le[::-1])


def _item(model, rng, order, npts, k_first, chain=INVERSE):
    return dict(model=model, rng=rng, chain=chain, A=A, B=B, order=order, k_first=k_first, n_points=npts)


@pytest.mark.parametrize("count", [2, 31, 33, 1023, 1025])
def test_batch_equals_calls(ctx, count):
    m = ctx.model(10.0, *_tables("plain"))
    rngs = {n: ctx.sobol(n) for n in (1, 2, 3, 5)}
    items = [_item(m, rngs[(1, 2, 3, 5)[i % 4]], (1, 2, 3, 5)[i % 4], (i * 7) % 23, 1 + i) for i in range(count)]
    batch = capi.integrate(ctx, items)
    for i in sorted({0, 1, count // 3, count // 2, count - 2, count - 1}):
        single, = capi.integrate(ctx, [items[i]])
        assert single == batch[i], i
    assert [r[1] for r in batch] == [it["n_points"] for it in items]


@pytest.mark.parametrize("chain", [INVERSE, EXPONENTIAL])
@pytest.mark.parametrize("order", [1, 2, 4, 6, 9])
def test_guarded_items_among_others(ctx, oracle, order, chain):
    rng = ctx.sobol(order)
    items, want = [], []
    for i, kind in enumerate(("plain", "guarded", "plain")):
        items.append(_item(ctx.model(10.0, *_tables(kind)), rng, order, 37 + i, 3 + i, chain))
        want.append(oracle.integrate(oracle.model(10.0, *_tables(kind)), A, B, chain, order, 37 + i, seed=2 + i))
    for (s, npt, nd, nfb), (w, onp, ond, sc), kind in zip(capi.integrate(ctx, items), want, ("plain", "guarded", "plain")):
        assert (npt, nd) == (onp, ond)
        assert (nfb > 0) == (kind == "guarded" and order > 1 and ond > 0)
        assert abs(s - w) <= 1e-12 * sc, (kind, abs(s - w) / sc)


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10])
def test_groups_of_several_quads(ctx, oracle, order):
    """Enough points for full groups: fewer are spread over the warps in smaller ones."""
    npts = 7203 if order <= 6 else 3601
    m = ctx.model(10.0, *_tables("plain"))
    (s, npt, nd, nfb), = capi.integrate(ctx, [_item(m, ctx.sobol(order), order, npts, 6, EXPONENTIAL)])
    w, onp, ond, sc = oracle.integrate(oracle.model(10.0, *_tables("plain")), A, B, EXPONENTIAL, order, npts, seed=5)
    assert (npt, nd, nfb) == (onp, ond, 0) and nd > npts // 2
    assert abs(s - w) <= 1e-12 * sc


@pytest.mark.parametrize("chunk", [1, 5, 33, 64, 128])
@pytest.mark.parametrize("order,npts", [(2, 1), (2, 6), (3, 131), (5, 300), (7, 66)])
def test_guarded_points_of_a_chunk(ctx, oracle, order, npts, chunk):
    """The pivoted-LU pass over chunks with one, some and all points guarded (those outside the domain
    are not), sums and bins; sums of a call and of the allocation-free call are the same."""
    gm, om = ctx.model(10.0, *_tables("guarded")), oracle.model(10.0, *_tables("guarded"))
    before = ctx.get_launch(order)
    try:
        ctx.set_launch(-1, chunk)
        for chain in (INVERSE, EXPONENTIAL):
            item = _item(gm, ctx.sobol(order), order, npts, 4, chain)
            (s, npt, nd, nfb, bins, counts, dropped), = capi.integrate_binned(ctx, [item], 9, 0.5, 9.0)
            w, onp, ond, sc, ob, oc, od = oracle.integrate_binned(om, A, B, chain, order, npts, 9, 0.5, 9.0, seed=3)
            assert (npt, nd, nfb, dropped) == (onp, ond, ond, od) and np.array_equal(counts, oc)
            assert abs(s - w) <= 1e-12 * sc and np.abs(bins - ob).max() <= 1e-12 * sc
            assert capi.integrate_noalloc(ctx, [item]) == capi.integrate(ctx, [item]) == [(s, npt, nd, nfb)]
    finally:
        ctx.set_launch(-1, *before)


def test_times_of_a_call_with_guarded_points(ctx):
    """The pivoted-LU time is its launch's own: for 40 points beside 2^18 ordinary ones with 4,096 bins
    less than the sums over the bins (168 MB), which are formed before it and after it."""
    rng = ctx.sobol(2)
    items = [_item(ctx.model(10.0, *_tables(k)), rng, 2, n, 1, EXPONENTIAL) for k, n in (("plain", 1 << 18), ("guarded", 40))]
    ctx.set_timing(True)
    try:
        for _ in range(3):
            res = capi.integrate_binned(ctx, items, 4096, 0.0, 10.0)
            integrand, lu, sums, launches = ctx.last_timing()
    finally:
        ctx.set_timing(False)
    assert res[1][3] == 40 and launches == 6
    assert 0.0 < lu < sums and integrand > 0.0
