"""The warp-per-group tree kernel where its layout changes: point counts around a pass (256 >> n
points), a group (32, 16 above order 8) and a chunk, at every order's first level; times equal
to each other and to the external times, and vertices later than one or both external points on
either branch. Against the CPU oracle; |gpu - cpu| <= 1e-12 sum_a |det up det down|, as for the
other integrand tests."""
import numpy as np
import pytest

from keldy_b200 import capi

pytestmark = pytest.mark.gpu

ENDS = [((7.0, 0, 0, 0, 0), (7.0, 0, 1, 0, 0)), ((6.0, 0, 1, 0, 0), (3.0, 0, 0, 0, 0)),
        ((2.5, 1, 0, 0, 0), (8.0, 1, 0, 0, 0)), ((5.0, 0, 1, 0, 0), (5.0, 0, 1, 0, 0))]


def _models(ctx, oracle, golden, alpha=0.4):
    le, gr = golden["table_beta20_lesser"], golden["table_beta20_greater"]
    return ctx.model(10.0, le, gr, alpha), oracle.model(10.0, le, gr, alpha)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 11])
def test_point_counts_ties_and_external_order(ctx, oracle, golden, n):
    gm, om = _models(ctx, oracle, golden)
    rng = np.random.default_rng(40 + n)
    per_pass = 32 if n <= 3 else max(1, 256 >> n)
    counts = {1, per_pass + 1, 33, 2 * per_pass - 1} if n <= 8 else {1, 2, 17} if n == 9 else {2}
    for k, count in enumerate(sorted(counts)):
        A, B = ENDS[(n + k) % len(ENDS)]
        t = rng.random((count, n)) * 10.0
        if n > 1:
            t[::2, n - 1] = t[::2, 0]  # equal vertex times
        t[-1, 0] = A[0]  # a vertex at each external time
        t[-1, n // 2] = B[0]
        for scale in (False, True):
            v, d, *gsc = gm.integrand(A, B, t, algo=capi.ALGO_TREE, want_scale=scale)
            w, dw, sc = oracle.integrand(om, A, B, t)
            np.testing.assert_array_equal(d, dw)
            assert np.all(np.abs(v - w) <= 1e-12 * sc), (n, count, scale)
            if scale:
                np.testing.assert_allclose(gsc[0], sc, rtol=1e-9)


@pytest.mark.parametrize("chunk", [1, 13, 33, 100, 128])
def test_chunk_sizes(ctx, oracle, golden, chunk):
    """Ragged chunks and groups of an integration, with out-of-domain points among the others."""
    gm, om = _models(ctx, oracle, golden, 0.0)
    chain = [(capi.WARPER_PLASMA_UV, 10.0, 0.0), (capi.WARPER_INVERSE, 10.0, 2.0)]
    A, B = (10.0, 0, 0, 0, 0), (10.0, 0, 1, 0, 0)
    before = ctx.get_launch(3)
    try:
        ctx.set_launch(-1, chunk)
        for n, npts in ((1, 301), (3, 301), (5, 203), (8, 101), (9, 35)):
            (s, np_, nd, nfb), = capi.integrate(ctx, [dict(model=gm, rng=ctx.sobol(n), chain=chain, A=A, B=B, order=n,
                                                           k_first=29, n_points=npts)])
            w, onp, ond, sc = oracle.integrate(om, A, B, [(1, 10.0, 0.0), (3, 10.0, 2.0)], n, npts, seed=28)
            assert (np_, nd, nfb) == (onp, ond, 0)
            assert abs(s - w) <= 1e-12 * sc, (n, abs(s - w) / sc)
    finally:
        ctx.set_launch(-1, *before)


def test_order_0_after_other_kernels(ctx, oracle, golden):
    """Order 0 is g0(A, B) at every point, whatever the kernels before left in shared memory: the
    kernel method's nodes, or times below zero (more chunks than resident warps, full groups)."""
    gm, om = _models(ctx, oracle, golden)
    rng = np.random.default_rng(9)
    none = np.zeros((1 << 17, 0))
    A, B = ENDS[0]
    want = oracle.integrand(om, A, B, none[:1])[0][0]
    before = [lambda n=n: gm.integrand_kernel(A, rng.random((8192, n)) * 10.0) for n in (1, 3, 6, 8)]
    before += [lambda n=n: gm.integrand(A, B, -3.0 * rng.random((1 << 16, n)), keep_u_hypercube=False) for n in (1, 5, 8)]
    for fill in before:
        for call in (lambda: gm.integrand(A, B, none), lambda: gm.evaluate_warped(A, B, [], none)[::2]):
            fill()
            v, d = call()
            assert np.all(d == 1) and np.all(np.abs(v - want) <= 1e-12 * abs(want))


def window_models(ctx, oracle, tmax, mesh, interp):
    t = np.linspace(-tmax, tmax, mesh)
    le = 0.5j * np.exp(-np.abs(t)) + 0.1 * np.sin(t) * np.exp(-np.abs(t))
    tables = le, -np.conj(le[::-1])
    gm, om = ctx.model(tmax, *tables), oracle.model(tmax, *tables, interp=interp)
    gm.set_interpolation(interp)
    return gm, om, 2.0 * tmax / (mesh - 1)


@pytest.mark.parametrize("interp", [1, 3])
@pytest.mark.parametrize("tmax,mesh", [(9.0, 1001), (11.0, 2001), (10.0, 2001), (14.0, 25001)])
def test_window_upper_end(ctx, oracle, tmax, mesh, interp):
    """Time differences of t_max, where 2 t_max / delta may round above the last mesh point's number
    (not at t_max = 10), and beyond it by less than a mesh step: the window is floor(position) <=
    npts - 1 for the tree, the pivoted LU and the oracle alike."""
    gm, om, delta = window_models(ctx, oracle, tmax, mesh, interp)
    rng = np.random.default_rng(3)
    for n in (1, 2, 4, 7, 9):
        t = rng.random((5, n)) * tmax
        t[0, 0], t[1, n - 1] = 0.0, tmax
        t[2, [0, n - 1]] = 0.0, tmax if n > 1 else 0.0
        for A, B in (((tmax, 0, 0, 0, 0), (tmax, 0, 1, 0, 0)), ((tmax, 0, 1, 0, 0), (0.0, 0, 0, 0, 0))):
            w, dw, sc = oracle.integrand(om, A, B, t)
            for algo in (capi.ALGO_TREE, capi.ALGO_DIRECT):
                v, d = gm.integrand(A, B, t, algo=algo)
                assert np.array_equal(d, dw) and np.all(np.abs(v - w) <= 1e-12 * sc), (n, algo)
        A, B = (tmax, 0, 0, 0, 0), (0.5 * tmax, 0, 1, 0, 0)
        t = rng.random((5, n)) * 0.9 * tmax
        t[1, 0], t[3, n - 1] = -0.4 * delta, -0.7 * delta
        w, dw, sc = oracle.integrand(om, A, B, t, keep_u_hypercube=False)
        for algo in (capi.ALGO_TREE, capi.ALGO_DIRECT):
            v, d = gm.integrand(A, B, t, algo=algo, keep_u_hypercube=False)
            assert np.array_equal(d, dw) and np.all(np.abs(v - w) <= 1e-12 * sc), (n, algo)
            t[1, 0] = -1.2 * delta
            with pytest.raises(capi.KbError) as e:
                gm.integrand(A, B, t, algo=algo, keep_u_hypercube=False)
            assert e.value.code == capi.KB_E_RANGE
            t[1, 0] = -0.4 * delta


def one_sided_models(ctx, oracle, ratio, small):
    """A nearly empty (small: "lesser") or full level: one of g^<, g^> `ratio` times the other."""
    t = np.linspace(-10, 10, 2001)
    big, little = np.exp(-np.abs(t) * (1 + 0.3j * np.sign(t))), ratio * np.exp(-0.5 * np.abs(t)) * np.cos(t)
    tables = (1j * little, -1j * big) if small == "lesser" else (1j * big, -1j * little)
    return ctx.model(10.0, *tables), oracle.model(10.0, *tables)


@pytest.mark.parametrize("small", ["lesser", "greater"])
@pytest.mark.parametrize("ratio", [1e-1, 1e-3, 1e-5])
def test_nearly_empty_and_full_levels(ctx, oracle, ratio, small):
    """The small function's entries keep their digits beside the other's."""
    gm, om = one_sided_models(ctx, oracle, ratio, small)
    for n in (1, 2, 3, 4, 5, 6, 7, 8, 9):
        t = np.random.default_rng(n).random((40 if n < 8 else 8, n)) * 10.0
        for A, B in ENDS[:2]:
            v, d, gsc = gm.integrand(A, B, t, algo=capi.ALGO_TREE, want_scale=True)
            w, dw, sc = oracle.integrand(om, A, B, t)
            assert np.array_equal(d, dw) and np.all(np.abs(v - w) <= 1e-12 * sc), n
            np.testing.assert_allclose(gsc, sc, rtol=1e-9)


@pytest.mark.parametrize("interp", [1, 3])
@pytest.mark.parametrize("n,count", [(10, 3), (13, 3), (14, 3), (15, 2), (16, 2)])
def test_depth_first_layouts(ctx, oracle, golden, n, count, interp):
    """Where the depth-first levels' nodes lie changes at orders 10 (level 9's node leaves shared memory),
    14 (level 8's pair as well, and level 9's is back) and 16 (neither); several points per group."""
    le, gr = golden["table_beta20_lesser"], golden["table_beta20_greater"]
    gm, om = ctx.model(10.0, le, gr, 0.4), oracle.model(10.0, le, gr, 0.4, interp=interp)
    gm.set_interpolation(interp)
    A, B = ENDS[n % 2]
    t = np.random.default_rng(n).random((count, n)) * 10.0
    v, d = gm.integrand(A, B, t, algo=capi.ALGO_TREE)
    w, dw, sc = oracle.integrand(om, A, B, t)
    assert np.array_equal(d, dw) and np.all(np.abs(v - w) <= 1e-12 * sc)
