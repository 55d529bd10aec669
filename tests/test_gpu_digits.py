"""The mixed path's gradient and objective products by exact digits on the
tensor cores (csrc/tc_digits.cuh) against the FP64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _instance(M, N, D, width, flat, seed):
    """Bands of `width` columns drifting over M; values positive and uneven
    over 40 binary orders, or all equal (every digit of one sign: the level
    sums at their largest)."""
    from pqdts_gb300.synth import Instance

    rng = np.random.default_rng(seed)
    lo = np.round(np.linspace(0, M - width, D)).astype(np.int64)
    hi = lo + width - 1
    n = D * width
    val = np.full(n, 0.7) if flat else rng.random(n) * 2.0 ** -rng.integers(0, 40, n)
    P = rng.random((D, N))
    return Instance(M, N, D, 1e-3, 1e-6, lo, hi, val, P / P.sum(1, keepdims=True))


def _bounds(inst, X):
    """Errors of O and F^T.R that the digits allow: per term and in units of
    the scales, both operands' rounding to 48 bits (2^-49 each) and the five
    and fewer pairs of the dropped levels (at most 2^14 2^-64 each, the next
    levels 2^-8 of that): below 2^-47, and 16 x the largest magnitudes are
    at least the scales; K terms, plus an ulp of level 4 a drain."""
    F = inst.dense_F()
    fm = np.abs(F).max()
    K = int((F != 0).sum(1).max())
    Kt = int((F != 0).sum(0).max())
    eO = 16 * (K + 16) * 2.0 ** -47 * fm * np.abs(X).max()
    R = 2 * (F @ X - inst.P)
    eG = 2 * np.abs(F).sum(0).max() * eO + 16 * (Kt + 16) * 2.0 ** -47 * fm * np.abs(R).max()
    return eO, eG, 2 * np.abs(R / 2).sum() * eO + R.size * eO * eO


# tile edges: 128-row blocks, N tiles of 16..64, K chunks of 32 and drains of 256
CASES = [(129, 1, 127, 20, False), (128, 17, 300, 64, False), (700, 65, 513, 300, False), (700, 64, 256, 600, True),
         (257, 130, 129, 256, True), (2, 3, 1, 2, False), (1200, 200, 1500, 257, False)]


@pytest.mark.parametrize("M,N,D,width,flat", CASES)
@pytest.mark.parametrize("sparse", [False, True])
def test_digit_products(built, M, N, D, width, flat, sparse):
    import pqdts_gb300 as pq
    from oracle.oracle import Oracle

    inst = _instance(M, N, D, width, flat, seed=M + N)
    rng = np.random.default_rng(5)
    X = rng.random((M, N)) + 0.1
    if sparse:
        X[rng.random((M, N)) < 0.8] = 0.0
        X[:, 0] += 0.01
    X = np.asfortranarray(X / X.sum(1, keepdims=True))
    eO, eG, eL = _bounds(inst, X)
    o = Oracle.from_instance(inst)
    o.set_space(True, None)
    with pq.Solver(0) as s:
        s.set_instance(inst, pq.MIXED)
        assert s.get_option("sched.dg_fwd") == 1 and s.get_option("sched.dg_trans") == 1
        s.set_x(X)
        L, G = s.L(), s.dL()
    Lo, _ = o.L(X)
    Go, _ = o.dL(X)
    assert abs(L - Lo) <= eL + 1e-13 * abs(Lo), (L, Lo, eL)
    assert np.max(np.abs(G - Go)) <= eG + 1e-13 * np.max(np.abs(Go)), (np.max(np.abs(G - Go)), eG)


@pytest.mark.parametrize("M,N,D,width", [(129, 5, 200, 20), (300, 16, 257, 200)])
def test_digit_products_residual(built, M, N, D, width):
    """Data that X reproduces to 1e-4: the residual's error is
    that of 56-bit operands (_bounds' 48-bit one by 2^-8, and the roundings
    of the sum and of the difference), and the gradient's what it grows to in
    F^T.R with its 48 bits of the small R.  The reference has at least 64
    bits of mantissa."""
    import pqdts_gb300 as pq

    inst = _instance(M, N, D, width, False, seed=M)
    rng = np.random.default_rng(6)
    X = rng.random((M, N)) + 0.1
    X = np.asfortranarray(X / X.sum(1, keepdims=True))
    F = inst.dense_F()
    inst.P = F @ X * (1 + 1e-4 * rng.standard_normal((D, N)))
    inst.gamma = 0.0
    with pq.Solver(0) as s:
        s.set_instance(inst, pq.MIXED)
        s.set_x(X)
        G = s.dL()
    Fl = F.astype(np.longdouble)
    R = 2 * (Fl @ X.astype(np.longdouble) - inst.P)
    exact = Fl.T @ R
    fm, Kt = np.abs(F).max(), int((F != 0).sum(0).max())
    eO = 16 * (width + 16) * 2.0 ** -55 * fm * X.max() + 2.0 ** -51 * np.abs(inst.P).max()
    eG = 2 * np.abs(F).sum(0).max() * eO + 16 * (Kt + 16) * 2.0 ** -47 * fm * float(np.abs(R).max())
    eG += 2.0 ** -51 * float(np.abs(exact).max())
    err = float(np.max(np.abs(G - exact)))
    assert err <= eG, (err, eG)


@pytest.mark.parametrize("width,digits", [(8191, 1), (8192, 0)])
def test_digit_products_widest(built, width, digits):
    """Terms of one sign at the scales' limit up to the width that the 64-bit
    sums hold; wider rows in double-FP32."""
    import pqdts_gb300 as pq

    inst = _instance(width, 2, 2, width, True, seed=4)
    most = 1 - 2.0 ** -53
    inst.band_val[:] = most
    inst.gamma = 0.0
    X = np.full((width, 2), most, order="F")
    with pq.Solver(0) as s:
        s.set_instance(inst, pq.MIXED)
        assert s.get_option("sched.dg_fwd") == digits
        s.set_x(X)
        G = s.dL()
    R = 2 * (width - inst.P)
    exact = np.broadcast_to(R.sum(0), (width, 2))
    # the double-FP32 sums: 2^-47 of the sum so far for each of 2^13 terms
    assert np.allclose(G, exact, rtol=2.0 ** -34, atol=0), np.abs(G / exact - 1).max()


@pytest.mark.parametrize("D,digits", [(2**17 - 1, 1), (2**17, 0)])
def test_digit_products_tallest(built, D, digits):
    """The same for F^T.R and the height of F's columns."""
    import pqdts_gb300 as pq

    inst = _instance(2, 2, D, 2, True, seed=4)
    most = 1 - 2.0 ** -53
    inst.band_val[:] = most
    inst.gamma = 0.0
    X = np.full((2, 2), most, order="F")
    with pq.Solver(0) as s:
        s.set_option("autotune", 0)
        s.set_instance(inst, pq.MIXED)
        assert s.get_option("sched.dg_fwd") == 1 and s.get_option("sched.dg_trans") == digits
        s.set_x(X)
        G = s.dL()
    exact = np.broadcast_to((2 * (2 - inst.P)).sum(0), (2, 2))
    # the double-FP32 sums: 2^-47 of the sum so far for each of 2^17 terms
    assert np.allclose(G, exact, rtol=2.0 ** -30, atol=0), np.abs(G / exact - 1).max()


def test_digit_products_not_finite(built):
    """A NaN or an infinity in X reaches exactly the entries whose sums hold
    it: the rows of F with X's row in their band, then the columns of F with
    such a row in theirs, and the gamma stencil's neighbours."""
    import pqdts_gb300 as pq

    inst = _instance(300, 20, 400, 40, False, seed=1)
    X = np.full((300, 20), 1 / 20, order="F")
    X[100, 3] = np.nan
    X[200, 7] = np.inf
    with pq.Solver(0) as s:
        s.set_instance(inst, pq.MIXED)
        assert s.get_option("sched.dg_fwd") == 1
        s.set_x(X)
        G = s.dL()
    band = inst.dense_F() != 0
    bad = ~np.isfinite(X)
    reach = band.T @ (band @ bad)  # booleans: any path
    reach[1:] |= bad[:-1]
    reach[:-1] |= bad[1:]
    assert np.array_equal(~np.isfinite(G), reach | bad)


def test_digit_products_options(built):
    """df_products = 1 and tensor_cores = 0 keep the double-FP32 kernels."""
    import pqdts_gb300 as pq

    inst = _instance(129, 8, 130, 20, False, seed=2)
    for name, value in (("df_products", 1), ("tensor_cores", 0), ("df_products", 0)):
        with pq.Solver(0) as s:
            s.set_option(name, value)
            s.set_instance(inst, pq.MIXED)
            assert s.get_option("sched.dg_fwd") == 0 and s.get_option("sched.dg_trans") == 0
            assert s.get_option("sched.df_fwd") == (value == 1 or name == "tensor_cores")
