"""The mixed path's gradient and residual products entry by entry: a sum that
is small beside the scales of its row of F and its column of X (or R) is as
accurate as double-FP32 leaves it, however the operands' magnitudes spread."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spread(M, N, D, width, seed):
    """Bands of `width` columns that fall off by 2^-30 from their middle, and
    (D, N) and (M, N) arrays that fall off by 2^-50 from a diagonal, with a
    column and a tenth of the entries zero."""
    from pqdts_gb300.synth import Instance

    rng = np.random.default_rng(seed)
    lo = np.round(np.linspace(0, M - width, D)).astype(np.int64)
    u = np.linspace(-1, 1, width)
    val = (rng.random((D, width)) + 0.5) * 2.0 ** (-30 * u * u)

    def profile(rows):
        away = np.abs(np.linspace(0, 1, rows)[:, None] - np.linspace(0, 1, N)[None, :])
        a = (rng.random((rows, N)) + 0.5) * 2.0 ** (-50 * away)
        a[rng.random((rows, N)) < 0.1] = 0.0
        a[:, N // 2] = 0.0
        return a

    inst = Instance(M, N, D, 0.0, 1e-6, lo, lo + width - 1, val.ravel(), profile(D))
    return inst, np.asfortranarray(profile(M))


def _dense(inst):
    return inst.dense_F().astype(np.longdouble)


def _check(G, exact, size, K, products):
    """Double-FP32 rounds a sum of K terms by ~0.2 sqrt(K) 2^-48 of its terms'
    magnitudes (rms): within 40 times that for each of the products."""
    bound = products * 8 * np.sqrt(K) * 2.0 ** -48 * size
    err = np.abs(G - exact)
    assert np.all(err <= bound), float(np.max(err[size > 0] / bound[size > 0]))


# the last two leave their outputs to double-FP32, the others to FP64
SIZES = [(300, 27, 555, 60), (900, 40, 700, 300), (129, 70, 400, 100), (200, 2, 3000, 40), (1200, 70, 1500, 400),
         (3000, 33, 2600, 700)]


@pytest.mark.parametrize("M,N,D,width", SIZES)
def test_gradient_entries(built, M, N, D, width):
    """F^T.R alone: X = 0, so R = -2 P exactly."""
    import pqdts_gb300 as pq

    inst, _ = _spread(M, N, D, width, seed=D)
    F = _dense(inst)
    with pq.Solver(0) as s:
        s.set_option("autotune", 0)
        s.set_instance(inst, pq.MIXED)
        assert s.get_option("sched.dg_trans") == 1
        s.set_x(np.zeros((M, N), order="F"))
        G = s.dL()
    K = int((F != 0).sum(0).max())
    _check(G, F.T @ (-2 * inst.P), F.T @ (2 * inst.P), K, 1)


@pytest.mark.parametrize("M,N,D,width", SIZES)
def test_residual_entries(built, M, N, D, width):
    """F.X, then F^T of it (P = 0; every term positive)."""
    import pqdts_gb300 as pq

    inst, X = _spread(M, N, D, width, seed=M)
    inst.P = np.zeros((D, N))
    F = _dense(inst)
    with pq.Solver(0) as s:
        s.set_option("autotune", 0)
        s.set_instance(inst, pq.MIXED)
        assert s.get_option("sched.dg_fwd") == 1
        s.set_x(X)
        G, L = s.dL(), s.L()
    O = F @ X
    exact = F.T @ (2 * O)
    K = max(width, int((F != 0).sum(0).max()))
    _check(G, exact, exact, K, 2)
    assert abs(L - float((O * O).sum())) <= 16 * np.sqrt(K) * 2.0 ** -48 * L


def test_subnormal_scales(built):
    """Columns of X whose largest magnitude is subnormal, against an F large
    enough for a normal product: right, or as in double-FP32 (which has no such
    numbers)."""
    import pqdts_gb300 as pq

    M, N, D, width = 140, 5, 150, 33
    inst, _ = _spread(M, N, D, width, seed=3)
    rng = np.random.default_rng(4)
    inst.P = np.zeros((D, N))
    X = np.asfortranarray(np.ldexp(rng.integers(1, 1025, (M, N)).astype(float), -1060))
    inst.band_val = np.ldexp(rng.random(D * width) + 0.5, 100)
    G = []
    for df in (-1, 1):
        with pq.Solver(0) as s:
            s.set_option("autotune", 0)
            s.set_option("df_products", df)
            s.set_instance(inst, pq.MIXED)
            s.set_x(X)
            G.append(s.dL())
    F = _dense(inst)
    exact = F.T @ (2 * (F @ X.astype(np.longdouble)))
    assert np.all((G[0] == G[1]) | (np.abs(G[0] - exact) <= 2.0 ** -40 * exact))
