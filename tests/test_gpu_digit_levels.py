"""Both digit products hold their seventh digit and sixth level: outputs whose
terms are all of one size are off by no more than the last rounding and eight
times the root mean square of what the 28 digit pairs leave out.  The same
bound rejects an emulation with six digits, or without the last level."""
import numpy as np
import pytest

W, ROWS, COLS = 24, 20, 17  # terms of a sum, and outputs


def _operands(seed):
    rng = np.random.default_rng(seed)
    return 0.5 + rng.random((ROWS, W)) / 2, 0.5 + rng.random((W, COLS)) / 2


def _digits(A, S, axis):
    """A scaled along the other axis to [1/4, 1/2), its S base-256 digits."""
    E = np.frexp(np.abs(A).max(axis=axis, keepdims=True))[1] + 1
    t = np.rint(np.ldexp(A, 8 * S - E)).astype(np.int64)
    t = t + sum(128 << 8 * q for q in range(S))
    return [((t >> 8 * (S - 1 - q)) & (255 if q else -1)) - 128.0 for q in range(S)], E


def _emulate(A, B, S, levels):
    """The product by digit pairs p + q < levels (their sums are exact)."""
    a, EA = _digits(A, S, 1)
    b, EB = _digits(B, S, 0)
    out = np.zeros((A.shape[0], B.shape[1]), np.longdouble)
    for p in range(S):
        for q in range(min(S, levels - p)):
            out += (a[p] @ b[q]).astype(np.longdouble) * np.longdouble(2.0) ** (-8 * (p + q + 2))
    return out * np.exp2((EA + EB).astype(np.longdouble))


def _bound(exact, scale):
    """Half an ulp, and 8 x sqrt(W) 2^-58 of the scales (six pairs of level 7 a
    term, digits of ~74 and weight 2^-72: 2^-58.3; the operands' rounding to
    2^-57, times values below 1/2: 2^-58.8)."""
    return 2.0 ** -53 * np.abs(exact) + 8 * np.sqrt(W) * 2.0 ** -58 * scale


def test_bound_rejects_fewer():
    A, B = _operands(1)
    exact = A.astype(np.longdouble) @ B.astype(np.longdouble)
    bound = _bound(exact, 4.0)  # 2^1 x 2^1
    for S, levels, held in ((7, 7, True), (7, 6, False), (6, 6, False)):
        err = np.abs(_emulate(A, B, S, levels).astype(np.float64) - exact)
        assert bool(np.all(err <= bound)) == held, (S, levels, float((err / bound).max()))


def _solver(M, N, D, lo, val, P, X):
    import pqdts_gb300 as pq
    from pqdts_gb300.synth import Instance

    s = pq.Solver(0)
    s.set_option("autotune", 0)
    s.set_instance(Instance(M, N, D, 0.0, 1e-6, lo, lo + len(val) // D - 1, val, P), pq.MIXED)
    assert s.get_option("sched.dg_fwd") == 1 and s.get_option("sched.dg_trans") == 1
    s.set_x(np.asfortranarray(X))
    return s


@pytest.mark.gpu
def test_gradient_levels(built):
    """F^T.R: X = 0, so R = -2 P; F's rows all cover the same columns."""
    A, P = _operands(2)
    with _solver(ROWS, COLS, W, np.zeros(W, np.int64), np.ascontiguousarray(A.T).ravel(), P, np.zeros((ROWS, COLS))) as s:
        G = s.dL()
    exact = A.astype(np.longdouble) @ (-2 * P.astype(np.longdouble))
    assert np.all(np.abs(G - exact) <= _bound(exact, 8.0))  # 2^1 x 2^2


@pytest.mark.gpu
def test_residual_levels(built):
    """F.X: rows of F that share no column, so each entry of the gradient is one
    of F times the residual of its row, and P the product's nearest double."""
    M = ROWS * W
    F, _ = _operands(3)
    rng = np.random.default_rng(4)
    X = 0.5 + rng.random((M, COLS)) / 2
    O = np.stack([F[d].astype(np.longdouble) @ X[d * W : (d + 1) * W].astype(np.longdouble) for d in range(ROWS)])
    P = O.astype(np.float64)
    with _solver(M, COLS, ROWS, np.arange(ROWS, dtype=np.int64) * W, F.ravel(), P, X) as s:
        G = s.dL()
    R = (G.reshape(ROWS, W, COLS) / F[:, :, None]) / 2
    exact = (O - P)[:, None, :]
    bound = _bound(O, 4.0)[:, None, :] + 2.0 ** -45 * np.abs(R)  # and what F^T.R adds
    assert np.all(np.abs(R - exact) <= bound)
