"""The exact-order sums run by a block a chain (block_chain in
csrc/kernels.cuh) against the oracle's sequential ones, bit for bit, at the
edges of its rounds (32 terms) and of its 64-round chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(kind, M, N, rng):
    if kind == "positive":  # a few binade changes, then a long plateau
        return rng.random((M, N)) * 10.0 ** rng.uniform(-12, 0, (M, N)), rng.random((M, N))
    if kind == "signed":  # the sum crosses zero and binades both ways
        return rng.standard_normal((M, N)), rng.standard_normal((M, N)) * 10.0 ** rng.uniform(-3, 0, (M, N))
    if kind == "sparse":  # whole rounds of exact zeros, -0 among them
        A = rng.standard_normal((M, N))
        A[(np.arange(M) // 40) % 3 > 0] = 0.0
        A[::7] *= -1.0
        return A, np.abs(rng.standard_normal((M, N)))
    # growing by orders of magnitude: guesses of the binade that fail, values
    # outside the range of a float, ties at the accumulator's grid
    A = 2.0 ** np.round(np.linspace(-400, 300, M))[:, None] * rng.choice([1.0, -1.0, 0.5, 1.0 + 2.0 ** -52], (M, N))
    return A, np.ones((M, N))


@pytest.mark.parametrize("M", [2, 31, 32, 33, 65, 257, 2047, 2048, 2049, 4130])
@pytest.mark.parametrize("kind", ["positive", "signed", "sparse", "growing"])
def test_pdot_chain_edges(built, M, kind):
    import pqdts_gb300 as pq
    from oracle.oracle import Oracle
    from pqdts_gb300.synth import Instance

    N, D = 33, 40
    rng = np.random.default_rng(M)
    lo = np.zeros(D, np.int64)
    inst = Instance(M, N, D, 1e-3, 1e-6, lo, lo + 1, rng.random(2 * D), rng.random((D, N)))
    o = Oracle.from_instance(inst)
    with pq.Solver(0) as s:
        s.set_instance(inst)
        for seed in range(3):
            A, B = (np.asfortranarray(a) for a in _data(kind, M, N, np.random.default_rng(100 * M + seed)))
            g, r = s.pdot(A, B), o.pdot(A, B)
            assert np.float64(g).tobytes() == np.float64(r).tobytes(), (g, r)


@pytest.mark.parametrize("D", [1, 32, 33, 2048, 2049, 5000])
def test_objective_chain_edges(built, D):
    """L adds D row sums, and the gamma term's M - 1 terms a column."""
    import pqdts_gb300 as pq
    from oracle.oracle import Oracle
    from pqdts_gb300.synth import Instance

    M, N = 2050, 5
    rng = np.random.default_rng(D)
    lo = rng.integers(0, M - 3, D)
    inst = Instance(M, N, D, 0.3, 1e-6, lo, lo + 2, rng.random(3 * D), rng.random((D, N)) * 10.0 ** rng.uniform(-6, 2, (D, N)))
    X = np.asfortranarray(rng.random((M, N)))
    o = Oracle.from_instance(inst)
    o.set_space(True, None)
    with pq.Solver(0) as s:
        s.set_instance(inst)
        s.set_x(X)
        assert np.float64(s.L()).tobytes() == np.float64(o.L(X)[0]).tobytes()
