"""FP64 results formed again only where a max-column rebuild moved X."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,D", [(33, 3, 40), (200, 20, 400), (257, 65, 300)])
@pytest.mark.parametrize("masks", [1, 0])
def test_rebuilt_columns_bitwise(built, M, N, D, masks):
    """A sequence of L, dL and conv_test in the reduced space, each starting
    with a rebuild, with set_x, doproj2 and space changes between them: the
    oracle's bits all along (column lists on and off)."""
    import pqdts_gb300 as pq
    from oracle.oracle import Oracle
    from pqdts_gb300 import synth

    inst = synth.make_instance(M=M, N=N, D=D, xmax=0.9 * M, eta=0.7, shots=10**6, gamma=1e-4, eps=1e-6, seed=M)
    o = Oracle.from_instance(inst)
    rng = np.random.default_rng(9)
    with pq.Solver(0) as s:
        s.set_option("row_masks", masks)
        s.set_instance(inst)
        X = None
        for step in ["set", "L", "dL", "dL", "L", "dL", "conv", "reduced", "dL", "proj", "dL", "dL", "redO", "dL", "set",
                     "dL", "conv", "full", "L", "dL", "reduced", "L", "dL", "dL"]:
            if step == "set":
                X = rng.random((M, N)) ** 3
                X[rng.random(X.shape) < 0.3] = 0.0
                X[:, -1] += 0.01
                X = np.asfortranarray(X / X.sum(1, keepdims=True))
                s.set_x(X)
            if step in ("set", "reduced", "full"):
                m = None if step == "full" else np.argmax(X, 1).astype(np.int32)
                s.set_space(step == "full", m)
                o.set_space(step == "full", m)
            elif step == "L":
                v, X = o.L(X)
                assert s.L() == v
            elif step == "dL":
                G, X = o.dL(X)
                assert np.array_equal(s.dL(), G)
            elif step == "conv":
                v, X, _ = o.conv_test(X)
                assert s.conv_test() == v
            elif step == "redO":
                assert np.array_equal(s.redO(), o.redO(X))
            elif step == "proj":
                X, xmin = o.doproj2(X)
                assert s.doproj2() == xmin
            assert np.array_equal(s.get_x(), X), step
